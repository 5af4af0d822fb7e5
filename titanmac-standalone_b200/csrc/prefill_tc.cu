// Tensor-core prefill kernel for B200: sliding-window attention with persistent prefix
// keys on tcgen05 (5th-generation tensor cores) with accumulators in tensor memory.
//
// A CTA owns one query tile: 128 consecutive rows of one (batch, head).  Its eight warps have fixed roles:
//   warp  0    TMA producer: Q, then the K tiles of the window
//   warp  1    TMA producer: persistent K/V tile, then the V tiles; allocates / frees tensor memory
//   warp  2    issues the tcgen05.mma (one elected thread)
//   warps 4-7  softmax, one thread per query row
// (the issuing warp comes early so that it is among the oldest warps of its scheduler)
// Key positions are cut into 64-key tiles anchored at (first query position - w); tiles that lie outside the query
// tile's window are neither loaded nor multiplied.  The persistent keys are extra, always-first tiles kept in their
// own shared-memory buffer.
//
// Per key tile:  S = Q Kᵀ (fp32, tensor memory)  ->  the softmax warps read their rows of S, update the running maximum
// lazily (the output accumulator in tensor memory is only rescaled when the maximum grew by more than 2^8), write
// P = exp2(S·c - m) as 16-bit values back into tensor memory over S  ->  O += P V with P read from tensor memory.
//
// What bounds it, and why this split: the exponentials (16 a clock and SM: 1024 clocks for 128 x 128 scores) take as long
// as head_dim 128's products and twice as long as head_dim 64's, and a key tile's chain - products, hand-over, load,
// maximum, exponentials, hand-over - is several times that.  So the chain is filled with other tiles' work:
//   head_dim 64   128 tensor-memory columns (S | O) and 64 registers a thread: FOUR CTAs per SM
//   head_dim 128  256 columns (S | S | O): two CTAs per SM, and the next scores are multiplied while these are
//                 exponentiated
// Measured before (128-key tiles; two CTAs per SM at head_dim 64, one CTA of two query tiles with one S each at 128) and
// now, us: 8 x 10 heads x 4112 rows of 64, window 128 | 512 | 2048: 82.2 | 133.8 | 283 and 63.4 | 105 | 242 (by itself, one
// input again or four in turn alike; 120 between the products of a layer, which hold the clock at 1760 MHz); 16 heads x
// 131 088 rows of 128, window 1024: 1604 and 1290 (two query tiles sharing K and V in one CTA: 1469; a hundred calls in a row,
// under the power cap: 1466, 1515 without the straight body below).
//
// Every wait on an mbarrier is bounded: on expiry the kernel records
// TMW_ERR_DEVICE_TIMEOUT in the device status word, stops waiting anywhere and runs
// to completion (with meaningless output) so that tensor memory is freed and the
// context stays usable.
#include <cuda.h>

#include <cstdio>
#include <mutex>
#include <type_traits>

#include "tc_ptx.cuh"
#include "tensor_map.cuh"
#include "tmw_common.cuh"

namespace tmw {
namespace {

using namespace ptx;

// Threads and register budget.  The four producer / issuing warps shrink to kRegsService, the softmax warps grow to
// kRegsSoftmax; setmaxnreg.inc blocks until the registers it asks for have been released INSIDE THE CTA and nothing bounds
// that wait, so the numbers must add up.
constexpr int kTcThreads = 256;
template <int DH>
struct Budget {
    static constexpr int kCtasPerSm = DH == 64 ? 4 : 2;
    static constexpr int kRegsLaunch = DH == 64 ? 64 : 128;
    static constexpr int kRegsService = DH == 64 ? 32 : 56;
    static constexpr int kRegsSoftmax = DH == 64 ? 96 : 200;
    static_assert(kTcThreads * kRegsLaunch <= 65536 / kCtasPerSm, "register file");
    static_assert(kRegsLaunch - kRegsService >= kRegsSoftmax - kRegsLaunch,
                  "setmaxnreg: the issuing warps must release what the softmax warps request");
};
constexpr int BM = 128;  // query rows per tile
constexpr int BN = 64;   // keys per tile

// Tensor-memory columns (32-bit each, 128 lanes): the S buffers, then O; P is written over its S.
template <int DH>
struct TmemMap {
    static constexpr int kSBufs = DH == 64 ? 1 : 2;
    static constexpr uint32_t kO = kSBufs * BN;
    static constexpr uint32_t kCols = kO + DH;  // 128 or 256
};

struct TcParams {
    int q_rows, k_rows, window, np, np_pad, q_pos0, k_pos0;
    int block;        // 0 or the block size of the block-granular window (first_visible_pos)
    int window_plan;  // window + block - 1: the widest window any row can have, used to lay out the key tiles
    int dim_order;  // bit i set: tensor i (0=q,1=k,2=v,3=o) has its head axis before its row axis in the map
    float scale_log2;
    int drain;  // a dependent launch follows: the stores have to be complete when the kernel ends
    int* status;
    float* lse;  // optional [batch, heads, q_rows]: log2 of the row's softmax denominator, in the scaled-by-log2(e) domain
    // Sequence-sharded call whose K/V buffer is filled by other GPUs (tmw_halo_push): key rows [0, np) may be read
    // once *pers_flag >= flag_value, key rows [np, np + halo_rows) once *halo_flag >= flag_value.  nullptr: no wait.
    const int* pers_flag;
    const int* halo_flag;
    int flag_value;
    int halo_rows;
    long long flag_wait_limit;
};

// Bounded wait of a producer warp for a flag that another GPU raises in this GPU's memory after it has written
// rows of the K/V buffer (release at system scope).  The rows are then read by TMA, i.e. through the asynchronous
// proxy, hence the proxy fence after the acquire.  On expiry: TMW_ERR_DEVICE_TIMEOUT in the status word
// (status[1] = -1 marks a flag, not an mbarrier), and nobody in the CTA waits any more.
__device__ __forceinline__ void flag_wait(const int* flag, int value, long long limit, volatile int* abort_flag,
                                          int* status) {
    if ((threadIdx.x & 31) == 0) {
        const long long t0 = clock64();
        for (;;) {
            int v;
            asm volatile("ld.acquire.sys.global.s32 %0, [%1];" : "=r"(v) : "l"(flag) : "memory");
            if (v >= value || *abort_flag) break;
            if (clock64() - t0 > limit) {
                *abort_flag = 1;
                if (atomicCAS(status, 0, (int)TMW_ERR_DEVICE_TIMEOUT) == 0) {
                    status[1] = -1;
                    status[2] = (int)(blockIdx.x | (blockIdx.y << 16));
                    status[3] = (int)(blockIdx.z | ((threadIdx.x >> 5) << 16));
                }
                break;
            }
            __nanosleep(100);
        }
        asm volatile("fence.proxy.async;" ::: "memory");
    }
    __syncwarp();
}

// ---------------------------------------------------------------------------------
// PTX wrappers beyond tc_ptx.cuh
// ---------------------------------------------------------------------------------
__device__ __forceinline__ void tma_store_commit_and_wait(bool drain) {
    tma_store_commit();
    if (drain) tma_store_wait_all();
    else tma_store_wait_read();
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
// Shared-memory matrix descriptors (128-byte swizzle, version 1 for sm_100) are built in the kernel as
//   bits [0,14)  start address >> 4       bits [16,30) leading byte offset >> 4
//   bits [32,46) stride byte offset >> 4  bits [46,48) version = 1    bits [61,64) layout = 2 (SWIZZLE_128B)

// Instruction descriptor for kind::f16: fp32 accumulate, A K-major; B K-major or MN-major.
//   [4,6) D format (1 = f32)  [7,10) A format  [10,13) B format (0 = f16, 1 = bf16)
//   [15] A major  [16] B major (1 = MN)  [17,23) N >> 3  [24,29) M >> 4
__device__ __forceinline__ uint32_t make_idesc(uint32_t fmt, uint32_t b_mn_major, uint32_t n) {
    return (1u << 4) | (fmt << 7) | (fmt << 10) | (b_mn_major << 16) | ((n >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
}

// ---------------------------------------------------------------------------------
// Schedule of one CTA, computed identically by every role
// ---------------------------------------------------------------------------------
struct Plan {
    int p_lo;     // position of the tile's first query row
    int rows;     // valid query rows
    int anchor;   // position of key 0 of window tile 0
    int a;        // first window tile index
    int n_win;    // number of window tiles
    int n_pers;   // items 0 .. n_pers - 1 are the persistent tiles
    int n_items;  // n_pers + n_win
};

__device__ __forceinline__ int floor_div(int a, int b) { return (a >= 0) ? a / b : -((-a + b - 1) / b); }

// `wblock`: the block-granular window; the kernel instantiated for the plain windowed mask passes a constant, so that it
// does not cost it an instruction
__device__ __forceinline__ Plan make_plan(const TcParams& p, int block, int wblock) {
    Plan q;
    const int r0 = block * BM;
    q.p_lo = p.q_pos0 + r0;
    q.rows = min(BM, p.q_rows - r0);
    q.anchor = q.p_lo - (wblock > 0 ? p.window_plan : p.window);
    q.n_pers = (p.np_pad + BN - 1) / BN;
    q.a = 0;
    q.n_win = 0;
    const int p_hi = q.p_lo + q.rows - 1;
    if (p_hi >= p.np) {
        const int g_lo = first_visible_pos(max(q.p_lo, p.np), p.np, p.window, wblock);
        q.a = floor_div(g_lo - q.anchor, BN);
        q.n_win = floor_div(p_hi - q.anchor, BN) - q.a + 1;
    }
    q.n_items = q.n_pers + q.n_win;
    return q;
}

// ---------------------------------------------------------------------------------
// The kernel
// ---------------------------------------------------------------------------------
template <int DH>
struct TcSmem {
    static constexpr int KS = 2, VS = 2;  // stages of the K and V rings
    // tiles are stored as sub-tiles of 64 columns: rows x 128 bytes
    static constexpr int kQSub = BM * 128, kQTile = kQSub * (DH / 64);
    static constexpr int kSub = BN * 128, kTile = kSub * (DH / 64);  // a K or V tile
    static constexpr int kQ = 0;
    static constexpr int kK = kQ + kQTile;
    static constexpr int kV = kK + KS * kTile;
    static constexpr int kP = kV + VS * kTile;  // persistent K then V: np_pad x DH x 2 bytes each
    static int total_bytes(int np_pad) { return kP + 2 * np_pad * DH * 2 + 512 /*barriers*/ + 1024 /*alignment*/; }
};

// barrier slots inside the barrier area
enum BarSlot {
    BAR_Q_FULL = 0,
    BAR_KP_FULL = 1,  // persistent K and V
    BAR_S_FULL = 2,   // [S buffer]
    BAR_P_READY = 4,  // [S buffer] (the softmax warps may be one item ahead of the products)
    BAR_O_DONE = 6,
    BAR_PV_DONE = 7,  // P V of the last item but one has finished (two S buffers)
    BAR_K_FULL = 8,   // [KS]
    BAR_K_EMPTY = 10,
    BAR_V_FULL = 12,  // [VS]
    BAR_V_EMPTY = 14,
    BAR_COUNT = 16
};

// GENERAL = false: the plain windowed mask (per-token);
// GENERAL = true: block-granular window, read from the parameters.
// STRAIGHT: key tiles that every row sees in full have a body of their own without mask and chunk tests, one run of
// instructions (head_dim 128; at head_dim 64 the 96 registers of a softmax thread do not hold it).  See straight_pays.
template <int DH, bool BF16, bool GENERAL, bool STRAIGHT>
__global__ void __launch_bounds__(kTcThreads, Budget<DH>::kCtasPerSm)
prefill_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                  const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_o,
                  const __grid_constant__ CUtensorMap map_kp, const __grid_constant__ CUtensorMap map_vp,
                  const TcParams p) {
    using L = TcSmem<DH>;
    using TM = TmemMap<DH>;
    constexpr uint32_t kTmemCols = TM::kCols;
    constexpr int SB = TM::kSBufs, KS = L::KS, VS = L::VS;
    constexpr int NSUB = DH / 64;  // 64-column sub-tiles per tile
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const uint32_t smem_base = smem_u32(smem);
    const uint32_t pers_bytes = (uint32_t)p.np_pad * DH * 2;
    const uint32_t bar_base = smem_base + L::kP + 2 * pers_bytes;
    uint8_t* bar_area = smem + L::kP + 2 * pers_bytes;
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(bar_area + BAR_COUNT * 8);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(bar_area + BAR_COUNT * 8 + 8);
    auto bar = [&](int slot) -> uint32_t { return bar_base + slot * 8; };

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int head = blockIdx.y, batch = blockIdx.z;
    const int wblock = GENERAL ? p.block : 0;
    const Plan q = make_plan(p, blockIdx.x, wblock);

    if (threadIdx.x == 0) {
        // the tensor maps live in the kernel parameters; fetch them into the descriptor cache early
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_q) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_k) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_v) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_kp) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_vp) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_o) : "memory");
        for (int i = 0; i < BAR_COUNT; ++i)  // P_READY: one arrival per softmax warp
            mbar_init(bar(i), i == BAR_P_READY || i == BAR_P_READY + 1 ? BM / 32 : 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32((const void*)tmem_slot)),
                     "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_trigger();  // (with its tensor memory in hand: a dependent that took it first would wait for this CTA forever)
    pdl_wait();

    // coordinate order of each tensor map: (dh, rows, heads, batch) or (dh, heads, rows, batch)
    auto coords = [&](int which, int row, int& c1, int& c2) {
        if ((p.dim_order >> which) & 1) { c1 = head; c2 = row; } else { c1 = row; c2 = head; }
    };

    if (warp < 4) {
        // register budget: see Budget
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(Budget<DH>::kRegsService) : "memory");
        if (warp == 0) {
            // ---------------- producer: Q, then K tiles ----------------
            if (elect_one()) {
                mbar_expect_tx(bar(BAR_Q_FULL), L::kQTile);
                int c1, c2;
                coords(0, blockIdx.x * BM, c1, c2);
                for (int s = 0; s < NSUB; ++s)
                    tma_load_4d(smem_base + L::kQ + s * L::kQSub, &map_q, bar(BAR_Q_FULL), s * 64, c1, c2, batch);
            }
            int n = 0;
            bool halo_seen = p.halo_flag == nullptr;
            for (int x = q.a; x < q.a + q.n_win; ++x, ++n) {
                const int s = n % KS;
                if (!halo_seen && p.np + q.anchor + x * BN - p.k_pos0 < p.np + p.halo_rows) {
                    flag_wait(p.halo_flag, p.flag_value, p.flag_wait_limit, abort_flag, p.status);
                    halo_seen = true;
                }
                mbar_wait(bar(BAR_K_EMPTY + s), ((n / KS) & 1) ^ 1, abort_flag, p.status);
                if (elect_one()) {
                    mbar_expect_tx(bar(BAR_K_FULL + s), L::kTile);
                    int c1, c2;
                    coords(1, p.np + q.anchor + x * BN - p.k_pos0, c1, c2);
                    for (int u = 0; u < NSUB; ++u)
                        tma_load_4d(smem_base + L::kK + s * L::kTile + u * L::kSub, &map_k,
                                    bar(BAR_K_FULL + s), u * 64, c1, c2, batch);
                }
                __syncwarp();
            }
        } else if (warp == 1) {
            // ---------------- producer: persistent K/V, then V tiles ----------------
            // (the persistent maps end at row np: rows np .. np_pad - 1 of the tile arrive as zeros)
            if (p.np > 0 && p.pers_flag != nullptr)
                flag_wait(p.pers_flag, p.flag_value, p.flag_wait_limit, abort_flag, p.status);
            if (p.np > 0 && elect_one()) {
                mbar_expect_tx(bar(BAR_KP_FULL), 2 * pers_bytes);
                int c1, c2;
                coords(1, 0, c1, c2);
                for (int u = 0; u < NSUB; ++u)
                    tma_load_4d(smem_base + L::kP + u * p.np_pad * 128, &map_kp, bar(BAR_KP_FULL), u * 64, c1, c2, batch);
                coords(2, 0, c1, c2);
                for (int u = 0; u < NSUB; ++u)
                    tma_load_4d(smem_base + L::kP + pers_bytes + u * p.np_pad * 128, &map_vp, bar(BAR_KP_FULL), u * 64,
                                c1, c2, batch);
            }
            int n = 0;
            bool halo_seen = p.halo_flag == nullptr;
            for (int x = q.a; x < q.a + q.n_win; ++x, ++n) {
                const int s = n % VS;
                if (!halo_seen && p.np + q.anchor + x * BN - p.k_pos0 < p.np + p.halo_rows) {
                    flag_wait(p.halo_flag, p.flag_value, p.flag_wait_limit, abort_flag, p.status);
                    halo_seen = true;
                }
                mbar_wait(bar(BAR_V_EMPTY + s), ((n / VS) & 1) ^ 1, abort_flag, p.status);
                if (elect_one()) {
                    mbar_expect_tx(bar(BAR_V_FULL + s), L::kTile);
                    int c1, c2;
                    coords(2, p.np + q.anchor + x * BN - p.k_pos0, c1, c2);
                    for (int u = 0; u < NSUB; ++u)
                        tma_load_4d(smem_base + L::kV + s * L::kTile + u * L::kSub, &map_v,
                                    bar(BAR_V_FULL + s), u * 64, c1, c2, batch);
                }
                __syncwarp();
            }
        } else if (warp == 2 && elect_one()) {  // (one thread runs the whole role, see elect_one)
            // ---------------- tensor-core issue ----------------
            // The QK that re-uses an S buffer is issued right after the PV that reads the P in it (tcgen05 operations of one
            // thread execute in issue order), and only then the commits that hand K and V stages back: a commit costs
            // the thread a few hundred cycles, and the softmax warps wait for the scores.
            const uint32_t fmt = BF16 ? 1u : 0u;
            const uint32_t idesc_qk = make_idesc(fmt, 0, BN);
            const uint32_t idesc_pv = make_idesc(fmt, 1, DH);
            // high word of every descriptor: stride byte offset 1024, version 1, 128-byte swizzle
            constexpr uint32_t kDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);
            auto desc_of = [](uint32_t lo) -> uint64_t { return ((uint64_t)kDescHi << 32) | lo; };
            // low word: start address >> 4 | leading byte offset >> 4 << 16
            auto lo_of = [](uint32_t addr, uint32_t lbo) -> uint32_t { return ((addr >> 4) & 0x3fffu) | ((lbo >> 4) << 16); };
            const uint32_t o_tmem = tmem_base + TM::kO;
            const uint32_t a_lo = lo_of(smem_base + L::kQ, 16);
            int k_stage = 0, v_stage = 0;  // ring cursors
            uint32_t k_par = 0, v_par = 0;
            // the scores of item i into its S buffer (the K tile, or the persistent tiles, have landed)
            auto qk = [&](int i) {
                const uint32_t d = tmem_base + (SB == 2 ? (i & 1) * BN : 0);
                const bool pers = i < q.n_pers;
                const uint32_t b_lo = pers ? lo_of(smem_base + L::kP + i * L::kSub, 16)
                                           : lo_of(smem_base + L::kK + k_stage * L::kTile, 16);
                const uint32_t b_sub = pers ? (uint32_t)p.np_pad * 8 : (uint32_t)(L::kSub >> 4);  // sub-tile stride >> 4
                const uint32_t idesc = pers ? make_idesc(fmt, 0, (uint32_t)min(BN, p.np_pad - i * BN)) : idesc_qk;
#pragma unroll
                for (int kk = 0; kk < DH / 16; ++kk)
                    mma_ss(d, desc_of(a_lo + (kk / 4) * (L::kQSub >> 4) + (kk % 4) * 2), desc_of(b_lo + (kk / 4) * b_sub + (kk % 4) * 2),
                           idesc, kk > 0 ? 1u : 0u);
                tc_commit(bar(BAR_S_FULL + (SB == 2 ? (i & 1) : 0)));
            };
            auto wait_keys = [&](int i) {
                if (i >= q.n_pers) mbar_wait(bar(BAR_K_FULL + k_stage), k_par, abort_flag, p.status);
            };
            auto free_keys = [&](int i) {
                if (i >= q.n_pers) {
                    tc_commit(bar(BAR_K_EMPTY + k_stage));
                    if (++k_stage == KS) { k_stage = 0; k_par ^= 1u; }
                }
            };
            mbar_wait(bar(BAR_Q_FULL), 0, abort_flag, p.status);
            if (q.n_pers > 0) mbar_wait(bar(BAR_KP_FULL), 0, abort_flag, p.status);
#pragma unroll
            for (int i = 0; i < SB; ++i)
                if (i < q.n_items) {
                    wait_keys(i);
                    tc_fence_after();
                    qk(i);
                    free_keys(i);
                }
#pragma unroll 1
            for (int i = 0; i < q.n_items; ++i) {
                const int next = i + SB;
                const bool pers = i < q.n_pers, more = next < q.n_items;
                if (!pers) mbar_wait(bar(BAR_V_FULL + v_stage), v_par, abort_flag, p.status);
                if (more) wait_keys(next);
                mbar_wait(bar(BAR_P_READY + (SB == 2 ? (i & 1) : 0)), (SB == 2 ? i >> 1 : i) & 1, abort_flag, p.status);
                tc_fence_after();
                // O += P V: B = V tile, MN-major, 16 keys = two 8-row groups of 1024 bytes per k-step
                const uint32_t pt = tmem_base + (SB == 2 ? (i & 1) * BN : 0);
                const uint32_t acc0 = i > 0 ? 1u : 0u;
                if (pers) {
                    const uint32_t b_lo = lo_of(smem_base + L::kP + pers_bytes + i * L::kSub, (uint32_t)p.np_pad * 128);
                    const int steps = min(BN, p.np_pad - i * BN) / 16;
                    for (int kk = 0; kk < steps; ++kk)
                        mma_ts(o_tmem, pt + kk * 8, desc_of(b_lo + kk * 128), idesc_pv, kk > 0 ? 1u : acc0);
                } else {
                    const uint32_t b_lo = lo_of(smem_base + L::kV + v_stage * L::kTile, L::kSub);
#pragma unroll
                    for (int kk = 0; kk < BN / 16; ++kk)
                        mma_ts(o_tmem, pt + kk * 8, desc_of(b_lo + kk * 128), idesc_pv, kk > 0 ? 1u : acc0);
                }
                if (more) qk(next);
                else if (SB == 2 && i == q.n_items - 2) tc_commit(bar(BAR_PV_DONE));
                else {  // the last item.  (Its V stage is not handed back: behind O_DONE nothing would keep the CTA's shared
                        // memory until that arrival has come in.)
                    tc_commit(bar(BAR_O_DONE));
                    break;
                }
                if (!pers) {
                    tc_commit(bar(BAR_V_EMPTY + v_stage));
                    if (++v_stage == VS) { v_stage = 0; v_par ^= 1u; }
                }
                if (more) free_keys(next);
            }
        }
    } else {
        // ---------------- softmax: one thread per row ----------------
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(Budget<DH>::kRegsSoftmax) : "memory");
        const int row = threadIdx.x & (BM - 1);  // row of the tile == tensor-memory lane
        constexpr int NCH = BN / 32;             // 32-column chunks
        const uint32_t lane_addr = (uint32_t)((warp & 3) * 32) << 16;
        const uint32_t s_base = tmem_base + lane_addr;
        const uint32_t o_addr = tmem_base + lane_addr + TM::kO;
        const int pos = q.p_lo + row;
        float m_used = -INFINITY;  // maximum the stored P and O are relative to (log2 domain)
        float l_sum = 0.f;

        // window tiles that every row of the query tile sees in full: items [full0, full1)
        int full0 = 0, full1 = 0;
        if (STRAIGHT && q.p_lo >= p.np) {
            const int lo = max(p.np, first_visible_pos(q.p_lo + BM - 1, p.np, p.window, wblock)) - q.anchor;
            full0 = max(1, q.n_pers + max(0, (lo + BN - 1) / BN - q.a));
            full1 = min(q.n_items, q.n_pers + floor_div(q.p_lo + 1 - q.anchor, BN) - q.a);
        }

        for (int item = 0; item < q.n_items; ++item) {
            if (STRAIGHT && item >= full0 && item < full1) {
                const int buf = SB == 2 ? (item & 1) : 0;
                const uint32_t s_addr = s_base + buf * BN;
                mbar_wait(bar(BAR_S_FULL + buf), (SB == 2 ? item >> 1 : item) & 1, abort_flag, p.status);
                tc_fence_after();
                const float neg_m = (m_used == -INFINITY) ? 0.f : -m_used;
                const uint64_t scale2 = pack2(p.scale_log2, p.scale_log2), negm2 = pack2(neg_m, neg_m);
                uint64_t lacc[2] = {0ull, 0ull};
                uint32_t s[NCH][32];
#pragma unroll
                for (int c = 0; c < NCH; ++c) tmem_ld32(s_addr + c * 32, s[c]);
                tc_wait_ld();
                float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
                for (int c = 0; c < NCH; ++c)
#pragma unroll
                    for (int i = 0; i < 16; ++i) mx[i & 3] = max3(mx[i & 3], __uint_as_float(s[c][2 * i]), __uint_as_float(s[c][2 * i + 1]));
                const float tile_max = max3(fmaxf(mx[0], mx[1]), mx[2], mx[3]) * p.scale_log2;
                if (!__any_sync(0xffffffffu, tile_max > m_used + 8.0f)) {  // (otherwise the general body does it all over again)
#pragma unroll
                    for (int c = 0; c < NCH; ++c) {
                        uint32_t packed[16];
#pragma unroll
                        for (int i = 0; i < 16; ++i) {
                            const float s0 = __uint_as_float(s[c][2 * i]), s1 = __uint_as_float(s[c][2 * i + 1]);
                            float x0, x1;
                            unpack2(fma2(pack2(s0, s1), scale2, negm2), x0, x1);
                            const float e0 = fast_exp2(x0), e1 = fast_exp2(x1);
                            lacc[i & 1] = add2(lacc[i & 1], pack2(e0, e1));
                            if (BF16) {
                                const __nv_bfloat162 h = __floats2bfloat162_rn(e0, e1);
                                packed[i] = *reinterpret_cast<const uint32_t*>(&h);
                            } else {
                                const __half2 h = __floats2half2_rn(e0, e1);
                                packed[i] = *reinterpret_cast<const uint32_t*>(&h);
                            }
                        }
                        tmem_st16(s_addr + c * 16, packed);
                    }
                    float a0, a1, a2, a3;
                    unpack2(lacc[0], a0, a1);
                    unpack2(lacc[1], a2, a3);
                    l_sum += (a0 + a1) + (a2 + a3);
                    tc_wait_st();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar(BAR_P_READY + buf));
                    continue;
                }
            }
            // visible columns of this row inside the tile: [j_lo, j_hi]
            int j_lo, j_hi, ncols;
            bool full;
            if (item < q.n_pers) {
                j_lo = 0;
                j_hi = p.np - 1 - item * BN;
                ncols = min(BN, p.np_pad - item * BN);
                full = j_hi >= BN - 1;
            } else {
                const int g0 = q.anchor + (q.a + item - q.n_pers) * BN;
                if (pos >= p.np) {
                    j_lo = first_visible_pos(pos, p.np, p.window, wblock) - g0;
                    j_hi = pos - g0;
                } else {
                    j_lo = 1;
                    j_hi = 0;
                }
                ncols = BN;
                // every row of the tile sees every key of the tile (decided per tile, not per row)
                full = q.p_lo >= p.np && g0 >= p.np && g0 + BN - 1 <= q.p_lo &&
                       g0 >= first_visible_pos(q.p_lo + BM - 1, p.np, p.window, wblock);
            }
            const int nchunks = (ncols + 31) / 32;
            // 32-column chunks in which no row of this warp sees a key (beyond the diagonal, or before the
            // window's left edge): not loaded, not exponentiated, P = 0
            bool hid[NCH];
#pragma unroll
            for (int c = 0; c < NCH; ++c)
                hid[c] = !full && __all_sync(0xffffffffu, j_hi - c * 32 < 0 || j_lo - c * 32 > 31);

            const int buf = SB == 2 ? (item & 1) : 0;
            const uint32_t s_addr = s_base + buf * BN;
            mbar_wait(bar(BAR_S_FULL + buf), (SB == 2 ? item >> 1 : item) & 1, abort_flag, p.status);
            tc_fence_after();

            uint32_t s[NCH][32];
#pragma unroll
            for (int c = 0; c < NCH; ++c)
                if (c < nchunks && !hid[c]) tmem_ld32(s_addr + c * 32, s[c]);
            tc_wait_ld();

            // mask (only the chunks in which some row of the warp has a hidden key), then the row maximum
            // over four independent chains of 3-input max
            if (!full) {
#pragma unroll
                for (int c = 0; c < NCH; ++c)
                    if (c < nchunks && !hid[c]) {
                        const int lo = j_lo - c * 32, hi = j_hi - c * 32;  // visible columns of the chunk: [lo, hi]
                        if (!__all_sync(0xffffffffu, lo <= 0 && hi >= 31)) {
#pragma unroll
                            for (int j = 0; j < 32; ++j)
                                if (j < lo || j > hi) s[c][j] = 0xff800000u;  // -inf
                        }
                    }
            }
            float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int c = 0; c < NCH; ++c)
                if (c < nchunks && !hid[c]) {
#pragma unroll
                    for (int j = 0; j < 32; j += 8) {
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            mx[k] = max3(mx[k], __uint_as_float(s[c][j + 2 * k]), __uint_as_float(s[c][j + 2 * k + 1]));
                        }
                    }
                }
            float tile_max = max3(fmaxf(mx[0], mx[1]), mx[2], mx[3]);
            tile_max *= p.scale_log2;  // scale > 0, so the maximum commutes with the scaling
            // lazy maximum: keep the old reference unless the new maximum is more than 2^8 above it
            const bool grow = tile_max > m_used + 8.0f;
            if (item == 0) {
                m_used = tile_max;
            } else if (__any_sync(0xffffffffu, grow)) {
                // the P V before this one must have finished before O is rescaled: with one S buffer it has (these scores
                // were issued behind it), with two the scores after these are what was issued behind it
                if (SB == 2) {
                    if (item + 1 < q.n_items)
                        mbar_wait(bar(BAR_S_FULL + (buf ^ 1)), ((item + 1) >> 1) & 1, abort_flag, p.status);
                    else
                        mbar_wait(bar(BAR_PV_DONE), 0, abort_flag, p.status);
                    tc_fence_after();
                }
                const float m_new = fmaxf(m_used, tile_max);
                const float alpha = (m_new == -INFINITY) ? 1.f : fast_exp2(m_used - m_new);
                m_used = m_new;
                l_sum *= alpha;
                // 16 columns at a time: the scores stay live in registers
#pragma unroll
                for (int c = 0; c < DH / 16; ++c) {
                    uint32_t o[16];
                    tmem_ld16(o_addr + c * 16, o);
                    tc_wait_ld();
#pragma unroll
                    for (int j = 0; j < 16; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * alpha);
                    tmem_st16(o_addr + c * 16, o);
                }
            }

            // P = exp2(S * c - m) on the special-function unit, packed two 16-bit values per column
            const float neg_m = (m_used == -INFINITY) ? 0.f : -m_used;
            const uint64_t scale2 = pack2(p.scale_log2, p.scale_log2);
            const uint64_t negm2 = pack2(neg_m, neg_m);
            uint64_t lacc[2] = {0ull, 0ull};  // four partial row sums
#pragma unroll
            for (int c = 0; c < NCH; ++c)
                if (c < nchunks) {
                    // 32 score columns -> 16 packed columns, eight per store (fewer registers in flight)
#pragma unroll
                    for (int part = 0; part < 2; ++part) {
                        uint32_t packed[8];
                        if (hid[c]) {
#pragma unroll
                            for (int i = 0; i < 8; ++i) packed[i] = 0u;
                        } else {
#pragma unroll
                            for (int i = 0; i < 8; ++i) {
                                const int j = (part * 8 + i) * 2;
                                const uint64_t x = fma2(pack2(__uint_as_float(s[c][j]), __uint_as_float(s[c][j + 1])),
                                                        scale2, negm2);
                                float x0, x1;
                                unpack2(x, x0, x1);
                                const float e0 = fast_exp2(x0);
                                const float e1 = fast_exp2(x1);
                                lacc[i & 1] = add2(lacc[i & 1], pack2(e0, e1));
                                if (BF16) {
                                    const __nv_bfloat162 h = __floats2bfloat162_rn(e0, e1);
                                    packed[i] = *reinterpret_cast<const uint32_t*>(&h);
                                } else {
                                    const __half2 h = __floats2half2_rn(e0, e1);
                                    packed[i] = *reinterpret_cast<const uint32_t*>(&h);
                                }
                            }
                        }
                        tmem_st8(s_addr + c * 16 + part * 8, packed);
                    }
                }
            {
                float a0, a1, a2, a3;
                unpack2(lacc[0], a0, a1);
                unpack2(lacc[1], a2, a3);
                l_sum += (a0 + a1) + (a2 + a3);
            }
            tc_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(BAR_P_READY + buf));
        }

        if (q.n_items > 0) {
            // ---------------- epilogue: O / l -> shared memory (swizzled) -> TMA store ----------------
            mbar_wait(bar(BAR_O_DONE), 0, abort_flag, p.status);
            tc_fence_after();
            const float inv = l_sum > 0.f ? 1.f / l_sum : 0.f;
            if (p.lse != nullptr && row < q.rows)
                p.lse[((long long)batch * gridDim.y + head) * p.q_rows + blockIdx.x * BM + row] =
                    m_used + log2f(l_sum);
            uint8_t* stage = smem + L::kQ;  // the Q tile is no longer needed
#pragma unroll
            for (int c = 0; c < DH / 32; ++c) {
                uint32_t o[32];
                tmem_ld32(o_addr + c * 32, o);
                tc_wait_ld();
#pragma unroll
                for (int g = 0; g < 4; ++g) {  // 8 columns = one 16-byte chunk
                    uint32_t w[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float a = __uint_as_float(o[g * 8 + 2 * e]) * inv;
                        const float b = __uint_as_float(o[g * 8 + 2 * e + 1]) * inv;
                        if (BF16) {
                            const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
                            w[e] = *reinterpret_cast<const uint32_t*>(&h);
                        } else {
                            const __half2 h = __floats2half2_rn(a, b);
                            w[e] = *reinterpret_cast<const uint32_t*>(&h);
                        }
                    }
                    const int col = c * 32 + g * 8;          // first column of the chunk
                    const int sub = col / 64;                // 64-column sub-tile
                    const int chunk = (col % 64) / 8;        // 16-byte chunk inside the 128-byte row
                    uint8_t* dst = stage + sub * L::kQSub + row * 128 + ((chunk ^ (row & 7)) * 16);
                    *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
                }
            }
            fence_proxy_async_smem();
            named_barrier_sync(1, BM);
            if (row == 0) {
                int c1, c2;
                coords(3, blockIdx.x * BM, c1, c2);
                for (int u = 0; u < NSUB; ++u)
                    tma_store_4d(&map_o, smem_u32(stage + u * L::kQSub), u * 64, c1, c2, batch);
                tma_store_commit_and_wait(p.drain);
            }
        }
    }

    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        if (*abort_flag) {
            // a wait expired somewhere in this CTA: give asynchronous copies and matrix products that may
            // still be in flight time to finish before tensor memory and shared memory are handed back
            const long long t0 = clock64();
            while (clock64() - t0 < 400000) __nanosleep(1000);
        }
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
    }
}

// ---------------------------------------------------------------------------------
// Host side: tensor maps and launch
// ---------------------------------------------------------------------------------
int np_pad_of(int np) { return np > 0 ? ((np + 15) / 16) * 16 : 0; }

// Whether the body for whole key tiles pays (never below 512, where few tiles of a window are such: 8 heads x 30 000 rows, window
// 300, 94.2 us without and 96.6 with it).  It does with block-granular windows (3 x 8 heads x 2747 rows, blocks of 64, windows 512 | 1024:
// 51.0 | 70.3 and 48.2 | 62.8 us), with windows of 1024 and more (30 000 rows: 169.9 and 162.8), with few query tiles to an SM, where
// one tile's time counts (1040 rows, window 640: 16.5 and 15.7), and in long sequences (30 000 rows, 512 | 896: 108.9 | 153.5 and
// 106.6 | 150.0; 4 x 8208, 896: 154.9 and 152.2).  Many sequences of a few windows each are slower with it (8 x 2064 rows, 512 | 640: 60.6 |
// 66.6 and 62.2 | 67.6; 16 x 2064, 896: 160.4 and 164.0; 8 x 4112, 512: 116.5 and 118.3).
bool straight_pays(const tmw_prefill_desc& d, bool block_window) {
    if (d.window < 512) return false;
    const long long tiles = (long long)((d.q_rows + BM - 1) / BM) * d.heads * d.batch;
    return block_window || d.window >= 1024 || tiles <= 4 * sm_count() || d.q_rows >= 9ll * d.window;
}

template <int DH>
int launch_tc(const tmw_prefill_desc& d, const void* q, const void* k, const void* v, void* o, cudaStream_t stream,
              int window_block, float* lse, const tmw_halo_wait* wait, int chain) {
    using L = TcSmem<DH>;
    const int np_pad = np_pad_of(d.n_persistent);
    CUtensorMap mq, mk, mv, mo, mkp, mvp;
    const MapStrides sq = map_strides(d.batch, d.heads, d.q_rows, DH, d.q_stride);
    const MapStrides sk = map_strides(d.batch, d.heads, d.k_rows, DH, d.k_stride);
    const MapStrides sv = map_strides(d.batch, d.heads, d.k_rows, DH, d.v_stride);
    const MapStrides so = map_strides(d.batch, d.heads, d.q_rows, DH, d.o_stride);
    // The persistent tile is a box of np_pad rows of a map that ENDS at row np: the rows between np and
    // np_pad are zero-filled instead of being read from the first sequence rows (whatever those hold - even
    // Inf or NaN bits of a buffer that is still being filled - must not reach 0 x V in the P V product).
    const int np_rows = d.n_persistent > 0 ? d.n_persistent : 1;
    if (!make_map_4d(&mq, q, d.dtype, d.batch, d.heads, d.q_rows, DH, sq, BM) ||
        !make_map_4d(&mk, k, d.dtype, d.batch, d.heads, d.k_rows, DH, sk, BN) ||
        !make_map_4d(&mv, v, d.dtype, d.batch, d.heads, d.k_rows, DH, sv, BN) ||
        !make_map_4d(&mo, o, d.dtype, d.batch, d.heads, d.q_rows, DH, so, BM) ||
        !make_map_4d(&mkp, k, d.dtype, d.batch, d.heads, np_rows, DH, sk, np_pad > 0 ? np_pad : 16) ||
        !make_map_4d(&mvp, v, d.dtype, d.batch, d.heads, np_rows, DH, sv, np_pad > 0 ? np_pad : 16))
        return TMW_ERR_CUDA;
    TcParams p;
    p.q_rows = d.q_rows; p.k_rows = d.k_rows; p.window = d.window; p.np = d.n_persistent; p.np_pad = np_pad;
    p.block = window_block;
    p.window_plan = d.window + (window_block > 0 ? window_block - 1 : 0);
    p.lse = lse;
    p.drain = chain & kChainFollowed;
    p.pers_flag = wait != nullptr ? wait->pers_flag : nullptr;
    p.halo_flag = wait != nullptr ? wait->halo_flag : nullptr;
    p.flag_value = wait != nullptr ? wait->value : 0;
    p.halo_rows = wait != nullptr ? wait->halo_rows : 0;
    p.flag_wait_limit = wait != nullptr && wait->wait_limit_cycles > 0 ? wait->wait_limit_cycles : kWaitLimitCycles;
    p.q_pos0 = d.q_pos0; p.k_pos0 = d.k_pos0;
    p.dim_order = (sq.heads_first ? 1 : 0) | (sk.heads_first ? 2 : 0) | (sv.heads_first ? 4 : 0) | (so.heads_first ? 8 : 0);
    const float scale = d.scale != 0.f ? d.scale : 1.0f / sqrtf((float)DH);
    p.scale_log2 = scale * 1.4426950408889634f;
    p.status = device_status_word();
    if (p.status == nullptr) return TMW_ERR_CUDA;
    const int smem_bytes = L::total_bytes(np_pad);
    dim3 grid((d.q_rows + BM - 1) / BM, d.heads, d.batch);
    auto run = [&](auto kern) -> int {
        const int rc = allow_shared_memory(reinterpret_cast<const void*>(kern), smem_bytes);
        if (rc != TMW_OK) return rc;
        TMW_CUDA_TRY(launch_ex(kern, grid, dim3(kTcThreads), smem_bytes, stream, chain & kChainDependent, 1, mq, mk, mv, mo, mkp, mvp, p));
        return TMW_OK;
    };
    auto pick = [&](auto bf16, auto general) -> int {
        constexpr bool BF16 = decltype(bf16)::value, GENERAL = decltype(general)::value;
        if (DH == 128 && straight_pays(d, GENERAL)) return run(prefill_tc_kernel<DH, BF16, GENERAL, DH == 128>);
        return run(prefill_tc_kernel<DH, BF16, GENERAL, false>);
    };
    if (d.dtype == TMW_BF16) return window_block > 0 ? pick(std::true_type{}, std::true_type{}) : pick(std::true_type{}, std::false_type{});
    return window_block > 0 ? pick(std::false_type{}, std::true_type{}) : pick(std::false_type{}, std::false_type{});
}

constexpr int kMaxDynamicSmem = 232448;  // 227 KB per CTA on sm_100

}  // namespace

bool prefill_tc_supports(const tmw_prefill_desc& d, const void*, const void*, const void*, const void*) {
    if (d.dtype != TMW_BF16 && d.dtype != TMW_F16) return false;
    if (d.head_dim != 64 && d.head_dim != 128) return false;
    if (d.batch > 65535 || d.heads > 65535) return false;
    const int np_pad = np_pad_of(d.n_persistent);
    if (np_pad > 128) return false;
    const int need = d.head_dim == 64 ? TcSmem<64>::total_bytes(np_pad) : TcSmem<128>::total_bytes(np_pad);
    if (need > kMaxDynamicSmem) return false;
    // positions are combined in 32-bit arithmetic inside the kernel
    if ((int64_t)d.q_pos0 + d.q_rows + d.window + 4 * BN >= (int64_t)1 << 30) return false;
    // layouts a tensor map cannot describe
    if (!map_strides(d.batch, d.heads, d.q_rows, d.head_dim, d.q_stride).ok ||
        !map_strides(d.batch, d.heads, d.k_rows, d.head_dim, d.k_stride).ok ||
        !map_strides(d.batch, d.heads, d.k_rows, d.head_dim, d.v_stride).ok ||
        !map_strides(d.batch, d.heads, d.q_rows, d.head_dim, d.o_stride).ok)
        return false;
    return true;
}

int launch_prefill_tc(const tmw_prefill_desc& d, const void* q, const void* k, const void* v, void* o,
                      cudaStream_t stream, int window_block, float* lse, const tmw_halo_wait* wait, int chain) {
    return d.head_dim == 64 ? launch_tc<64>(d, q, k, v, o, stream, window_block, lse, wait, chain)
                            : launch_tc<128>(d, q, k, v, o, stream, window_block, lse, wait, chain);
}

}  // namespace tmw
