// Products on tcgen05: C[M, N] = epilogue(sum over k of A(m, k) B(n, k)), 16-bit operands, fp32 accumulation in tensor memory,
// 16-bit output (or, with k cut into ranges, fp32 sums of each).  The linear layer of torch.nn.functional.linear has both
// operands K-major ([M, K] activations, [N, K] weight); a gradient's operands lie transposed and are read MN-major, B alone
// for the input's gradient, A and B for the weight's.  No transposes in memory anywhere.  Epilogues: see GemmEpilogue.
//
// gemm_tc_kernel: a persistent CTA per SM walks over 128 x BN output tiles (consecutive tiles share their rows of A, so those
// stay in L2 while the panels of B change).  Warp roles:
//   warp 0      TMA producer: A and B tiles of 64 K-elements into a ring of shared-memory stages
//   warp 1      issues the tcgen05.mma of every stage (one elected thread); allocates / frees tensor memory
//   warps 2-9   epilogue: tensor memory -> registers -> bias, GELU, ... -> 16-bit -> global memory, a row per lane in whole
//               32-byte sectors; warp w reads the 32 lanes of its number modulo 4 and takes every second panel of 32 columns
// The accumulator is double-buffered in tensor memory (2 x BN columns): the epilogue of a tile runs under the
// matrix products of the next one.  gemm_tc_pair_kernel, below, does the same on CTA pairs.  Every mbarrier wait is bounded
// and reports TMW_ERR_DEVICE_TIMEOUT through the device status word.
#include <cuda.h>

#include <cmath>
#include <type_traits>
#include <mutex>

#include "tc_ptx.cuh"
#include "tensor_map.cuh"
#include "tmw_common.cuh"

namespace tmw {
namespace {

using namespace ptx;

constexpr int GM = 128;        // rows of an output tile
constexpr int GK = 64;         // K elements per stage: one 128-byte swizzle row
constexpr int kPanel = 32;     // columns that an epilogue warp finishes at a time
constexpr int kBiasSlot = 96;  // bytes: an epilogue warp's bias of a panel and the eight columns behind it
constexpr int kEpiWarps = 8;
constexpr int kGemmThreads = 32 * (2 + kEpiWarps);
// The pair kernel's tiles are ready every 4 to 5 us at K = 640; with GELU the epilogue of one is 128 x 256 x 24 instructions a
// CTA.  16416 x 2560 x 640 with GELU, us: 75 with eight warps behind block-wide barriers, 72 with sixteen, 58 with sixteen that
// do not wait for one another (QKV, N = 1920, no epilogue: 42 -> 38).
constexpr int kPairEpiWarps = 16;
constexpr int kPairThreads = 32 * (2 + kPairEpiWarps);

template <int BN>
struct GemmSmem {
    // 64-wide slices of K per stage: a tcgen05.commit costs the issuing thread about 220 cycles, which the products of
    // one slice cover only where the tile is wide (K = 2560, us: 128 columns 10.4 -> 8.7, 32 columns 9.3 -> 7.0)
    static constexpr int kSlices = BN <= 128 ? 2 : 1;
    static constexpr int kStageA = kSlices * GM * GK * 2;
    static constexpr int kStageB = kSlices * BN * GK * 2;
    static constexpr int kStage = kStageA + kStageB;
    static constexpr int kStages = (232448 - 2048) / kStage;
    static constexpr int kBars = kStages * kStage;      // offset of the barrier area
    static constexpr int kTotal = kBars + 1024 + 1024;  // barriers and, from 256 on, the warps' bias; alignment slack
    static_assert(256 + kEpiWarps * kBiasSlot <= 1024, "bias slots");
    static_assert(kStages >= 3, "pipeline depth");
};

struct GemmParams {
    int m, n, k;
    int epilogue;        // GemmEpilogue
    const void* bias;    // [n] in the dtype of the operands, or nullptr
    void* aux;           // [m, n] beside the output (see GemmEpilogue), contiguous
    float* partial;      // k cut into `splits` ranges: their fp32 sums go to [splits][m][n] here instead of to the output
    int splits;
    int width;           // pair kernel: columns of a tile (a multiple of 32)
    int group;           // pair kernel: row bands that a wide output is walked in (group_bands)
    void* c;             // the output, rows of ldc elements
    long long ldc;
    int wide;            // rows of what is written (c, or the fp32 sums) and of aux start on 32-byte boundaries
    int* status;
};

template <bool BF16>
__device__ __forceinline__ uint4 pack8(const float* v) {
    uint32_t w[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        if (BF16) {
            const __nv_bfloat162 hh = __floats2bfloat162_rn(v[2 * e], v[2 * e + 1]);
            w[e] = *reinterpret_cast<const uint32_t*>(&hh);
        } else {
            const __half2 hh = __floats2half2_rn(v[2 * e], v[2 * e + 1]);
            w[e] = *reinterpret_cast<const uint32_t*>(&hh);
        }
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
}

// Rows that start on a sector (32 bytes; WIDE: all of the output and of what the epilogue reads do) go out as they lie in tensor
// memory, 32 columns of a row per lane and panel.  Rows that do not (every second one of 16 n + 8 values, all of an output 16 bytes
// into its allocation) would cost L2 two accesses of half a sector for each sector: their lane takes its columns 8 further on,
// where sectors start, and the first eight of the tile with the last panel.  (In kernels of their own: another form chosen at run
// time beside the plain one cost that its registers, 16416 x 2560 x 640 with GELU 54 -> 62 us.)  us, staged for TMA stores as before |
// halves of sectors | shifted: 16416 x 50008 x 640 1098 | 1390 | 912, 32896 x 1928 x 640 70.8 | 86.1 | 63.8, 16416 x 2568 x 640 with
// GELU_KEEP 77.6 | 134 | 71.5; an output 16 bytes off, 16416 x 50000 x 640 1234 | 1573 | 925.
// Columns [c0, c0 + 8) and [c1, c1 + 8) of a row, of which those below n exist (a multiple of 8):
template <bool WIDE>
__device__ __forceinline__ bool one_sector(const void* at, int c0, int c1, int n) {
    return WIDE ? c1 < n : c1 == c0 + 8 && c1 < n && (reinterpret_cast<uintptr_t>(at) & 31u) == 0;
}
// The stores pass L1 by: lines that it keeps for them are lines that the next ones wait for, most where K is short and the output is
// all there is (8320 x 1024 | 4096 x 256 us: 9.6 | 25.3 with them, 8.7 | 21.8 so, staged for TMA stores 9.8 | 22.5; 8320 x 2560 x 640
// keeping GELU's argument, with bias 39.7 and 38.5; 8320 x 2560 x 640 with GELU's derivative 49.5 and 39.8).
template <bool WIDE>
__device__ __forceinline__ void store16(void* row, int c0, int c1, int n, const uint4& a, const uint4& b) {
    uint16_t *dst = static_cast<uint16_t*>(row) + c0, *dst1 = static_cast<uint16_t*>(row) + c1;
    if (one_sector<WIDE>(dst, c0, c1, n)) {
        asm volatile("st.global.L1::no_allocate.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                     ::"l"(dst), "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w)
                     : "memory");
        return;
    }
    if (c0 < n) *reinterpret_cast<uint4*>(dst) = a;
    if (!WIDE && c1 < n) *reinterpret_cast<uint4*>(dst1) = b;
}
template <bool WIDE>
__device__ __forceinline__ void load16(const void* row, int c0, int c1, int n, uint4& a, uint4& b) {
    const uint16_t *src = static_cast<const uint16_t*>(row) + c0, *src1 = static_cast<const uint16_t*>(row) + c1;
    if (one_sector<WIDE>(src, c0, c1, n)) {
        asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w), "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w)
                     : "l"(src)
                     : "memory");
        return;
    }
    a = c0 < n ? *reinterpret_cast<const uint4*>(src) : make_uint4(0, 0, 0, 0);
    b = !WIDE && c1 < n ? *reinterpret_cast<const uint4*>(src1) : make_uint4(0, 0, 0, 0);
}

// The columns that a lane has of a panel: [col, col + 24) and [col3, col3 + 8).
struct PanelColumns {
    int col, col3;
};
template <bool WIDE>
__device__ __forceinline__ PanelColumns panel_columns(bool shifted, int col0, int panel, int panels) {
    const int col = col0 + panel * kPanel;
    if (WIDE || !shifted) return {col, col + 24};
    return {col + 8, panel + 1 < panels ? col + 32 : col0};
}

// What the epilogue of a panel reads beside the accumulator (GEMM_ADD, GEMM_GELU_GRAD): a lane's row of its 32 columns.
// Asked for before the accumulator is waited for.
struct PanelAux { uint4 v[4]; };

template <bool WIDE, bool AUX>
__device__ __forceinline__ void load_aux(PanelAux& in, const GemmParams& p, int row, const PanelColumns& c) {
    if (!AUX || row >= p.m) return;
    const uint16_t* src = static_cast<const uint16_t*>(p.aux) + (long long)row * p.n;
    load16<WIDE>(src, c.col, c.col + 8, p.n, in.v[0], in.v[1]);
    load16<WIDE>(src, c.col + 16, c.col3, p.n, in.v[2], in.v[3]);
}

// The bias of a panel and of the eight columns behind it (at the tile's end: its first eight), two columns for each of 20 lanes.  It is
// asked for a panel ahead and passes through a slot of the warp's own in shared memory.  Loaded by every lane where it is added, 64
// bytes four times, it came from L2 - the outputs that the lanes store push it out of L1 - and the warps are at the latency of their
// instructions as it is.  With GELU, N = 2560, K = 640, rows 8320 | 16416 | 32896, us: 38.1 | 72.5 | 142 so, 38.9 | 75.3 | 147 by
// shuffles, 33.0 | 62.8 | 120 now (panels staged for TMA stores 33.4 | 62.1 | 119).
__device__ __forceinline__ uint32_t load_bias(const GemmParams& p, int col0, int panel, int panels, int lane) {
    if (p.bias == nullptr || lane >= 20) return 0u;
    const int c = col0 + (lane >= 16 && panel + 1 == panels ? 2 * lane - 32 : panel * kPanel + 2 * lane);
    return c < p.n ? *reinterpret_cast<const uint32_t*>(static_cast<const uint16_t*>(p.bias) + c) : 0u;
}

// 32 accumulator columns of one row per lane -> epilogue -> the output, sixteen at a time.  A row per lane and 32 bytes per access: every
// sector is written once and whole, without a detour through shared memory, which leaves that to two more stages of operands.
// Against panels of 32 x 32 staged for TMA stores, us, K = 640: 16416 x 50000 863 -> 800, 16416 x 2560 46.6 -> 43.5, 32896 x 1920
// 66.4 -> 64.8, 32896 x 640 30.5 -> 28.5; 8320 x 640 x 2560 28.0 -> 25.0; 8192^3 718 -> 715.  Sixteen columns at a time, and the epilogues
// that read a second operand (AUX) in kernels of their own, leave the registers that GELU's instructions overlap in: with GELU and
// bias, 16416 x 2560 x 640 65.5 us with 32 at a time, 63.7 with one kernel for all, 62.8 so (a chip that is warm).
template <bool BF16, bool WIDE, bool AUX>
__device__ __forceinline__ void finish_panel(float (&v)[32], const GemmParams& p, const PanelAux& in, int row, const PanelColumns& c) {
    using T = typename std::conditional<BF16, __nv_bfloat16, __half>::type;
    uint16_t* out = static_cast<uint16_t*>(p.c) + (long long)row * p.ldc;
    uint16_t* aux = static_cast<uint16_t*>(p.aux) + (long long)row * p.n;
    const int n = row < p.m ? p.n : 0;  // (nothing of a row beyond the output is stored)
#pragma unroll
    for (int j = 0; j < 32; j += 16) {
        const int c0 = c.col + j, c1 = j ? c.col3 : c.col + 8;
        if (!AUX && p.epilogue == GEMM_GELU) {
#pragma unroll
            for (int e = 0; e < 16; ++e) v[j + e] = gelu_erf(v[j + e]);
        } else if (!AUX && p.epilogue == GEMM_GELU_KEEP) {
            const uint4 raw[2] = {pack8<BF16>(v + j), pack8<BF16>(v + j + 8)};
            store16<WIDE>(aux, c0, c1, n, raw[0], raw[1]);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float x[8];
                load8<T>(reinterpret_cast<const T*>(&raw[h]), x);
#pragma unroll
                for (int e = 0; e < 8; ++e) v[j + 8 * h + e] = gelu_erf(x[e]);
            }
        } else if (AUX) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float x[8];
                load8<T>(reinterpret_cast<const T*>(&in.v[j / 8 + h]), x);
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    float& y = v[j + 8 * h + e];
                    y = p.epilogue == GEMM_ADD ? x[e] + to_f32<T>(from_f32<T>(y)) : y * gelu_slope(x[e]);
                }
            }
        }
        store16<WIDE>(out, c0, c1, n, pack8<BF16>(v + j), pack8<BF16>(v + j + 8));
    }
}

// the fp32 sums of a k range: whole sectors where `partial` lies on one (n is a multiple of 8), halves where the caller's scratch is
// aligned to 16 bytes only
__device__ __forceinline__ void store_partial(const uint32_t (&v)[32], const GemmParams& p, int split, int row, int col) {
    if (row >= p.m) return;
    float* dst = p.partial + ((long long)split * p.m + row) * p.n + col;
#pragma unroll
    for (int j = 0; j < 32; j += 8) {
        if (col + j >= p.n) continue;
        if (p.wide) {
            asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                         ::"l"(dst + j), "r"(v[j]), "r"(v[j + 1]), "r"(v[j + 2]), "r"(v[j + 3]), "r"(v[j + 4]), "r"(v[j + 5]),
                           "r"(v[j + 6]), "r"(v[j + 7])
                         : "memory");
        } else {
            *reinterpret_cast<uint4*>(dst + j) = make_uint4(v[j], v[j + 1], v[j + 2], v[j + 3]);
            *reinterpret_cast<uint4*>(dst + j + 4) = make_uint4(v[j + 4], v[j + 5], v[j + 6], v[j + 7]);
        }
    }
}

// A warp's panels (first, first + step, ...) of a finished tile: tensor memory -> global memory.  No warp waits for another.
// `in` and `bias` hold what the first panel needs; `all_read` is called once the accumulator has been read.
template <bool BF16, bool WIDE, bool AUX, typename F>
__device__ __forceinline__ void epilogue_panels(const GemmParams& p, PanelAux& in, uint32_t bias, uint8_t* slot, uint32_t t_addr,
                                                bool shifted, int row, int col0, int first, int panels, int step, int split, F all_read) {
    using T = typename std::conditional<BF16, __nv_bfloat16, __half>::type;
    const int lane = row & 31;
    if (first >= panels) all_read();
    for (int pn = first; pn < panels; pn += step) {
        uint32_t acc[32], next[8];
        __syncwarp();
        if (p.bias != nullptr) {
            if (lane < 20) reinterpret_cast<uint32_t*>(slot)[lane] = bias;
            __syncwarp();
        }
        tmem_ld32(t_addr + pn * kPanel, acc);
        if (!WIDE) tmem_ld8(t_addr + (pn + 1 < panels ? (pn + 1) * kPanel : 0), next);
        tc_wait_ld();
        if (pn + step >= panels) {
            tc_fence_before();
            __syncwarp();
            all_read();
        }
        if (WIDE && p.partial != nullptr) {
            store_partial(acc, p, split, row, col0 + pn * kPanel);
            continue;
        }
        float v[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(WIDE || !shifted ? acc[j] : j < 24 ? acc[j + 8] : next[j - 24]);
        if (p.bias != nullptr) {
            const T* b = reinterpret_cast<const T*>(slot) + (!WIDE && shifted ? 8 : 0);
#pragma unroll
            for (int i = 0; i < 32; i += 8) {
                float x[8];
                load8<T>(b + i, x);
#pragma unroll
                for (int e = 0; e < 8; ++e) v[i + e] += x[e];
            }
            if (pn + step < panels) bias = load_bias(p, col0, pn + step, panels, lane);
        }
        finish_panel<BF16, WIDE, AUX>(v, p, in, row, panel_columns<WIDE>(shifted, col0, pn, panels));
        if (pn + step < panels) load_aux<WIDE, AUX>(in, p, row, panel_columns<WIDE>(shifted, col0, pn + step, panels));
    }
}
// whether a row of the output starts in the middle of a sector (its columns from col0 on, a multiple of 32)
template <bool WIDE>
__device__ __forceinline__ bool off_sector(const GemmParams& p, int row) {
    return !WIDE && (reinterpret_cast<uintptr_t>(static_cast<uint16_t*>(p.c) + (long long)row * p.ldc) & 31u) != 0;
}

// An operand tile of R rows (of the product: M or N) x 64 k-elements in shared memory, 128 bytes per swizzled row.
// K-major (the matrix is [R, k] row-major): R rows of 64 k.  MN-major (the matrix is [k, R]): R / 64 sub-tiles of 64 k-rows
// x 64 columns.
template <int R, bool MN>
__device__ __forceinline__ uint64_t tile_desc(uint32_t addr) {
    return MN ? mnmajor_desc(addr, 64 * 128) : kmajor_desc(addr);
}
template <bool MN>
constexpr uint64_t kStepDesc = MN ? 128 : 2;  // 16 k-elements on, in units of 16 bytes

template <int BN, bool BF16, bool AMN, bool BMN, bool WIDE, bool AUX>
__global__ void __launch_bounds__(kGemmThreads, 1)
gemm_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, const GemmParams p) {
    using L = GemmSmem<BN>;
    constexpr int S = L::kStages;
    constexpr uint32_t kTmemCols = 512;  // two accumulators of BN <= 256 columns
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const uint32_t smem_base = smem_u32(smem);
    uint8_t* bar_area = smem + L::kBars;
    const uint32_t bar_base = smem_base + L::kBars;
    // barrier slots: full[S] | empty[S] | acc_full[2] | acc_empty[2]
    auto full = [&](int s) -> uint32_t { return bar_base + 8 * s; };
    auto empty = [&](int s) -> uint32_t { return bar_base + 8 * (S + s); };
    auto acc_full = [&](int b) -> uint32_t { return bar_base + 8 * (2 * S + b); };
    auto acc_empty = [&](int b) -> uint32_t { return bar_base + 8 * (2 * S + 2 + b); };
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(bar_area + 8 * (2 * S + 4));
    volatile int* abort_flag = reinterpret_cast<volatile int*>(bar_area + 8 * (2 * S + 4) + 8);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n_tiles = (p.n + BN - 1) / BN, m_tiles = (p.m + GM - 1) / GM;
    const int tiles = n_tiles * m_tiles * p.splits;  // (tile, k range)
    const int k_blocks = (p.k + L::kSlices * GK - 1) / (L::kSlices * GK);

    if (threadIdx.x == 0) {
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_a) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w) : "memory");
        for (int s = 0; s < S; ++s) {
            mbar_init(full(s), 1);
            mbar_init(empty(s), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(acc_full(b), 1);
            mbar_init(acc_empty(b), kEpiWarps);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) tmem_alloc(smem_u32((const void*)tmem_slot), kTmemCols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_trigger();  // (with its tensor memory in hand: a dependent that took it first would wait for this CTA forever)
    pdl_wait();

    constexpr int SL = L::kSlices;
    if (warp == 0) {
        // ---------------- producer ----------------
        if (elect_one()) {
            int s = 0;
            uint32_t parity = 1;
            for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
                const int mn = tile / p.splits, split = tile % p.splits;
                const int row0 = (mn / n_tiles) * GM, col0 = (mn % n_tiles) * BN;
                const int kb1 = k_blocks * (split + 1) / p.splits;
                for (int kb = k_blocks * split / p.splits; kb < kb1; ++kb) {
                    mbar_wait(empty(s), parity, abort_flag, p.status);
                    mbar_expect_tx(full(s), L::kStage);
                    const uint32_t dst = smem_base + s * L::kStage;
#pragma unroll
                    for (int u = 0; u < SL; ++u) {  // (slices beyond K arrive as zeros)
                        const int k0 = (kb * SL + u) * GK;
                        const uint32_t da = dst + u * (GM * GK * 2), db = dst + L::kStageA + u * (BN * GK * 2);
                        if (AMN) {
#pragma unroll
                            for (int c = 0; c < GM / 64; ++c) tma_load_2d(da + c * 8192, &map_a, full(s), row0 + c * 64, k0);
                        } else {
                            tma_load_2d(da, &map_a, full(s), k0, row0);
                        }
                        if (BMN) {
#pragma unroll
                            for (int c = 0; c < BN / 64; ++c) tma_load_2d(db + c * 8192, &map_w, full(s), col0 + c * 64, k0);
                        } else {
                            tma_load_2d(db, &map_w, full(s), k0, col0);
                        }
                    }
                    if (++s == S) { s = 0; parity ^= 1u; }
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ---------------- tensor-core issue ----------------
        if (elect_one()) {
            const uint32_t idesc = idesc_kmajor(BF16 ? 1u : 0u, BN) | (AMN ? 1u << 15 : 0u) | (BMN ? 1u << 16 : 0u);
            int s = 0, t = 0;
            uint32_t parity = 0;
            for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, ++t) {
                const int buf = t & 1;
                mbar_wait(acc_empty(buf), ((t >> 1) & 1) ^ 1, abort_flag, p.status);  // the epilogue has drained it
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + buf * BN;
                const int split = tile % p.splits, kb0 = k_blocks * split / p.splits, kb1 = k_blocks * (split + 1) / p.splits;
                for (int kb = kb0; kb < kb1; ++kb) {
                    mbar_wait(full(s), parity, abort_flag, p.status);
                    tc_fence_after();
                    const uint64_t a_desc = tile_desc<GM, AMN>(smem_base + s * L::kStage);
                    const uint64_t b_desc = tile_desc<BN, BMN>(smem_base + s * L::kStage + L::kStageA);
#pragma unroll
                    for (int u = 0; u < SL; ++u)
#pragma unroll
                        for (int kk = 0; kk < GK / 16; ++kk)
                            mma_ss(d_tmem, a_desc + u * (GM * GK * 2 / 16) + kStepDesc<AMN> * kk,
                                   b_desc + u * (BN * GK * 2 / 16) + kStepDesc<BMN> * kk, idesc, (kb > kb0 || (u | kk)) ? 1u : 0u);
                    tc_commit(empty(s));  // the stage is free once these products have read it
                    if (kb == kb1 - 1) tc_commit(acc_full(buf));
                    if (++s == S) { s = 0; parity ^= 1u; }
                }
            }
        }
        __syncwarp();
    } else {
        // ---------------- epilogue ----------------
        const int g = warp & 3;             // lane group of tensor memory this warp may read
        const int sub = (warp - 2) >> 2;    // its first panel
        constexpr int kPanels = BN / kPanel;
        int t = 0;
        for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, ++t) {
            const int buf = t & 1;
            const int mn = tile / p.splits, row = (mn / n_tiles) * GM + g * 32 + lane, col0 = (mn % n_tiles) * BN;
            PanelAux in;
            const bool shifted = off_sector<WIDE>(p, row);
            if (sub < kPanels) load_aux<WIDE, AUX>(in, p, row, panel_columns<WIDE>(shifted, col0, sub, kPanels));
            const uint32_t bias = load_bias(p, col0, sub, kPanels, lane);
            mbar_wait(acc_full(buf), (t >> 1) & 1, abort_flag, p.status);
            tc_fence_after();
            epilogue_panels<BF16, WIDE, AUX>(p, in, bias, bar_area + 256 + (warp - 2) * kBiasSlot,
                                             tmem_base + ((uint32_t)(g * 32) << 16) + buf * BN, shifted, row, col0, sub, kPanels,
                                             kEpiWarps / 4, tile % p.splits, [&] { if (lane == 0) mbar_arrive(acc_empty(buf)); });
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        if (*abort_flag) {
            // a wait expired in this CTA: give copies and products that may still be in flight time to finish
            const long long t0 = clock64();
            while (clock64() - t0 < 400000) __nanosleep(1000);
        }
        tmem_dealloc(tmem_base, kTmemCols);
    }
}

// ---------------------------------------------------------------------------------
// The same product on CTA pairs: two CTAs of a cluster (two SMs) share 256 x BN output tiles.  Each CTA
// loads its 128 rows of A and its BN / 2 rows of W, so a W tile crosses L2 -> SM once per 256 output rows instead
// of once per 128 (the single-CTA kernel is bound by exactly that traffic).  The first CTA of the pair issues
// tcgen05.mma.cta_group::2 for both; each CTA keeps its 128 x BN half of the accumulator in its own tensor
// memory and runs its own epilogue.  Barriers: "full" lives in the first CTA and counts the bytes of both CTAs'
// loads; "empty" and "accumulator full" are arrived on in both CTAs by one commit; "accumulator empty" lives in
// the first CTA and collects the epilogue warps of both.
// ---------------------------------------------------------------------------------
// Outputs of kGroupFrom or more column tiles are walked in groups of row bands, column by column: the tiles in flight then share
// few rows of W as well as of A.  W is read once per group, so a group is as large as its rows of A stay in L2 beside the rest:
// 32 MiB of them, from 8 up to 48 bands (of 256 rows).  us with groups of 8 | 16 | 24 | 32 | 48 | 128: 16416 x 50000 x 640
// 777 | 762 | 755 | 755 | 753 | 754; 32896 x 50000 x 640 1583 | 1550 | 1538 | 1535 | 1533 | 1632; 16384^2 x 4096
// 1385 | 1350 | 1373 | 1447 | 1534 | 1650; 8192^3 695 | 698 | 713 | 740 | 739 | 738.
constexpr int kGroupFrom = 16;
int group_bands(int k) {
    const int bands = (32 << 20) / (2 * GM * 2) / k;
    return bands < 8 ? 8 : bands > 48 ? 48 : bands;
}

// Shared memory of the pair kernel is a ring of as many stages as fit at the tile's width (256 columns: 7, 160: 8).  The bytes
// in flight are what the rate hangs on: 16416 x 50000 x 640 took 976 | 875 | 847 | 823 us with 3 | 4 | 5 | 6 stages of a form on the
// way to this one, whose seven took 800 (753 since wide outputs are walked in larger groups).
struct PairSmem {
    static constexpr int kStageA = GM * GK * 2;
    static constexpr int kMost = 10;  // stages (barriers)
    static constexpr int kBars = 229376;  // (what the ring takes at most)
    static constexpr int kTotal = kBars + 256 + kPairEpiWarps * kBiasSlot + 1024;  // barriers, bias, alignment slack
    static_assert(kTotal <= 232448, "shared memory");
};

template <int BN, bool BF16, bool AMN, bool BMN, bool WIDE, bool AUX>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPairThreads, 1)
gemm_tc_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, const GemmParams p) {
    using L = PairSmem;
    constexpr int M = L::kMost;
    constexpr uint32_t kTmemCols = 512;
    extern __shared__ uint8_t smem_raw[];
    // the same offsets in both CTAs of the pair (the dynamic shared memory of a kernel starts at the same
    // address in every CTA)
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const uint32_t smem_base = smem_u32(smem);
    uint8_t* bar_area = smem + L::kBars;
    const uint32_t bar_base = smem_base + L::kBars;
    auto full = [&](int s) -> uint32_t { return bar_base + 8 * s; };
    auto empty = [&](int s) -> uint32_t { return bar_base + 8 * (M + s); };
    auto acc_full = [&](int b) -> uint32_t { return bar_base + 8 * (2 * M + b); };
    auto acc_empty = [&](int b) -> uint32_t { return bar_base + 8 * (2 * M + 2 + b); };
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(bar_area + 8 * (2 * M + 4));
    volatile int* abort_flag = reinterpret_cast<volatile int*>(bar_area + 8 * (2 * M + 4) + 8);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();  // 0: issues the products, 1: partner
    const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    const int n_tiles = (p.n + p.width - 1) / p.width, m_tiles = (p.m + 2 * GM - 1) / (2 * GM);
    const int tiles = n_tiles * m_tiles * p.splits;  // (tile, k range)
    const int k_blocks = (p.k + GK - 1) / GK;
    auto locate = [&](int tile, int& band, int& col) {  // its band of 256 rows and first column
        const int mn = tile / p.splits;
        if (n_tiles < kGroupFrom) {
            band = mn / n_tiles;
            col = (mn % n_tiles) * p.width;
        } else {
            const int first = mn / (p.group * n_tiles) * p.group, r = mn - first * n_tiles, bands = min(p.group, m_tiles - first);
            band = first + r % bands;
            col = r / bands * p.width;
        }
    };
    // columns a tile multiplies: its width, or for the last tile of a row what is left of N (in steps of 32) - a product
    // over columns that do not exist would cost its full time
    auto columns = [&](int col) -> int { return min(p.width, (p.n - col + 31) / 32 * 32); };
    const int b_boxes = (p.width + 127) / 128;  // boxes of 64 columns that an MN-major half takes
    const uint32_t stage = L::kStageA + (BMN ? b_boxes * 8192 : p.width * 64);  // (a multiple of 1024: swizzled tiles)
    const int S = min(M, (int)(L::kBars / stage));

    if (threadIdx.x == 0) {
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_a) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w) : "memory");
        for (int s = 0; s < M; ++s) {
            mbar_init(full(s), 1);
            mbar_init(empty(s), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(acc_full(b), 1);
            mbar_init(acc_empty(b), 2 * kPairEpiWarps);  // the epilogue warps of both CTAs
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) tmem_alloc_pair(smem_u32((const void*)tmem_slot), kTmemCols);
    tc_fence_before();
    __syncthreads();
    cluster_sync();  // the partner's barriers exist before anything is signalled across
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_trigger();  // (with its tensor memory in hand: a dependent that took it first would wait for this CTA forever)
    pdl_wait();

    if (warp == 0) {
        // ---------------- producer (both CTAs) ----------------
        if (elect_one()) {
            int s = 0;
            uint32_t parity = 1, dst = smem_base;
            for (int tile = pair; tile < tiles; tile += pairs) {
                const int split = tile % p.splits;
                int band, col;
                locate(tile, band, col);
                const int row0 = band * (2 * GM) + (int)rank * GM;
                // each CTA supplies half of the tile's columns (the box is half of p.width; a narrow tile uses its first rows)
                const int col0 = col + (int)rank * (columns(col) / 2);
                const int kb1 = k_blocks * (split + 1) / p.splits;
                for (int kb = k_blocks * split / p.splits; kb < kb1; ++kb) {
                    mbar_wait(empty(s), parity, abort_flag, p.status);
                    if (rank == 0) mbar_expect_tx(full(s), 2 * stage);  // both CTAs' bytes
                    const uint32_t bar0 = map_to_cta(full(s), 0);
                    if (AMN) {
#pragma unroll
                        for (int c = 0; c < GM / 64; ++c) tma_load_2d_pair(dst + c * 8192, &map_a, bar0, row0 + c * 64, kb * GK);
                    } else {
                        tma_load_2d_pair(dst, &map_a, bar0, kb * GK, row0);
                    }
                    if (BMN) {
                        for (int c = 0; c < b_boxes; ++c)
                            tma_load_2d_pair(dst + L::kStageA + c * 8192, &map_w, bar0, col0 + c * 64, kb * GK);
                    } else {
                        tma_load_2d_pair(dst + L::kStageA, &map_w, bar0, kb * GK, col0);
                    }
                    dst += stage;
                    if (++s == S) { s = 0; dst = smem_base; parity ^= 1u; }
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ---------------- tensor-core issue (first CTA of the pair only) ----------------
        if (rank == 0 && elect_one()) {
            int s = 0, t = 0;
            uint32_t parity = 0, src = smem_base;
            for (int tile = pair; tile < tiles; tile += pairs, ++t) {
                const int buf = t & 1;
                int band, col;
                locate(tile, band, col);
                const uint32_t idesc = idesc_kmajor(BF16 ? 1u : 0u, (uint32_t)columns(col), 2 * GM) | (AMN ? 1u << 15 : 0u) |
                                       (BMN ? 1u << 16 : 0u);
                mbar_wait(acc_empty(buf), ((t >> 1) & 1) ^ 1, abort_flag, p.status);
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + buf * BN;
                const int split = tile % p.splits, kb0 = k_blocks * split / p.splits, kb1 = k_blocks * (split + 1) / p.splits;
                for (int kb = kb0; kb < kb1; ++kb) {
                    mbar_wait(full(s), parity, abort_flag, p.status);
                    tc_fence_after();
                    const uint64_t a_desc = tile_desc<GM, AMN>(src);
                    const uint64_t b_desc = tile_desc<BN / 2, BMN>(src + L::kStageA);
#pragma unroll
                    for (int kk = 0; kk < GK / 16; ++kk)
                        mma_ss_pair(d_tmem, a_desc + kStepDesc<AMN> * kk, b_desc + kStepDesc<BMN> * kk, idesc,
                                    (kb > kb0 || kk) ? 1u : 0u);
                    tc_commit_pair(empty(s));
                    if (kb == kb1 - 1) tc_commit_pair(acc_full(buf));
                    src += stage;
                    if (++s == S) { s = 0; src = smem_base; parity ^= 1u; }
                }
            }
        }
        __syncwarp();
    } else {
        // ---------------- epilogue (both CTAs, each its own 128 rows) ----------------
        const int g = warp & 3;
        const int sub = (warp - 2) >> 2;
        int t = 0;
        for (int tile = pair; tile < tiles; tile += pairs, ++t) {
            const int buf = t & 1;
            int band, col0;
            locate(tile, band, col0);
            const int row = band * (2 * GM) + (int)rank * GM + g * 32 + lane;
            const int panels = columns(col0) / kPanel;
            PanelAux in;
            const bool shifted = off_sector<WIDE>(p, row);
            if (sub < panels) load_aux<WIDE, AUX>(in, p, row, panel_columns<WIDE>(shifted, col0, sub, panels));
            const uint32_t bias = load_bias(p, col0, sub, panels, lane);
            mbar_wait(acc_full(buf), (t >> 1) & 1, abort_flag, p.status);
            tc_fence_after();
            epilogue_panels<BF16, WIDE, AUX>(p, in, bias, bar_area + 256 + (warp - 2) * kBiasSlot,
                                             tmem_base + ((uint32_t)(g * 32) << 16) + buf * BN, shifted, row, col0, sub, panels,
                                             kPairEpiWarps / 4, tile % p.splits, [&] { if (lane == 0) mbar_arrive_cluster(map_to_cta(acc_empty(buf), 0)); });
        }
    }

    tc_fence_before();
    __syncthreads();
    cluster_sync();  // nothing of the partner (its barriers, its shared memory) is touched after this
    if (warp == 1) {
        tc_fence_after();
        if (*abort_flag) {
            const long long t0 = clock64();
            while (clock64() - t0 < 400000) __nanosleep(1000);
        }
        tmem_dealloc_pair(tmem_base, kTmemCols);
    }
}

// ---------------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------------
bool make_maps(const GemmCall& g, int b_rows, CUtensorMap* ma, CUtensorMap* mb) {
    const auto sw = CU_TENSOR_MAP_SWIZZLE_128B;
    return (g.a_mn ? make_map_2d(ma, g.a, g.dtype, g.k, g.m, g.lda, GK, 64, sw) : make_map_2d(ma, g.a, g.dtype, g.m, g.k, g.lda, GM, GK, sw)) &&
           (g.b_mn ? make_map_2d(mb, g.b, g.dtype, g.k, g.n, g.ldb, GK, 64, sw)
                   : make_map_2d(mb, g.b, g.dtype, g.n, g.k, g.ldb, b_rows, GK, sw));
}

int gemm_params(const GemmCall& g, GemmParams* p) {
    p->m = g.m; p->n = g.n; p->k = g.k;
    p->epilogue = g.epilogue;
    p->bias = g.bias;
    p->aux = g.aux;
    p->splits = g.splits;
    p->partial = g.splits > 1 ? g.partial : nullptr;
    p->c = g.c;
    p->ldc = g.ldc;
    auto on32 = [](const void* q, int64_t ld) { return (reinterpret_cast<uintptr_t>(q) & 31u) == 0 && ld % 16 == 0; };
    p->wide = p->partial != nullptr ? on32(p->partial, 16) : on32(g.c, g.ldc) && (g.aux == nullptr || on32(g.aux, g.n));
    p->status = device_status_word();
    if (p->status == nullptr) return TMW_ERR_CUDA;
    auto on16 = [](const void* q, int64_t ld) { return (reinterpret_cast<uintptr_t>(q) & 15u) == 0 && ld % 8 == 0; };
    if (g.c == nullptr || !on16(g.c, g.ldc) || (g.aux != nullptr && !on16(g.aux, g.n))) {
        set_error_text("product: rows of the output and of what the epilogue reads must start on 16-byte boundaries");
        return TMW_ERR_INVALID_ARGUMENT;
    }
    return TMW_OK;
}

// The kernels by data type, operand layouts (built with MN-major ones: 256 x 256, 128 and 64 columns) and alignment of the rows.
template <int BN>
struct Single {
    static constexpr bool kMn = BN == 64 || BN == 128;
    template <bool BF16, bool AMN, bool BMN, bool WIDE, bool AUX>
    static auto kernel() { return gemm_tc_kernel<BN, BF16, AMN, BMN, WIDE, AUX>; }
};
template <int BN>
struct Pair {
    static constexpr bool kMn = true;
    template <bool BF16, bool AMN, bool BMN, bool WIDE, bool AUX>
    static auto kernel() { return gemm_tc_pair_kernel<BN, BF16, AMN, BMN, WIDE, AUX>; }
};
template <typename F>
int with_bool(bool value, F f) { return value ? f(std::true_type{}) : f(std::false_type{}); }
// `run` is called with the call's kernel
template <typename Family, typename F>
int with_kernel(const GemmCall& g, const GemmParams& p, F run) {
    const bool wide = p.partial != nullptr || p.wide;  // (fp32 sums have a path of their own)
    const bool aux = p.partial == nullptr && (g.epilogue == GEMM_ADD || g.epilogue == GEMM_GELU_GRAD);
    return with_bool(g.dtype == TMW_BF16, [&](auto bf16) {
        return with_bool(wide, [&](auto w) {
            constexpr bool B = decltype(bf16)::value, W = decltype(w)::value;
            if (g.a_mn) {
                if constexpr (Family::kMn) {
                    if (g.b_mn && !aux) return run(Family::template kernel<B, true, true, W, false>());
                }
                return (int)TMW_ERR_UNSUPPORTED;
            }
            return with_bool(aux, [&](auto a) {
                constexpr bool A = decltype(a)::value;
                if (!g.b_mn) return run(Family::template kernel<B, false, false, W, A>());
                if constexpr (Family::kMn) return run(Family::template kernel<B, false, true, W, A>());
                return (int)TMW_ERR_UNSUPPORTED;
            });
        });
    });
}

template <int BN>
int launch_gemm(const GemmCall& g, cudaStream_t stream) {
    using L = GemmSmem<BN>;
    CUtensorMap ma, mb;
    GemmParams p;
    if (!make_maps(g, BN, &ma, &mb)) return TMW_ERR_CUDA;
    if (const int rc = gemm_params(g, &p); rc != TMW_OK) return rc;
    const int tiles = ((g.m + GM - 1) / GM) * ((g.n + BN - 1) / BN) * g.splits;
    const int grid = tiles < sm_count() ? tiles : sm_count();
    auto run = [&](auto kern) -> int {
        const int rc = allow_shared_memory(reinterpret_cast<const void*>(kern), L::kTotal);
        if (rc != TMW_OK) return rc;
        TMW_CUDA_TRY(launch_ex(kern, dim3(grid), dim3(kGemmThreads), L::kTotal, stream, g.chain & kChainDependent, 1, ma, mb, p));
        return TMW_OK;
    };
    return with_kernel<Single<BN>>(g, p, run);
}

// How many CTA pairs of the kernel the device runs at once (asked once per kernel and device).
int max_active_pairs(const void* kern, int smem_bytes) {
    constexpr int kMaxDevices = 64, kMaxKernels = 32;
    struct Entry { const void* kern; int pairs[kMaxDevices]; };
    static std::mutex mutex;
    static Entry table[kMaxKernels] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return sm_count() / 2;
    std::lock_guard<std::mutex> lock(mutex);
    Entry* e = nullptr;
    for (int i = 0; i < kMaxKernels && e == nullptr; ++i) {
        if (table[i].kern == kern) e = &table[i];
        else if (table[i].kern == nullptr) { table[i].kern = kern; e = &table[i]; }
    }
    if (e != nullptr && e->pairs[dev] > 0) return e->pairs[dev];
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(sm_count() & ~1, 1, 1);
    cfg.blockDim = dim3(kPairThreads, 1, 1);
    cfg.dynamicSmemBytes = smem_bytes;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n <= 0) {
        (void)cudaGetLastError();
        n = sm_count() / 2;
    }
    if (e != nullptr) e->pairs[dev] = n;
    return n;
}

template <int BN>
int launch_gemm_pair(const GemmCall& g, int width, cudaStream_t stream) {
    using L = PairSmem;
    CUtensorMap ma, mb;
    GemmParams p;
    if (!make_maps(g, width / 2, &ma, &mb)) return TMW_ERR_CUDA;
    if (const int rc = gemm_params(g, &p); rc != TMW_OK) return rc;
    p.width = width;
    p.group = group_bands(g.k);
    const int tiles = ((g.m + 2 * GM - 1) / (2 * GM)) * ((g.n + width - 1) / width) * g.splits;
    auto run = [&](auto kern) -> int {
        const void* fn = reinterpret_cast<const void*>(kern);
        const int rc = allow_shared_memory(fn, L::kTotal);
        if (rc != TMW_OK) return rc;
        const int resident = max_active_pairs(fn, L::kTotal);
        const int pairs = tiles < resident ? tiles : resident;
        TMW_CUDA_TRY(launch_ex(kern, dim3(2 * pairs), dim3(kPairThreads), L::kTotal, stream, g.chain & kChainDependent, 1, ma, mb, p));
        return TMW_OK;
    };
    return with_kernel<Pair<BN>>(g, p, run);
}

// What a single-CTA kernel was measured to need (us): a launch without its K, what a 64-wide slice of K takes where a tile is
// alone on the chip, and where all SMs stream operands.  The pair kernel moves the fewest operand bytes per product and wins
// wherever it has enough tiles: measured at K = 640 for 1056 | 2528 | 8256 | 32 896 rows of N = 1920, pair | 128 | 64
// columns: 7.8 | 10.0 | 21.1 | 73.8, 6.2 | 11.1 | 24.9 | 102.9, 7.0 | 12.1 | 30.8 | 129.7 us (one after the other, the chip warm).  The
// constants are older than the present epilogue and ring.  What they choose is within 4 % of the best kernel and width for the four
// products of a layer of width 640 at 144 to 32 896 rows; elsewhere it is up to a sixth off (2112 x 1024 x 4096, second operand
// MN-major: 19.1 against 16.5).
struct Variant {
    int rows, cols;
    float launch, alone, full;
};
constexpr Variant kVariants[] = {{2 * GM, 256, 6.1f, 0.f, 0.f},  // (see pair_cost)
                                 {GM, 256, 5.0f, 0.305f, 0.54f}, {GM, 128, 4.2f, 0.167f, 0.306f},
                                 {GM, 64, 3.7f, 0.128f, 0.186f}, {GM, 32, 3.5f, 0.117f, 0.135f}};

// The pair kernel's cost and tile width.  A 64-wide slice of a tile of w columns takes 0.12 + 0.00105 w us on a busy chip
// and the chip as a whole 0.465 us per 256 columns of a pair; few waves of wide tiles leave a last one that is nearly empty,
// which narrower tiles fill.  8256 x 640 x 2560: 33 bands over 74 pairs are two waves at 256 columns and at 160; 30.7 and
// 23.8 us (64 columns a CTA, single: 35.2).  16416 x 640 x 2560: 52.1 at 256, 48.4 at 224, 50.5 at 160 (the chip warm).
float pair_cost(const GemmCall& g, int splits, int sms, int* width) {
    const float slices = (float)((g.k + GK - 1) / GK) / (float)splits;
    const int bands = (g.m + 2 * GM - 1) / (2 * GM), pairs = sms / 2 > 0 ? sms / 2 : 1;
    const float busy = (float)bands * (float)((g.n + 31) / 32) / 8.f * (float)splits / (float)pairs;
    auto slice = [](int w) { return 0.12f + 0.00105f * (float)w; };
    float least = 0.f;
    for (int w = 256; w >= 128; w -= 32) {
        const int n_tiles = (g.n + w - 1) / w, last = g.n - (n_tiles - 1) * w;
        const long long tiles = (long long)n_tiles * bands * splits, waves = (tiles + pairs - 1) / pairs, narrow = waves / n_tiles;
        float t = (float)(waves - narrow) * slice(w) + (float)narrow * slice(last);
        if (waves == 1) t *= 0.72f + 0.28f * (float)tiles / (float)pairs;  // operands arrive faster on a chip half idle
        t = t > 0.465f * busy ? t : 0.465f * busy;
        if (w == 256 || t < 0.97f * least) {
            least = t;
            *width = w;
        }
    }
    return kVariants[0].launch + slices * least;
}

float variant_cost(int i, const GemmCall& g, int splits, int sms, int* width) {
    if (i == 0) return pair_cost(g, splits, sms, width);
    const Variant& v = kVariants[i];
    const float slices = (float)((g.k + GK - 1) / GK) / (float)splits;
    const float load = (float)((g.m + v.rows - 1) / v.rows) * (float)((g.n + v.cols - 1) / v.cols) * (float)splits / (float)sms;
    return v.launch + slices * (load <= 1.f ? v.alone + (v.full - v.alone) * load : v.full * ceilf(load));
}

int launch_variant(int i, const GemmCall& g, int width, cudaStream_t stream) {
    switch (i) {
        case 0: return launch_gemm_pair<256>(g, width, stream);
        case 1: return launch_gemm<256>(g, stream);
        case 2: return launch_gemm<128>(g, stream);
        case 3: return launch_gemm<64>(g, stream);
        default: return launch_gemm<32>(g, stream);
    }
}

}  // namespace

int launch_gemm_call(const GemmCall& call, cudaStream_t stream) {
    GemmCall g = call;
    const int sms = sm_count();
    g.splits = 1;
    // a long K over few tiles goes to the kernel that cuts K (144 rows, N = 640, K = 2560: 7.6 us against 8.2)
    if (!g.a_mn && !g.b_mn && g.epilogue <= GEMM_ADD && g.k >= 16 * GK && 2 * ((g.m + GM - 1) / GM) * ((g.n + 31) / 32) <= sms &&
        g.lda == g.k && g.ldb == g.k && g.ldc == g.n && (g.epilogue != GEMM_ADD || g.aux == g.c))
        return launch_rows_tc(g.dtype, g.m, g.n, g.k, g.a, g.b, g.bias, g.c, g.epilogue, stream, g.chain & kChainDependent);
    int best = -1, width = 256;
    float least = 0.f;
    for (int i = 0; i < 5; ++i) {
        if ((g.a_mn || g.b_mn) && (i == 1 || i == 4)) continue;  // built for the layouts of a backward pass: 256 x 256, 128, 64
        const float t = variant_cost(i, g, 1, sms, &width);
        if (best < 0 || t < least) {
            best = i;
            least = t;
        }
    }
    return launch_variant(best, g, width, stream);
}

int gemm_most_splits(int k) { return k / (4 * GK) < 32 ? k / (4 * GK) : 32; }

// A product with a long k and a small output (a weight gradient: k = rows of the batch): k is cut into as many ranges as
// pays, each leaving fp32 sums in `partial`, and *splits says how many (1: the output itself was written).  Every range
// costs a trip of m x n fp32 values through memory and back, at about 4 TB/s, and a launch.
int launch_gemm_splitk(const GemmCall& call, size_t partial_bytes, int* splits, cudaStream_t stream) {
    GemmCall g = call;
    const int sms = sm_count();
    const size_t out = (size_t)g.m * g.n * sizeof(float);
    int best = 0, best_s = 1, best_width = 256;
    float least = 0.f;
    for (int i = 0; i < 4; ++i) {
        if (i == 1) continue;
        for (int s = 1; s == 1 || (s <= gemm_most_splits(g.k) && s * out <= partial_bytes); ++s) {
            int width = 256;
            const float t = variant_cost(i, g, s, sms, &width) + (s > 1 ? 2.5f + 2.f * (float)(s * out) / 4e6f : 0.f);
            if ((i == 0 && s == 1) || t < least) {
                best = i;
                best_s = s;
                best_width = width;
                least = t;
            }
        }
    }
    *splits = g.splits = best_s;
    return launch_variant(best, g, best_width, stream);
}

int launch_linear(const tmw_linear_desc& d, const void* a, const void* w, const void* bias, void* c, cudaStream_t stream,
                  int chain) {
    GemmCall g;
    g.dtype = d.dtype; g.m = d.m; g.n = d.n; g.k = d.k;
    g.a = a; g.lda = d.lda; g.b = w; g.ldb = d.ldw; g.c = c; g.ldc = d.ldc;
    g.bias = bias; g.epilogue = d.epilogue; g.chain = chain;
    return launch_gemm_call(g, stream);
}

}  // namespace tmw
