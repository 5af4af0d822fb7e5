// A decode step of up to 8 sequences as ONE kernel that stays on the chip: one CTA per SM, all layers and the head.
//
// With a launch per product and attention (decode_step.cu) a layer is five dependent launches of 3 to 4 us for 10 MB of
// weights, which the memory delivers in 1.5: a link costs its launch, its drain and the cold start of its loads, whatever it
// computes.  Here a link is one exchange through L2, and what does not depend on the step is under way long before it is
// needed: a pair's keys and values in shared memory one layer ahead, weights in L2 one layer ahead and in registers before a
// phase's input has arrived, the head's weights in L2 under the layers.
//
// Exchange.  Rows travel as 8-byte words of two 16-bit values and a 32-bit tag, written and read as single 64-bit accesses:
// a reader that sees the tag of its phase has the values with it, so there is no barrier, no fence and no flag to fetch first
// (store -> poll is one trip through L2; a grid-wide barrier is a fence, an arrival, a poll and then the load, about three).
// The words are zeroed in front of the first step, and a tag is used once.  A buffer is written again one layer later, by CTAs
// whose input depends on every reader of the layer before: a CTA sends nothing of a phase before its own reads of it are done,
// and every phase takes in the whole rows of the phase in front.
//
// All CTAs have to be resident (a reader polls for what another CTA sends): the launch is cooperative, and a device that
// cannot hold it gets the chain of launches.  Every wait is bounded; when one expires, the polls of all CTAs end, the status
// word says so, and the copies in flight are still waited for.
//
// What bounds it: instructions.  A layer is about 17 000 cycles for five exchanges of 500 to 900 (store to load, within a die
// and across); the rest is what the warps issue between a poll that succeeds and the words that they send, about 10 cycles per
// instruction and warp, a third of them waiting for the slowest warp at a barrier.  So the code of a phase stands once, in a
// loop over the half layers, sums of squares and scores are mma, and nothing is computed twice.  Twelve warps, three per
// scheduler, without register spills: 159 us for 16 layers with a vocabulary of 8000 and one sequence, 211 with eight; sixteen
// warps (which spill) 171 and 220, ten 183 and 235, eight 175 and 228.  Tried in an earlier form with sixteen warps: scores and
// weighted sums on CUDA cores took 5000 cycles per layer, as mma 3200, the most of it shared memory (135 KB per pair); code of
// its own for each of the four products, a phase's weights loaded a phase ahead, pauses between polls, a poll of one word in
// front of the full one and a barrier behind every send gained nothing or lost.
//
// 16 layers of width 640, vocabulary 50 000, window 512, one sequence: 313 us as a chain of launches, 172 as one kernel; eight
// prompts of 300 continued by 48 tokens: 17.3 and 10.9 ms.
#include <math_constants.h>

#include "tc_ptx.cuh"
#include "tmw_common.cuh"

namespace tmw {
namespace {

constexpr int kWarps = 12, kThreads = 32 * kWarps, kRows = 8;  // kRows: sequences at most, half an mma's rows
constexpr int kHeadDim = 64, kRowBytes = kHeadDim * 2;
constexpr int kMaxLayers = 32;                       // the table travels as a kernel parameter (4 KB)
constexpr int kMaxDim = 768, kMaxHidden = 3072;
constexpr int kInChunks = (kMaxDim / 32 + kWarps - 1) / kWarps;  // chunks of 32 elements of k that a warp has, at most
constexpr int kMaxGroup = (768 / kWarps + 15) / 16 * 16;                        // keys that a warp has on chip: four tiles of 16
constexpr int kSmemLimit = 227 * 1024;

struct HalfLayer {  // norm -> product -> (attention | GELU) -> product + residual
    const void *norm, *w_in, *b_in, *w_out, *b_out;
};
struct LayerTable {
    HalfLayer half[2];  // attention, MLP
    void *k_ring, *v_ring;
    const void *k_pers, *v_pers;
    float scale_log2;
};

struct ResidentParams {
    LayerTable layer[kMaxLayers];
    const void *tokens, *positions, *norm, *head;
    const int64_t* ids;
    const int32_t* pos;
    const unsigned long long* best_in;  // the step's tokens as [CTA][rows] keys of the step before, or nullptr: ids
    unsigned long long* best_out;       // this step's keys, or nullptr
    int64_t* out;                       // where the tokens of best_in go
    long long out_stride;
    void* logits;
    uint64_t *x, *qkv, *o, *y, *f;      // exchange buffers
    int *abort, *status;
    uint32_t tag0;                      // of the embedded rows; layer l uses tag0 + l + 1
    int rows, layers, dim, hidden, heads, vocab, slots, np, max_pos, advance, group_keys, nt_qkv, nt_fc1;
    float eps, inv_dim;
};

__device__ __forceinline__ uint4 ld_weights(const void* p) {  // read once per step: past L1
    uint4 r;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p));
    return r;
}
__device__ __forceinline__ void prefetch_l2(const void* p, long long bytes) {
    if (bytes > 0) asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"((uint32_t)bytes) : "memory");
}
__device__ __forceinline__ void ld_words(const uint64_t* p, uint64_t& a, uint64_t& b) {
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}
// Rows that all CTAs wait for are sent to kCopies places, `copy` words apart, and a CTA polls one of them, so that fewer poll the
// same lines of L2 (16 layers, one | eight sequences, us: with a vocabulary of 8000 one copy 163 | 211, two 159 | 211, four
// 160 | 212; with 50 000 172 | 222, 175 | 222, 176 | 223).
constexpr int kCopies = 2;
__device__ __forceinline__ void st_word(uint64_t* p, uint32_t bits, uint32_t tag) {
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(((uint64_t)tag << 32) | bits) : "memory");
}

__device__ __forceinline__ void st_copies(uint64_t* p, int copy, uint32_t bits, uint32_t tag) {
#pragma unroll
    for (int i = 0; i < kCopies; ++i) st_word(p + i * copy, bits, tag);
}

// what a CTA shares; the variable part (partial sums, ring rows) follows in dynamic shared memory
struct KeyRange {  // a warp's keys of a pair
    int lo, hi, slot_new, sequence, head;
};
constexpr int kSums = (kWarps + 3) / 4 * 4;
struct Shared {
    LayerTable layer[kMaxLayers];  // (out of the parameters: a first touch in the constant cache is a trip to L2, every layer)
    long long id[kRows];
    int pos[kRows], bad[kRows];
    unsigned long long best[kRows];
    __align__(16) float ss[kRows][kSums];
    __align__(16) float part[kWarps][kHeadDim + 2];
    KeyRange range[kWarps];
    int abort;
};

// asked by a poll now and then: whether to give up, because it has waited for about a second or another poll of the grid has
__device__ __noinline__ bool patience_over(volatile int* grid_abort, int* status, volatile int* local, long long t0) {
    if (*local) return true;
    const bool late = clock64() - t0 > ptx::kWaitLimitCycles;
    if (late || *grid_abort) {
        *local = 1;
        *grid_abort = 1;
        if (late) atomicCAS(status, 0, (int)TMW_ERR_DEVICE_TIMEOUT);
        return true;
    }
    return false;
}

// Eight values from four words, of up to N places `kWarps` chunks of 32 columns apart, as soon as all of them carry the tag.  `n`:
// how many places there are for this lane; the others are zeros.  The warp leaves together.
constexpr int kPlace = kWarps * 32 / 2;  // words

template <int N>
__device__ __forceinline__ void receive(uint4 (&out)[N], const uint64_t* src, int n, uint32_t tag, const ResidentParams& p, Shared& sh) {
    uint64_t v[N][4] = {};
    long long t0 = 0;
    uint32_t spins = 0;
#pragma unroll 1
    for (;;) {
#pragma unroll
        for (int i = 0; i < N; ++i)
            if (i < n) {
                ld_words(src + i * kPlace, v[i][0], v[i][1]);
                ld_words(src + i * kPlace + 2, v[i][2], v[i][3]);
            }
        uint32_t other = 0u;
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const uint32_t want = i < n ? tag : 0u;
#pragma unroll
            for (int j = 0; j < 4; ++j) other |= (uint32_t)(v[i][j] >> 32) ^ want;
        }
        if (!__any_sync(0xffffffffu, other != 0u)) break;
        if (++spins == 1u) t0 = clock64();
        if ((spins & 63u) == 0u && __any_sync(0xffffffffu, patience_over(p.abort, p.status, &sh.abort, t0))) break;
    }
#pragma unroll
    for (int i = 0; i < N; ++i) out[i] = make_uint4((uint32_t)v[i][0], (uint32_t)v[i][1], (uint32_t)v[i][2], (uint32_t)v[i][3]);
}

// N words per lane, at `stride` words from each other, the first only or (`all`) every one of them
template <int N>
__device__ __forceinline__ void receive_words(uint32_t (&out)[N], const uint64_t* src, int stride, bool all, uint32_t tag,
                                              const ResidentParams& p, Shared& sh) {
    uint64_t v[N] = {};
    long long t0 = 0;
    uint32_t spins = 0;
#pragma unroll 1
    for (;;) {
        uint32_t other = 0u;
#pragma unroll
        for (int i = 0; i < N; ++i)
            if (i == 0 || all) asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v[i]) : "l"(src + i * stride) : "memory");
#pragma unroll
        for (int i = 0; i < N; ++i)
            if (i == 0 || all) other |= (uint32_t)(v[i] >> 32) ^ tag;
        if (!__any_sync(0xffffffffu, other != 0u)) break;
        if (++spins == 1u) t0 = clock64();
        if ((spins & 63u) == 0u && __any_sync(0xffffffffu, patience_over(p.abort, p.status, &sh.abort, t0))) break;
    }
#pragma unroll
    for (int i = 0; i < N; ++i) out[i] = (uint32_t)v[i];
}

template <typename T>
__device__ __forceinline__ uint32_t pack(float a, float b) {
    T w[2] = {from_f32<T>(a), from_f32<T>(b)};
    return *reinterpret_cast<const uint32_t*>(w);
}
template <typename T>
__device__ __forceinline__ float2 unpack(uint32_t raw) {
    const T* w = reinterpret_cast<const T*>(&raw);
    return make_float2(to_f32<T>(w[0]), to_f32<T>(w[1]));
}

// Partial sums of the warps, [warp][row][column], in rows of 24 floats for the products with a norm (up to 24 columns) and of
// 8 for those with the residual; the 8-byte accesses meet no bank twice.
// Outputs: a lane has row lane % 8 and two columns of an eight, a warp an eight.
constexpr int kInStride = 24, kOutStride = 8;

__device__ __forceinline__ void put_partial(float* red, int stride, const float (&acc)[4], int warp, int g, int t) {
    *reinterpret_cast<float2*>(red + (warp * kRows + g) * stride + 2 * t) = make_float2(acc[0], acc[1]);
}
__device__ __forceinline__ float2 sum_partial(const float* red, int stride, int row) {
    float2 v[4] = {};
    const float* from = red + row * stride;
#pragma unroll
    for (int s = 0; s < kWarps; ++s) {
        const float2 u = *reinterpret_cast<const float2*>(from + s * kRows * stride);
        v[s & 3].x += u.x;
        v[s & 3].y += u.y;
    }
    return make_float2((v[0].x + v[1].x) + (v[2].x + v[3].x), (v[0].y + v[1].y) + (v[2].y + v[3].y));
}

// Rows from the exchange, normalised, as the mma fragments of this warp's `n` chunks of 32 columns: a thread of a quad takes
// eight adjacent values of a chunk, the same ones for both operands, so their order does not matter.  The sums of squares are
// the diagonal of x x^T, two more mma per chunk.
template <typename T>
__device__ __forceinline__ void normed_rows(uint4 (&a)[kInChunks], const uint4 (&gain)[kInChunks], const uint64_t* x, int n, uint32_t tag,
                                            const ResidentParams& p, Shared& sh, int warp, int g, int t) {
    float gains[kInChunks][8];
#pragma unroll
    for (int i = 0; i < kInChunks; ++i) load8<T>(reinterpret_cast<const T*>(&gain[i]), gains[i]);
    receive<kInChunks>(a, x + ((blockIdx.x % kCopies * p.rows + g) * p.dim + warp * 32 + t * 8) / 2, g < p.rows ? n : 0, tag, p, sh);
    if (n > 0) {
        float c[4] = {};
#pragma unroll
        for (int i = 0; i < kInChunks; ++i)
            if (i == 0 || i < n) {
                mma_16816<T>(c, a[i].x, 0u, a[i].y, 0u, a[i].x, a[i].y);
                mma_16816<T>(c, a[i].z, 0u, a[i].w, 0u, a[i].z, a[i].w);
            }
        if (t == g >> 1) sh.ss[g][warp] = (g & 1) ? c[1] : c[0];
    }
    __syncthreads();
    if (n <= 0) return;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);  // (warps without a chunk left zeros at the start)
#pragma unroll
    for (int q = 0; q < kSums / 4; ++q) {
        const float4 u = *reinterpret_cast<const float4*>(&sh.ss[g][q * 4]);
        s.x += u.x;
        s.y += u.y;
        s.z += u.z;
        s.w += u.w;
    }
    // (one rounded function: 0.7 us of a step of 170 more than the hardware's approximation with a step of Newton's method;
    // 1 / sqrtf of a divided sum, which rounds three times, takes 8 us)
    const float inv = __frsqrt_rn(fmaf((s.x + s.y) + (s.z + s.w), p.inv_dim, p.eps));
#pragma unroll
    for (int i = 0; i < kInChunks; ++i)
        if (i == 0 || i < n) {
            float v[8];
            load8<T>(reinterpret_cast<const T*>(&a[i]), v);
#pragma unroll
            for (int e = 0; e < 8; ++e) v[e] = v[e] * inv * gains[i][e];
            store8<T>(reinterpret_cast<T*>(&a[i]), v);
        }
}

// The weights of a phase are loaded into registers in front of its poll.  In: nt * 8 rows
// of this CTA; out: eight rows.
constexpr int kInTiles = 3;
struct InWeights {
    uint4 w[kInChunks][kInTiles], gain[kInChunks];
};
template <typename T>
__device__ __forceinline__ void load_in(InWeights& r, const ResidentParams& p, const HalfLayer& l, int n, int nt) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const int n0 = blockIdx.x * nt * 8, mine = n0 < n ? (p.dim / 32 - warp + kWarps - 1) / kWarps : 0, k = warp * 32 + t * 8;
    const T* src = static_cast<const T*>(l.w_in) + (n0 + g) * p.dim + k;
    const T* gain = static_cast<const T*>(l.norm) + k;
#pragma unroll
    for (int i = 0; i < kInChunks; ++i) {
#pragma unroll
        for (int j = 0; j < kInTiles; ++j) {
            r.w[i][j] = make_uint4(0u, 0u, 0u, 0u);
            if (i < mine && j < nt && n0 + j * 8 < n) r.w[i][j] = ld_weights(src + j * 8 * p.dim + i * (kWarps * 32));  // (n: eights)
        }
        r.gain[i] = make_uint4(0u, 0u, 0u, 0u);
        if (i < mine) r.gain[i] = ld_weights(gain + i * (kWarps * 32));
    }
}
template <typename T, int CH>
__device__ __forceinline__ void load_out(uint4 (&w)[CH], const ResidentParams& p, const HalfLayer& l, int k) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const int n0 = blockIdx.x * 8, mine = n0 < p.dim ? (k / 32 - warp + kWarps - 1) / kWarps : 0;
    const T* src = static_cast<const T*>(l.w_out) + (n0 + g) * k + warp * 32 + t * 8;
#pragma unroll
    for (int i = 0; i < CH; ++i) {
        w[i] = make_uint4(0u, 0u, 0u, 0u);
        if (i < mine) w[i] = ld_weights(src + i * (kWarps * 32));
    }
}

// dst = round(norm(x) w^T + bias), or its GELU.  A CTA has nt * 8 columns, its warps interleaved chunks of k.
template <typename T>
__device__ __forceinline__ void norm_product(const ResidentParams& p, Shared& sh, float* red, const InWeights& in, const HalfLayer& l, int n,
                                             int nt, bool gelu, const uint64_t* x, uint32_t tag_in, uint64_t* dst, uint32_t tag_out) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const int n0 = blockIdx.x * nt * 8, mine = (p.dim / 32 - warp + kWarps - 1) / kWarps;  // this warp's chunks (0 or less: none)
    if (n0 >= n) return;
    const int row = lane & 7, col = warp * 8 + (lane >> 3) * 2;
    const bool out = warp < nt && row < p.rows && n0 + col < n;
    uint32_t bias = 0u;
    if (l.b_in != nullptr && out) bias = *reinterpret_cast<const uint32_t*>(static_cast<const T*>(l.b_in) + n0 + col);
    uint4 a[kInChunks];
    normed_rows<T>(a, in.gain, x, mine, tag_in, p, sh, warp, g, t);
#pragma unroll
    for (int j = 0; j < kInTiles; ++j)
        if (j < nt) {
            float acc[4] = {};
#pragma unroll
            for (int i = 0; i < kInChunks; ++i)
                if (i < mine) {
                    mma_16816<T>(acc, a[i].x, 0u, a[i].y, 0u, in.w[i][j].x, in.w[i][j].y);
                    mma_16816<T>(acc, a[i].z, 0u, a[i].w, 0u, in.w[i][j].z, in.w[i][j].w);
                }
            put_partial(red + j * 8, kInStride, acc, warp, g, t);
        }
    __syncthreads();
    if (out) {
        float2 v = sum_partial(red + col, kInStride, row);
        const float2 b = unpack<T>(bias);
        v.x += b.x;
        v.y += b.y;
        if (gelu) {
            v.x = gelu_erf(v.x);
            v.y = gelu_erf(v.y);
        }
        uint64_t* to = dst + (row * n + n0 + col) / 2;
        if (gelu) st_copies(to, p.rows * n / 2, pack<T>(v.x, v.y), tag_out);
        else st_word(to, pack<T>(v.x, v.y), tag_out);  // (queries, keys and values have few readers)
    }
}

// x' = x + round(a w^T + bias) for eight columns of every row; x stays in the thread that computes it
constexpr int kOutChunks = (kMaxHidden / 32 + kWarps - 1) / kWarps;  // chunks of k that a warp has at most
template <typename T>
__device__ __forceinline__ void residual_product(const ResidentParams& p, Shared& sh, float* red, const uint4 (&w)[kOutChunks],
                                                 const HalfLayer& l, const uint64_t* src, int k, uint64_t* dst, uint32_t tag, uint32_t& x) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const int n0 = blockIdx.x * 8, mine = (k / 32 - warp + kWarps - 1) / kWarps;
    if (n0 >= p.dim) return;
    const int row = lane & 7, col = (lane >> 3) * 2;
    const bool out = warp == 0 && row < p.rows;
    uint32_t bias = 0u;
    if (l.b_out != nullptr && out) bias = *reinterpret_cast<const uint32_t*>(static_cast<const T*>(l.b_out) + n0 + col);
    float acc[4] = {};
    uint4 a[kOutChunks];
    receive<kOutChunks>(a, src + ((blockIdx.x % kCopies * p.rows + g) * k + warp * 32 + t * 8) / 2, g < p.rows ? mine : 0, tag, p, sh);
#pragma unroll
    for (int i = 0; i < kOutChunks; ++i)
        if (i < mine) {
            mma_16816<T>(acc, a[i].x, 0u, a[i].y, 0u, w[i].x, w[i].y);
            mma_16816<T>(acc, a[i].z, 0u, a[i].w, 0u, w[i].z, w[i].w);
        }
    put_partial(red, kOutStride, acc, warp, g, t);
    __syncthreads();
    if (out) {
        const float2 v = sum_partial(red + col, kOutStride, row), old = unpack<T>(x), b = unpack<T>(bias);
        const float2 r = unpack<T>(pack<T>(v.x + b.x, v.y + b.y));
        x = pack<T>(old.x + r.x, old.y + r.y);
        st_copies(dst + (row * p.dim + n0 + col) / 2, p.rows * p.dim / 2, x, tag);
    }
}

// The keys of a (sequence, head) pair - persistent rows, then the ring slots in use - are cut into a range per warp.
// A warp has up to kMaxGroup keys and values of its range in shared memory of its own and, once it is done with them, fetches
// the next: of the same range where it is longer, else of the next layer, whose rows are then on their way while the products of
// this one run.  A CTA has one pair or none.
__device__ __forceinline__ KeyRange key_range(const ResidentParams& p, const Shared& sh, int pair, int warp) {
    KeyRange r;
    r.sequence = pair / p.heads;
    r.head = pair - r.sequence * p.heads;
    const int t = max(sh.pos[r.sequence], 0);
    const int n = p.np + min(t, p.slots - 1) + 1, per = (n + kWarps - 1) / kWarps;  // (t may be 2^31 - 1: no t + 1)
    r.lo = min(n, warp * per);
    r.hi = min(n, r.lo + per);
    r.slot_new = t % p.slots;
    return r;
}

// rows of 128 bytes, their 16-byte units exchanged by the row (ldmatrix reads eight rows without bank conflicts)
__device__ __forceinline__ uint32_t unit_offset(int row, int unit) { return (uint32_t)(row * kRowBytes + ((unit ^ (row & 7)) << 4)); }

// (as much of a range as there is room for, of the keys or of the values)
__device__ __forceinline__ void fetch_rows(const ResidentParams& p, const void* ring_, const void* pers_, const KeyRange& range, int pair, int at,
                                           uint32_t mem, int lane) {
    const int n = min(p.group_keys, range.hi - at), unit = lane & 7;
    const char* ring = static_cast<const char*>(ring_) + ((long long)pair * p.slots - p.np) * kRowBytes + unit * 16;
    const char* pers = static_cast<const char*>(pers_) + range.head * p.np * kRowBytes + unit * 16;
#pragma unroll 3
    for (int row = lane >> 3; row < n; row += 4) {
        const int i = at + row;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(mem + unit_offset(row, unit)),
                     "l"((i < p.np ? pers : ring) + (long long)i * kRowBytes)
                     : "memory");
    }
}

__device__ __forceinline__ void ldmatrix(uint32_t (&r)[4], uint32_t at) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at) : "memory");
}
__device__ __forceinline__ void ldmatrix_trans(uint32_t (&r)[4], uint32_t at) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at) : "memory");
}

// Scores of 16 keys are q K^T with q in all rows of the product, so that every lane has those of the keys 2t, 2t + 1, 2t + 8
// and 2t + 9: as the second product, V^T P, wants its P.  The weights keep their 24 bits: columns 0, 1 and 2 of P are their
// first, second and third 16-bit part.  fp16 has not the exponents for that: its weights are 2^15 times larger (accumulators and
// sums with them, so the quotient is the same), and the second and third part 2^11 and 2^22 times, until the warps are merged.
// So a weight has its 24 bits down to 2^-37 of the largest of its warp, and what is lost of a smaller one is below 2^-62.
// (16 layers, window 512, one sequence: 1 us of 170 more than unscaled parts.)
template <typename T>
struct Parts {
    static constexpr float kRaise = 1.f, kNext = 1.f;  // how many times larger the weights are; a part, relative to the one before
};
template <>
struct Parts<__half> {
    static constexpr float kRaise = 32768.f, kNext = 2048.f;
};
template <typename T>
__device__ __forceinline__ void attention(const ResidentParams& p, Shared& sh, int pair, unsigned char* mem, int layer, uint32_t tag) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const LayerTable& l = sh.layer[layer];
    const uint32_t k_mem = ptx::smem_u32(mem), v_mem = k_mem + p.group_keys * kRowBytes;
    const float part1 = g >= 1 ? -1.f : 0.f, part2 = g >= 2 ? -1.f : 0.f;  // what a lane's column leaves out of a weight
    const float raise1 = g >= 1 ? Parts<T>::kNext : 1.f, raise2 = g >= 2 ? Parts<T>::kNext : 1.f;
    const uint32_t mask = g <= 2 ? 0xffffffffu : 0u;
    const KeyRange range = sh.range[warp];
    const int i_new = p.np + range.slot_new;
    const bool brings = i_new >= range.lo && i_new < range.hi;
    // query and, in the warp whose range holds the new token's slot, its key and value: two elements per lane
    uint32_t got[3];
    receive_words<3>(got, p.qkv + (range.sequence * 3 * p.dim + range.head * kHeadDim) / 2 + lane, p.dim / 2, brings, tag, p, sh);
    uint32_t q[4][2];
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
        q[kk][0] = __shfl_sync(0xffffffffu, got[0], kk * 8 + t);
        q[kk][1] = __shfl_sync(0xffffffffu, got[0], kk * 8 + 4 + t);
    }
    float m = -CUDART_INF_F, sum = 0.f, acc[4][4] = {};
    int at = range.lo;
    do {
        const int n = min(p.group_keys, range.hi - at);
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncwarp();
        if (brings && i_new >= at && i_new < at + n) {  // the copy brought what falls out of the window
            const uint32_t to = unit_offset(i_new - at, lane >> 2) + (lane & 3) * 4;
            *reinterpret_cast<uint32_t*>(mem + to) = got[1];
            *reinterpret_cast<uint32_t*>(mem + p.group_keys * kRowBytes + to) = got[2];
            __syncwarp();
        }
        uint32_t off[kMaxGroup / 16];
        float s[kMaxGroup / 16][4], top = -CUDART_INF_F;
        bool any = false;
#pragma unroll
        for (int c = 0; c < kMaxGroup / 16; ++c)
            if (c * 16 < n) {
                const int row = min(c * 16 + (lane & 7) + (lane >> 4) * 8, n - 1);  // (no key of its own: the last one, at weight zero)
                off[c] = unit_offset(row, (lane >> 3) & 1);
                float lo[4] = {}, hi[4] = {};
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) {
                    uint32_t k[4];
                    ldmatrix(k, k_mem + (off[c] ^ (kk << 5)));
                    mma_16816<T>(lo, q[kk][0], 0u, q[kk][1], 0u, k[0], k[1]);
                    mma_16816<T>(hi, q[kk][0], 0u, q[kk][1], 0u, k[2], k[3]);
                }
                const int left = n - c * 16 - 2 * t;
                s[c][0] = left > 0 ? lo[0] * l.scale_log2 : -CUDART_INF_F;
                s[c][1] = left > 1 ? lo[1] * l.scale_log2 : -CUDART_INF_F;
                s[c][2] = left > 8 ? hi[0] * l.scale_log2 : -CUDART_INF_F;
                s[c][3] = left > 9 ? hi[1] * l.scale_log2 : -CUDART_INF_F;
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    top = fmaxf(top, s[c][e]);
                    any = any || s[c][e] != -CUDART_INF_F;  // (NaN too)
                }
            }
        top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
        top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
        any = __any_sync(0xffffffffu, any);
        const float m_new = fmaxf(m, top), base = any ? m_new : 0.f;
        if (at > range.lo) {
            const float alpha = any ? exp2f(m - m_new) : 1.f;
            sum *= alpha;
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[j][e] *= alpha;
        }
        m = m_new;
#pragma unroll
        for (int c = 0; c < kMaxGroup / 16; ++c)
            if (c * 16 < n) {
                uint32_t b[2];
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    // (raised behind the exponential: 15 more in front of it would be rounded by the size of the scores)
                    float2 w = make_float2(exp2f(s[c][2 * e] - base) * Parts<T>::kRaise, exp2f(s[c][2 * e + 1] - base) * Parts<T>::kRaise);
                    sum += w.x + w.y;
                    float2 h = unpack<T>(pack<T>(w.x, w.y));
                    w = make_float2(fmaf(h.x, part1, w.x) * raise1, fmaf(h.y, part1, w.y) * raise1);
                    h = unpack<T>(pack<T>(w.x, w.y));
                    b[e] = pack<T>(fmaf(h.x, part2, w.x) * raise2, fmaf(h.y, part2, w.y) * raise2) & mask;
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    uint32_t v[4];
                    ldmatrix_trans(v, v_mem + (off[c] ^ (j << 5)));
                    mma_16816<T>(acc[j], v[0], v[1], v[2], v[3], b[0], b[1]);
                }
            }
        at += p.group_keys;
        if (at < range.hi) {  // more of this range
            __syncwarp();
            fetch_rows(p, l.k_ring, l.k_pers, range, pair, at, k_mem, lane);
            fetch_rows(p, l.v_ring, l.v_pers, range, pair, at, v_mem, lane);
        }
    } while (at < range.hi);
    // merge the warps (the sums of the layer before have been read: this layer's query depends on what came of them)
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float lower0 = t == 0 ? 1.f : 1.f / (Parts<T>::kNext * Parts<T>::kNext), lower1 = 1.f / Parts<T>::kNext;
        float2 v = make_float2(fmaf(acc[j][1], lower1, acc[j][0] * lower0), fmaf(acc[j][3], lower1, acc[j][2] * lower0));
        v.x += __shfl_xor_sync(0xffffffffu, v.x, 1);
        v.y += __shfl_xor_sync(0xffffffffu, v.y, 1);
        if (t == 0) {
            sh.part[warp][j * 16 + g] = v.x;
            sh.part[warp][j * 16 + 8 + g] = v.y;
        }
    }
    if (lane == 0) *reinterpret_cast<float2*>(&sh.part[warp][kHeadDim]) = make_float2(m, sum);
    __syncthreads();
    if (warp == 0) {
        const float2 ml = lane < kWarps ? *reinterpret_cast<const float2*>(&sh.part[lane][kHeadDim]) : make_float2(-CUDART_INF_F, 0.f);
        float top = ml.x;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
        const float w = exp2f(ml.x - (top > -CUDART_INF_F ? top : 0.f));
        float all = ml.y * w;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) all += __shfl_xor_sync(0xffffffffu, all, o);
        float2 r = make_float2(0.f, 0.f);
#pragma unroll
        for (int i = 0; i < kWarps; ++i) {
            const float w_i = __shfl_sync(0xffffffffu, w, i);
            const float2 v = *reinterpret_cast<const float2*>(&sh.part[i][lane * 2]);
            r.x = fmaf(v.x, w_i, r.x);
            r.y = fmaf(v.y, w_i, r.y);
        }
        const float inv = all == 0.f ? 0.f : 1.f / all;
        st_copies(p.o + (range.sequence * p.dim + range.head * kHeadDim) / 2 + lane, p.rows * p.dim / 2, pack<T>(r.x * inv, r.y * inv),
                  tag);
    }
    // nobody waits for the rest: the new token's row for the steps behind (the next layer's first rows: see the kernel)
    if (brings) {
        const long long to = ((long long)pair * p.slots + range.slot_new) * (kHeadDim / 2) + lane;
        static_cast<uint32_t*>(l.k_ring)[to] = got[1];
        static_cast<uint32_t*>(l.v_ring)[to] = got[2];
    }
}

// order of the greedy choice: larger value first (NaN largest), then smaller index
__device__ __forceinline__ unsigned long long choice_key(float v, int index) {
    const uint32_t u = __float_as_uint(v + 0.0f);  // (-0 equals +0)
    const uint32_t order = v != v ? 0xffffffffu : (u & 0x80000000u) ? ~u : u | 0x80000000u;
    return ((unsigned long long)order << 32) | (uint32_t)~index;
}
__device__ __forceinline__ unsigned long long larger(unsigned long long a, unsigned long long b) { return a > b ? a : b; }

// the token that the CTAs' keys [ctas][rows] decide for a row; the whole warp gets it
__device__ __forceinline__ long long chosen(const unsigned long long* best, int ctas, int rows, int row, int lane) {
    unsigned long long key = 0;
    for (int i = lane; i < ctas; i += 32) key = larger(key, best[(long long)i * rows + row]);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) key = larger(key, __shfl_xor_sync(0xffffffffu, key, off));
    return (long long)(uint32_t)~(uint32_t)key;
}

// logits = norm(x) head^T: the rows, normalised, in shared memory for all warps; a warp takes tiles of eight vocabulary rows
// with the whole of k, kHeadDepth loads of 16 bytes per lane in flight
// half layers in front of the head under which its weights go into L2 (under all of them: 178 us instead of 175)
constexpr int kHeadSteps = 8;
constexpr int kHeadDepth = 20;

template <typename T>
__device__ __forceinline__ void head_product(const ResidentParams& p, Shared& sh, unsigned char* mem, uint32_t tag) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int chunks = p.dim / 32, tiles = (p.vocab + 7) / 8, step = gridDim.x * kWarps;
    // a tile's chunks in equal groups of at most kHeadDepth; the group behind the one in use is being loaded
    const int groups = (chunks + kHeadDepth - 1) / kHeadDepth, per = (chunks + groups - 1) / groups;
    int tile = warp * gridDim.x + blockIdx.x, group = 0;
    const T* base = static_cast<const T*>(p.head) + t * 8;
    uint4 w[kHeadDepth] = {};
    auto source = [&](int tl, int gr) { return base + (long long)min(tl * 8 + g, p.vocab - 1) * p.dim + gr * per * 32; };
    {
        const T* src = source(tile, 0);
#pragma unroll
        for (int d = 0; d < kHeadDepth; ++d)
            if (d < per && tile < tiles) w[d] = ld_weights(src + d * 32);
    }
    const int stride = p.dim * 2 + 64;  // bytes of a row: eight lanes of a 16-byte access fall on different banks
    {
        uint4 gain[kInChunks], a[kInChunks];
#pragma unroll
        for (int i = 0; i < kInChunks; ++i) {
            gain[i] = make_uint4(0u, 0u, 0u, 0u);
            if (warp + kWarps * i < chunks)
                gain[i] = *reinterpret_cast<const uint4*>(static_cast<const T*>(p.norm) + (warp + kWarps * i) * 32 + t * 8);
        }
        normed_rows<T>(a, gain, p.x, (chunks - warp + kWarps - 1) / kWarps, tag, p, sh, warp, g, t);
#pragma unroll
        for (int i = 0; i < kInChunks; ++i)
            if (warp + kWarps * i < chunks) *reinterpret_cast<uint4*>(mem + g * stride + (warp + kWarps * i) * 64 + t * 16) = a[i];
    }
    __syncthreads();
    unsigned long long best = 0ull;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    const bool wide = (p.vocab & 1) == 0;
    while (tile < tiles) {
        const int n = min(per, chunks - group * per);
        const bool last = group + 1 == groups;
        const int tile_next = last ? tile + step : tile, group_next = last ? 0 : group + 1;
        const int n_next = tile_next < tiles ? min(per, chunks - group_next * per) : 0;
        const T* src = source(tile_next, group_next);
        const unsigned char* row = mem + g * stride + group * per * 64 + t * 16;
#pragma unroll
        for (int d = 0; d < kHeadDepth; ++d) {
            if (d < n) {
                const uint4 v = *reinterpret_cast<const uint4*>(row + d * 64);
                mma_16816<T>(acc, v.x, 0u, v.y, 0u, w[d].x, w[d].y);
                mma_16816<T>(acc, v.z, 0u, v.w, 0u, w[d].z, w[d].w);
            }
            if (d < n_next) w[d] = ld_weights(src + d * 32);
        }
        if (last) {
            const int col = tile * 8 + 2 * t;
            const uint32_t two = pack<T>(acc[0], acc[1]);
            if (g < p.rows && col < p.vocab) {
                const float2 v = unpack<T>(two);
                T* dst = static_cast<T*>(p.logits) + (long long)g * p.vocab + col;
                best = larger(best, choice_key(v.x, col));
                if (col + 1 < p.vocab) best = larger(best, choice_key(v.y, col + 1));
                if (wide) {
                    *reinterpret_cast<uint32_t*>(dst) = two;
                } else {
                    dst[0] = from_f32<T>(acc[0]);
                    if (col + 1 < p.vocab) dst[1] = from_f32<T>(acc[1]);
                }
            }
            acc[0] = acc[1] = 0.f;
        }
        tile = tile_next;
        group = group_next;
    }
    if (p.best_out != nullptr) {
        best = larger(best, __shfl_xor_sync(0xffffffffu, best, 1));
        best = larger(best, __shfl_xor_sync(0xffffffffu, best, 2));
        if (t == 0) atomicMax(&sh.best[g], best);
        __syncthreads();
        if (tid < p.rows) p.best_out[(long long)blockIdx.x * p.rows + tid] = sh.best[tid];
    }
}

template <typename T>
__global__ void __launch_bounds__(kThreads, 1) decode_resident_kernel(const __grid_constant__ ResidentParams p) {
    extern __shared__ __align__(128) unsigned char dynamic[];
    __shared__ Shared sh;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, cta = blockIdx.x, ctas = gridDim.x;
    // Partial sums: one buffer for the products with a norm (whose sums of squares bring a barrier between the last readers and
    // the next writes), one each for the two with the residual (each has the other's barrier in between).  Then the ring rows.
    float *red = reinterpret_cast<float*>(dynamic), *red_out = red + kWarps * kRows * kInStride, *red_fc2 = red_out + kWarps * kRows * kOutStride;
    unsigned char* rows_mem = reinterpret_cast<unsigned char*>(red_fc2 + kWarps * kRows * kOutStride);
    unsigned char* mem = rows_mem + warp * (2 * p.group_keys * kRowBytes);
    for (int i = tid; i < p.layers * (int)(sizeof(LayerTable) / 8); i += kThreads)
        reinterpret_cast<uint64_t*>(sh.layer)[i] = reinterpret_cast<const uint64_t*>(p.layer)[i];
    if (tid == 0) sh.abort = 0;
    if (tid < kRows) sh.best[tid] = 0ull;
    for (int i = tid; i < kRows * kSums; i += kThreads) sh.ss[i / kSums][i % kSums] = 0.f;
    if (warp < p.rows) {
        long long id = 0;
        if (p.best_in != nullptr) {
            id = chosen(p.best_in, ctas, p.rows, warp, lane);
            if (cta == 0 && lane == 0) p.out[warp * p.out_stride] = id;
        } else {
            id = p.ids[warp];
        }
        if (lane == 0) {
            const int pos = p.pos[warp] + p.advance;
            const bool bad = id < 0 || id >= p.vocab || pos < 0 || pos >= p.max_pos;
            if (bad && cta == 0) atomicCAS(p.status, 0, (int)TMW_ERR_INVALID_ARGUMENT);
            sh.id[warp] = bad ? 0 : id;
            sh.pos[warp] = pos;
            sh.bad[warp] = bad;
        }
    }
    __syncthreads();
    // the embedded rows; from here on a thread keeps its two values of the residual stream (see residual_product)
    uint32_t x = 0;
    {
        const int row = lane & 7, col = cta * 8 + (lane >> 3) * 2;
        if (warp == 0 && row < p.rows && col < p.dim) {
            const int pos = sh.bad[row] ? 0 : sh.pos[row];  // (outside the table: a row of NaN, but a ring position all the same)
            const float2 a = unpack<T>(*reinterpret_cast<const uint32_t*>(static_cast<const T*>(p.tokens) + sh.id[row] * p.dim + col));
            const float2 b = unpack<T>(*reinterpret_cast<const uint32_t*>(static_cast<const T*>(p.positions) + (long long)pos * p.dim + col));
            x = sh.bad[row] ? pack<T>(CUDART_NAN_F, CUDART_NAN_F) : pack<T>(a.x + b.x, a.y + b.y);
            st_copies(p.x + (row * p.dim + col) / 2, p.rows * p.dim / 2, x, p.tag0);
        }
    }
    // (the pairs from the last CTA on: the first ones have the residual's columns as well)
    const int pair = ctas - 1 - cta;
    const bool attends = pair < p.rows * p.heads;
    if (attends) {
        const KeyRange r = key_range(p, sh, pair, warp);
        const LayerTable& l = sh.layer[0];
        fetch_rows(p, l.k_ring, l.k_pers, r, pair, r.lo, ptx::smem_u32(mem), lane);
        fetch_rows(p, l.v_ring, l.v_pers, r, pair, r.lo, ptx::smem_u32(mem) + p.group_keys * kRowBytes, lane);
        if (lane == 0) sh.range[warp] = r;
    }
    __syncwarp();

    // weights of half a layer that this CTA will read, into L2: by one lane of the last warp, at times when all wait
    auto prefetch = [&](const HalfLayer& h, bool mlp) {
        auto rows = [&](const void* w, int per, int total, int row_bytes) {
            const int r0 = cta * per, r1 = min(total, r0 + per);
            if (r0 < r1) prefetch_l2(static_cast<const char*>(w) + (long long)r0 * row_bytes, (r1 - r0) * row_bytes);
        };
        rows(h.w_in, (mlp ? p.nt_fc1 : p.nt_qkv) * 8, mlp ? p.hidden : 3 * p.dim, p.dim * 2);
        rows(h.w_out, 8, p.dim, (mlp ? p.hidden : p.dim) * 2);
        if (cta == ctas - 1) {
            prefetch_l2(h.norm, p.dim * 2);
            if (h.b_in != nullptr) prefetch_l2(h.b_in, p.hidden * 2);
            if (h.b_out != nullptr) prefetch_l2(h.b_out, p.dim * 2);
        }
    };
    if (warp == kWarps - 1 && ptx::elect_one()) {
        prefetch(sh.layer[0].half[0], false);
        prefetch(sh.layer[0].half[1], true);
    }
    __syncwarp();
    const int head_from = max(0, 2 * p.layers - kHeadSteps);
    const long long head_part = ((long long)p.vocab * p.dim * 2 / ((long long)ctas * (2 * p.layers - head_from))) & ~15ll;
    // (one loop over the halves of all layers: each phase's code once, which the instruction caches hold)
#pragma unroll 1
    for (int step = 0; step < 2 * p.layers; ++step) {
        const int l = step >> 1;
        const bool mlp = step & 1;
        const HalfLayer& half = sh.layer[l].half[mlp];
        const uint32_t tag = p.tag0 + l + 1;
        {
            InWeights in;
            load_in<T>(in, p, half, mlp ? p.hidden : 3 * p.dim, mlp ? p.nt_fc1 : p.nt_qkv);
            norm_product<T>(p, sh, red, in, half, mlp ? p.hidden : 3 * p.dim, mlp ? p.nt_fc1 : p.nt_qkv, mlp, mlp ? p.y : p.x,
                                mlp ? tag : tag - 1, mlp ? p.f : p.qkv, tag);
        }
        if (!mlp && attends) attention<T>(p, sh, pair, mem, l, tag);
        if (warp == kWarps - 1 && ptx::elect_one()) {  // this half of the next layer, and a part of the head
            if (l + 1 < p.layers) prefetch(sh.layer[l + 1].half[mlp], mlp);
            if (step >= head_from)
                prefetch_l2(static_cast<const char*>(p.head) + ((long long)(step - head_from) * ctas + cta) * head_part, head_part);
        }
        __syncwarp();
        {
            uint4 w[kOutChunks];
            load_out<T>(w, p, half, mlp ? p.hidden : p.dim);
            residual_product<T>(p, sh, mlp ? red_fc2 : red_out, w, half, mlp ? p.f : p.o, mlp ? p.hidden : p.dim, mlp ? p.x : p.y, tag, x);
        }
        // the next layer's keys, then its values, at times when the rows of the next phase are on their way (135 KB keep the load
        // path of an SM busy for 2700 cycles)
        if (attends && l + 1 < p.layers) {
            const LayerTable& next = sh.layer[l + 1];
            const KeyRange r = sh.range[warp];
            fetch_rows(p, mlp ? next.v_ring : next.k_ring, mlp ? next.v_pers : next.k_pers, r, pair, r.lo,
                       ptx::smem_u32(mem) + (mlp ? p.group_keys * kRowBytes : 0), lane);
        }
    }
    head_product<T>(p, sh, rows_mem, p.tag0 + p.layers);
    asm volatile("cp.async.wait_all;" ::: "memory");  // (nothing is in flight, unless a wait expired)
}

// the last choice of a generation: tokens[row], out[row * out_stride], pos[row] += advance
__global__ void __launch_bounds__(kThreads) decode_choice_kernel(const unsigned long long* best, int ctas, int rows, int64_t* tokens,
                                                                 int64_t* out, long long out_stride, int32_t* pos, int advance) {
    const int row = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (row >= rows) return;
    const long long id = chosen(best, ctas, rows, row, lane);
    if (lane == 0) {
        tokens[row] = id;
        out[row * out_stride] = id;
        pos[row] += advance;
    }
}

int columns_per_cta(int n) { return (n / 8 + sm_count() - 1) / sm_count(); }  // in units of eight

struct ResidentBuffers {
    int64_t abort, x, qkv, o, y, f, cleared, best, total;  // byte offsets; [0, cleared) is zero in front of the first step
};
ResidentBuffers resident_buffers(const tmw_stack_desc& d) {
    const int64_t words = (int64_t)d.batch * d.d_model / 2 * 8;  // of rows of the model's width
    ResidentBuffers s;
    s.abort = 0;
    s.x = 256;
    s.qkv = s.x + kCopies * words;
    s.o = s.qkv + 3 * words;
    s.y = s.o + kCopies * words;
    s.f = s.y + kCopies * words;
    s.cleared = s.f + kCopies * ((int64_t)d.batch * d.d_ff / 2 * 8);
    s.best = s.cleared;
    s.total = s.best + 2 * (int64_t)sm_count() * d.batch * 8;
    return s;
}

template <typename T>
int launch(const ResidentParams& p, int ctas, int smem, cudaStream_t stream) {
    auto kern = decode_resident_kernel<T>;
    const int rc = allow_shared_memory(reinterpret_cast<const void*>(kern), smem);
    if (rc != TMW_OK) return rc;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeCooperative;
    attr.val.cooperative = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, p);
    if (e == cudaErrorCooperativeLaunchTooLarge) {  // (a context that may use only a part of the device)
        (void)cudaGetLastError();
        return TMW_ERR_UNSUPPORTED;
    }
    TMW_CUDA_TRY(e);
    return TMW_OK;
}

}  // namespace

// The line is where the registers and the used half of the mma's rows end: eight sequences, three tiles of eight columns per
// CTA, chunks of k as declared above.  us per step as one kernel / as a chain (8 layers, vocabulary 8000, 16 persistent rows):
//   width 640, window 64: 1 sequence 79 / 162, 4: 84 / 162, 8: 95 / 163       512: 1: 84 / 170, 4: 92 / 178, 8: 113 / 186
//              window 1024: 1: 108 / 171, 4: 130 / 205, 8: 147 / 211           3000: 1: 172 / 214, 4: 194 / 299, 8: 225 / 307
//   width 512, window 512: 1: 79 / 161, 8: 93 / 173                            width 768: 8: 124 / 207
// With the mma's other eight rows in use (tried with sixteen warps only): 9 sequences 162 / 187 and 16 208 / 190 at window 512,
// 274 / 216 at 1024: not kept.  Windows that the chain splits over the chip (decode_step_splits) stay with it.
bool decode_step_is_resident(const tmw_stack_desc& d, const tmw_block* blocks) {
    const int sms = sm_count();
    static_assert(kRows * 8 <= kHeadDim, "a CTA per eight columns of the model is a CTA per pair: 8 heads = d_model / 8");
    if (d.batch < 1 || d.batch > kRows || d.layers < 1 || d.layers > kMaxLayers || d.head_dim != kHeadDim || d.d_model > kMaxDim ||
        d.d_ff > kMaxHidden || d.d_ff % 32 != 0 || d.d_model / 8 > sms || columns_per_cta(3 * d.d_model) > kInTiles ||
        columns_per_cta(d.d_ff) > kInTiles)
        return false;
    tmw_cache_desc c = {};
    c.batch = d.batch; c.heads = d.heads; c.head_dim = d.head_dim; c.window = d.window;
    if (decode_step_splits(c) > 0) return false;
    for (int l = 0; blocks != nullptr && l < d.layers; ++l)  // biases are read in pairs and fetched in units of 16 bytes
        if (((reinterpret_cast<uintptr_t>(blocks[l].b_fc1) | reinterpret_cast<uintptr_t>(blocks[l].b_fc2)) & 15u) != 0) return false;
    return true;
}

size_t decode_resident_workspace(const tmw_stack_desc& d) { return (size_t)resident_buffers(d).total; }

int decode_resident_begin(const tmw_stack_desc& d, void* workspace, cudaStream_t stream) {
    TMW_CUDA_TRY(cudaMemsetAsync(workspace, 0, (size_t)resident_buffers(d).cleared, stream));
    return TMW_OK;
}

int launch_decode_resident(const tmw_stack_desc& d, const tmw_block* blocks, const int64_t* ids, const int32_t* pos, void* logits,
                           int step, bool choose, int64_t* out, int64_t out_stride, void* workspace, cudaStream_t stream) {
    const ResidentBuffers off = resident_buffers(d);
    char* ws = static_cast<char*>(workspace);
    const int ctas = sm_count();
    ResidentParams p = {};
    for (int l = 0; l < d.layers; ++l) {
        const tmw_block& b = blocks[l];
        LayerTable& t = p.layer[l];
        t.half[0] = {b.norm_attn, b.w_qkv, nullptr, b.w_out, nullptr};
        t.half[1] = {b.norm_mlp, b.w_fc1, b.b_fc1, b.w_fc2, b.b_fc2};
        t.k_ring = b.k_ring; t.v_ring = b.v_ring; t.k_pers = b.k_pers; t.v_pers = b.v_pers;
        t.scale_log2 = (b.cache_scale != 0.f ? b.cache_scale : 1.0f / sqrtf((float)d.head_dim)) * 1.4426950408889634f;
    }
    unsigned long long* best = reinterpret_cast<unsigned long long*>(ws + off.best);
    const int64_t half = (int64_t)ctas * d.batch;
    p.tokens = d.embed_tokens; p.positions = d.embed_positions; p.norm = d.norm; p.head = d.head;
    p.ids = ids; p.pos = pos; p.logits = logits;
    p.best_in = choose && step > 0 ? best + (step & 1) * half : nullptr;
    p.best_out = choose ? best + ((step + 1) & 1) * half : nullptr;
    p.out = out; p.out_stride = out_stride;
    p.x = reinterpret_cast<uint64_t*>(ws + off.x); p.qkv = reinterpret_cast<uint64_t*>(ws + off.qkv);
    p.o = reinterpret_cast<uint64_t*>(ws + off.o); p.y = reinterpret_cast<uint64_t*>(ws + off.y);
    p.f = reinterpret_cast<uint64_t*>(ws + off.f);
    p.abort = reinterpret_cast<int*>(ws + off.abort);
    p.status = device_status_word();
    if (p.status == nullptr) return TMW_ERR_CUDA;
    p.tag0 = (uint32_t)step * (uint32_t)(d.layers + 1) + 1u;  // (zero is an empty word)
    p.rows = d.batch; p.layers = d.layers; p.dim = d.d_model; p.hidden = d.d_ff; p.heads = d.heads; p.vocab = d.vocab;
    p.slots = d.window + 1; p.np = d.n_persistent; p.max_pos = d.max_positions; p.advance = step; p.eps = d.eps; p.inv_dim = 1.0f / (float)d.d_model;
    p.nt_qkv = columns_per_cta(3 * d.d_model);
    p.nt_fc1 = columns_per_cta(d.d_ff);
    const int red = kWarps * kRows * (kInStride + 2 * kOutStride) * (int)sizeof(float);
    const int head = kRows * (d.d_model * 2 + 64), per_key = kWarps * 2 * kRowBytes;
    const int64_t range = ((int64_t)d.n_persistent + d.window + 1 + kWarps - 1) / kWarps;
    const int keys = range > kMaxGroup ? kMaxGroup : (int)range, room = (kSmemLimit - (int)sizeof(Shared) - 128 - red) / per_key;
    p.group_keys = keys < room ? keys : room;
    const int smem = red + (p.group_keys * per_key > head ? p.group_keys * per_key : head);
    return d.dtype == TMW_BF16 ? launch<__nv_bfloat16>(p, ctas, smem, stream) : launch<__half>(p, ctas, smem, stream);
}

int launch_decode_choice(const tmw_stack_desc& d, int steps, int64_t* tokens, int64_t* out, int64_t out_stride, int32_t* pos,
                         void* workspace, cudaStream_t stream) {
    const unsigned long long* best =
        reinterpret_cast<const unsigned long long*>(static_cast<char*>(workspace) + resident_buffers(d).best) +
        (steps & 1) * (int64_t)sm_count() * d.batch;
    decode_choice_kernel<<<1, kThreads, 0, stream>>>(best, sm_count(), d.batch, tokens, out, out_stride, pos, steps);
    TMW_CUDA_TRY(cudaGetLastError());
    return TMW_OK;
}

}  // namespace tmw
