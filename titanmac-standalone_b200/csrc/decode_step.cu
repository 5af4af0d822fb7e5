// One decode step of the whole model: embedding, `layers` blocks (norm, QKV, attention against the ring cache, output
// projection, norm, MLP) and the head, as one chain of five launches per block issued by one C call.
//
// A step has one row per sequence, so every product is a few rows against a weight matrix: nothing in it is bound by
// arithmetic, and with separate norm, GEMM, activation and residual kernels (eight launches per block, each started
// from Python) the step was bound by the host: 2.55 ms for one sequence and 2.64 ms for 256, of which the GPU was busy
// 0.63 and 1.49 ms.  Here
//   * the RMSNorm rides on the A operand of the product that consumes it, bias / GELU / residual add on the epilogue;
//     the row sums of squares that the norm needs are left by the product that wrote the row (per column tile, added
//     up in a fixed order);
//   * the kernels are launched as programmatic dependents: a kernel's weights are on their way into registers before
//     its predecessor has finished.
// Up to eight sequences with heads of 64 the step is one kernel instead (decode_resident.cu).
#include <math_constants.h>

#include "tmw_common.cuh"

namespace tmw {
namespace {

constexpr int kRowsThreads = 256;

struct RowsGemmParams {
    const void* a;       // [m, k] rows, leading dimension lda
    const void* w;       // [n, k] contiguous
    const void* bias;    // [n] or nullptr
    void* c;             // [m, n], leading dimension ldc; residual epilogue: x, read and written
    const void* gain;    // NORM: [k]
    const float* ss_in;  // NORM: [ss_parts][m] partial sums of squares of the rows of a
    float* ss_out;       // residual epilogue: [column tiles][m]
    long long lda, ldc;
    int m, n, k, ss_parts;
    float eps;
};

enum { EPI_STORE = 0, EPI_GELU = 1, EPI_RESIDUAL = 2 };

__device__ __forceinline__ uint4 ld_weights(const void* p) {  // read once per step: past L1
    uint4 r;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p));
    return r;
}

// Eight 16-bit values h -> round(h * inv * gain), the RMSNorm of the row they belong to.
template <typename T>
__device__ __forceinline__ uint4 norm8(const uint4& raw, float inv, const uint4& gain) {
    float h[8], g[8];
    load8<T>(reinterpret_cast<const T*>(&raw), h);
    load8<T>(reinterpret_cast<const T*>(&gain), g);
#pragma unroll
    for (int e = 0; e < 8; ++e) h[e] = h[e] * inv * g[e];
    uint4 out;
    store8<T>(reinterpret_cast<T*>(&out), h);
    return out;
}

// c[m, n] = epilogue(norm(a)[m, k] · w[n, k]ᵀ) for few rows m.  A CTA owns BM rows x BN columns, its eight warps
// interleaved slices of k.
//
// Operands go from global memory straight into the mma fragments: k is consumed in chunks of 32, of which a thread of
// a quad takes eight adjacent values (one 16-byte load) of its row - the same ones for A and B, so the order of k inside
// the chunk does not matter - and DEPTH chunks are in flight per warp.  Shared memory only adds up the k slices.
template <typename T, int BM, int BN, int DEPTH, bool NORM, int EPI>
__global__ void __launch_bounds__(kRowsThreads, DEPTH > 5 ? 1 : 2) rows_gemm_kernel(const RowsGemmParams p) {
    constexpr int WK = 8, MT = BM / 16, NT = BN / 8;
    constexpr int STR = BN == 8 ? 8 : BN + 8;  // row stride of the partial sums (bank conflicts of 8-byte stores)
    extern __shared__ __align__(16) float red[];  // [WK][BM][STR]
    __shared__ float s_part[kRowsThreads];
    __shared__ float s_inv[BM];
    pdl_trigger();

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int tile = blockIdx.x, n0 = tile * BN, m0 = blockIdx.y * BM;
    const int n_my = max(0, (p.k / 32 - warp + WK - 1) / WK);  // this warp's chunks: warp, + WK, ...
    const int k_first = warp * 32 + t * 8;

    // rows and columns beyond the matrix are computed on a row that exists and not stored
    const T* wrow[NT];
    const T* arow[MT][2];
#pragma unroll
    for (int j = 0; j < NT; ++j)
        wrow[j] = static_cast<const T*>(p.w) + (long long)min(n0 + j * 8 + g, p.n - 1) * p.k + k_first;
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int hh = 0; hh < 2; ++hh)
            arow[i][hh] = static_cast<const T*>(p.a) +
                          (long long)min(m0 + i * 16 + hh * 8 + g, p.m - 1) * p.lda + k_first;
    uint4 bw[DEPTH][NT], ba[DEPTH][MT][2], bg[NORM ? DEPTH : 1];
    auto load_w = [&](int d, int i) {
#pragma unroll
        for (int j = 0; j < NT; ++j) bw[d][j] = ld_weights(wrow[j] + i * (32 * WK));
        if (NORM) bg[d] = *reinterpret_cast<const uint4*>(static_cast<const T*>(p.gain) + k_first + i * (32 * WK));
    };
    auto load_a = [&](int d, int i) {
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) ba[d][m][hh] = *reinterpret_cast<const uint4*>(arow[m][hh] + i * (32 * WK));
    };
#pragma unroll
    for (int d = 0; d < DEPTH; ++d)
        if (d < n_my) load_w(d, d);
    pdl_wait();
#pragma unroll
    for (int d = 0; d < DEPTH; ++d)
        if (d < n_my) load_a(d, d);
    // what this thread's first pair of outputs needs besides the product
    constexpr int PR = BN / 2;   // column pairs per row: adjacent threads
    const int gm_first = m0 + tid / PR, gn_first = n0 + (tid % PR) * 2;
    const bool first_ok = tid < BM * PR && gm_first < p.m && gn_first + 1 < p.n;
    uint32_t res_first = 0u;
    if (EPI == EPI_RESIDUAL && first_ok)
        res_first = *reinterpret_cast<const uint32_t*>(static_cast<const T*>(p.c) + (long long)gm_first * p.ldc + gn_first);
    float inv[NORM ? MT : 1][2];
    if (NORM) {
        // the rows' sums of squares: kRowsThreads / BM threads per row, partial sums in a fixed order
        constexpr int LPR = kRowsThreads / BM;
        const int r = tid % BM, l = tid / BM;
        float s = 0.f;
        if (m0 + r < p.m) {
            for (int q0 = l; q0 < p.ss_parts; q0 += 8 * LPR) {  // eight loads in flight
                float part[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const int q = q0 + u * LPR;
                    part[u] = q < p.ss_parts ? p.ss_in[(long long)q * p.m + m0 + r] : 0.f;
                }
#pragma unroll
                for (int u = 0; u < 8; ++u) s += part[u];
            }
        }
        s_part[l * BM + r] = s;
        __syncthreads();
        if (tid < BM) {
            float sum = 0.f;
#pragma unroll
            for (int q = 0; q < LPR; ++q) sum += s_part[q * BM + tid];
            s_inv[tid] = 1.0f / sqrtf(sum / (float)p.k + p.eps);
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) inv[i][hh] = s_inv[i * 16 + hh * 8 + g];
    }
    float acc[MT][NT][4];
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.f;
    for (int i0 = 0; i0 < n_my; i0 += DEPTH) {
#pragma unroll
        for (int d = 0; d < DEPTH; ++d) {
            if (i0 + d < n_my) {
#pragma unroll
                for (int i = 0; i < MT; ++i) {
                    uint4 a0 = ba[d][i][0], a1 = ba[d][i][1];
                    if (NORM) {
                        a0 = norm8<T>(a0, inv[i][0], bg[d]);
                        a1 = norm8<T>(a1, inv[i][1], bg[d]);
                    }
#pragma unroll
                    for (int j = 0; j < NT; ++j) {
                        mma_16816<T>(acc[i][j], a0.x, a1.x, a0.y, a1.y, bw[d][j].x, bw[d][j].y);
                        mma_16816<T>(acc[i][j], a0.z, a1.z, a0.w, a1.w, bw[d][j].z, bw[d][j].w);
                    }
                }
                if (i0 + d + DEPTH < n_my) {
                    load_w(d, i0 + d + DEPTH);
                    load_a(d, i0 + d + DEPTH);
                }
            }
        }
    }

    // add up the k slices of the warps
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int hh = 0; hh < 2; ++hh)
                *reinterpret_cast<float2*>(red + (warp * BM + i * 16 + hh * 8 + g) * STR + j * 8 + 2 * t) =
                    make_float2(acc[i][j][2 * hh], acc[i][j][2 * hh + 1]);
    __syncthreads();
    for (int q = tid; q < BM * PR; q += kRowsThreads) {
        const int row = q / PR, col = (q % PR) * 2;
        float v0 = 0.f, v1 = 0.f;
#pragma unroll
        for (int s = 0; s < WK; ++s) {
            const float2 x = *reinterpret_cast<const float2*>(red + (s * BM + row) * STR + col);
            v0 += x.x;
            v1 += x.y;
        }
        const int gm = m0 + row, gn = n0 + col;
        const bool ok0 = gm < p.m && gn < p.n, ok1 = gm < p.m && gn + 1 < p.n;
        if (p.bias != nullptr) {
            if (ok0) v0 += to_f32<T>(static_cast<const T*>(p.bias)[gn]);
            if (ok1) v1 += to_f32<T>(static_cast<const T*>(p.bias)[gn + 1]);
        }
        if (EPI == EPI_GELU) {
            v0 = gelu_erf(v0);
            v1 = gelu_erf(v1);
        }
        T* dst = static_cast<T*>(p.c) + (long long)gm * p.ldc + gn;
        const bool wide = ok1 && (p.ldc & 1) == 0;
        T w2[2] = {from_f32<T>(v0), from_f32<T>(v1)};
        if (EPI == EPI_RESIDUAL) {  // (n = d_model and ldc are even)
            float ss = 0.f;
            if (ok1) {
                const uint32_t raw = q == tid ? res_first : *reinterpret_cast<const uint32_t*>(dst);
                const T* r2 = reinterpret_cast<const T*>(&raw);
                w2[0] = from_f32<T>(to_f32<T>(r2[0]) + to_f32<T>(w2[0]));
                w2[1] = from_f32<T>(to_f32<T>(r2[1]) + to_f32<T>(w2[1]));
                ss = fmaf(to_f32<T>(w2[1]), to_f32<T>(w2[1]), to_f32<T>(w2[0]) * to_f32<T>(w2[0]));
            }
#pragma unroll
            for (int off = PR / 2; off > 0; off >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, off);
            if (q % PR == 0 && gm < p.m) p.ss_out[(long long)tile * p.m + gm] = ss;
        }
        if (wide) {
            *reinterpret_cast<uint32_t*>(dst) = *reinterpret_cast<const uint32_t*>(w2);
        } else {
            if (ok0) dst[0] = w2[0];
            if (ok1) dst[1] = w2[1];
        }
    }
}

template <typename T, int BM, int BN, int DEPTH, bool NORM, int EPI>
int launch_rows_tile(const RowsGemmParams& p, cudaStream_t stream) {
    constexpr int STR = BN == 8 ? 8 : BN + 8;
    constexpr int smem = 8 * BM * STR * (int)sizeof(float);
    auto kern = rows_gemm_kernel<T, BM, BN, DEPTH, NORM, EPI>;
    if (smem > 40 * 1024) {
        const int rc = allow_shared_memory(reinterpret_cast<const void*>(kern), smem);
        if (rc != TMW_OK) return rc;
    }
    const dim3 grid((p.n + BN - 1) / BN, (p.m + BM - 1) / BM);
    TMW_CUDA_TRY(launch_ex(kern, grid, dim3(kRowsThreads), smem, stream, true, 1, p));
    return TMW_OK;
}

// The head of up to 16 rows: norm(a)[m, k] · w[n, k]ᵀ against a whole vocabulary, a stream of weights.  The normalised rows
// stay in registers as mma fragments and two CTAs per SM walk over tiles of 16 columns, the next tile's weights in
// flight while this one's are used (one tile per CTA, each with its own norm and cold start, measured 20 us for
// 50 000 x 640; this 64 MB at the rate of a copy is 10).
template <typename T, int NCH>  // NCH: chunks of 32 k-elements per warp
__global__ void __launch_bounds__(kRowsThreads, 2) rows_head_kernel(const RowsGemmParams p) {
    constexpr int STR = 24;
    __shared__ __align__(16) float red[2][8][16][STR];
    __shared__ float s_part[kRowsThreads];
    __shared__ float s_inv[16];
    pdl_trigger();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int tiles = (p.n + 15) / 16, n_my = max(0, (p.k / 32 - warp + 7) / 8);
    const int k_first = warp * 32 + t * 8;
    uint4 cur[NCH][2], nxt[NCH][2], a[NCH][2];
    auto load_w = [&](uint4 (&w)[NCH][2], int tile) {
#pragma unroll
        for (int i = 0; i < NCH; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j)
                if (i < n_my)
                    w[i][j] = ld_weights(static_cast<const T*>(p.w) + (long long)min(tile * 16 + j * 8 + g, p.n - 1) * p.k + k_first +
                                         i * 256);
    };
    load_w(cur, blockIdx.x);
    pdl_wait();
#pragma unroll
    for (int i = 0; i < NCH; ++i)
#pragma unroll
        for (int hh = 0; hh < 2; ++hh)
            if (i < n_my)
                a[i][hh] = *reinterpret_cast<const uint4*>(static_cast<const T*>(p.a) +
                                                           (long long)min(hh * 8 + g, p.m - 1) * p.lda + k_first + i * 256);
    {
        const int r = tid % 16, l = tid / 16;
        float s = 0.f;
        if (r < p.m) {
#pragma unroll 8
            for (int q = l; q < p.ss_parts; q += 16) s += p.ss_in[(long long)q * p.m + r];
        }
        s_part[l * 16 + r] = s;
        __syncthreads();
        if (tid < 16) {
            float sum = 0.f;
#pragma unroll
            for (int q = 0; q < 16; ++q) sum += s_part[q * 16 + tid];
            s_inv[tid] = 1.0f / sqrtf(sum / (float)p.k + p.eps);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < NCH; ++i)
        if (i < n_my) {
            const uint4 gain = *reinterpret_cast<const uint4*>(static_cast<const T*>(p.gain) + k_first + i * 256);
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) a[i][hh] = norm8<T>(a[i][hh], s_inv[hh * 8 + g], gain);
        }
    int buf = 0;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, buf ^= 1) {
        if (tile + (int)gridDim.x < tiles) load_w(nxt, tile + gridDim.x);
        float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
        for (int i = 0; i < NCH; ++i)
            if (i < n_my) {
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    mma_16816<T>(acc[j], a[i][0].x, a[i][1].x, a[i][0].y, a[i][1].y, cur[i][j].x, cur[i][j].y);
                    mma_16816<T>(acc[j], a[i][0].z, a[i][1].z, a[i][0].w, a[i][1].w, cur[i][j].z, cur[i][j].w);
                }
            }
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int hh = 0; hh < 2; ++hh)
                *reinterpret_cast<float2*>(&red[buf][warp][hh * 8 + g][j * 8 + 2 * t]) = make_float2(acc[j][2 * hh], acc[j][2 * hh + 1]);
        __syncthreads();  // (the other buffer is written next: its readers are behind this barrier by then)
        if (tid < 128) {
            const int row = tid / 8, col = (tid % 8) * 2, gn = tile * 16 + col;
            float v0 = 0.f, v1 = 0.f;
#pragma unroll
            for (int w = 0; w < 8; ++w) {
                const float2 x = *reinterpret_cast<const float2*>(&red[buf][w][row][col]);
                v0 += x.x;
                v1 += x.y;
            }
            if (row < p.m) {
                T* dst = static_cast<T*>(p.c) + (long long)row * p.ldc + gn;
                T w2[2] = {from_f32<T>(v0), from_f32<T>(v1)};
                if (gn + 1 < p.n && (p.ldc & 1) == 0) {
                    *reinterpret_cast<uint32_t*>(dst) = *reinterpret_cast<const uint32_t*>(w2);
                } else {
                    if (gn < p.n) dst[0] = w2[0];
                    if (gn + 1 < p.n) dst[1] = w2[1];
                }
            }
        }
#pragma unroll
        for (int i = 0; i < NCH; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j) cur[i][j] = nxt[i][j];
    }
}

template <typename T>
int launch_rows_head(const RowsGemmParams& p, cudaStream_t stream) {
    const int tiles = (p.n + 15) / 16, grid = tiles < 2 * sm_count() ? tiles : 2 * sm_count();
    auto run = [&](auto kern) -> int {
        TMW_CUDA_TRY(launch_ex(kern, dim3(grid), dim3(kRowsThreads), 0, stream, true, 1, p));
        return TMW_OK;
    };
    const int nch = (p.k / 32 + 7) / 8;
    return nch <= 2 ? run(rows_head_kernel<T, 2>) : nch == 3 ? run(rows_head_kernel<T, 3>) : run(rows_head_kernel<T, 4>);
}

// Tile for m <= 32 rows (or, more rows against a vocabulary of a ragged size, tiles of 32).  The weights are read once per
// row tile; columns are cut narrow enough that most SMs get a tile, and the eight warps of a CTA share its k.  A tile of
// eight columns keeps ten chunks per warp in flight: the whole k of 2560 (32 rows: 8.1 us against 13.8 with three).
template <typename T, bool NORM, int EPI>
int launch_rows(const RowsGemmParams& p, int* tiles_out, cudaStream_t stream) {
    const int sms = sm_count();
    const int bn = p.n >= 32 * 3 * sms ? 32 : p.n >= 16 * (sms / 2) ? 16 : 8;
    *tiles_out = (p.n + bn - 1) / bn;
    if (p.m <= 16) {
        if (bn == 32) return launch_rows_tile<T, 16, 32, 3, NORM, EPI>(p, stream);
        if (bn == 16) return launch_rows_tile<T, 16, 16, 4, NORM, EPI>(p, stream);
        return launch_rows_tile<T, 16, 8, NORM ? 5 : 10, NORM, EPI>(p, stream);
    }
    if (bn == 32) return launch_rows_tile<T, 32, 32, 2, NORM, EPI>(p, stream);
    if (bn == 16) return launch_rows_tile<T, 32, 16, 3, NORM, EPI>(p, stream);
    return launch_rows_tile<T, 32, 8, NORM ? 3 : 10, NORM, EPI>(p, stream);
}

// x[b] = round(tokens[ids[b]] + positions[pos[b]]), and the row's sum of squares; one warp per row
struct EmbedParams {
    const void *tokens, *positions;
    const int64_t* ids;
    const int32_t* pos;
    void* x;
    float* ss;
    int* status;
    int rows, dim, vocab, max_pos;
};

template <typename T>
__global__ void __launch_bounds__(128) embed_rows_kernel(const EmbedParams p) {
    const int row = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (row >= p.rows) return;
    long long id = p.ids[row];
    int pos = p.pos[row];
    const bool bad = id < 0 || id >= p.vocab || pos < 0 || pos >= p.max_pos;
    if (bad) {  // outside the tables: a row of NaN, and the status word says so
        if (lane == 0) atomicCAS(p.status, 0, (int)TMW_ERR_INVALID_ARGUMENT);
        id = pos = 0;
    }
    const T* a = static_cast<const T*>(p.tokens) + id * p.dim;
    const T* b = static_cast<const T*>(p.positions) + (long long)pos * p.dim;
    T* x = static_cast<T*>(p.x) + (long long)row * p.dim;
    float ss = 0.f;
    for (int v = lane; v < p.dim / 8; v += 32) {
        float u[8], w[8];
        load8<T>(a + v * 8, u);
        load8<T>(b + v * 8, w);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            u[e] = bad ? CUDART_NAN_F : to_f32<T>(from_f32<T>(u[e] + w[e]));
            ss = fmaf(u[e], u[e], ss);
        }
        store8<T>(x + v * 8, u);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if (lane == 0) p.ss[row] = ss;
}

// The greedy choice: token[b] = the first index of row b's largest logit (NaN counts as largest), out[b * out_stride] the
// same, pos[b] += advance.  A cluster of CTAs shares a row (one CTA per row: 14 us for 8 rows of 50 000).
struct ArgmaxParams {
    const void* logits;
    int64_t *token, *out;
    int32_t* pos;
    long long out_stride;
    int vocab, cluster, advance;
};

template <typename T>
__global__ void __launch_bounds__(256) argmax_rows_kernel(const ArgmaxParams p) {
    __shared__ unsigned long long best[8], mine;
    pdl_trigger();
    pdl_wait();
    const int cs = p.cluster, rank = blockIdx.x % cs, row = blockIdx.x / cs, tid = threadIdx.x;
    const T* x = static_cast<const T*>(p.logits) + (long long)row * p.vocab;
    // larger value first, then smaller index: the value as an unsigned number in the same order, above the index inverted
    unsigned long long key = 0;
    auto take = [&](float v, int i) {
        const uint32_t u = __float_as_uint(v + 0.0f);  // (-0 equals +0)
        const uint32_t order = v != v ? 0xffffffffu : (u & 0x80000000u) ? ~u : u | 0x80000000u;
        const unsigned long long k = ((unsigned long long)order << 32) | (uint32_t)~i;
        key = k > key ? k : key;
    };
    const bool wide = (p.vocab & 7) == 0;
    const int n = wide ? p.vocab / 8 : p.vocab, lo = (int)((long long)n * rank / cs), hi = (int)((long long)n * (rank + 1) / cs);
    if (wide) {
        for (int v0 = lo + tid; v0 < hi; v0 += 256 * 4) {
            Vec8<T> raw[4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (v0 + u * 256 < hi) raw[u].load(x + (long long)(v0 + u * 256) * 8);
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (v0 + u * 256 < hi) {
                    float f[8];
                    raw[u].unpack(f);
#pragma unroll
                    for (int e = 0; e < 8; ++e) take(f[e], (v0 + u * 256) * 8 + e);
                }
        }
    } else {
        for (int i = lo + tid; i < hi; i += 256) take(to_f32<T>(x[i]), i);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long other = __shfl_xor_sync(0xffffffffu, key, o);
        key = other > key ? other : key;
    }
    if ((tid & 31) == 0) best[tid >> 5] = key;
    __syncthreads();
    if (tid == 0) {
        for (int i = 1; i < 8; ++i) key = best[i] > key ? best[i] : key;
        mine = key;
    }
    if (cs > 1) {
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
    if (rank == 0 && tid == 0) {
        for (int r = 1; r < cs; ++r) {
            uint32_t a = (uint32_t)__cvta_generic_to_shared(&mine);
            unsigned long long k;
            asm volatile("mapa.shared::cluster.u32 %0, %0, %1;" : "+r"(a) : "r"(r));
            asm volatile("ld.shared::cluster.u64 %0, [%1];" : "=l"(k) : "r"(a) : "memory");
            key = k > key ? k : key;
        }
        const int64_t id = (int64_t)(uint32_t)~(uint32_t)key;
        p.token[row] = id;
        p.out[row * p.out_stride] = id;
        p.pos[row] += p.advance;
    }
    if (cs > 1) {
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
}

template <typename T>
int launch_argmax(int rows, int vocab, const void* logits, int64_t* token, int64_t* out, int64_t out_stride, int32_t* pos, int advance,
                  bool pdl, cudaStream_t stream) {
    ArgmaxParams p;
    p.logits = logits; p.token = token; p.out = out; p.pos = pos; p.out_stride = out_stride; p.vocab = vocab; p.advance = advance;
    p.cluster = 1;
    while (p.cluster < 8 && rows * p.cluster * 2 <= 2 * sm_count()) p.cluster *= 2;
    TMW_CUDA_TRY(launch_ex(argmax_rows_kernel<T>, dim3(rows * p.cluster), dim3(256), 0, stream, pdl, p.cluster, p));
    return TMW_OK;
}

int64_t align256(int64_t n) { return (n + 255) & ~(int64_t)255; }

tmw_cache_desc cache_of(const tmw_stack_desc& d) {
    tmw_cache_desc c = {};
    c.dtype = d.dtype; c.batch = d.batch; c.heads = d.heads; c.head_dim = d.head_dim; c.window = d.window;
    c.n_persistent = d.n_persistent;
    return c;
}

struct StepBuffers {
    int64_t x, qkv, o, f, y, ss, parts, counters, total;  // byte offsets
    int splits;                                           // of the attention (decode_step_splits)
};
StepBuffers step_buffers(const tmw_stack_desc& d) {
    StepBuffers s;
    const int64_t row = (int64_t)d.batch * 2;
    s.x = 0;
    s.qkv = s.x + align256(row * d.d_model);
    s.o = s.qkv + align256(row * 3 * d.d_model);
    s.f = s.o + align256(row * d.d_model);
    s.y = s.f + align256(row * d.d_ff);
    s.ss = s.y + align256(row * d.d_model);
    s.parts = s.ss + align256((int64_t)d.batch * ((d.d_model + 7) / 8) * 4);
    s.splits = decode_step_splits(cache_of(d));
    s.counters = s.parts + (s.splits > 0 ? align256((int64_t)decode_partials_bytes(d.batch, d.heads, d.head_dim, s.splits)) : 0);
    s.total = s.counters + (s.splits > 0 ? align256((int64_t)d.batch * d.heads * 4) : 0);
    if (decode_step_is_resident(d, nullptr)) {  // (which needs nothing of the above)
        const int64_t resident = (int64_t)decode_resident_workspace(d);
        s.total = s.total > resident ? s.total : resident;
    }
    return s;
}

// the split attention's counters: zero in front of the first step (every launch leaves them so)
int clear_counters(const tmw_stack_desc& d, char* ws, cudaStream_t stream) {
    const StepBuffers off = step_buffers(d);
    if (off.splits > 0) TMW_CUDA_TRY(cudaMemsetAsync(ws + off.counters, 0, (size_t)(off.total - off.counters), stream));
    return TMW_OK;
}

template <typename T>
int decode_step_t(const tmw_stack_desc& d, const tmw_block* blocks, const int64_t* ids, const int32_t* pos, void* logits,
                  char* ws, cudaStream_t stream) {
    const StepBuffers off = step_buffers(d);
    const int B = d.batch, D = d.d_model, F = d.d_ff;
    void *x = ws + off.x, *qkv = ws + off.qkv, *o = ws + off.o, *f = ws + off.f, *y = ws + off.y;
    float* ss = reinterpret_cast<float*>(ws + off.ss);
    int parts = 1;
    EmbedParams e;
    e.tokens = d.embed_tokens; e.positions = d.embed_positions; e.ids = ids; e.pos = pos; e.x = x; e.ss = ss;
    e.status = device_status_word();
    if (e.status == nullptr) return TMW_ERR_CUDA;
    e.rows = B; e.dim = D; e.vocab = d.vocab; e.max_pos = d.max_positions;
    // an ordinary launch: whatever the caller's stream held before (new weights, say) has finished when it starts, so
    // the kernels behind it may read their weights early
    embed_rows_kernel<T><<<(B + 3) / 4, 128, 0, stream>>>(e);
    TMW_CUDA_TRY(cudaGetLastError());

    RowsGemmParams p = {};
    p.m = B;
    p.eps = d.eps;
    // up to 32 rows the fragment kernels with the norm inside (16 layers, 32 rows: 480 us against 650), above them the
    // norm as a launch of its own and tcgen05 tiles of 128 rows (64 rows: 760 us against 1080)
    const bool tc = B > 32;
    auto normed = [&](const void* gain, const void* w, const void* bias, int n, void* c, int epi) {
        if (tc) {
            const int rc = launch_rows_norm(d.dtype, B, D, x, gain, d.eps, y, stream);
            return rc != TMW_OK ? rc : launch_rows_tc(d.dtype, B, n, D, y, w, bias, c, epi, stream, true);
        }
        p.a = x; p.lda = D; p.k = D; p.w = w; p.bias = bias; p.n = n; p.c = c; p.ldc = n;
        p.gain = gain; p.ss_in = ss; p.ss_parts = parts; p.ss_out = nullptr;
        int unused;
        return epi == EPI_GELU ? launch_rows<T, true, EPI_GELU>(p, &unused, stream)
                               : launch_rows<T, true, EPI_STORE>(p, &unused, stream);
    };
    auto back = [&](const void* a, int k, const void* w, const void* bias) {
        if (tc) return launch_rows_tc(d.dtype, B, D, k, a, w, bias, x, EPI_RESIDUAL, stream, true);
        p.a = a; p.lda = k; p.k = k; p.w = w; p.bias = bias; p.n = D; p.c = x; p.ldc = D; p.ss_out = ss;
        return launch_rows<T, false, EPI_RESIDUAL>(p, &parts, stream);
    };
    const int64_t row3[2] = {3 * (int64_t)D, d.head_dim}, row1[2] = {D, d.head_dim};
    for (int l = 0; l < d.layers; ++l) {
        const tmw_block& b = blocks[l];
        int rc = normed(b.norm_attn, b.w_qkv, nullptr, 3 * D, qkv, EPI_STORE);
        if (rc != TMW_OK) return rc;
        tmw_cache_desc c = cache_of(d);
        c.k_ring = b.k_ring; c.v_ring = b.v_ring; c.k_pers = b.k_pers; c.v_pers = b.v_pers; c.scale = b.cache_scale;
        const T* q = static_cast<const T*>(qkv);
        rc = launch_decode(c, q, q + D, q + 2 * D, o, row3, row3, row1, pos, off.splits, reinterpret_cast<float*>(ws + off.parts),
                           reinterpret_cast<unsigned int*>(ws + off.counters), stream, off.splits == 0);
        if (rc == TMW_OK) rc = back(o, D, b.w_out, nullptr);
        if (rc == TMW_OK) rc = normed(b.norm_mlp, b.w_fc1, b.b_fc1, F, f, EPI_GELU);
        if (rc == TMW_OK) rc = back(f, F, b.w_fc2, b.b_fc2);
        if (rc != TMW_OK) return rc;
    }
    if (B <= 16 && D <= 1024) {
        p.a = x; p.lda = D; p.k = D; p.w = d.head; p.n = d.vocab; p.c = logits; p.ldc = d.vocab;
        p.gain = d.norm; p.ss_in = ss; p.ss_parts = parts;
        return launch_rows_head<T>(p, stream);
    }
    int rc = launch_rows_norm(d.dtype, B, D, x, d.norm, d.eps, y, stream);
    if (rc != TMW_OK) return rc;
    if (d.vocab % 8 != 0) {  // the wide stores of the tcgen05 product need whole 16-byte units
        p.a = y; p.lda = D; p.k = D; p.w = d.head; p.bias = nullptr; p.n = d.vocab; p.c = logits; p.ldc = d.vocab;
        return launch_rows<T, false, EPI_STORE>(p, &parts, stream);
    }
    tmw_linear_desc ld = {};
    ld.dtype = d.dtype; ld.m = B; ld.n = d.vocab; ld.k = D; ld.epilogue = TMW_EPILOGUE_NONE;
    ld.lda = D; ld.ldw = D; ld.ldc = d.vocab;
    return launch_linear(ld, y, d.head, nullptr, logits, stream);
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

int validate_step(const tmw_stack_desc* d) {
    if (d == nullptr) return TMW_ERR_INVALID_ARGUMENT;
    if (d->dtype != TMW_BF16 && d->dtype != TMW_F16) return TMW_ERR_UNSUPPORTED;
    if (d->batch < 0 || d->layers < 0 || d->heads <= 0 || d->d_ff <= 0 || d->vocab <= 0 || d->max_positions <= 0 ||
        d->n_persistent < 0 || !(d->eps >= 0.f))
        return TMW_ERR_INVALID_ARGUMENT;
    if (d->window < 0) return TMW_ERR_NEGATIVE_WINDOW;
    if (d->head_dim != 64 && d->head_dim != 128) return TMW_ERR_UNSUPPORTED;
    if (d->d_model != d->heads * d->head_dim) return TMW_ERR_INVALID_ARGUMENT;
    if (d->d_ff % 32 != 0 || d->d_model > 4096) return TMW_ERR_UNSUPPORTED;  // (launch_rows_norm keeps a row in registers)
    if (d->batch > 65535) return TMW_ERR_TOO_LARGE;
    return TMW_OK;
}

int validate_step_arrays(const tmw_stack_desc& d, const tmw_block* blocks, const void* token_ids, const void* pos, const void* logits,
                         const void* workspace, size_t workspace_bytes) {
    if ((d.layers > 0 && blocks == nullptr) || token_ids == nullptr || pos == nullptr || logits == nullptr ||
        workspace == nullptr || d.embed_tokens == nullptr || d.embed_positions == nullptr || d.norm == nullptr ||
        d.head == nullptr)
        return TMW_ERR_INVALID_ARGUMENT;
    if (workspace_bytes < (size_t)step_buffers(d).total) return TMW_ERR_TOO_LARGE;
    if (!aligned16(d.embed_tokens) || !aligned16(d.embed_positions) || !aligned16(d.norm) || !aligned16(d.head) ||
        !aligned16(logits) || !aligned16(workspace))
        return TMW_ERR_INVALID_ARGUMENT;
    for (int l = 0; l < d.layers; ++l) {
        const tmw_block& b = blocks[l];
        const void* need[] = {b.norm_attn, b.w_qkv, b.w_out, b.norm_mlp, b.w_fc1, b.w_fc2, b.k_ring, b.v_ring};
        for (const void* q : need)
            if (q == nullptr || !aligned16(q)) return TMW_ERR_INVALID_ARGUMENT;
        if (d.n_persistent > 0 && (b.k_pers == nullptr || b.v_pers == nullptr || !aligned16(b.k_pers) || !aligned16(b.v_pers)))
            return TMW_ERR_INVALID_ARGUMENT;
        if (!(b.cache_scale >= 0.f)) return TMW_ERR_INVALID_ARGUMENT;
    }
    return TMW_OK;
}

}  // namespace
}  // namespace tmw

extern "C" size_t tmw_decode_step_workspace(const tmw_stack_desc* desc) {
    return tmw::validate_step(desc) != TMW_OK ? 0 : (size_t)tmw::step_buffers(*desc).total;
}

extern "C" int tmw_decode_step(const tmw_stack_desc* desc, const tmw_block* blocks, const int64_t* token_ids,
                               const int32_t* pos, void* logits, void* workspace, size_t workspace_bytes, void* stream) {
    using namespace tmw;
    int rc = validate_step(desc);
    if (rc != TMW_OK || desc->batch == 0) return rc;
    rc = validate_step_arrays(*desc, blocks, token_ids, pos, logits, workspace, workspace_bytes);
    if (rc != TMW_OK) return rc;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    char* ws = static_cast<char*>(workspace);
    if (decode_step_is_resident(*desc, blocks)) {
        rc = decode_resident_begin(*desc, ws, s);
        if (rc == TMW_OK) rc = launch_decode_resident(*desc, blocks, token_ids, pos, logits, 0, false, nullptr, 0, ws, s);
        if (rc != TMW_ERR_UNSUPPORTED) return rc;
    }
    rc = clear_counters(*desc, ws, s);
    if (rc != TMW_OK) return rc;
    return desc->dtype == TMW_BF16 ? decode_step_t<__nv_bfloat16>(*desc, blocks, token_ids, pos, logits, ws, s)
                                   : decode_step_t<__half>(*desc, blocks, token_ids, pos, logits, ws, s);
}

extern "C" int tmw_generate(const tmw_stack_desc* desc, const tmw_block* blocks, void* logits, int32_t tokens, int64_t* token_ids,
                            int32_t* pos, int64_t* out, int64_t out_stride, void* workspace, size_t workspace_bytes, void* stream) {
    using namespace tmw;
    int rc = validate_step(desc);
    if (rc != TMW_OK || desc->batch == 0 || tokens == 0) return rc;
    if (tokens < 0 || out == nullptr) return TMW_ERR_INVALID_ARGUMENT;
    rc = validate_step_arrays(*desc, blocks, token_ids, pos, logits, workspace, workspace_bytes);
    if (rc != TMW_OK) return rc;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    char* ws = static_cast<char*>(workspace);
    const tmw_stack_desc& d = *desc;
    // (a tag is used once: 32 bits of them)
    if (tokens > 1 && (int64_t)tokens * (d.layers + 1) < 0x7fffffff && decode_step_is_resident(d, blocks)) {
        rc = d.dtype == TMW_BF16 ? launch_argmax<__nv_bfloat16>(d.batch, d.vocab, logits, token_ids, out, out_stride, pos, 0, false, s)
                                 : launch_argmax<__half>(d.batch, d.vocab, logits, token_ids, out, out_stride, pos, 0, false, s);
        if (rc == TMW_OK) rc = decode_resident_begin(d, ws, s);
        if (rc != TMW_OK) return rc;
        int step = 0;
        for (; step < tokens - 1 && rc == TMW_OK; ++step)
            rc = launch_decode_resident(d, blocks, token_ids, pos, logits, step, true, out + step, out_stride, ws, s);
        if (rc == TMW_OK) return launch_decode_choice(d, step, token_ids, out + step, out_stride, pos, ws, s);
        if (rc != TMW_ERR_UNSUPPORTED || step != 1) return rc;  // (refused: the first launch was; `step` counts it)
    }
    rc = clear_counters(d, ws, s);
    if (rc != TMW_OK) return rc;
    auto run = [&](auto type) -> int {
        using T = decltype(type);
        // (an ordinary launch first; every step starts with one as well, so that a step's early reads of the rings see
        // what the step before has written)
        int st = launch_argmax<T>(d.batch, d.vocab, logits, token_ids, out, out_stride, pos, 0, false, s);
        for (int i = 1; i < tokens && st == TMW_OK; ++i) {
            st = decode_step_t<T>(d, blocks, token_ids, pos, logits, ws, s);
            if (st == TMW_OK) st = launch_argmax<T>(d.batch, d.vocab, logits, token_ids, out + i, out_stride, pos, 1, true, s);
        }
        return st;
    };
    return d.dtype == TMW_BF16 ? run(__nv_bfloat16{}) : run(__half{});
}
