// Kernels of the training step beside the products and the attention cores: backward of RMSNorm, column sums, the sums of
// split products, shifted cross-entropy and the embedding gradients.  All of them are bound by HBM (or, in a small
// model, by their launch): one pass over their operands, 16-byte accesses, fp32 inside, and sums whose order does not
// depend on the schedule except where tokens repeat (embed_scatter_kernel).
#include <math_constants.h>

#include "train_ops.cuh"

namespace tmw {
namespace {

constexpr int kNormWarps = 8;

// y = x inv gain with inv = 1 / sqrt(mean(x^2) + eps).  Given dy: dx = inv (dy gain - x̂ mean(dy gain x̂)), x̂ = x inv, and
// out = add + dx (the residual branch's gradient rides along).  A warp walks over rows with its columns of the two column
// sums - dgain = sum dy x̂, and sum out, the bias gradient of the linear whose output the residual stream is - in registers;
// the CTA adds its warps' up and leaves one partial row of each.  Bound by HBM and, with three or four rows to a warp, by the
// first row's latency and the tail; 8320 rows of 640 (32 MB in, 11 MB out: 6.5 us), cold caches, us: 21.1 -> 15.2 with both sums,
// 17.6 -> 14.6 with dgain alone, since the warps' sums are added up side by side and not one warp after the other, and the
// next row loads under a row.
// Two CTAs to an SM, as many as are launched, up to 768 columns, and up to 1024 without the second sum (32896 rows of 1024, us:
// 49.8, with one 66.9).  With both sums 1024 columns take 179 registers; at 128 they spill (fp16, 8320 rows: 23.4 against 20.4).
constexpr bool norm_two_ctas(int nv, bool sums) { return nv <= (sums ? 3 : 4); }
template <typename T, int NV, bool SUMS>
__global__ void __launch_bounds__(kNormWarps * 32, norm_two_ctas(NV, SUMS) ? 2 : 1) rmsnorm_bwd_kernel(const NormBwd p) {
    extern __shared__ float sums[];  // [dgain | sum of out][warp][dim]
    pdl_trigger();
    pdl_wait();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nvec = p.dim / 8;
    float ds[NV][8], os[SUMS ? NV : 1][8];
#pragma unroll
    for (int j = 0; j < NV; ++j)
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            ds[j][e] = 0.f;
            if (SUMS) os[j][e] = 0.f;
        }
    const long long warps = (long long)gridDim.x * kNormWarps;
    // the next row loads under this one, where two rows beside the sums come close to 128 registers (of a thread's, 16 bytes spill at
    // 520 to 768 columns without the second sum; the bound itself spills 56 there in fp16 with it and 16 up to 1024 without)
    constexpr bool AHEAD = NV <= 2 || (NV == 3 && !SUMS);
    Vec8<T> xv[NV], dv[NV], av[NV];
    auto fetch = [&](long long row) {
        if (row >= p.rows) return;
#pragma unroll
        for (int j = 0; j < NV; ++j)
            if (lane + j * 32 < nvec) {
                const long long o = row * p.dim + (lane + j * 32) * 8;
                xv[j].load(static_cast<const T*>(p.x) + o);
                dv[j].load(static_cast<const T*>(p.dy) + o);
                if (p.add != nullptr) av[j].load(static_cast<const T*>(p.add) + o);
            }
    };
    const long long first = (long long)blockIdx.x * kNormWarps + warp;
    if (AHEAD) fetch(first);
    for (long long row = first; row < p.rows; row += warps) {
        const long long at = row * p.dim;
        if (!AHEAD) fetch(row);
        Vec8<T> x0[NV], d0[NV], a0[NV];
#pragma unroll
        for (int j = 0; j < NV; ++j) { x0[j] = xv[j]; d0[j] = dv[j]; a0[j] = av[j]; }
        if (AHEAD) fetch(row + warps);
        float ss = 0.f, dot = 0.f;
#pragma unroll
        for (int j = 0; j < NV; ++j)
            if (lane + j * 32 < nvec) {
                float x[8], d[8], g[8];
                x0[j].unpack(x);
                d0[j].unpack(d);
                load8<T>(static_cast<const T*>(p.gain) + (lane + j * 32) * 8, g);
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    ss = fmaf(x[e], x[e], ss);
                    dot = fmaf(d[e] * g[e], x[e], dot);
                }
            }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            ss += __shfl_xor_sync(0xffffffffu, ss, o);
            dot += __shfl_xor_sync(0xffffffffu, dot, o);
        }
        const float inv = 1.0f / sqrtf(ss / (float)p.dim + p.eps);
        const float c = dot * inv * inv * inv / (float)p.dim;  // x̂ mean(dy gain x̂) inv = x inv^3 mean(dy gain x)
#pragma unroll
        for (int j = 0; j < NV; ++j)
            if (lane + j * 32 < nvec) {
                float x[8], d[8], g[8], a[8];
                x0[j].unpack(x);
                d0[j].unpack(d);
                load8<T>(static_cast<const T*>(p.gain) + (lane + j * 32) * 8, g);
                if (p.add != nullptr) a0[j].unpack(a);
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    ds[j][e] = fmaf(d[e], x[e] * inv, ds[j][e]);
                    float v = d[e] * g[e] * inv - x[e] * c;
                    if (p.add != nullptr) v += a[e];
                    a[e] = to_f32<T>(from_f32<T>(v));
                    if (SUMS) os[j][e] += a[e];
                }
                store8<T>(static_cast<T*>(p.out) + at + (lane + j * 32) * 8, a);
            }
    }
    // every warp leaves its columns, then each column's eight values are added up in the order of the warps (neighbouring lanes
    // in neighbouring banks)
#pragma unroll
    for (int j = 0; j < NV; ++j)
        if (lane + j * 32 < nvec) {
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const int col = e * nvec + lane + j * 32;
                sums[warp * p.dim + col] = ds[j][e];
                if (SUMS) sums[(kNormWarps + warp) * p.dim + col] = os[j][e];
            }
        }
    __syncthreads();
    for (int i = threadIdx.x; i < p.dim; i += kNormWarps * 32) {
        const int at = (i & 7) * nvec + (i >> 3);
        float a = 0.f, b = 0.f;
#pragma unroll
        for (int w = 0; w < kNormWarps; ++w) {
            a += sums[w * p.dim + at];
            if (SUMS) b += sums[(kNormWarps + w) * p.dim + at];
        }
        p.dgain_part[(long long)blockIdx.x * p.dim + i] = a;
        if (SUMS) p.sum_part[(long long)blockIdx.x * p.dim + i] = b;
    }
}

// partial column sums of a [rows, cols] matrix: CTA (x: 256 columns, y: a strip of rows), 8 columns per thread, the
// CTA's eight row lanes added up in shared memory
template <typename T>
__global__ void __launch_bounds__(256) colsum_kernel(const void* src, float* part, int rows, int cols, int strip) {
    __shared__ float s[8][32][9];
    pdl_trigger();
    pdl_wait();
    const int c8 = threadIdx.x & 31, r = threadIdx.x >> 5, col = (blockIdx.x * 32 + c8) * 8;
    const int r0 = blockIdx.y * strip, r1 = min(rows, r0 + strip);
    float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (col < cols) {
        const T* p = static_cast<const T*>(src) + col;
#pragma unroll 4
        for (int i = r0 + r; i < r1; i += 8) {
            float v[8];
            load8<T>(p + (long long)i * cols, v);
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[e] += v[e];
        }
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) s[r][c8][e] = acc[e];
    __syncthreads();
    const int cc = threadIdx.x >> 3, e = threadIdx.x & 7, out = (blockIdx.x * 32 + cc) * 8 + e;
    if (out < cols) {
        float t = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) t += s[i][cc][e];
        part[(long long)blockIdx.y * cols + out] = t;
    }
}

// dst[j] = round(sum over parts of src[part][j]) for several arrays at once (blockIdx.y).  Up to kManyParts parts (split products): a
// thread per group of four columns, one chain.  More: eight chains (parts sub, sub + 8, ...), then their sums in the order of sub,
// whatever the threads are shared out to: 32 groups x 8 threads where the columns fill the chip (weight gradients cut into 17 to
// 32 ranges), and where they do not - column sums, 296 parts of 640 columns are a matter of latency - 8 groups x 32 threads
// that bring 128 parts at a time into shared memory for the eight chains.  us, cold caches (back to back), 32 x 8 | 8 x 32: 296 parts
// of 640 columns 16.4 (6.2) | 9.2 (3.4), 64 of 2560 9.2 (2.8) | 6.2 (2.4); 24 of 400 000 14.4 (5.8) | 28.7 (15.7).
constexpr int kManyParts = 16, kWide = 32, kNarrow = 8, kChunk = 128;
constexpr long long kNarrowColumns = 4096;  // (a CTA per 32 of them is less than one per SM)
__host__ __device__ inline int sum_groups(const SumParts::Item& it) {
    return it.parts <= kManyParts ? 256 : it.n <= kNarrowColumns ? kNarrow : kWide;
}

__device__ __forceinline__ void add4(float4& t, const float4& v) { t.x += v.x; t.y += v.y; t.z += v.z; t.w += v.w; }
template <typename T>
__device__ __forceinline__ void store_sum(const SumParts::Item& it, long long g, const float4& t) {
    T o[4] = {from_f32<T>(t.x), from_f32<T>(t.y), from_f32<T>(t.z), from_f32<T>(t.w)};
    *reinterpret_cast<uint2*>(static_cast<T*>(it.dst) + g * 4) = *reinterpret_cast<const uint2*>(o);
}

template <typename T>
__global__ void __launch_bounds__(256) sum_parts_kernel(const SumParts p) {
    __shared__ float4 s[kChunk * kNarrow];
    pdl_trigger();
    pdl_wait();
    const SumParts::Item it = p.item[blockIdx.y];
    const long long groups = (it.n + 3) / 4;
    if (sum_groups(it) == kNarrow) {
        const int at = threadIdx.x % kNarrow, sub = threadIdx.x / kNarrow;
        for (long long g0 = (long long)blockIdx.x * kNarrow; g0 < groups; g0 += (long long)gridDim.x * kNarrow) {
            const bool mine = g0 + at < groups;
            const float* src = it.src + (g0 + at) * 4;
            float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int q0 = 0; q0 < it.parts; q0 += kChunk) {
                const int n = min(kChunk, it.parts - q0);
                if (mine)
                    for (int q = sub; q < n; q += 256 / kNarrow)
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;"
                                     ::"r"((uint32_t)__cvta_generic_to_shared(s + q * kNarrow + at)), "l"(src + (q0 + q) * it.n) : "memory");
                asm volatile("cp.async.wait_all;" ::: "memory");
                __syncthreads();
                if (mine && sub < 8)
                    for (int q = sub; q < n; q += 8) add4(t, s[q * kNarrow + at]);
                __syncthreads();
            }
            if (sub < 8) s[sub * kNarrow + at] = t;
            __syncthreads();
            if (mine && sub == 0) {
                for (int q = 1; q < 8; ++q) add4(t, s[q * kNarrow + at]);
                store_sum<T>(it, g0 + at, t);
            }
            __syncthreads();
        }
        return;
    }
    const bool many = it.parts > kManyParts;
    const int lanes = many ? kWide : 256, sub = many ? threadIdx.x >> 5 : 0, step = many ? 8 : 1;
    for (long long g0 = (long long)blockIdx.x * lanes; g0 < groups; g0 += (long long)gridDim.x * lanes) {
        const long long g = g0 + (many ? threadIdx.x & 31 : threadIdx.x);
        float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
        if (g < groups) {
#pragma unroll 4
            for (int q = sub; q < it.parts; q += step) add4(t, *reinterpret_cast<const float4*>(it.src + (long long)q * it.n + g * 4));
        }
        if (many) {
            s[sub * kWide + (threadIdx.x & 31)] = t;
            __syncthreads();
            if (sub == 0) {
                for (int q = 1; q < 8; ++q) add4(t, s[q * kWide + threadIdx.x]);
            }
            __syncthreads();
        }
        if (g < groups && sub == 0) store_sum<T>(it, g, t);
    }
}

// ---- shifted cross-entropy ---------------------------------------------------------------------------------
// Row (b, i) of the logits [batch, np + seq, vocab] predicts labels[b, i - np + 1]; rows without a label (the persistent
// ones, the last, label = kIgnore) do not count.  A label outside the vocabulary makes loss and gradient NaN, and the status
// word says so.
constexpr long long kIgnore = -100, kBadLabel = -1;
__device__ __forceinline__ long long label_of(const CrossEntropy& p, int row) {
    const int len = p.np + p.seq, b = row / len, t = row - b * len - p.np;
    if (t < 0 || t + 1 >= p.seq) return kIgnore;
    const long long y = p.labels[(long long)b * p.seq + t + 1];
    if (y == kIgnore) return y;
    if (y < 0 || y >= p.vocab) {
        if (threadIdx.x == 0) atomicCAS(p.status, 0, (int)TMW_ERR_INVALID_ARGUMENT);
        return kBadLabel;
    }
    return y;
}

template <typename T>
__global__ void __launch_bounds__(256) ce_forward_kernel(const CrossEntropy p) {
    __shared__ float sm[8], sl[8];
    const int row = blockIdx.x, tid = threadIdx.x;
    const long long y = label_of(p, row);
    if (y < 0) {
        if (tid == 0) p.row_loss[row] = y == kIgnore ? -1.f : CUDART_NAN_F;  // (a loss is never negative)
        return;
    }
    const T* x = static_cast<const T*>(p.logits) + (long long)row * p.vocab;
    float m = -CUDART_INF_F, l = 0.f;
    const int nvec = p.vocab / 8;
    for (int v0 = tid; v0 < nvec; v0 += 256 * 4) {
        Vec8<T> raw[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (v0 + u * 256 < nvec) raw[u].load(x + (long long)(v0 + u * 256) * 8);
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (v0 + u * 256 < nvec) {
                float f[8];
                raw[u].unpack(f);
                float mx = f[0];
#pragma unroll
                for (int e = 1; e < 8; ++e) mx = fmaxf(mx, f[e]);
                if (mx > m) {
                    l *= __expf(m - mx);
                    m = mx;
                }
                // while only hidden logits (-inf) or NaN have been seen, the former count nothing; a NaN reaches the sum anyway
                const float base = m > -CUDART_INF_F ? m : 0.f;
#pragma unroll
                for (int e = 0; e < 8; ++e) l += __expf(f[e] - base);
            }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float mo = __shfl_xor_sync(0xffffffffu, m, o), lo = __shfl_xor_sync(0xffffffffu, l, o);
        const float mn = fmaxf(m, mo);
        l = (mn > -CUDART_INF_F) ? l * __expf(m - mn) + lo * __expf(mo - mn) : l + lo;  // (zeros, or NaN)
        m = mn;
    }
    if ((tid & 31) == 0) {
        sm[tid >> 5] = m;
        sl[tid >> 5] = l;
    }
    __syncthreads();
    if (tid == 0) {
        float ma = sm[0];
        for (int i = 1; i < 8; ++i) ma = fmaxf(ma, sm[i]);
        float la = 0.f;
        for (int i = 0; i < 8; ++i) la += sl[i] * __expf(sm[i] - ma);
        const float lse = ma + logf(la);
        const float loss = lse - to_f32<T>(x[y]);
        p.lse[row] = lse;
        p.row_loss[row] = loss < 0.f ? 0.f : loss;  // (by rounding; not fmaxf, which makes 0 of NaN)
    }
}

// loss = mean over the counted rows (NaN without any, like the library's); count[0] = their number
template <typename T>
__global__ void __launch_bounds__(1024) ce_mean_kernel(const CrossEntropy p) {
    __shared__ float s[32], c[32];
    float sum = 0.f, n = 0.f;
    for (int i = threadIdx.x; i < p.rows; i += 1024) {
        const float v = p.row_loss[i];
        if (v >= 0.f || v != v) {
            sum += v;
            n += 1.f;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        sum += __shfl_xor_sync(0xffffffffu, sum, o);
        n += __shfl_xor_sync(0xffffffffu, n, o);
    }
    if ((threadIdx.x & 31) == 0) {
        s[threadIdx.x >> 5] = sum;
        c[threadIdx.x >> 5] = n;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 1; i < 32; ++i) {
            sum += s[i];
            n += c[i];
        }
        *static_cast<T*>(p.loss) = from_f32<T>(sum / n);
        p.count[0] = n;
    }
}

// d_logits = (softmax - onehot) * grad / count on the counted rows, zero on the others
template <typename T>
__global__ void __launch_bounds__(256) ce_backward_kernel(const CrossEntropy p) {
    const int row = blockIdx.x, tid = threadIdx.x;
    const T* x = static_cast<const T*>(p.logits) + (long long)row * p.vocab;
    T* d = static_cast<T*>(p.d_logits) + (long long)row * p.vocab;
    const int nvec = p.vocab / 8;
    const long long y = label_of(p, row);
    if (y < 0) {
        float f[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] = y == kIgnore ? 0.f : CUDART_NAN_F;
        for (int v = tid; v < nvec; v += 256) store8<T>(d + (long long)v * 8, f);
        return;
    }
    const float scale = to_f32<T>(*static_cast<const T*>(p.grad)) / p.count[0], lse = p.lse[row];
    for (int v0 = tid; v0 < nvec; v0 += 256 * 4) {
        Vec8<T> raw[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (v0 + u * 256 < nvec) raw[u].load(x + (long long)(v0 + u * 256) * 8);
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (v0 + u * 256 < nvec) {
                const int v = v0 + u * 256;
                float f[8];
                raw[u].unpack(f);
#pragma unroll
                for (int e = 0; e < 8; ++e) f[e] = __expf(f[e] - lse) * scale;
                if (v == (int)(y >> 3)) {
#pragma unroll
                    for (int e = 0; e < 8; ++e)
                        if (e == (int)(y & 7)) f[e] -= scale;
                }
                store8<T>(d + (long long)v * 8, f);
            }
    }
}

// ---- embedding gradients -----------------------------------------------------------------------------------
// g [batch, np + seq, dim] is the gradient of the embedded rows.  Tokens that repeat share a row of the table: the first
// position to claim a token (owner) lends its row of `acc` (fp32, zero) to all of them, and adds the sum to the table's
// gradient once.  (Adding 16-bit values into the table one by one would round every time.)
template <typename T>
__global__ void __launch_bounds__(256) embed_claim_kernel(const EmbedBwd p) {
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= p.batch * p.seq) return;
    const long long id = p.ids[i];
    if (id >= 0 && id < p.vocab) atomicCAS(p.owner + id, -1, i);
}
template <typename T>
__global__ void __launch_bounds__(256) embed_scatter_kernel(const EmbedBwd p) {
    const int i = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (i >= p.batch * p.seq) return;
    const long long id = p.ids[i];
    if (id < 0 || id >= p.vocab) return;
    const int b = i / p.seq;
    const T* g = static_cast<const T*>(p.g) + ((long long)i + (long long)(b + 1) * p.np) * p.dim;
    float* acc = p.acc + (long long)p.owner[id] * p.dim;
    for (int v = lane; v < p.dim / 4; v += 32) {
        const uint2 raw = *reinterpret_cast<const uint2*>(g + v * 4);
        const T* h = reinterpret_cast<const T*>(&raw);
        asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(acc + v * 4), "f"(to_f32<T>(h[0])), "f"(to_f32<T>(h[1])),
                     "f"(to_f32<T>(h[2])), "f"(to_f32<T>(h[3])) : "memory");
    }
}
template <typename T>
__global__ void __launch_bounds__(256) embed_merge_kernel(const EmbedBwd p) {
    const int i = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (i >= p.batch * p.seq) return;
    const long long id = p.ids[i];
    if (id < 0 || id >= p.vocab || p.owner[id] != i) return;
    const float* acc = p.acc + (long long)i * p.dim;
    T* d = static_cast<T*>(p.d_tokens) + id * p.dim;
    for (int v = lane; v < p.dim / 8; v += 32) {
        float a[8], t[8];
        load8<float>(acc + v * 8, a);
        load8<T>(d + v * 8, t);
#pragma unroll
        for (int e = 0; e < 8; ++e) t[e] += a[e];
        store8<T>(d + v * 8, t);
    }
}
// position rows and persistent rows: sums over the batch
template <typename T>
__global__ void __launch_bounds__(256) embed_rows_bwd_kernel(const EmbedBwd p) {
    const int i = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31, len = p.np + p.seq;
    if (i >= len) return;
    T* d = i < p.np ? static_cast<T*>(p.d_persistent) + (long long)i * p.dim
                    : static_cast<T*>(p.d_positions) + (long long)(i - p.np) * p.dim;
    for (int v = lane; v < p.dim / 8; v += 32) {
        float t[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll 4
        for (int b = 0; b < p.batch; ++b) {
            float g[8];
            load8<T>(static_cast<const T*>(p.g) + ((long long)b * len + i) * p.dim + v * 8, g);
#pragma unroll
            for (int e = 0; e < 8; ++e) t[e] += g[e];
        }
        store8<T>(d + v * 8, t);
    }
}

template <typename T, int NV>
int launch_rmsnorm_bwd_nv(const NormBwd& p, int blocks, cudaStream_t stream) {
    const dim3 grid(blocks), block(kNormWarps * 32);
    auto run = [&](auto kern, int sums) -> int {
        const int smem = sums * kNormWarps * p.dim * (int)sizeof(float);
        if (smem > 48 * 1024) {  // (the default limit)
            const int rc = allow_shared_memory(reinterpret_cast<const void*>(kern), smem);
            if (rc != TMW_OK) return rc;
        }
        TMW_CUDA_TRY(launch_ex(kern, grid, block, smem, stream, true, 1, p));
        return TMW_OK;
    };
    return p.sum_part != nullptr ? run(rmsnorm_bwd_kernel<T, NV, true>, 2) : run(rmsnorm_bwd_kernel<T, NV, false>, 1);
}

template <typename T>
int launch_rmsnorm_bwd_t(const NormBwd& p, int blocks, cudaStream_t stream) {
    const int nv = (p.dim / 8 + 31) / 32;
    if (nv == 1) return launch_rmsnorm_bwd_nv<T, 1>(p, blocks, stream);
    if (nv == 2) return launch_rmsnorm_bwd_nv<T, 2>(p, blocks, stream);
    if (nv == 3) return launch_rmsnorm_bwd_nv<T, 3>(p, blocks, stream);
    if (nv <= 4) return launch_rmsnorm_bwd_nv<T, 4>(p, blocks, stream);
    if (nv <= 8) return launch_rmsnorm_bwd_nv<T, 8>(p, blocks, stream);
    return TMW_ERR_UNSUPPORTED;
}

}  // namespace

int norm_bwd_blocks(long long rows) {
    const long long want = (rows + kNormWarps - 1) / kNormWarps;
    return (int)(want < 2 * sm_count() ? want : 2 * sm_count());
}
int launch_rmsnorm_bwd(int dtype, const NormBwd& p, cudaStream_t stream) {
    const int blocks = norm_bwd_blocks(p.rows);
    return dtype == TMW_BF16 ? launch_rmsnorm_bwd_t<__nv_bfloat16>(p, blocks, stream) : launch_rmsnorm_bwd_t<__half>(p, blocks, stream);
}

int colsum_strips(int rows) {
    const int want = (rows + 63) / 64;
    return want < 64 ? want : 64;
}
int launch_colsum(int dtype, const void* src, float* part, int rows, int cols, cudaStream_t stream) {
    const int strips = colsum_strips(rows), strip = (rows + strips - 1) / strips;
    const dim3 grid((cols + 255) / 256, strips), block(256);
    if (dtype == TMW_BF16) TMW_CUDA_TRY(launch_ex(colsum_kernel<__nv_bfloat16>, grid, block, 0, stream, true, 1, src, part, rows, cols, strip));
    else TMW_CUDA_TRY(launch_ex(colsum_kernel<__half>, grid, block, 0, stream, true, 1, src, part, rows, cols, strip));
    return TMW_OK;
}

int launch_sum_parts(int dtype, const SumParts& p, cudaStream_t stream) {
    if (p.count == 0) return TMW_OK;
    long long most = 1;
    for (int i = 0; i < p.count; ++i) {
        const long long lanes = sum_groups(p.item[i]), blocks = ((p.item[i].n + 3) / 4 + lanes - 1) / lanes;
        most = blocks > most ? blocks : most;
    }
    const dim3 grid((unsigned)(most < 8 * sm_count() ? most : 8 * sm_count()), p.count), block(256);
    if (dtype == TMW_BF16) TMW_CUDA_TRY(launch_ex(sum_parts_kernel<__nv_bfloat16>, grid, block, 0, stream, true, 1, p));
    else TMW_CUDA_TRY(launch_ex(sum_parts_kernel<__half>, grid, block, 0, stream, true, 1, p));
    return TMW_OK;
}

int launch_cross_entropy(int dtype, const CrossEntropy& p, bool backward, cudaStream_t stream) {
    const bool bf16 = dtype == TMW_BF16;
    if (backward) {
        if (bf16) ce_backward_kernel<__nv_bfloat16><<<p.rows, 256, 0, stream>>>(p);
        else ce_backward_kernel<__half><<<p.rows, 256, 0, stream>>>(p);
    } else {
        if (bf16) ce_forward_kernel<__nv_bfloat16><<<p.rows, 256, 0, stream>>>(p);
        else ce_forward_kernel<__half><<<p.rows, 256, 0, stream>>>(p);
        if (bf16) ce_mean_kernel<__nv_bfloat16><<<1, 1024, 0, stream>>>(p);
        else ce_mean_kernel<__half><<<1, 1024, 0, stream>>>(p);
    }
    TMW_CUDA_TRY(cudaGetLastError());
    return TMW_OK;
}

template <typename T>
static int launch_embed_bwd_t(const EmbedBwd& p, cudaStream_t stream) {
    const int n = p.batch * p.seq, len = p.np + p.seq;
    TMW_CUDA_TRY(cudaMemsetAsync(p.owner, 0xff, (size_t)p.vocab * sizeof(int), stream));
    TMW_CUDA_TRY(cudaMemsetAsync(p.acc, 0, (size_t)n * p.dim * sizeof(float), stream));
    embed_claim_kernel<T><<<(n + 255) / 256, 256, 0, stream>>>(p);
    embed_scatter_kernel<T><<<(n + 7) / 8, 256, 0, stream>>>(p);
    embed_merge_kernel<T><<<(n + 7) / 8, 256, 0, stream>>>(p);
    embed_rows_bwd_kernel<T><<<(len + 7) / 8, 256, 0, stream>>>(p);
    TMW_CUDA_TRY(cudaGetLastError());
    return TMW_OK;
}
int launch_embed_bwd(int dtype, const EmbedBwd& p, cudaStream_t stream) {
    return dtype == TMW_BF16 ? launch_embed_bwd_t<__nv_bfloat16>(p, stream) : launch_embed_bwd_t<__half>(p, stream);
}

}  // namespace tmw
