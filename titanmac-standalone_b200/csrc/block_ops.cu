// Element-wise kernels around the attention call (all HBM-bound, 16-byte accesses).
//
// Residual add + RMSNorm in one pass over the rows: the element-wise work that surrounds the
// attention module in a TitanBlock (titans_core/blocks/titan_block.py:92-100 of the reference,
// norm formula titans_core/blocks/norms.py:55-58).  In PyTorch the residual add and the norm are
// seven small kernels and as many trips through HBM; here a row is read once, the sum is stored
// (it is the new residual stream) and the normalised row is written.  HBM-bound: one warp per row,
// 16-byte accesses, the row stays in registers between the two passes when it is short enough.
#include "tmw_common.cuh"

namespace tmw {
namespace {

constexpr int kWarpsPerBlock = 8;

// CTAs of `kernel` that fit on the whole GPU at once (the grid of a kernel whose threads loop over the work)
template <typename K>
int resident_ctas(K kernel, int threads) {
    int sms = 148, dev = 0, per_sm = 1;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, 0) != cudaSuccess || per_sm < 1) per_sm = 1;
    return sms * per_sm;
}

// NV = 8-element vectors per lane kept in registers; NV == 0: the row is read again for the second pass
// (it comes out of L1/L2: the same warp has just read or written it).
template <typename T, int NV, bool RES>
__global__ void __launch_bounds__(kWarpsPerBlock * 32)
add_rmsnorm_kernel(const T* x, const T* residual, const T* __restrict__ scale, float eps, T* sum_out, T* y, long long rows,
                   int dim) {
    pdl_trigger();
    pdl_wait();
    const T* res = RES ? residual : nullptr;  // (without a residual its registers are not there either)
    const int lane = threadIdx.x & 31;
    const long long warps = (long long)gridDim.x * kWarpsPerBlock;
    // a resident grid: every warp walks over rows (a block that lives for one row per warp spends most of
    // its life being scheduled), the next row's loads in flight under the current one's reduction and stores (65664 rows of
    // 640, us: 36.7 without, 30.8 with; 16416 rows of 1024: 13.2, 9.2)
    constexpr int kN = NV > 0 ? NV : 1;
    Vec8<T> nx[kN], nr[kN], gain[kN];
    auto fetch = [&](long long row) {
#pragma unroll
        for (int j = 0; j < NV; ++j)
            if (row < rows && lane + j * 32 < dim / 8) {
                nx[j].load(x + row * dim + (lane + j * 32) * 8);
                if (res != nullptr) nr[j].load(res + row * dim + (lane + j * 32) * 8);
            }
    };
    if (NV > 0) {
#pragma unroll
        for (int j = 0; j < NV; ++j)
            if (lane + j * 32 < dim / 8) gain[j].load(scale + (lane + j * 32) * 8);
        fetch((long long)blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5));
    }
    for (long long row = (long long)blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5); row < rows; row += warps) {
    const T* xr = x + row * dim;
    const T* rr = res != nullptr ? res + row * dim : nullptr;
    T* sr = sum_out != nullptr ? sum_out + row * dim : nullptr;
    T* yr = y + row * dim;
    const int nvec = dim / 8;

    // h = x + residual, rounded to the storage type like the reference's `x + f(x)`; the norm is taken of
    // the rounded values, in fp32
    auto load_h = [&](int v, float (&h)[8]) {
        load8<T>(xr + v * 8, h);
        if (rr != nullptr) {
            float r[8];
            load8<T>(rr + v * 8, r);
#pragma unroll
            for (int i = 0; i < 8; ++i) h[i] = to_f32<T>(from_f32<T>(h[i] + r[i]));
        }
    };

    float keep[NV > 0 ? NV : 1][8];
    float ss = 0.f;
    if constexpr (NV > 0) {
        // (all loads before the first store, which may be to the same rows)
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            if (lane + j * 32 < nvec) {
                nx[j].unpack(keep[j]);
                if (rr != nullptr) {
                    float r[8];
                    nr[j].unpack(r);
#pragma unroll
                    for (int i = 0; i < 8; ++i) keep[j][i] = to_f32<T>(from_f32<T>(keep[j][i] + r[i]));
                }
            }
        }
        fetch(row + warps);
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            const int v = lane + j * 32;
            if (v < nvec) {
                if (rr != nullptr && sr != nullptr) store8<T>(sr + v * 8, keep[j]);
#pragma unroll
                for (int i = 0; i < 8; ++i) ss = fmaf(keep[j][i], keep[j][i], ss);
            }
        }
    } else {
        for (int v = lane; v < nvec; v += 32) {
            float h[8];
            load_h(v, h);
            if (sr != nullptr && rr != nullptr) store8<T>(sr + v * 8, h);
#pragma unroll
            for (int i = 0; i < 8; ++i) ss = fmaf(h[i], h[i], ss);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    // the reference computes x / rms * scale; multiplying by the reciprocal differs by at most one fp32 ulp
    const float inv = 1.0f / sqrtf(ss / (float)dim + eps);

    auto emit = [&](int v, const float (&h)[8], const Vec8<T>* kept) {
        float g[8], out[8];
        if (kept != nullptr) kept->unpack(g); else load8<T>(scale + v * 8, g);
#pragma unroll
        for (int i = 0; i < 8; ++i) out[i] = h[i] * inv * g[i];
        store8<T>(yr + v * 8, out);
    };
    if (NV > 0) {
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            const int v = lane + j * 32;
            if (v < nvec) emit(v, keep[j], &gain[j]);
        }
    } else {
        for (int v = lane; v < nvec; v += 32) {
            float h[8];
            if (sr != nullptr && rr != nullptr) load8<T>(sr + v * 8, h); else load_h(v, h);
            emit(v, h, nullptr);
        }
    }
    }  // rows
}

template <typename T>
int launch_add_rmsnorm_t(long long rows, int dim, const void* x, const void* res, const void* scale, float eps,
                         void* sum_out, void* y, cudaStream_t stream, bool pdl) {
    const long long want = (rows + kWarpsPerBlock - 1) / kWarpsPerBlock;
    const int nv = (dim / 8 + 31) / 32;
    // one resident wave: every warp walks over its rows, nothing waits for a slot
#define TMW_NORM_CASE(N)                                                                                     \
    {                                                                                                        \
        static int waves[2] = {0, 0};                                                                        \
        auto kern = res != nullptr ? add_rmsnorm_kernel<T, N, true> : add_rmsnorm_kernel<T, N, false>;       \
        int& wave = waves[res != nullptr];                                                                   \
        if (wave == 0) wave = resident_ctas(kern, kWarpsPerBlock * 32);                                      \
        const unsigned blocks = (unsigned)(want < wave ? want : wave);                                       \
        TMW_CUDA_TRY(launch_ex(kern, dim3(blocks), dim3(kWarpsPerBlock * 32), 0, stream, pdl, 1,      \
                               static_cast<const T*>(x), static_cast<const T*>(res), static_cast<const T*>(scale), eps,  \
                               static_cast<T*>(sum_out), static_cast<T*>(y), rows, dim));                                \
    }
    switch (nv) {
        case 1: TMW_NORM_CASE(1); break;
        case 2: TMW_NORM_CASE(2); break;
        case 3: TMW_NORM_CASE(3); break;
        case 4: TMW_NORM_CASE(4); break;
        default: TMW_NORM_CASE(0); break;
    }
#undef TMW_NORM_CASE
    return TMW_OK;
}

// ---- exact GELU --------------------------------------------------------------------------------------
// 0.5 x (1 + erf(x / sqrt 2)), the default nn.GELU() of the reference's MLP (titans_core/blocks/mlp.py:58-65).
// erf by the rational approximation of gelu_erf (tmw_common.cuh), so that the kernel stays bound by HBM (one read, one
// write) and not by arithmetic.
constexpr int kGeluUnroll = 4;  // 16-byte loads in flight per thread

template <typename T>
__global__ void __launch_bounds__(256) gelu_kernel(const T* x, T* y, long long nvec) {
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long v0 = (long long)blockIdx.x * blockDim.x + threadIdx.x; v0 < nvec; v0 += stride * kGeluUnroll) {
        float a[kGeluUnroll][8];
#pragma unroll
        for (int u = 0; u < kGeluUnroll; ++u)
            if (v0 + u * stride < nvec) load8<T>(x + (v0 + u * stride) * 8, a[u]);
#pragma unroll
        for (int u = 0; u < kGeluUnroll; ++u)
            if (v0 + u * stride < nvec) {
#pragma unroll
                for (int i = 0; i < 8; ++i) a[u][i] = gelu_erf(a[u][i]);
                store8<T>(y + (v0 + u * stride) * 8, a[u]);
            }
    }
}

template <typename T>
int launch_gelu(long long n, const void* x, void* y, cudaStream_t stream) {
    static int wave = 0;
    if (wave == 0) wave = resident_ctas(gelu_kernel<T>, 256);
    const long long nvec = n / 8;
    const long long want = (nvec + 256 * kGeluUnroll - 1) / (256 * kGeluUnroll);
    const unsigned blocks = (unsigned)(want < wave ? want : wave);
    gelu_kernel<T><<<blocks, 256, 0, stream>>>(static_cast<const T*>(x), static_cast<T*>(y), nvec);
    TMW_CUDA_TRY(cudaGetLastError());
    return TMW_OK;
}

// ---- causal depthwise convolution along the rows ---------------------------------------------------------
// y[b, t, c] = sum_j w[c, j] * x[b, t - (TAPS-1) + j, c]: the Conv1d(groups = channels, padding = TAPS-1),
// trimmed to the input length, that the reference's block-sparse attention applies to Q, K and V
// (titans_core/attn/block_sparse_attention.py:77-92, 241-256).  Bound by HBM (or L2) where the tensors are large and by the
// length of a thread's chain of loads where they are not: a warp owns 32 x 8 adjacent channels and a strip of rows, four
// rows requested at a time (one thread walking 64 rows one by one took 18.8 us for 8241 x 1920 values of 16 bits and 14.9 us
// for 2112 x 768).  The taps - 1 rows in front of a warp's own come out of L1 or L2.
constexpr int kConvWarps = 8;   // warps per CTA, one below the other
constexpr int kConvThreads = 32 * kConvWarps;
constexpr int kConvBatch = 4;   // rows in flight per thread
constexpr int kConvMinRows = 8, kConvMaxRows = 16;  // rows per warp

// eight rows per warp, or sixteen where that still leaves every SM two CTAs (fewer filter loads and rows read twice)
int conv_rows_per_warp(int batch, int rows, int channels) {
    const long long ctas = (long long)batch * ((channels + 255) / 256) * ((rows + kConvWarps * kConvMaxRows - 1) / (kConvWarps * kConvMaxRows));
    return ctas >= 2 * sm_count() ? kConvMaxRows : kConvMinRows;
}

// The filters [channels, taps] in up to three arrays of `per` channels each (Q, K and V keep theirs apart).
struct ConvWeights {
    const void* w[3];
    int per;
};

// the filters of 8 adjacent channels: 8 * TAPS adjacent values
template <typename T, int TAPS>
__device__ __forceinline__ void load_filters(const ConvWeights& f, int channel, float (&wr)[TAPS][8]) {
    const int part = channel / f.per, first = channel - part * f.per;  // (`per` is a multiple of 8)
    const T* w = static_cast<const T*>(part == 0 ? f.w[0] : part == 1 ? f.w[1] : f.w[2]) + (long long)first * TAPS;
    float v[TAPS][8];
    if ((reinterpret_cast<uintptr_t>(w) & 15) == 0) {
#pragma unroll
        for (int i = 0; i < TAPS; ++i) load8<T>(w + i * 8, v[i]);
    } else {
#pragma unroll
        for (int i = 0; i < TAPS * 8; ++i) v[i / 8][i % 8] = to_f32<T>(w[i]);
    }
#pragma unroll
    for (int c = 0; c < 8; ++c)
#pragma unroll
        for (int j = 0; j < TAPS; ++j) wr[j][c] = v[(c * TAPS + j) / 8][(c * TAPS + j) % 8];
}

template <typename T, int TAPS>
__global__ void __launch_bounds__(kConvThreads)
dwconv_kernel(const T* x, const ConvWeights f, T* y, int rows, int channels, int per_warp) {
    const int vec = blockIdx.x * 32 + (threadIdx.x & 31);  // which group of 8 channels
    const int t0 = (blockIdx.y * kConvWarps + (threadIdx.x >> 5)) * per_warp, t1 = min(rows, t0 + per_warp);
    if (vec * 8 >= channels || t0 >= rows) return;
    const long long base = (long long)blockIdx.z * rows * channels + vec * 8;
    float wr[TAPS][8], hist[TAPS][8];  // hist[j] = x[t - (TAPS-1) + j]
    load_filters<T, TAPS>(f, vec * 8, wr);
    // A link of the chain that does not trigger its successor early: the CTAs of the persistent rows' kernel and, behind them,
    // of the attention would sit in registers and shared memory while this one's later waves still wait for room.  Layer of
    // 3 x 2747 | 8 x 4112 rows, us: 97.5 | 284 as an ordinary launch, 98.4 | 292 with the trigger, 95.3 | 280 without.
    pdl_wait();
#pragma unroll
    for (int j = 0; j < TAPS - 1; ++j) {
        const int t = t0 - (TAPS - 1) + j;
        if (t >= 0) {
            load8<T>(x + base + (long long)t * channels, hist[j + 1]);
        } else {
#pragma unroll
            for (int c = 0; c < 8; ++c) hist[j + 1][c] = 0.f;
        }
    }
    for (int tb = t0; tb < t1; tb += kConvBatch) {
        Vec8<T> raw[kConvBatch];
#pragma unroll
        for (int u = 0; u < kConvBatch; ++u)
            if (tb + u < t1) raw[u].load(x + base + (long long)(tb + u) * channels);
#pragma unroll
        for (int u = 0; u < kConvBatch; ++u)
            if (tb + u < t1) {
#pragma unroll
                for (int j = 0; j < TAPS - 1; ++j)
#pragma unroll
                    for (int c = 0; c < 8; ++c) hist[j][c] = hist[j + 1][c];
                raw[u].unpack(hist[TAPS - 1]);
                float out[8];
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    float a = 0.f;
#pragma unroll
                    for (int j = 0; j < TAPS; ++j) a = fmaf(wr[j][c], hist[j][c], a);
                    out[c] = a;
                }
                store8<T>(y + base + (long long)(tb + u) * channels, out);
            }
    }
}

template <typename T, int TAPS>
int launch_dwconv_taps(int batch, int rows, int channels, const void* x, const ConvWeights& w, void* y, cudaStream_t stream, bool pdl) {
    const int per_warp = conv_rows_per_warp(batch, rows, channels), strip = kConvWarps * per_warp;
    const dim3 grid((channels / 8 + 31) / 32, (rows + strip - 1) / strip, batch);
    TMW_CUDA_TRY(launch_ex(dwconv_kernel<T, TAPS>, grid, dim3(kConvThreads), 0, stream, pdl, 1, static_cast<const T*>(x), w,
                           static_cast<T*>(y), rows, channels, per_warp));
    return TMW_OK;
}

// Backward of the convolution in one pass over x and dy: dx[t] = sum_j w[j] dy[t + (TAPS-1) - j] from the TAPS rows of dy at
// and behind t, dw[c][j] = sum over batch and rows of dy[t][c] x[t - (TAPS-1) + j][c] from the TAPS rows of x up to t.  The
// filter's gradient is added up over the CTA's warps in shared memory and from there, with atomics, into an fp32 buffer
// [channels, TAPS] (zero on entry).  (2112 x 768 values: 34.3 us as two passes over strips of 64 rows, 11.3 us.)
template <typename T, int TAPS>
__global__ void __launch_bounds__(kConvThreads)
dwconv_bwd_kernel(const T* __restrict__ x, const ConvWeights f, const T* __restrict__ dy, T* __restrict__ dx,
                  float* __restrict__ dw, int rows, int channels, int per_warp) {
    __shared__ float sums[256 * TAPS];  // [tap][channel of the CTA]
    constexpr int kBatch = TAPS <= 4 ? kConvBatch : 1;  // (registers)
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int vec = blockIdx.x * 32 + lane;
    const int t0 = (blockIdx.y * kConvWarps + warp) * per_warp, t1 = min(rows, t0 + per_warp);
    const bool live = vec * 8 < channels && t0 < rows;
    const long long base = (long long)blockIdx.z * rows * channels + vec * 8;
    float acc[TAPS][8];
#pragma unroll
    for (int j = 0; j < TAPS; ++j)
#pragma unroll
        for (int c = 0; c < 8; ++c) acc[j][c] = 0.f;
    if (live) {
        float wr[TAPS][8], hist[TAPS][8], ahead[TAPS][8];  // hist[j] = x[t - (TAPS-1) + j], ahead[m] = dy[t + m]
        load_filters<T, TAPS>(f, vec * 8, wr);
        auto row_or_zero = [&](const T* src, int t, float (&out)[8]) {
            if (t >= 0 && t < rows) {
                load8<T>(src + base + (long long)t * channels, out);
            } else {
#pragma unroll
                for (int c = 0; c < 8; ++c) out[c] = 0.f;
            }
        };
#pragma unroll
        for (int j = 0; j < TAPS - 1; ++j) {
            row_or_zero(x, t0 - (TAPS - 1) + j, hist[j + 1]);
            row_or_zero(dy, t0 + j, ahead[j + 1]);
        }
        for (int tb = t0; tb < t1; tb += kBatch) {
            Vec8<T> xr[kBatch], dr[kBatch];
#pragma unroll
            for (int u = 0; u < kBatch; ++u) {
                if (tb + u < t1) xr[u].load(x + base + (long long)(tb + u) * channels);
                if (tb + u + TAPS - 1 < rows) dr[u].load(dy + base + (long long)(tb + u + TAPS - 1) * channels);
            }
#pragma unroll
            for (int u = 0; u < kBatch; ++u)
                if (tb + u < t1) {
#pragma unroll
                    for (int j = 0; j < TAPS - 1; ++j)
#pragma unroll
                        for (int c = 0; c < 8; ++c) {
                            hist[j][c] = hist[j + 1][c];
                            ahead[j][c] = ahead[j + 1][c];
                        }
                    xr[u].unpack(hist[TAPS - 1]);
                    if (tb + u + TAPS - 1 < rows) {
                        dr[u].unpack(ahead[TAPS - 1]);
                    } else {
#pragma unroll
                        for (int c = 0; c < 8; ++c) ahead[TAPS - 1][c] = 0.f;
                    }
                    float out[8];
#pragma unroll
                    for (int c = 0; c < 8; ++c) {
                        float a = 0.f;
#pragma unroll
                        for (int j = 0; j < TAPS; ++j) {
                            a = fmaf(wr[j][c], ahead[TAPS - 1 - j][c], a);
                            acc[j][c] = fmaf(ahead[0][c], hist[j][c], acc[j][c]);
                        }
                        out[c] = a;
                    }
                    store8<T>(dx + base + (long long)(tb + u) * channels, out);
                }
        }
    }
    for (int w = 0; w < kConvWarps; ++w) {
        if (warp == w) {
#pragma unroll
            for (int j = 0; j < TAPS; ++j)
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    float* p = sums + j * 256 + c * 32 + lane;
                    *p = w ? *p + acc[j][c] : acc[j][c];
                }
        }
        __syncthreads();
    }
    for (int i = threadIdx.x; i < 256 * TAPS; i += kConvThreads) {
        const int j = i / 256, c = i % 256 / 32, channel = (blockIdx.x * 32 + i % 32) * 8 + c;
        if (channel < channels) atomicAdd(dw + (long long)channel * TAPS + j, sums[i]);
    }
}

template <typename T, int TAPS>
int launch_dwconv_bwd_taps(int batch, int rows, int channels, const void* x, const ConvWeights& w, const void* dy, void* dx,
                           float* dw, cudaStream_t stream) {
    const int per_warp = conv_rows_per_warp(batch, rows, channels), strip = kConvWarps * per_warp;
    const dim3 grid((channels / 8 + 31) / 32, (rows + strip - 1) / strip, batch);
    dwconv_bwd_kernel<T, TAPS><<<grid, kConvThreads, 0, stream>>>(static_cast<const T*>(x), w,
                                                                  static_cast<const T*>(dy), static_cast<T*>(dx), dw,
                                                                  rows, channels, per_warp);
    TMW_CUDA_TRY(cudaGetLastError());
    return TMW_OK;
}

template <typename T>
int launch_dwconv_bwd(int batch, int rows, int channels, int taps, const void* x, const ConvWeights& w, const void* dy,
                      void* dx, float* dw, cudaStream_t stream) {
    switch (taps) {
        case 1: return launch_dwconv_bwd_taps<T, 1>(batch, rows, channels, x, w, dy, dx, dw, stream);
        case 2: return launch_dwconv_bwd_taps<T, 2>(batch, rows, channels, x, w, dy, dx, dw, stream);
        case 3: return launch_dwconv_bwd_taps<T, 3>(batch, rows, channels, x, w, dy, dx, dw, stream);
        case 4: return launch_dwconv_bwd_taps<T, 4>(batch, rows, channels, x, w, dy, dx, dw, stream);
        case 5: return launch_dwconv_bwd_taps<T, 5>(batch, rows, channels, x, w, dy, dx, dw, stream);
        case 6: return launch_dwconv_bwd_taps<T, 6>(batch, rows, channels, x, w, dy, dx, dw, stream);
        case 7: return launch_dwconv_bwd_taps<T, 7>(batch, rows, channels, x, w, dy, dx, dw, stream);
        case 8: return launch_dwconv_bwd_taps<T, 8>(batch, rows, channels, x, w, dy, dx, dw, stream);
        default: return TMW_ERR_UNSUPPORTED;
    }
}

template <typename T>
int launch_dwconv_t(int batch, int rows, int channels, int taps, const void* x, const ConvWeights& w, void* y,
                    cudaStream_t stream, bool pdl) {
    switch (taps) {
        case 1: return launch_dwconv_taps<T, 1>(batch, rows, channels, x, w, y, stream, pdl);
        case 2: return launch_dwconv_taps<T, 2>(batch, rows, channels, x, w, y, stream, pdl);
        case 3: return launch_dwconv_taps<T, 3>(batch, rows, channels, x, w, y, stream, pdl);
        case 4: return launch_dwconv_taps<T, 4>(batch, rows, channels, x, w, y, stream, pdl);
        case 5: return launch_dwconv_taps<T, 5>(batch, rows, channels, x, w, y, stream, pdl);
        case 6: return launch_dwconv_taps<T, 6>(batch, rows, channels, x, w, y, stream, pdl);
        case 7: return launch_dwconv_taps<T, 7>(batch, rows, channels, x, w, y, stream, pdl);
        case 8: return launch_dwconv_taps<T, 8>(batch, rows, channels, x, w, y, stream, pdl);
        default: return TMW_ERR_UNSUPPORTED;
    }
}

}  // namespace

int launch_add_rmsnorm(int dtype, long long rows, int dim, const void* x, const void* residual, const void* scale, float eps,
                       void* sum_out, void* y, cudaStream_t stream, bool pdl) {
    switch (dtype) {
        case TMW_F32: return launch_add_rmsnorm_t<float>(rows, dim, x, residual, scale, eps, sum_out, y, stream, pdl);
        case TMW_BF16: return launch_add_rmsnorm_t<__nv_bfloat16>(rows, dim, x, residual, scale, eps, sum_out, y, stream, pdl);
        default: return launch_add_rmsnorm_t<__half>(rows, dim, x, residual, scale, eps, sum_out, y, stream, pdl);
    }
}

int launch_dwconv(int dtype, int batch, int rows, int channels, int taps, const void* x, const void* const* w, int n_w, void* y,
                  cudaStream_t stream, bool pdl) {
    ConvWeights f;
    f.per = channels / n_w;
    for (int i = 0; i < 3; ++i) f.w[i] = w[i < n_w ? i : 0];
    switch (dtype) {
        case TMW_F32: return launch_dwconv_t<float>(batch, rows, channels, taps, x, f, y, stream, pdl);
        case TMW_BF16: return launch_dwconv_t<__nv_bfloat16>(batch, rows, channels, taps, x, f, y, stream, pdl);
        default: return launch_dwconv_t<__half>(batch, rows, channels, taps, x, f, y, stream, pdl);
    }
}

int launch_dwconv_backward(int dtype, int batch, int rows, int channels, int taps, const void* x, const void* const* w, int n_w,
                           const void* dy, void* dx, float* dw, cudaStream_t stream) {
    ConvWeights f;
    f.per = channels / n_w;
    for (int i = 0; i < 3; ++i) f.w[i] = w[i < n_w ? i : 0];
    switch (dtype) {
        case TMW_F32: return launch_dwconv_bwd<float>(batch, rows, channels, taps, x, f, dy, dx, dw, stream);
        case TMW_BF16: return launch_dwconv_bwd<__nv_bfloat16>(batch, rows, channels, taps, x, f, dy, dx, dw, stream);
        default: return launch_dwconv_bwd<__half>(batch, rows, channels, taps, x, f, dy, dx, dw, stream);
    }
}

}  // namespace tmw

extern "C" int tmw_causal_dwconv(int32_t dtype, int32_t batch, int32_t rows, int32_t channels, int32_t taps,
                                 const void* x, const void* weight, void* y, void* stream) {
    using namespace tmw;
    if (batch < 0 || rows < 0 || channels <= 0) return TMW_ERR_INVALID_ARGUMENT;
    if (dtype != TMW_F32 && dtype != TMW_BF16 && dtype != TMW_F16) return TMW_ERR_INVALID_ARGUMENT;
    if (taps < 1 || taps > 8 || channels % 8 != 0) {
        set_error_text("tmw_causal_dwconv: 1 to 8 taps and a multiple of 8 channels");
        return TMW_ERR_UNSUPPORTED;
    }
    if (batch == 0 || rows == 0) return TMW_OK;
    if (x == nullptr || weight == nullptr || y == nullptr || x == y) return TMW_ERR_INVALID_ARGUMENT;
    if ((((uintptr_t)x | (uintptr_t)y) & 15) != 0) {
        set_error_text("tmw_causal_dwconv: x and y must be 16-byte aligned");
        return TMW_ERR_INVALID_ARGUMENT;
    }
    if (batch > 65535 || (rows + kConvWarps * kConvMinRows - 1) / (kConvWarps * kConvMinRows) > 65535) return TMW_ERR_TOO_LARGE;
    return launch_dwconv(dtype, batch, rows, channels, taps, x, &weight, 1, y, static_cast<cudaStream_t>(stream));
}

extern "C" int tmw_causal_dwconv_backward(int32_t dtype, int32_t batch, int32_t rows, int32_t channels, int32_t taps,
                                          const void* x, const void* weight, const void* dy, void* dx, float* dw,
                                          void* stream) {
    using namespace tmw;
    if (batch < 0 || rows < 0 || channels <= 0) return TMW_ERR_INVALID_ARGUMENT;
    if (dtype != TMW_F32 && dtype != TMW_BF16 && dtype != TMW_F16) return TMW_ERR_INVALID_ARGUMENT;
    if (taps < 1 || taps > 8 || channels % 8 != 0) return TMW_ERR_UNSUPPORTED;
    if (batch == 0 || rows == 0) return TMW_OK;
    if (x == nullptr || weight == nullptr || dy == nullptr || dx == nullptr || dw == nullptr || dx == dy)
        return TMW_ERR_INVALID_ARGUMENT;
    if ((((uintptr_t)x | (uintptr_t)dy | (uintptr_t)dx) & 15) != 0) return TMW_ERR_INVALID_ARGUMENT;
    if (batch > 65535 || (rows + kConvWarps * kConvMinRows - 1) / (kConvWarps * kConvMinRows) > 65535) return TMW_ERR_TOO_LARGE;
    return launch_dwconv_backward(dtype, batch, rows, channels, taps, x, &weight, 1, dy, dx, dw, static_cast<cudaStream_t>(stream));
}

extern "C" int tmw_gelu(int32_t dtype, int64_t n, const void* x, void* y, void* stream) {
    using namespace tmw;
    if (n < 0 || (n > 0 && (x == nullptr || y == nullptr))) {
        set_error_text("tmw_gelu: null pointer or negative size");
        return TMW_ERR_INVALID_ARGUMENT;
    }
    if (dtype != TMW_F32 && dtype != TMW_BF16 && dtype != TMW_F16) return TMW_ERR_INVALID_ARGUMENT;
    if (n % 8 != 0) {
        set_error_text("tmw_gelu: the element count must be a multiple of 8");
        return TMW_ERR_UNSUPPORTED;
    }
    if ((((uintptr_t)x | (uintptr_t)y) & 15) != 0) {
        set_error_text("tmw_gelu: both pointers must be 16-byte aligned");
        return TMW_ERR_INVALID_ARGUMENT;
    }
    if (n == 0) return TMW_OK;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    switch (dtype) {
        case TMW_F32: return launch_gelu<float>(n, x, y, s);
        case TMW_BF16: return launch_gelu<__nv_bfloat16>(n, x, y, s);
        default: return launch_gelu<__half>(n, x, y, s);
    }
}

extern "C" int tmw_add_rmsnorm(int32_t dtype, int64_t rows, int32_t dim, const void* x, const void* residual,
                               const void* scale, float eps, void* sum_out, void* y, void* stream) {
    using namespace tmw;
    if (rows < 0 || dim <= 0 || x == nullptr || scale == nullptr || y == nullptr || !(eps >= 0.f)) {
        set_error_text("tmw_add_rmsnorm: null pointer, negative size or negative eps");
        return TMW_ERR_INVALID_ARGUMENT;
    }
    if (dtype != TMW_F32 && dtype != TMW_BF16 && dtype != TMW_F16) return TMW_ERR_INVALID_ARGUMENT;
    if (dim % 8 != 0) {
        set_error_text("tmw_add_rmsnorm: the row length must be a multiple of 8");
        return TMW_ERR_UNSUPPORTED;
    }
    const uintptr_t all = (uintptr_t)x | (uintptr_t)residual | (uintptr_t)scale | (uintptr_t)sum_out | (uintptr_t)y;
    if (all % 16 != 0) {
        set_error_text("tmw_add_rmsnorm: every pointer must be 16-byte aligned");
        return TMW_ERR_INVALID_ARGUMENT;
    }
    if (rows == 0) return TMW_OK;
    return launch_add_rmsnorm(dtype, rows, dim, x, residual, scale, eps, sum_out, y, static_cast<cudaStream_t>(stream));
}
