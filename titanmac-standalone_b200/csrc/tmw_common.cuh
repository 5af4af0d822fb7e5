// Shared declarations of libtmw's translation units (internal; the public ABI is
// include/tmw.h).
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <mutex>
#include <utility>

#include "tmw.h"

namespace tmw {

// ---- element conversion ---------------------------------------------------------
template <typename T>
__device__ __forceinline__ float to_f32(T x);
template <>
__device__ __forceinline__ float to_f32<float>(float x) { return x; }
template <>
__device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 x) { return __bfloat162float(x); }
template <>
__device__ __forceinline__ float to_f32<__half>(__half x) { return __half2float(x); }

template <typename T>
__device__ __forceinline__ T from_f32(float x);
template <>
__device__ __forceinline__ float from_f32<float>(float x) { return x; }
template <>
__device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float x) { return __float2bfloat16_rn(x); }
template <>
__device__ __forceinline__ __half from_f32<__half>(float x) { return __float2half_rn(x); }

// Loads 8 consecutive elements (16 B for 16-bit types, 32 B for float) as floats.
template <typename T>
__device__ __forceinline__ void load8(const T* p, float (&out)[8]);
template <>
__device__ __forceinline__ void load8<float>(const float* p, float (&out)[8]) {
    const float4 a = *reinterpret_cast<const float4*>(p);
    const float4 b = *reinterpret_cast<const float4*>(p + 4);
    out[0] = a.x; out[1] = a.y; out[2] = a.z; out[3] = a.w;
    out[4] = b.x; out[5] = b.y; out[6] = b.z; out[7] = b.w;
}
template <>
__device__ __forceinline__ void load8<__nv_bfloat16>(const __nv_bfloat16* p, float (&out)[8]) {
    const uint4 raw = *reinterpret_cast<const uint4*>(p);
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        out[2 * i] = __uint_as_float(w[i] << 16);
        out[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
}
template <>
__device__ __forceinline__ void load8<__half>(const __half* p, float (&out)[8]) {
    const uint4 raw = *reinterpret_cast<const uint4*>(p);
    const __half2* h = reinterpret_cast<const __half2*>(&raw);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 f = __half22float2(h[i]);
        out[2 * i] = f.x;
        out[2 * i + 1] = f.y;
    }
}

template <typename T>
__device__ __forceinline__ void store8(T* p, const float (&in)[8]);
template <>
__device__ __forceinline__ void store8<float>(float* p, const float (&in)[8]) {
    *reinterpret_cast<float4*>(p) = make_float4(in[0], in[1], in[2], in[3]);
    *reinterpret_cast<float4*>(p + 4) = make_float4(in[4], in[5], in[6], in[7]);
}
template <>
__device__ __forceinline__ void store8<__nv_bfloat16>(__nv_bfloat16* p, const float (&in)[8]) {
    uint4 raw;
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&raw);
#pragma unroll
    for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(in[2 * i], in[2 * i + 1]);
    *reinterpret_cast<uint4*>(p) = raw;
}
template <>
__device__ __forceinline__ void store8<__half>(__half* p, const float (&in)[8]) {
    uint4 raw;
    __half2* h = reinterpret_cast<__half2*>(&raw);
#pragma unroll
    for (int i = 0; i < 4; ++i) h[i] = __floats2half2_rn(in[2 * i], in[2 * i + 1]);
    *reinterpret_cast<uint4*>(p) = raw;
}

// Exact (erf-based) GELU, 0.5 x (1 + erf(x / sqrt 2)), with erf from the rational approximation 7.1.26 of
// Abramowitz & Stegun (absolute error below 1.5e-7, i.e. fp32 rounding noise against a 16-bit result): with z = |x| / sqrt 2
// and t = 1 / (1 + 0.3275911 z), erf(z) = 1 - Q(t) t exp(-z^2).  In the product's epilogue this is the longest part, so the
// result is put together from 1 - erf, max(x, 0) - |x| / 2 (1 - erf), and the reciprocal (of 1 or more) and the exponential
// (zero below 2^-126) take the forms without the care for subnormal numbers: 16416 x 2560 x 640 with GELU, 87 -> 75 us.
__device__ __forceinline__ float rcp_ftz(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float ex2_ftz(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// Q(t) t / 2 and exp(-x^2 / 2)
__device__ __forceinline__ float half_erfc_poly(float x) {
    const float t = rcp_ftz(fmaf(0.3275911f * 0.70710678118654752f, fabsf(x), 1.0f));
    float poly = fmaf(0.5f * 1.061405429f, t, 0.5f * -1.453152027f);
    poly = fmaf(poly, t, 0.5f * 1.421413741f);
    poly = fmaf(poly, t, 0.5f * -0.284496736f);
    poly = fmaf(poly, t, 0.5f * 0.254829592f);
    return poly * t;
}
__device__ __forceinline__ float gauss(float x) { return ex2_ftz(x * -0.72134752044448170f * x); }
__device__ __forceinline__ float gelu_erf(float x) {
    // (beyond 16 the exponential is zero: the bound keeps infinity times zero out)
    return fmaf(-fminf(fabsf(x), 16.0f) * half_erfc_poly(x), gauss(x), fmaxf(x, 0.0f));
}

// derivative of gelu_erf: Phi(x) + x phi(x)
__device__ __forceinline__ float gelu_slope(float x) {
    const float odd = fmaf(0.3989422804014327f, x, -copysignf(half_erfc_poly(x), x));
    return fmaf(gauss(x), odd, x > 0.0f ? 1.0f : 0.0f);
}

__host__ __device__ inline size_t dtype_size(int dtype) { return dtype == TMW_F32 ? 4 : 2; }

// Eight consecutive elements as raw bits: half the registers of their fp32 values for 16-bit types.
template <typename T>
struct Vec8 {
    uint4 raw[sizeof(T) / 2];
    __device__ __forceinline__ void load(const T* p) {
#pragma unroll
        for (int i = 0; i < (int)sizeof(T) / 2; ++i) raw[i] = reinterpret_cast<const uint4*>(p)[i];
    }
    __device__ __forceinline__ void unpack(float (&out)[8]) const { load8<T>(reinterpret_cast<const T*>(raw), out); }
};

// Position of the first sequence key that the sequence query at position `pos` (>= np) sees.
// block == 0: the query and its `window` predecessors (WindowedAttention, windowed_attention.py:136-150).
// block  > 0: the left edge moves in steps of `block` rows - the query in block b of the sequence sees the
//             keys from b * block - window on (BlockSparseAttention, block_sparse_attention.py:299-311).
__host__ __device__ inline int first_visible_pos(int pos, int np, int window, int block) {
    if (block > 0) {
        const int lo = ((pos - np) / block) * block - window;
        return np + (lo > 0 ? lo : 0);
    }
    const int lo = pos - window;
    return lo > np ? lo : np;
}

// d += a b for one 16 x 8 x 16 tile (mma.sync: tiles of a few rows, which tcgen05's 64 or 128 would waste)
template <typename T>
__device__ __forceinline__ void mma_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                          uint32_t b1);
template <>
__device__ __forceinline__ void mma_16816<__nv_bfloat16>(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                                         uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
template <>
__device__ __forceinline__ void mma_16816<__half>(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                                  uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// ---- host-side plumbing shared by the entry points ---------------------------------
void set_cuda_error(cudaError_t e, const char* where);
void set_error_text(const char* text);
int* device_status_word();  // per-device int in global memory, 0 = fine
// opt-in of a kernel to `bytes` of dynamic shared memory, made once per kernel and device
int allow_shared_memory(const void* kern, int bytes);

// a library-owned stream for work that may overlap the caller's stream, with the events of the fork / join
struct SideStream {
    cudaStream_t stream = nullptr;
    cudaEvent_t fork = nullptr, join = nullptr;
    std::mutex mutex;
};
SideStream* side_stream_of_current_device();  // nullptr if it cannot be made

// ---- programmatic dependent launch ---------------------------------------------------
// A chain of small kernels spends more time on launch, drain and cold loads than on work.  A kernel of such a chain
// triggers the launch of its successor at once (launching takes about 2.5 us), loads what no kernel of the chain writes
// (weights, cache rows) and then waits until its predecessor has finished - which has waited for its own.  The first
// kernel of a chain is an ordinary launch: what the stream held before is complete when the chain starts.
// Without the launch attribute both calls are no-ops.
// What another kernel of the chain writes must not be read through a `const __restrict__` pointer: the compiler takes such
// loads for invariant and moves them in front of pdl_wait().
// A kernel that stores through TMA has to see its stores complete, not just read, before it ends if a dependent follows:
// what it leaves in flight an ordinary launch waits for, pdl_wait() does not.
// A launch's place in a chain (0: none).  Products store from registers: kChainFollowed matters to the attention core alone.
enum : int { kChainDependent = 1, kChainFollowed = 2, kChainLink = 3 };
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// launch with the dependent-launch attribute and / or a cluster of `cluster` CTAs along x
template <typename... P, typename... A>
cudaError_t launch_ex(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, bool pdl, int cluster,
                      A&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (pdl) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (cluster > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = cluster;
        attr[n].val.clusterDim.y = 1;
        attr[n++].val.clusterDim.z = 1;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    return cudaLaunchKernelEx(&cfg, kern, std::forward<A>(args)...);
}

int sm_count();  // of the current device, asked once per device

#define TMW_CUDA_TRY(expr)                                   \
    do {                                                     \
        cudaError_t _e = (expr);                             \
        if (_e != cudaSuccess) {                             \
            ::tmw::set_cuda_error(_e, #expr);                \
            return TMW_ERR_CUDA;                             \
        }                                                    \
    } while (0)

// Argument checks shared by the decode entry points (defined with the entry points in api.cu).
int validate_decode_call(const tmw_cache_desc* cache, const void* q, const void* k_new, const void* v_new,
                         const void* o, const int64_t q_stride[2], const int64_t kv_new_stride[2],
                         const int64_t o_stride[2], const int32_t* pos);

// Kernel launchers (one per translation unit).
// window_block: 0 = per-token window, > 0 = block-granular left edge (see first_visible_pos);
// all_keys: every query row of the call sees every key, unmasked (the persistent rows of the block-sparse class)
// lse (optional): [batch, heads, q_rows] fp32, log2 of every row's softmax denominator in the domain of
// score * scale * log2(e) - what the backward pass needs to rebuild the probabilities
int launch_prefill_simt(const tmw_prefill_desc& d, const void* q, const void* k, const void* v, void* o,
                        cudaStream_t stream, int window_block = 0, bool all_keys = false, float* lse = nullptr);
// fp32, head_dim 64 / 128: register-tiled kernel (prefill_fp32.cu), which launch_prefill_simt hands those calls to
bool prefill_fp32_supports(const tmw_prefill_desc& d);
int launch_prefill_fp32(const tmw_prefill_desc& d, const void* q, const void* k, const void* v, void* o, cudaStream_t stream,
                        int window_block, bool all_keys, float* lse);
int launch_prefill_tc(const tmw_prefill_desc& d, const void* q, const void* k, const void* v, void* o,
                      cudaStream_t stream, int window_block = 0, float* lse = nullptr, const tmw_halo_wait* wait = nullptr,
                      int chain = 0);
// the query rows of the call see every key row, unmasked (16-bit types, head_dim 64 / 128): see pers_rows.cu
int launch_pers_rows(const tmw_prefill_desc& d, const void* q, const void* k, const void* v, void* o, float* lse,
                     cudaStream_t stream, bool pdl);
// window_block / pers_global select the mask of the block-sparse class (see first_visible_pos; pers_global: the
// persistent query rows see every key, and lse comes as [batch, heads, rows - np] followed by [batch, heads, np])
int launch_prefill_backward(const tmw_prefill_desc& d, const void* q, const void* k, const void* v, const void* o,
                            const void* d_o, const float* lse, void* dq, void* dk, void* dv, cudaStream_t stream,
                            int window_block = 0, bool pers_global = false);
// the same on the warp-level tensor-core path (16-bit types, head_dim 64 / 128)
bool prefill_backward_mma_supports(const tmw_prefill_desc& d);
int launch_prefill_backward_mma(const tmw_prefill_desc& d, const void* q, const void* k, const void* v, const void* o,
                                const void* d_o, const float* lse, void* dq, void* dk, void* dv, cudaStream_t stream,
                                int window_block = 0, bool pers_global = false);
// the same on tcgen05 (16-bit types, head_dim 64 / 128); window_block > 0: the block-sparse class's mask with its
// persistent query rows seeing every key and lse in two planes
bool prefill_backward_tc_supports(const tmw_prefill_desc& d);
int launch_prefill_backward_tc(const tmw_prefill_desc& d, const void* q, const void* k, const void* v, const void* o,
                               const void* d_o, const float* lse, void* dq, void* dk, void* dv, cudaStream_t stream,
                               int window_block = 0);
int launch_dwconv_backward(int dtype, int batch, int rows, int channels, int taps, const void* x, const void* const* w, int n_w,
                           const void* dy, void* dx, float* dw, cudaStream_t stream);
// x = embedded rows (persistent rows first), y = RMSNorm(x): see stack_forward.cu
int launch_embed_seq(const tmw_stack_desc& d, const int64_t* token_ids, int tokens, const void* gain, void* x, void* y,
                     cudaStream_t stream);
// tmw_prefill_block_sparse_lse as links of a chain of dependent launches
int prefill_block_sparse(const tmw_prefill_desc* desc, int block_size, const void* q, const void* k, const void* v, void* o,
                         float* lse, cudaStream_t s, int chain);
bool prefill_tc_supports(const tmw_prefill_desc& d, const void* q, const void* k, const void* v, const void* o);
int launch_decode(const tmw_cache_desc& c, const void* q, const void* k_new, const void* v_new, void* o,
                  const int64_t qs[2], const int64_t ns[2], const int64_t os[2], const int32_t* pos,
                  int splits, float* scratch, unsigned int* counters, cudaStream_t stream, bool pdl = false);
int decode_step_splits(const tmw_cache_desc& c);
// A decode step as one kernel (decode_resident.cu).  decode_resident_begin once, then steps 0, 1, ... in a row: `choose`: a step
// leaves what its greedy choice needs, and a step behind it takes its tokens from there (and writes them to out), at the
// positions pos + step; launch_decode_choice settles the last one.  TMW_ERR_UNSUPPORTED: the device cannot hold the kernel.
bool decode_step_is_resident(const tmw_stack_desc& d, const tmw_block* blocks);
size_t decode_resident_workspace(const tmw_stack_desc& d);
int decode_resident_begin(const tmw_stack_desc& d, void* workspace, cudaStream_t stream);
int launch_decode_resident(const tmw_stack_desc& d, const tmw_block* blocks, const int64_t* ids, const int32_t* pos, void* logits,
                           int step, bool choose, int64_t* out, int64_t out_stride, void* workspace, cudaStream_t stream);
int launch_decode_choice(const tmw_stack_desc& d, int steps, int64_t* tokens, int64_t* out, int64_t out_stride, int32_t* pos,
                         void* workspace, cudaStream_t stream);

// layout of the split-decode scratch memory: partial results, then (16-byte aligned) one counter per pair
inline size_t decode_partials_bytes(int batch, int heads, int head_dim, int splits) {
    const size_t n = (size_t)batch * heads * splits * ((size_t)head_dim + 2) * sizeof(float);
    return (n + 15) & ~(size_t)15;
}
// c[m, n] = epilogue(sum_k a(m, k) b(n, k)): a is [m, k] row-major, or [k, m] with a_mn; b is [n, k], or [k, n] with b_mn
// (a_mn needs b_mn)
enum GemmEpilogue {
    GEMM_NONE = 0,
    GEMM_GELU = 1,       // gelu(v)
    GEMM_ADD = 2,        // aux + round(v)
    GEMM_GELU_KEEP = 3,  // aux = round(v), c = gelu(aux)
    GEMM_GELU_GRAD = 4   // v * gelu'(aux)
};
struct GemmCall {
    int dtype = 0, m = 0, n = 0, k = 0;
    const void *a = nullptr, *b = nullptr, *bias = nullptr;
    void *c = nullptr, *aux = nullptr;  // aux: [m, n] contiguous
    long long lda = 0, ldb = 0, ldc = 0;
    bool a_mn = false, b_mn = false;
    int epilogue = GEMM_NONE, chain = 0;
    int splits = 1;
    float* partial = nullptr;
};
int launch_gemm_call(const GemmCall& g, cudaStream_t stream);
int gemm_most_splits(int k);  // into how many ranges launch_gemm_splitk cuts a k at most
int launch_gemm_splitk(const GemmCall& g, size_t partial_bytes, int* splits, cudaStream_t stream);
int launch_linear(const tmw_linear_desc& d, const void* a, const void* w, const void* bias, void* c,
                  cudaStream_t stream, int chain = 0);
int launch_add_rmsnorm(int dtype, long long rows, int dim, const void* x, const void* residual, const void* scale, float eps,
                       void* sum_out, void* y, cudaStream_t stream, bool pdl = false);
// w: the filters of channels [0, c/n), [c/n, 2c/n), ... in n arrays [c/n, taps]
int launch_dwconv(int dtype, int batch, int rows, int channels, int taps, const void* x, const void* const* w, int n_w, void* y,
                  cudaStream_t stream, bool pdl = false);
// links of a chain of dependent launches (see pdl_wait): a product of up to a few hundred rows (epi: 0 = store, 1 = GELU,
// 2 = added to c, which is read and written; n and k multiples of 8, contiguous rows), and the RMSNorm in front of it
int launch_rows_tc(int dtype, int m, int n, int k, const void* a, const void* w, const void* bias, void* c, int epi,
                   cudaStream_t stream, bool pdl);
int launch_rows_norm(int dtype, int rows, int dim, const void* x, const void* gain, float eps, void* y, cudaStream_t stream);
// pers_k / pers_v (optional): rows [0, n_persistent) of the first sequence at these addresses go into k_pers / v_pers
int launch_cache_fill(const tmw_cache_desc& c, const void* k, const void* v, const int64_t ks[3],
                      const int64_t vs[3], int rows, int t0, cudaStream_t stream, const void* pers_k = nullptr,
                      const void* pers_v = nullptr, bool pdl = false);

}  // namespace tmw
