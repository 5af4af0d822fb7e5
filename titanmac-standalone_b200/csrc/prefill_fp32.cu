// Sliding-window attention in fp32 for head_dim 64 and 128, forward: register-tiled multiply-adds on CUDA cores.
//
// The fp32 contract (max-abs 1e-5 against the reference) leaves the tensor cores out, so the multiply-add pipe is the bound.
// A kernel that gives every query row to a lane (prefill_simt.cu) reads a key element from shared memory for each of its
// multiply-adds.  Here a thread owns 4 x 4 scores and 4 x (head_dim / 16) outputs: eight 16-byte reads feed 64 multiply-adds.
// A CTA owns 32 query rows of one (batch, head) and has two groups of 128 threads, which take 64-key tiles in turn and keep
// softmax states of their own, merged at the end: short sequences leave few CTAs, and each must hold enough warps to hide
// its latencies.  Within a group K of the next tile arrives (cp.async) under P V, and V under Q K.
// Measured, us, 16 heads x 528 rows of 64, window 256: 69.8 with a row per lane, 30.4 here.
#include <math_constants.h>

#include "tmw_common.cuh"

namespace tmw {
namespace {

constexpr int FR = 32;        // query rows per CTA
constexpr int FK = 64;        // keys per tile
constexpr int kGroups = 2;    // groups of 128 threads
constexpr int kF32Threads = 128 * kGroups;

template <int DH>
struct F32Smem {
    static constexpr int kRow = DH + 4;   // floats per row of Q, K, V: rows of a quarter warp's keys in different banks
    static constexpr int kPRow = FK + 4;
    static constexpr int kQ = FR * kRow, kK = FK * kRow, kP = FR * kPRow;
    static constexpr int kGroup = 2 * kK + kP;
    static constexpr int kBytes = (kQ + kGroups * kGroup) * 4;
    static_assert(FR * DH + 2 * FR <= kGroup, "a group's result for the merge takes the place of its tiles");
};

struct F32Params {
    const float *q, *k, *v;
    float *o, *lse;  // lse optional: [batch, heads, q_rows], m + log2(l) of every row
    long long qs[3], ks[3], vs[3], os[3];
    int q_rows, k_rows, window, np, q_pos0, k_pos0, block, all_keys;
    float scale_log2;
};

__device__ __forceinline__ void cp_async16(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

template <int DH>
__global__ void __launch_bounds__(kF32Threads) prefill_fp32_kernel(const F32Params p) {
    using L = F32Smem<DH>;
    constexpr int DC = DH / 64;  // float4 columns of the output per thread
    extern __shared__ __align__(16) float f32_smem[];
    const int tid = threadIdx.x & 127, group = threadIdx.x >> 7;
    const int tx = tid & 15, ty = tid >> 4;  // rows ty * 4 + i; keys tx + 16 j; output columns (c * 16 + tx) * 4
    float* qs = f32_smem;
    float* ks = f32_smem + L::kQ + group * L::kGroup;
    float* vs = ks + L::kK;
    float* ps = vs + L::kK;
    const int r0 = blockIdx.x * FR, head = blockIdx.y, batch = blockIdx.z;
    const float* qg = p.q + batch * p.qs[0] + head * p.qs[1];
    const float* kg = p.k + batch * p.ks[0] + head * p.ks[1];
    const float* vg = p.v + batch * p.vs[0] + head * p.vs[1];
    auto group_sync = [&] { asm volatile("bar.sync %0, 128;" ::"r"(1 + group) : "memory"); };

    // the keys this CTA can need: virtual index u in [0, np) persistent, then the window's positions [glo, ghi]
    const int p_first = p.q_pos0 + r0, p_last = p.q_pos0 + min(r0 + FR, p.q_rows) - 1;
    const int glo = p.all_keys ? p.k_pos0 : first_visible_pos(max(p_first, p.np), p.np, p.window, p.block);
    const int ghi = p.all_keys ? p.k_pos0 + (p.k_rows - p.np) - 1 : p_last;
    const int n_win = (p.all_keys || p_last >= p.np) && ghi >= glo ? ghi - glo + 1 : 0;
    const int n_keys = p.np + n_win, n_tiles = (n_keys + FK - 1) / FK;
    int u_lo[4], u_hi[4];  // the window keys row i sees, as virtual indices [u_lo, u_hi] (beside the persistent ones)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int pos = p_first + ty * 4 + i;
        u_lo[i] = 1 << 30;
        u_hi[i] = -1;
        if (p.all_keys) {
            u_lo[i] = p.np;
            u_hi[i] = n_keys - 1;
        } else if (pos >= p.np) {
            u_lo[i] = p.np + first_visible_pos(pos, p.np, p.window, p.block) - glo;
            u_hi[i] = min(p.np + pos - glo, n_keys - 1);
        }
    }
    auto load_tile = [&](float* dst, const float* src, long long stride, int tile) {
#pragma unroll
        for (int i = 0; i < FK * DH / 4 / 128; ++i) {
            const int idx = i * 128 + tid, j = idx / (DH / 4), d4 = idx % (DH / 4);
            const int u = min(tile * FK + j, n_keys - 1);  // (rows beyond the last key are masked)
            const int row = min(max(u < p.np ? u : u + glo - p.k_pos0, 0), p.k_rows - 1);
            cp_async16(dst + j * L::kRow + d4 * 4, src + (long long)row * stride + d4 * 4);
        }
        cp_async_commit();
    };
    for (int idx = threadIdx.x; idx < FR * DH / 4; idx += kF32Threads) {
        const int r = idx / (DH / 4), d4 = idx % (DH / 4);
        cp_async16(qs + r * L::kRow + d4 * 4, qg + (long long)min(r0 + r, p.q_rows - 1) * p.qs[2] + d4 * 4);
    }
    cp_async_commit();
    if (group < n_tiles) load_tile(ks, kg, p.ks[2], group);
    cp_async_wait<0>();
    __syncthreads();  // Q is there for both groups

    float m[4], l[4], acc[4][DC][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        m[i] = -CUDART_INF_F;
        l[i] = 0.f;
#pragma unroll
        for (int c = 0; c < DC; ++c)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[i][c][e] = 0.f;
    }
    for (int tile = group; tile < n_tiles; tile += kGroups) {
        load_tile(vs, vg, p.vs[2], tile);
        cp_async_wait<1>();  // K
        group_sync();
        float s[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
#pragma unroll 4
        for (int d = 0; d < DH; d += 4) {
            float4 a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const float4*>(qs + (ty * 4 + i) * L::kRow + d);
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const float4*>(ks + (tx + 16 * j) * L::kRow + d);
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    s[i][j] = fmaf(a[i].x, b[j].x, s[i][j]);
                    s[i][j] = fmaf(a[i].y, b[j].y, s[i][j]);
                    s[i][j] = fmaf(a[i].z, b[j].z, s[i][j]);
                    s[i][j] = fmaf(a[i].w, b[j].w, s[i][j]);
                }
        }
        group_sync();  // K has been read
        if (tile + kGroups < n_tiles) load_tile(ks, kg, p.ks[2], tile + kGroups);
        else cp_async_commit();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float mx = m[i];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int u = tile * FK + tx + 16 * j;
                const bool vis = u < p.np || (u >= u_lo[i] && u <= u_hi[i]);
                s[i][j] = vis ? s[i][j] * p.scale_log2 : -CUDART_INF_F;
                mx = fmaxf(mx, s[i][j]);
            }
#pragma unroll
            for (int o = 1; o < 16; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            const float safe = mx > -CUDART_INF_F ? mx : 0.f;
            const float alpha = exp2f(m[i] - safe);  // m = -inf gives 0
            m[i] = mx;
            l[i] *= alpha;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float e = exp2f(s[i][j] - safe);
                l[i] += e;
                ps[(ty * 4 + i) * L::kPRow + tx + 16 * j] = e;
            }
#pragma unroll
            for (int c = 0; c < DC; ++c)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[i][c][e] *= alpha;
        }
        cp_async_wait<1>();  // V (the next K may still be on its way)
        group_sync();
#pragma unroll 4
        for (int j = 0; j < FK; j += 4) {
            float4 a[4], b[4][DC];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const float4*>(ps + (ty * 4 + i) * L::kPRow + j);
#pragma unroll
            for (int jj = 0; jj < 4; ++jj)
#pragma unroll
                for (int c = 0; c < DC; ++c)
                    b[jj][c] = *reinterpret_cast<const float4*>(vs + (j + jj) * L::kRow + (c * 16 + tx) * 4);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float w[4] = {a[i].x, a[i].y, a[i].z, a[i].w};
#pragma unroll
                for (int jj = 0; jj < 4; ++jj)
#pragma unroll
                    for (int c = 0; c < DC; ++c) {
                        acc[i][c][0] = fmaf(w[jj], b[jj][c].x, acc[i][c][0]);
                        acc[i][c][1] = fmaf(w[jj], b[jj][c].y, acc[i][c][1]);
                        acc[i][c][2] = fmaf(w[jj], b[jj][c].z, acc[i][c][2]);
                        acc[i][c][3] = fmaf(w[jj], b[jj][c].w, acc[i][c][3]);
                    }
            }
        }
        group_sync();  // V and P have been read
    }
    cp_async_wait<0>();
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int o = 1; o < 16; o <<= 1) l[i] += __shfl_xor_sync(0xffffffffu, l[i], o);
    __syncthreads();
    // the second group hands its state over through its own tiles' memory
    float* other = f32_smem + L::kQ + L::kGroup;
    if (group == 1) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = ty * 4 + i;
#pragma unroll
            for (int c = 0; c < DC; ++c)
                *reinterpret_cast<float4*>(other + r * DH + (c * 16 + tx) * 4) = make_float4(acc[i][c][0], acc[i][c][1], acc[i][c][2], acc[i][c][3]);
            if (tx == 0) {
                other[FR * DH + r] = m[i];
                other[FR * DH + FR + r] = l[i];
            }
        }
    }
    __syncthreads();
    if (group == 0) {
        float* og = p.o + batch * p.os[0] + head * p.os[1];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = ty * 4 + i;
            if (r0 + r >= p.q_rows) continue;
            const float m2 = other[FR * DH + r], l2 = other[FR * DH + FR + r];
            const float ma = fmaxf(m[i], m2), safe = ma > -CUDART_INF_F ? ma : 0.f;
            const float f1 = exp2f(m[i] - safe), f2 = exp2f(m2 - safe);
            const float la = l[i] * f1 + l2 * f2, inv = la > 0.f ? 1.f / la : 0.f;
#pragma unroll
            for (int c = 0; c < DC; ++c) {
                const float4 b = *reinterpret_cast<const float4*>(other + r * DH + (c * 16 + tx) * 4);
                *reinterpret_cast<float4*>(og + (long long)(r0 + r) * p.os[2] + (c * 16 + tx) * 4) =
                    make_float4((acc[i][c][0] * f1 + b.x * f2) * inv, (acc[i][c][1] * f1 + b.y * f2) * inv,
                                (acc[i][c][2] * f1 + b.z * f2) * inv, (acc[i][c][3] * f1 + b.w * f2) * inv);
            }
            if (tx == 0 && p.lse != nullptr) p.lse[((long long)batch * gridDim.y + head) * p.q_rows + r0 + r] = ma + log2f(la);
        }
    }
}

}  // namespace

bool prefill_fp32_supports(const tmw_prefill_desc& d) { return d.dtype == TMW_F32 && (d.head_dim == 64 || d.head_dim == 128); }

int launch_prefill_fp32(const tmw_prefill_desc& d, const void* q, const void* k, const void* v, void* o, cudaStream_t stream,
                        int window_block, bool all_keys, float* lse) {
    F32Params p;
    p.q = static_cast<const float*>(q); p.k = static_cast<const float*>(k); p.v = static_cast<const float*>(v);
    p.o = static_cast<float*>(o); p.lse = lse;
    for (int i = 0; i < 3; ++i) {
        p.qs[i] = d.q_stride[i]; p.ks[i] = d.k_stride[i]; p.vs[i] = d.v_stride[i]; p.os[i] = d.o_stride[i];
    }
    p.q_rows = d.q_rows; p.k_rows = d.k_rows; p.window = d.window; p.np = d.n_persistent;
    p.q_pos0 = d.q_pos0; p.k_pos0 = d.k_pos0; p.block = window_block; p.all_keys = all_keys ? 1 : 0;
    p.scale_log2 = (d.scale != 0.f ? d.scale : 1.0f / sqrtf((float)d.head_dim)) * 1.4426950408889634f;
    if (d.q_rows == 0 || d.batch == 0 || d.heads == 0) return TMW_OK;
    const dim3 grid((d.q_rows + FR - 1) / FR, d.heads, d.batch);
    auto run = [&](auto kern, int smem) -> int {
        const int rc = allow_shared_memory(reinterpret_cast<const void*>(kern), smem);
        if (rc != TMW_OK) return rc;
        kern<<<grid, kF32Threads, smem, stream>>>(p);
        TMW_CUDA_TRY(cudaGetLastError());
        return TMW_OK;
    };
    return d.head_dim == 64 ? run(prefill_fp32_kernel<64>, F32Smem<64>::kBytes) : run(prefill_fp32_kernel<128>, F32Smem<128>::kBytes);
}

}  // namespace tmw
