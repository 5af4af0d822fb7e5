// Attention of a few query rows over every key row, unmasked: the persistent rows of the block-sparse class
// (block_sparse_attention.py:283-291).  16-bit types, head_dim 64 or 128.
//
// Sixteen rows are one mma.sync tile and an eighth of a tcgen05 tile, and what they need - one pass over all keys and values
// of a (batch, head) - is a matter of bytes in flight: a cluster of up to eight CTAs shares a (batch, head, 16 rows), every
// warp walks over blocks of 32 (head_dim 128: 16) keys with its own running maximum, and the partial results are merged through shared memory
// and the cluster's.  As a query tile of 128 rows in the tcgen05 kernel the same rows walked 2747 keys one tile after the
// other, 37 us on a side stream of its own beside 35 us for all other rows.
// V of a warp's next block loads under this one, K does not: at head_dim 64 the second block of K takes 168 registers instead of 126,
// three CTAs to an SM instead of four, and these leave the attention behind no room to start.  Block-sparse layers of 10 heads, us, K
// ahead | not: 5 x 1400 rows, window 300 74.6 | 71.3; 5 x 2747, window 512 130.6 | 124.9; 1 x 316 30.0 | 30.3; 3 x 2747 89.7 | 89.7.
#include <math_constants.h>

#include "tmw_common.cuh"

namespace tmw {
namespace {

constexpr int kPersWarps = 4;
__host__ __device__ constexpr int pers_keys(int dh) { return dh == 64 ? 32 : 16; }  // keys per block of a warp

struct PersParams {
    const void *q, *k, *v;
    void* o;
    float* lse;  // [batch, heads, q_rows] or nullptr
    long long qs[3], ks[3], vs[3], os[3];
    int q_rows, k_rows, cluster;
    float scale_log2;
};

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
template <typename T>
__device__ __forceinline__ uint32_t pack16(float a, float b) {
    T h[2] = {from_f32<T>(a), from_f32<T>(b)};
    return *reinterpret_cast<const uint32_t*>(h);
}

template <typename T, int DH>
__global__ void __launch_bounds__(kPersWarps * 32) pers_rows_kernel(const PersParams p) {
    constexpr int KEYS = pers_keys(DH), KN = KEYS / 8;  // keys per block, in groups of 8
    constexpr int KC = DH / 32, NT = DH / 8;            // 32-wide chunks of head_dim; 8-wide output columns
    constexpr int ROWB = DH * 2 + 16;         // bytes per V row in shared memory (padding: no bank conflicts of ldmatrix)
    __shared__ __align__(16) uint8_t v_tile[kPersWarps][2][KEYS * ROWB];
    __shared__ float part[16][DH + 2];        // this CTA's merged result: accumulator, maximum, sum
    __shared__ float w_m[kPersWarps][16], w_l[kPersWarps][16];
    pdl_trigger();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const int cs = p.cluster, rank = blockIdx.x % cs, row0 = blockIdx.x / cs * 16, head = blockIdx.y, batch = blockIdx.z;
    const T* q = static_cast<const T*>(p.q) + batch * p.qs[0] + head * p.qs[1];
    const T* k = static_cast<const T*>(p.k) + batch * p.ks[0] + head * p.ks[1];
    const T* v = static_cast<const T*>(p.v) + batch * p.vs[0] + head * p.vs[1];
    const int blocks = (p.k_rows + KEYS - 1) / KEYS, first = rank * kPersWarps + warp, step = cs * kPersWarps;
    pdl_wait();

    // Q as mma fragments: of every 32 elements of head_dim a thread of a quad takes eight adjacent ones, the same for Q and K
    uint4 qa[KC][2];
#pragma unroll
    for (int c = 0; c < KC; ++c)
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
            const int r = min(row0 + hh * 8 + g, p.q_rows - 1);  // (rows that do not exist are not stored)
            qa[c][hh] = *reinterpret_cast<const uint4*>(q + r * p.qs[2] + c * 32 + t * 8);
        }
    auto fetch_v = [&](int block, int buf) {  // rows beyond the last: the last (their probabilities are zero)
        uint8_t* dst = v_tile[warp][buf];
#pragma unroll
        for (int i = 0; i < KEYS * DH / 8 / 32; ++i) {
            const int idx = i * 32 + lane, row = idx / (DH / 8), col = idx % (DH / 8);
            cp_async16(smem_addr(dst + row * ROWB + col * 16), v + min(block * KEYS + row, p.k_rows - 1) * p.vs[2] + col * 8);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    float m[2] = {-CUDART_INF_F, -CUDART_INF_F}, l[2] = {0.f, 0.f}, acc[NT][4];
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[n][e] = 0.f;
    if (first < blocks) fetch_v(first, 0);
    int buf = 0;
    for (int b = first; b < blocks; b += step, buf ^= 1) {
        uint4 kb[KN][KC];
#pragma unroll
        for (int n = 0; n < KN; ++n)
#pragma unroll
            for (int c = 0; c < KC; ++c)
                kb[n][c] = *reinterpret_cast<const uint4*>(k + min(b * KEYS + n * 8 + g, p.k_rows - 1) * p.ks[2] + c * 32 + t * 8);
        if (b + step < blocks) fetch_v(b + step, buf ^ 1);
        float s[KN][4], mx[2] = {m[0], m[1]};
#pragma unroll
        for (int n = 0; n < KN; ++n) {
#pragma unroll
            for (int e = 0; e < 4; ++e) s[n][e] = 0.f;
#pragma unroll
            for (int c = 0; c < KC; ++c) {
                mma_16816<T>(s[n], qa[c][0].x, qa[c][1].x, qa[c][0].y, qa[c][1].y, kb[n][c].x, kb[n][c].y);
                mma_16816<T>(s[n], qa[c][0].z, qa[c][1].z, qa[c][0].w, qa[c][1].w, kb[n][c].z, kb[n][c].w);
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int key = b * KEYS + n * 8 + 2 * t + (e & 1);
                s[n][e] = key < p.k_rows ? s[n][e] * p.scale_log2 : -CUDART_INF_F;
                mx[e >> 1] = fmaxf(mx[e >> 1], s[n][e]);
            }
        }
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
            mx[hh] = fmaxf(mx[hh], __shfl_xor_sync(0xffffffffu, mx[hh], 1));
            mx[hh] = fmaxf(mx[hh], __shfl_xor_sync(0xffffffffu, mx[hh], 2));
            const float alpha = ex2(m[hh] - mx[hh]);  // (a block holds a key that exists: mx is finite)
            m[hh] = mx[hh];
            l[hh] *= alpha;
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                acc[n][2 * hh] *= alpha;
                acc[n][2 * hh + 1] *= alpha;
            }
        }
        uint32_t pa[KN][2];  // P as A fragments: [8 keys][row g | row g + 8]
#pragma unroll
        for (int n = 0; n < KN; ++n) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                s[n][e] = ex2(s[n][e] - m[e >> 1]);
                l[e >> 1] += s[n][e];
            }
            pa[n][0] = pack16<T>(s[n][0], s[n][1]);
            pa[n][1] = pack16<T>(s[n][2], s[n][3]);
        }
        if (b + step < blocks) asm volatile("cp.async.wait_group 1;" ::: "memory");
        else asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncwarp();
        const uint32_t vt = smem_addr(v_tile[warp][buf]);
#pragma unroll
        for (int kk = 0; kk < KEYS / 16; ++kk)  // 16 keys each
#pragma unroll
            for (int n = 0; n < NT; n += 2) {
                // four 8 x 8 blocks, transposed: keys 0-7 | 8-15 of columns n and n + 1
                uint32_t r[4];
                const uint32_t a = vt + (kk * 16 + (lane & 15)) * ROWB + (n + (lane >> 4)) * 16;
                asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                             : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
                mma_16816<T>(acc[n], pa[2 * kk][0], pa[2 * kk][1], pa[2 * kk + 1][0], pa[2 * kk + 1][1], r[0], r[1]);
                mma_16816<T>(acc[n + 1], pa[2 * kk][0], pa[2 * kk][1], pa[2 * kk + 1][0], pa[2 * kk + 1][1], r[2], r[3]);
            }
        __syncwarp();  // everybody has read the tile that is filled next
    }
    // ---- merge: the quad's sums, then the warps of the CTA one after the other, then the CTAs of the cluster ----
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
        l[hh] += __shfl_xor_sync(0xffffffffu, l[hh], 1);
        l[hh] += __shfl_xor_sync(0xffffffffu, l[hh], 2);
        if (t == 0) {
            w_m[warp][hh * 8 + g] = m[hh];
            w_l[warp][hh * 8 + g] = l[hh];
        }
    }
    __syncthreads();
    float mc[2], f[2];  // the CTA's maximum of this thread's rows, and what scales this warp's sums to it
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
        mc[hh] = -CUDART_INF_F;
#pragma unroll
        for (int w = 0; w < kPersWarps; ++w) mc[hh] = fmaxf(mc[hh], w_m[w][hh * 8 + g]);
        f[hh] = m[hh] > -CUDART_INF_F ? ex2(m[hh] - mc[hh]) : 0.f;
    }
    for (int w = 0; w < kPersWarps; ++w) {
        if (warp == w) {
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
                float* dst = part[hh * 8 + g];
#pragma unroll
                for (int n = 0; n < NT; ++n)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const int col = n * 8 + 2 * t + e;
                        dst[col] = (w ? dst[col] : 0.f) + acc[n][2 * hh + e] * f[hh];
                    }
                if (t == 0) {
                    dst[DH] = mc[hh];
                    dst[DH + 1] = (w ? dst[DH + 1] : 0.f) + l[hh] * f[hh];
                }
            }
        }
        __syncthreads();
    }
    if (cs > 1) {
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
    const uint32_t base = smem_addr(&part[0][0]);
    auto at = [&](int r, int row, int what) -> float {
        uint32_t a = base + (row * (DH + 2) + what) * 4;
        float x;
        asm volatile("mapa.shared::cluster.u32 %0, %0, %1;" : "+r"(a) : "r"(r));
        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(x) : "r"(a) : "memory");
        return x;
    };
    // this CTA finishes rows rank, rank + cs, ...: a warp per row
    for (int row = rank + warp * cs; row < 16; row += cs * kPersWarps) {
        if (row0 + row >= p.q_rows) continue;
        float ma = -CUDART_INF_F, la = 0.f, fr[8];
#pragma unroll
        for (int r = 0; r < 8; ++r) fr[r] = r < cs ? at(r, row, DH) : -CUDART_INF_F;
#pragma unroll
        for (int r = 0; r < 8; ++r) ma = fmaxf(ma, fr[r]);
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            fr[r] = fr[r] > -CUDART_INF_F ? ex2(fr[r] - ma) : 0.f;
            if (r < cs) la = fmaf(at(r, row, DH + 1), fr[r], la);
        }
        T* dst = static_cast<T*>(p.o) + batch * p.os[0] + head * p.os[1] + (row0 + row) * p.os[2];
        for (int col = lane; col < DH; col += 32) {
            float a = 0.f;
#pragma unroll
            for (int r = 0; r < 8; ++r)
                if (r < cs && fr[r] > 0.f) a = fmaf(at(r, row, col), fr[r], a);
            dst[col] = from_f32<T>(a / la);
        }
        if (p.lse != nullptr && lane == 0) p.lse[((long long)batch * gridDim.y + head) * p.q_rows + row0 + row] = ma + log2f(la);
    }
    if (cs > 1) {  // nobody's shared memory goes away while a peer may still read it
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
}

}  // namespace

int launch_pers_rows(const tmw_prefill_desc& d, const void* q, const void* k, const void* v, void* o, float* lse,
                     cudaStream_t stream, bool pdl) {
    PersParams p;
    p.q = q; p.k = k; p.v = v; p.o = o; p.lse = lse;
    for (int i = 0; i < 3; ++i) {
        p.qs[i] = d.q_stride[i]; p.ks[i] = d.k_stride[i]; p.vs[i] = d.v_stride[i]; p.os[i] = d.o_stride[i];
    }
    p.q_rows = d.q_rows; p.k_rows = d.k_rows;
    p.scale_log2 = (d.scale != 0.f ? d.scale : 1.0f / sqrtf((float)d.head_dim)) * 1.4426950408889634f;
    // CTAs per (batch, head, 16 rows): up to eight, while they fit the chip four to an SM (head_dim 64; at 128 two are resident and the
    // rest a second wave) and have a block for every warp
    const long long groups = (long long)(d.q_rows + 15) / 16 * d.heads * d.batch;
    p.cluster = 1;
    while (p.cluster < 8 && groups * p.cluster * 2 <= 4 * sm_count() && p.cluster * 2 * kPersWarps * pers_keys(d.head_dim) <= d.k_rows) p.cluster *= 2;
    const dim3 grid((d.q_rows + 15) / 16 * p.cluster, d.heads, d.batch), block(kPersWarps * 32);
    auto run = [&](auto kern) -> int {
        TMW_CUDA_TRY(launch_ex(kern, grid, block, 0, stream, pdl, p.cluster, p));
        return TMW_OK;
    };
    if (d.head_dim == 64)
        return d.dtype == TMW_BF16 ? run(pers_rows_kernel<__nv_bfloat16, 64>) : run(pers_rows_kernel<__half, 64>);
    return d.dtype == TMW_BF16 ? run(pers_rows_kernel<__nv_bfloat16, 128>) : run(pers_rows_kernel<__half, 128>);
}

}  // namespace tmw
