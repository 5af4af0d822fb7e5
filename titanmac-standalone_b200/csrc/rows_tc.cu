// Products of a decode step with more rows than one mma tile (17 .. 256 sequences) on tcgen05:
// c[m, n] = epilogue(a[m, k] · w[n, k]ᵀ), and the RMSNorm in front of them, as links of a chain of dependent launches.
//
// The product is latency from end to end: 0.2 to 0.8 GFLOP, about 0.5 us at the tensor cores' rate.  So the work is cut for
// the shortest path, not for the fewest bytes: 128 rows x BN columns per CTA with BN small, and where that leaves SMs
// idle a cluster of up to eight CTAs shares a tile's k and adds up through distributed shared memory.  Barriers, tensor
// memory and the first tiles of w are ready before the predecessor has finished (pdl_wait); rows of a beyond m are
// filled in by TMA and cost no traffic.
#include <cuda.h>

#include <type_traits>

#include "tc_ptx.cuh"
#include "tensor_map.cuh"
#include "tmw_common.cuh"

namespace tmw {
namespace {

using namespace ptx;

constexpr int kTcThreads = 192;  // warps 0-3 epilogue (one row each thread), 4 TMA, 5 tcgen05.mma

struct RowsTcParams {
    void* c;           // [m, n], leading dimension ldc; EPI 2: x, read and written
    const void* bias;  // [n] or nullptr
    long long ldc;
    int m, n, k, cluster;
    int* status;
};

template <int BN>
struct RowsTcSmem {
    static constexpr int kA = 128 * 128, kW = BN * 128;  // 64 k-elements of a row = 128 bytes
    static constexpr int kStage = kA + kW;
    static constexpr int kStages = 5;  // two CTAs fit an SM: the successor's, or a grid's second wave
    static constexpr int kStr = BN + 4;  // floats per row of the partial sums
    static constexpr int kBars = kStages * kStage;
    static constexpr int kTotal = kBars + 256 + 1024;
    static_assert(128 * kStr * 4 <= kBars, "the partial sums take the place of the stages");
};

struct RowsTcArgs {
    CUtensorMap map_a, map_w;
    RowsTcParams p;
};

template <int BN, bool BF16, int EPI>
__global__ void __launch_bounds__(kTcThreads) rows_tc_kernel(const __grid_constant__ RowsTcArgs args) {
    using L = RowsTcSmem<BN>;
    constexpr int S = L::kStages;
    using T = typename std::conditional<BF16, __nv_bfloat16, __half>::type;
    const RowsTcParams& p = args.p;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const uint32_t smem_base = smem_u32(smem), bar_base = smem_base + L::kBars;
    auto full = [&](int s) -> uint32_t { return bar_base + 8 * s; };
    auto empty = [&](int s) -> uint32_t { return bar_base + 8 * (S + s); };
    const uint32_t done = bar_base + 16 * S;
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem + L::kBars + 16 * S + 8);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + L::kBars + 16 * S + 16);

    const int warp = threadIdx.x >> 5;
    const int cs = p.cluster, rank = (int)blockIdx.x % cs, n0 = (int)(blockIdx.x / cs) * BN, m0 = blockIdx.y * 128;
    const int blocks = (p.k + 63) / 64;
    const int b_lo = blocks * rank / cs, nb = blocks * (rank + 1) / cs - b_lo;  // this CTA's 64-wide slices of k

    if (threadIdx.x == 0) {
        for (int s = 0; s < S; ++s) {
            mbar_init(full(s), 1);
            mbar_init(empty(s), 1);
        }
        mbar_init(done, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 5) tmem_alloc(smem_u32((const void*)tmem_slot), BN);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    pdl_trigger();  // (with its tensor memory in hand: a dependent that took it first would wait for this CTA forever)

    if (warp == 4) {
        if (elect_one()) {
            for (int i = 0; i < nb && i < S; ++i) {  // weights of the first stages: nobody's output
                mbar_expect_tx(full(i), L::kStage);
                tma_load_2d(smem_base + i * L::kStage + L::kA, &args.map_w, full(i), (b_lo + i) * 64, n0);
            }
            pdl_wait();
            for (int i = 0; i < nb; ++i) {
                const int s = i % S;
                if (i >= S) {
                    mbar_wait(empty(s), ((i / S) & 1) ^ 1, abort_flag, p.status);
                    mbar_expect_tx(full(s), L::kStage);
                    tma_load_2d(smem_base + s * L::kStage + L::kA, &args.map_w, full(s), (b_lo + i) * 64, n0);
                }
                tma_load_2d(smem_base + s * L::kStage, &args.map_a, full(s), (b_lo + i) * 64, m0);
            }
        }
        __syncwarp();
    } else if (warp == 5) {
        if (elect_one()) {
            const uint32_t idesc = idesc_kmajor(BF16 ? 1u : 0u, BN);
            for (int i = 0; i < nb; ++i) {
                const int s = i % S;
                mbar_wait(full(s), (i / S) & 1, abort_flag, p.status);
                tc_fence_after();
                const uint64_t ad = kmajor_desc(smem_base + s * L::kStage);
                const uint64_t wd = kmajor_desc(smem_base + s * L::kStage + L::kA);
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) mma_ss(tmem, ad + 2 * kk, wd + 2 * kk, idesc, (i | kk) ? 1u : 0u);
                if (i + S < nb) tc_commit(empty(s));  // (a stage that is not filled again needs no hand-back)
            }
            tc_commit(done);
        }
        __syncwarp();
    }

    // ---- epilogue: CS threads per row, BN / CS columns each (one CTA: one thread per row), eight columns at a time ----
    const int rows_r = 128 / cs, cols_t = BN / cs;
    const int row = rank * rows_r + (int)threadIdx.x / cs, col0 = ((int)threadIdx.x % cs) * cols_t;
    const int gm = m0 + row;
    float* part = reinterpret_cast<float*>(smem);
    T* dst_row = static_cast<T*>(p.c) + (long long)gm * p.ldc + n0 + col0;
    auto live = [&](int v) { return warp < 4 && gm < p.m && v * 8 < cols_t && n0 + col0 + v * 8 < p.n; };
    uint4 bias[BN / 8], res[EPI == 2 ? BN / 8 : 1];  // on their way before the product is done
#pragma unroll
    for (int v = 0; v < BN / 8; ++v)
        if (live(v) && p.bias != nullptr)
            bias[v] = *reinterpret_cast<const uint4*>(static_cast<const T*>(p.bias) + n0 + col0 + v * 8);
    pdl_wait();  // (every thread: below is read and written what the predecessor may still be using)
    if (EPI == 2) {
#pragma unroll
        for (int v = 0; v < BN / 8; ++v)
            if (live(v)) res[v] = *reinterpret_cast<const uint4*>(dst_row + v * 8);
    }
    if (warp < 4) {
        mbar_wait(done, 0, abort_flag, p.status);
        tc_fence_after();
        // tensor memory -> shared memory: thread = lane = row of the tile
        float* mine = part + threadIdx.x * L::kStr;
#pragma unroll
        for (int c = 0; c < BN; c += 32) {
            uint32_t v[32];
            tmem_ld32(tmem + ((uint32_t)(warp * 32) << 16) + c, v);
            tc_wait_ld();
#pragma unroll
            for (int j = 0; j < 32; j += 4)
                *reinterpret_cast<uint4*>(mine + c + j) = make_uint4(v[j], v[j + 1], v[j + 2], v[j + 3]);
        }
    }
    if (cs > 1) cluster_sync();
    if (warp < 4) {
        const uint32_t part_addr = smem_u32(part);
#pragma unroll
        for (int v = 0; v < BN / 8; ++v) {
            if (!live(v)) continue;
            const int at = row * L::kStr + col0 + v * 8;
            float4 lo = *reinterpret_cast<const float4*>(part + at), hi = *reinterpret_cast<const float4*>(part + at + 4);
            for (int r = 0; r < cs; ++r) {
                if (r == rank) continue;
                const uint32_t a = map_to_cta(part_addr, r) + at * 4;
                float4 x, y;
                asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];"
                             : "=f"(x.x), "=f"(x.y), "=f"(x.z), "=f"(x.w) : "r"(a) : "memory");
                asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];"
                             : "=f"(y.x), "=f"(y.y), "=f"(y.z), "=f"(y.w) : "r"(a + 16) : "memory");
                lo.x += x.x; lo.y += x.y; lo.z += x.z; lo.w += x.w;
                hi.x += y.x; hi.y += y.y; hi.z += y.z; hi.w += y.w;
            }
            float o[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
            if (p.bias != nullptr) {
                float b[8];
                load8<T>(reinterpret_cast<const T*>(&bias[v]), b);
#pragma unroll
                for (int e = 0; e < 8; ++e) o[e] += b[e];
            }
            if (EPI == 1) {
#pragma unroll
                for (int e = 0; e < 8; ++e) o[e] = gelu_erf(o[e]);
            }
            if (EPI == 2) {
                float x[8];
                load8<T>(reinterpret_cast<const T*>(&res[v]), x);
#pragma unroll
                for (int e = 0; e < 8; ++e) o[e] = x[e] + to_f32<T>(from_f32<T>(o[e]));
            }
            store8<T>(dst_row + v * 8, o);
        }
    }
    if (cs > 1) cluster_sync();  // nobody's shared memory goes away while a peer may still read it
    tc_fence_before();
    __syncthreads();
    if (warp == 5) {
        tc_fence_after();
        if (*abort_flag) {
            const long long t0 = clock64();
            while (clock64() - t0 < 400000) __nanosleep(1000);
        }
        tmem_dealloc(tmem, BN);
    }
}

// y = x / sqrt(mean(x^2) + eps) * gain, one warp per row, the row in registers (dim <= 32 * 8 * NV)
struct RowsNormParams {
    const void *x, *gain;
    void* y;
    int rows, dim;
    float eps;
};

template <typename T, int NV>
__global__ void __launch_bounds__(64) rows_norm_kernel(const RowsNormParams p) {
    pdl_trigger();
    const int row = blockIdx.x * 2 + (threadIdx.x >> 5), lane = threadIdx.x & 31, nvec = p.dim / 8;
    uint4 g[NV], x[NV];
#pragma unroll
    for (int j = 0; j < NV; ++j)
        if (lane + j * 32 < nvec) g[j] = reinterpret_cast<const uint4*>(p.gain)[lane + j * 32];
    pdl_wait();
    if (row >= p.rows) return;
    const uint4* xr = reinterpret_cast<const uint4*>(static_cast<const T*>(p.x) + (long long)row * p.dim);
#pragma unroll
    for (int j = 0; j < NV; ++j) x[j] = lane + j * 32 < nvec ? xr[lane + j * 32] : make_uint4(0u, 0u, 0u, 0u);
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        float h[8];
        load8<T>(reinterpret_cast<const T*>(&x[j]), h);
#pragma unroll
        for (int e = 0; e < 8; ++e) ss = fmaf(h[e], h[e], ss);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    const float inv = 1.0f / sqrtf(ss / (float)p.dim + p.eps);
#pragma unroll
    for (int j = 0; j < NV; ++j)
        if (lane + j * 32 < nvec) {
            float h[8], w[8];
            load8<T>(reinterpret_cast<const T*>(&x[j]), h);
            load8<T>(reinterpret_cast<const T*>(&g[j]), w);
#pragma unroll
            for (int e = 0; e < 8; ++e) h[e] = h[e] * inv * w[e];
            store8<T>(static_cast<T*>(p.y) + (long long)row * p.dim + (lane + j * 32) * 8, h);
        }
}

}  // namespace

int launch_rows_norm(int dtype, int rows, int dim, const void* x, const void* gain, float eps, void* y, cudaStream_t stream) {
    RowsNormParams p;
    p.x = x; p.gain = gain; p.y = y; p.rows = rows; p.dim = dim; p.eps = eps;
    const dim3 grid((rows + 1) / 2), block(64);
    auto run = [&](auto kern) -> int {
        TMW_CUDA_TRY(launch_ex(kern, grid, block, 0, stream, true, 1, p));
        return TMW_OK;
    };
    const bool bf16 = dtype == TMW_BF16;
    if (dim <= 1024) return bf16 ? run(rows_norm_kernel<__nv_bfloat16, 4>) : run(rows_norm_kernel<__half, 4>);
    if (dim <= 2048) return bf16 ? run(rows_norm_kernel<__nv_bfloat16, 8>) : run(rows_norm_kernel<__half, 8>);
    if (dim <= 4096) return bf16 ? run(rows_norm_kernel<__nv_bfloat16, 16>) : run(rows_norm_kernel<__half, 16>);
    return TMW_ERR_UNSUPPORTED;
}

int launch_rows_tc(int dtype, int m, int n, int k, const void* a, const void* w, const void* bias, void* c, int epi,
                   cudaStream_t stream, bool pdl) {
    RowsTcArgs args;
    // 32 columns per tile, and the k of a tile over as many CTAs as fill the chip once (a CTA keeps at least two slices
    // of 64): one step of 16 layers for 64 | 128 | 256 rows took 784 | 1093 | 1461 us, with 64 columns 865 | 1261 | 1629
    constexpr int bn = 32;
    const int sms = sm_count(), m_tiles = (m + 127) / 128, blocks = (k + 63) / 64;
    const int tiles = (n + bn - 1) / bn * m_tiles;
    RowsTcParams& p = args.p;
    p.cluster = 1;
    while (p.cluster < bn / 8 && tiles * p.cluster * 2 <= sms * 9 / 8 && blocks / (p.cluster * 2) >= 2) p.cluster *= 2;
    if (!make_map_2d(&args.map_a, a, dtype, m, k, k, 128, 64, CU_TENSOR_MAP_SWIZZLE_128B) ||
        !make_map_2d(&args.map_w, w, dtype, n, k, k, bn, 64, CU_TENSOR_MAP_SWIZZLE_128B))
        return TMW_ERR_CUDA;
    p.c = c; p.bias = bias; p.ldc = n; p.m = m; p.n = n; p.k = k;
    p.status = device_status_word();
    if (p.status == nullptr) return TMW_ERR_CUDA;
    const dim3 grid((n + bn - 1) / bn * p.cluster, m_tiles);
    auto run = [&](auto kern, int smem) -> int {
        const int rc = allow_shared_memory(reinterpret_cast<const void*>(kern), smem);
        if (rc != TMW_OK) return rc;
        TMW_CUDA_TRY(launch_ex(kern, grid, dim3(kTcThreads), smem, stream, pdl, p.cluster, args));
        return TMW_OK;
    };
    auto pick = [&](auto bf16) -> int {
        constexpr bool BF16 = decltype(bf16)::value;
        const int smem = RowsTcSmem<bn>::kTotal;
        return epi == 0 ? run(rows_tc_kernel<bn, BF16, 0>, smem) : epi == 1 ? run(rows_tc_kernel<bn, BF16, 1>, smem)
                                                                            : run(rows_tc_kernel<bn, BF16, 2>, smem);
    };
    return dtype == TMW_BF16 ? pick(std::true_type{}) : pick(std::false_type{});
}

}  // namespace tmw
