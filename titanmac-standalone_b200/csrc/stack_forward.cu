// The attention module and the whole model over full sequences as one call each: the existing kernels, launched from
// here as a chain of dependent launches (see pdl_wait) instead of one by one from Python.  With six to eight calls per
// block at 15 - 20 us of host work each, a 16-layer model took 4 ms to issue - more than the GPU needs below about
// 8000 rows - and a single layer of 144 rows 80 us for 15 us of kernels.
#include <math_constants.h>

#include "tmw_common.cuh"

namespace tmw {
namespace {

int64_t align256(int64_t n) { return (n + 255) & ~(int64_t)255; }
bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// x[b, i] = persistent[i] for i < np, else round(tokens[ids[b, i - np]] + positions[i - np]); y = RMSNorm(x).
// One warp per row; replaces two gathers, an add, a concatenation and the first norm.
struct EmbedSeqParams {
    const void *tokens, *positions, *persistent, *gain;
    const int64_t* ids;
    void *x, *y;
    int* status;
    long long rows;
    int seq, np, dim, vocab;
    float eps;
};

constexpr int kEmbedWarps = 8;

template <typename T>
__global__ void __launch_bounds__(kEmbedWarps * 32) embed_seq_kernel(const EmbedSeqParams p) {
    const int lane = threadIdx.x & 31, len = p.seq + p.np;
    const long long warps = (long long)gridDim.x * kEmbedWarps;
    for (long long row = (long long)blockIdx.x * kEmbedWarps + (threadIdx.x >> 5); row < p.rows; row += warps) {
        const long long b = row / len;
        const int i = (int)(row - b * len) - p.np;
        const T *src = static_cast<const T*>(p.persistent) + (long long)(i + p.np) * p.dim, *add = nullptr;
        bool bad = false;
        if (i >= 0) {
            long long id = p.ids[b * p.seq + i];
            if (id < 0 || id >= p.vocab) {  // outside the table: a row of NaN, and the status word says so
                if (lane == 0) atomicCAS(p.status, 0, (int)TMW_ERR_INVALID_ARGUMENT);
                bad = true;
                id = 0;
            }
            src = static_cast<const T*>(p.tokens) + id * p.dim;
            add = static_cast<const T*>(p.positions) + (long long)i * p.dim;
        }
        T *x = static_cast<T*>(p.x) + row * p.dim, *y = static_cast<T*>(p.y) + row * p.dim;
        float ss = 0.f;
        for (int v = lane; v < p.dim / 8; v += 32) {
            float u[8];
            load8<T>(src + v * 8, u);
            if (add != nullptr) {
                float w[8];
                load8<T>(add + v * 8, w);
#pragma unroll
                for (int e = 0; e < 8; ++e) u[e] = bad ? CUDART_NAN_F : to_f32<T>(from_f32<T>(u[e] + w[e]));
            }
#pragma unroll
            for (int e = 0; e < 8; ++e) ss = fmaf(u[e], u[e], ss);
            store8<T>(x + v * 8, u);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        const float inv = 1.0f / sqrtf(ss / (float)p.dim + p.eps);
        for (int v = lane; v < p.dim / 8; v += 32) {  // (the row comes back out of L1)
            float u[8], g[8];
            load8<T>(x + v * 8, u);
            load8<T>(static_cast<const T*>(p.gain) + v * 8, g);
#pragma unroll
            for (int e = 0; e < 8; ++e) u[e] = u[e] * inv * g[e];
            store8<T>(y + v * 8, u);
        }
    }
}

// y[b] = RMSNorm(x[b, last]): the final norm of the last rows only
struct LastRowsParams {
    const void *x, *gain;
    void* y;
    int batch, len, dim;
    float eps;
};

template <typename T>
__global__ void __launch_bounds__(128) last_rows_norm_kernel(const LastRowsParams p) {
    pdl_trigger();
    pdl_wait();
    const int b = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (b >= p.batch) return;
    const long long at = ((long long)b * p.len + p.len - 1) * p.dim;
    T* y = static_cast<T*>(p.y) + (long long)b * p.dim;
    float ss = 0.f;
    for (int v = lane; v < p.dim / 8; v += 32) {
        float u[8];
        load8<T>(static_cast<const T*>(p.x) + at + v * 8, u);
#pragma unroll
        for (int e = 0; e < 8; ++e) ss = fmaf(u[e], u[e], ss);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    const float inv = 1.0f / sqrtf(ss / (float)p.dim + p.eps);
    for (int v = lane; v < p.dim / 8; v += 32) {
        float u[8], g[8];
        load8<T>(static_cast<const T*>(p.x) + at + v * 8, u);  // (out of L1)
        load8<T>(static_cast<const T*>(p.gain) + v * 8, g);
#pragma unroll
        for (int e = 0; e < 8; ++e) u[e] = u[e] * inv * g[e];
        store8<T>(y + v * 8, u);
    }
}

int linear(int dtype, int m, int n, int k, const void* a, const void* w, const void* bias, void* c, int epilogue,
           cudaStream_t stream, int chain) {
    tmw_linear_desc d = {};
    d.dtype = dtype; d.m = m; d.n = n; d.k = k; d.epilogue = epilogue;
    d.lda = k; d.ldw = k; d.ldc = n;
    return launch_linear(d, a, w, bias, c, stream, chain);
}

// x += round(a w^T + bias): the residual rides on the product, and the norm behind it reads one array and writes one, not two
// and two (16 layers over 2 x 8208 rows of 640, vocabulary 50 000: 5351 -> 5237 us, 1.01 to 1.03 times in six comparisons
// whose repeats of one side differ by up to 3.6 %)
int linear_onto(int dtype, int m, int n, int k, const void* a, const void* w, const void* bias, void* x, cudaStream_t stream, int chain) {
    GemmCall g;
    g.dtype = dtype; g.m = m; g.n = n; g.k = k;
    g.a = a; g.lda = k; g.b = w; g.ldb = k; g.c = x; g.ldc = n; g.aux = x;
    g.bias = bias; g.epilogue = GEMM_ADD; g.chain = chain;
    return launch_gemm_call(g, stream);
}

// qkv [B, L, 3, H, dh] -> o [B, L, H, dh] with the mask of the class
tmw_prefill_desc core_desc(const tmw_attention_desc& a) {
    tmw_prefill_desc d = {};
    d.dtype = a.dtype; d.algo = TMW_ALGO_AUTO; d.batch = a.batch; d.heads = a.heads; d.head_dim = a.head_dim;
    d.q_rows = d.k_rows = a.rows; d.window = a.window; d.n_persistent = a.n_persistent;
    d.q_pos0 = 0; d.k_pos0 = a.n_persistent; d.scale = a.scale;
    const int64_t D = (int64_t)a.heads * a.head_dim;
    const int64_t in[3] = {a.rows * 3 * D, a.head_dim, 3 * D}, out[3] = {a.rows * D, a.head_dim, D};
    for (int i = 0; i < 3; ++i) {
        d.q_stride[i] = d.k_stride[i] = d.v_stride[i] = in[i];
        d.o_stride[i] = out[i];
    }
    return d;
}

// *link: whether the launch behind may be a dependent one
int core(const tmw_attention_desc& a, const void* qkv, void* o, bool* link, cudaStream_t stream) {
    const tmw_prefill_desc d = core_desc(a);
    const int64_t D = (int64_t)a.heads * a.head_dim, esz = (int64_t)dtype_size(a.dtype);
    const char* q = static_cast<const char*>(qkv);
    const void *k = q + D * esz, *v = q + 2 * D * esz;
    *link = prefill_tc_supports(d, q, k, v, o);
    if (a.block_size > 0) return prefill_block_sparse(&d, a.block_size, q, k, v, o, nullptr, stream, kChainLink);
    if (*link) return launch_prefill_tc(d, q, k, v, o, stream, 0, nullptr, nullptr, kChainLink);
    return tmw_prefill(&d, q, k, v, o, stream);
}

int validate_attention(const tmw_attention_desc* a) {
    if (a == nullptr) return TMW_ERR_INVALID_ARGUMENT;
    if (a->dtype != TMW_BF16 && a->dtype != TMW_F16) return TMW_ERR_UNSUPPORTED;
    if (a->batch < 0 || a->rows < 0 || a->heads <= 0 || a->head_dim <= 0 || a->head_dim % 8 != 0 || a->n_persistent < 0 ||
        a->block_size < 0 || a->conv_taps < 0 || a->conv_taps > 8 || !(a->scale >= 0.f))
        return TMW_ERR_INVALID_ARGUMENT;
    if (a->window < 0) return TMW_ERR_NEGATIVE_WINDOW;
    if ((int64_t)a->batch * a->rows > 0x7fffffff) return TMW_ERR_TOO_LARGE;
    if (a->rows > 0 && a->n_persistent >= a->rows) return TMW_ERR_PERSISTENT_GE_LEN;
    return TMW_OK;
}

struct AttentionBuffers {
    int64_t qkv, conv, o, total;
};
AttentionBuffers attention_buffers(const tmw_attention_desc& a) {
    const int64_t row = (int64_t)a.batch * a.rows * a.heads * a.head_dim * 2;
    AttentionBuffers b;
    b.qkv = 0;
    b.conv = align256(3 * row);
    b.o = b.conv + (a.conv_taps > 0 ? align256(3 * row) : 0);
    b.total = b.o + align256(row);
    return b;
}

// x [rows, D] -> y [rows, D], or added to y (`onto`).  `first`: nothing of this chain is in front.  (Launching as
// dependents pays at every size: 2 x 8208 rows of 16 layers 5.96 -> 5.83 ms, 3000 rows of one layer 38.9 -> 32.8 us.)
int attention(const tmw_attention_desc& a, const void* x, const void* w_qkv, const void* const* conv, const void* w_out,
              void* qkv, void* conv_out, void* o, void* y, bool onto, bool first, cudaStream_t stream) {
    const int rows = a.batch * a.rows, D = a.heads * a.head_dim;
    int rc = linear(a.dtype, rows, 3 * D, D, x, w_qkv, nullptr, qkv, TMW_EPILOGUE_NONE, stream,
                    first ? 0 : kChainDependent);
    if (rc == TMW_OK && a.conv_taps > 0) {
        rc = launch_dwconv(a.dtype, a.batch, a.rows, 3 * D, a.conv_taps, qkv, conv, 3, conv_out, stream, true);
        qkv = conv_out;
    }
    bool dependent = false;
    if (rc == TMW_OK) rc = core(a, qkv, o, &dependent, stream);
    const int link = dependent ? kChainDependent : 0;
    if (rc != TMW_OK) return rc;
    return onto ? linear_onto(a.dtype, rows, D, D, o, w_out, nullptr, y, stream, link)
                : linear(a.dtype, rows, D, D, o, w_out, nullptr, y, TMW_EPILOGUE_NONE, stream, link);
}

struct StackBuffers {
    int64_t x, y, big, conv, total;  // big: [qkv | o] and, those two used up, the MLP's hidden rows
};
StackBuffers stack_buffers(const tmw_stack_desc& d, int64_t rows) {
    const int64_t row = rows * 2;
    StackBuffers s;
    s.x = 0;
    s.y = s.x + align256(row * d.d_model);
    s.big = s.y + align256(row * d.d_model);
    const int64_t attn = align256(row * 3 * d.d_model) + align256(row * d.d_model), mlp = align256(row * d.d_ff);
    s.conv = s.big + (attn > mlp ? attn : mlp);
    s.total = s.conv + (d.conv_taps > 0 ? align256(row * 3 * d.d_model) : 0);
    return s;
}

int validate_stack(const tmw_stack_desc* d, int tokens) {
    if (d == nullptr || tokens < 0) return TMW_ERR_INVALID_ARGUMENT;
    if (d->layers < 1 || d->d_ff <= 0 || d->d_ff % 8 != 0 || d->vocab <= 0 || d->vocab % 8 != 0 || tokens > d->max_positions ||
        !(d->eps >= 0.f) || d->d_model != d->heads * d->head_dim)
        return TMW_ERR_INVALID_ARGUMENT;
    return TMW_OK;
}

tmw_attention_desc attention_of(const tmw_stack_desc& d, int tokens) {
    tmw_attention_desc a = {};
    a.dtype = d.dtype; a.batch = d.batch; a.rows = tokens + d.n_persistent; a.heads = d.heads; a.head_dim = d.head_dim;
    a.window = d.window; a.n_persistent = d.n_persistent; a.block_size = d.block_size; a.conv_taps = d.conv_taps;
    a.scale = 0.f;
    return a;
}

}  // namespace

int launch_embed_seq(const tmw_stack_desc& d, const int64_t* token_ids, int tokens, const void* gain, void* x, void* y,
                     cudaStream_t stream) {
    EmbedSeqParams e;
    e.tokens = d.embed_tokens; e.positions = d.embed_positions; e.persistent = d.persistent; e.gain = gain;
    e.ids = token_ids; e.x = x; e.y = y; e.status = device_status_word();
    if (e.status == nullptr) return TMW_ERR_CUDA;
    e.rows = (long long)d.batch * (tokens + d.n_persistent); e.seq = tokens; e.np = d.n_persistent; e.dim = d.d_model; e.vocab = d.vocab; e.eps = d.eps;
    const int want = (int)((e.rows + kEmbedWarps - 1) / kEmbedWarps), grid = want < 8 * sm_count() ? want : 8 * sm_count();
    if (d.dtype == TMW_BF16) embed_seq_kernel<__nv_bfloat16><<<grid, kEmbedWarps * 32, 0, stream>>>(e);
    else embed_seq_kernel<__half><<<grid, kEmbedWarps * 32, 0, stream>>>(e);
    TMW_CUDA_TRY(cudaGetLastError());
    return TMW_OK;
}

}  // namespace tmw

extern "C" size_t tmw_attention_workspace(const tmw_attention_desc* desc) {
    return tmw::validate_attention(desc) != TMW_OK ? 0 : (size_t)tmw::attention_buffers(*desc).total;
}

extern "C" int tmw_attention_forward(const tmw_attention_desc* desc, const void* x, const void* w_qkv, const void* conv_q,
                                     const void* conv_k, const void* conv_v, const void* w_out, void* y, void* workspace,
                                     size_t workspace_bytes, void* stream) {
    using namespace tmw;
    const int rc = validate_attention(desc);
    if (rc != TMW_OK) return rc;
    if (desc->batch == 0 || desc->rows == 0) return TMW_OK;
    const void* conv[3] = {conv_q, conv_k, conv_v};
    const void* need[] = {x, w_qkv, w_out, y, workspace};
    for (const void* q : need)
        if (q == nullptr || !aligned16(q)) return TMW_ERR_INVALID_ARGUMENT;
    for (const void* q : conv)
        if (desc->conv_taps > 0 && q == nullptr) return TMW_ERR_INVALID_ARGUMENT;
    const AttentionBuffers off = attention_buffers(*desc);
    if (workspace_bytes < (size_t)off.total) return TMW_ERR_TOO_LARGE;
    char* ws = static_cast<char*>(workspace);
    return attention(*desc, x, w_qkv, conv, w_out, ws + off.qkv, ws + off.conv, ws + off.o, y,
                     false, true, static_cast<cudaStream_t>(stream));
}

extern "C" size_t tmw_stack_workspace(const tmw_stack_desc* desc, int32_t tokens) {
    if (tmw::validate_stack(desc, tokens) != TMW_OK) return 0;
    return (size_t)tmw::stack_buffers(*desc, (int64_t)desc->batch * (tokens + desc->n_persistent)).total;
}

extern "C" int tmw_stack_forward(const tmw_stack_desc* desc, const tmw_block* blocks, const int64_t* token_ids, int32_t tokens,
                                 int32_t last_only, void* logits, void* workspace, size_t workspace_bytes, void* stream) {
    using namespace tmw;
    int rc = validate_stack(desc, tokens);
    if (rc != TMW_OK) return rc;
    const tmw_stack_desc& d = *desc;
    const tmw_attention_desc a = attention_of(d, tokens);
    rc = validate_attention(&a);
    if (rc != TMW_OK) return rc;
    if (d.batch == 0 || tokens == 0) return TMW_OK;
    const void* tops[] = {blocks, token_ids, logits, workspace, d.embed_tokens, d.embed_positions, d.norm, d.head};
    for (const void* q : tops)
        if (q == nullptr) return TMW_ERR_INVALID_ARGUMENT;
    if (!aligned16(d.embed_tokens) || !aligned16(d.embed_positions) || !aligned16(d.norm) || !aligned16(d.head) ||
        !aligned16(logits) || !aligned16(workspace) || (d.n_persistent > 0 && (d.persistent == nullptr || !aligned16(d.persistent))))
        return TMW_ERR_INVALID_ARGUMENT;
    for (int l = 0; l < d.layers; ++l) {
        const tmw_block& b = blocks[l];
        const void* need[] = {b.norm_attn, b.w_qkv, b.w_out, b.norm_mlp, b.w_fc1, b.w_fc2};
        for (const void* q : need)
            if (q == nullptr || !aligned16(q)) return TMW_ERR_INVALID_ARGUMENT;
        if (d.conv_taps > 0 && (b.conv_q == nullptr || b.conv_k == nullptr || b.conv_v == nullptr)) return TMW_ERR_INVALID_ARGUMENT;
        const void* ring[] = {b.k_ring, b.v_ring, b.k_pers, b.v_pers};
        for (int i = 0; i < 4; ++i)
            if (b.k_ring != nullptr && (i < 2 || d.n_persistent > 0) && (ring[i] == nullptr || !aligned16(ring[i])))
                return TMW_ERR_INVALID_ARGUMENT;
    }
    const int L = a.rows, D = d.d_model, F = d.d_ff, rows = d.batch * L;
    const StackBuffers off = stack_buffers(d, rows);
    if (workspace_bytes < (size_t)off.total) return TMW_ERR_TOO_LARGE;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    char* ws = static_cast<char*>(workspace);
    void *x = ws + off.x, *y = ws + off.y, *big = ws + off.big;
    char* o = ws + off.big + align256((int64_t)rows * 6 * D);

    rc = launch_embed_seq(d, token_ids, tokens, blocks[0].norm_attn, x, y, s);
    for (int l = 0; l < d.layers && rc == TMW_OK; ++l) {
        const tmw_block& b = blocks[l];
        const void* conv[3] = {b.conv_q, b.conv_k, b.conv_v};
        rc = attention(a, y, b.w_qkv, conv, b.w_out, big, ws + off.conv, o, x, true, false, s);
        if (rc == TMW_OK && b.k_ring != nullptr) {
            // keys and values of the sequence rows into the ring, those of the persistent rows (the same for every
            // sequence) beside it
            tmw_cache_desc c = {};
            c.dtype = d.dtype; c.batch = d.batch; c.heads = d.heads; c.head_dim = d.head_dim; c.window = d.window;
            c.n_persistent = d.n_persistent;
            c.k_ring = b.k_ring; c.v_ring = b.v_ring; c.k_pers = b.k_pers; c.v_pers = b.v_pers;
            const int64_t st[3] = {(int64_t)L * 3 * D, d.head_dim, 3 * (int64_t)D};
            const char* k = static_cast<const char*>(big) + (int64_t)D * 2;
            const char* v = k + (int64_t)D * 2;
            const int64_t skip = (int64_t)d.n_persistent * 3 * D * 2;
            rc = launch_cache_fill(c, k + skip, v + skip, st, st, tokens, 0, s, d.n_persistent > 0 ? k : nullptr,
                                   d.n_persistent > 0 ? v : nullptr, true);
        }
        if (rc == TMW_OK) rc = launch_add_rmsnorm(d.dtype, rows, D, x, nullptr, b.norm_mlp, d.eps, nullptr, y, s, true);
        if (rc == TMW_OK) rc = linear(d.dtype, rows, F, D, y, b.w_fc1, b.b_fc1, big, TMW_EPILOGUE_GELU, s, kChainDependent);
        if (rc == TMW_OK) rc = linear_onto(d.dtype, rows, D, F, big, b.w_fc2, b.b_fc2, x, s, kChainDependent);
        if (rc == TMW_OK && (l + 1 < d.layers || !last_only))
            rc = launch_add_rmsnorm(d.dtype, rows, D, x, nullptr, l + 1 < d.layers ? blocks[l + 1].norm_attn : d.norm, d.eps, nullptr, y, s,
                                    true);
    }
    if (rc != TMW_OK) return rc;
    if (!last_only) return linear(d.dtype, rows, d.vocab, D, y, d.head, nullptr, logits, TMW_EPILOGUE_NONE, s, kChainDependent);
    LastRowsParams p;
    p.x = x; p.gain = d.norm; p.y = y; p.batch = d.batch; p.len = L; p.dim = D; p.eps = d.eps;
    const dim3 g((d.batch + 3) / 4), t(128);
    if (d.dtype == TMW_BF16) TMW_CUDA_TRY(launch_ex(last_rows_norm_kernel<__nv_bfloat16>, g, t, 0, s, true, 1, p));
    else TMW_CUDA_TRY(launch_ex(last_rows_norm_kernel<__half>, g, t, 0, s, true, 1, p));
    return linear(d.dtype, d.batch, d.vocab, D, y, d.head, nullptr, logits, TMW_EPILOGUE_NONE, s, kChainDependent);
}
