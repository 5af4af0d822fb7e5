// Forward and backward of the attention module and of the whole model as one call each, for training in 16-bit types.
//
// Autograd over the modules ran 380 - 510 small kernels per step of a 4- to 6-layer model, nine for each RMSNorm and its
// gradient alone, and issued them from Python in 5.6 - 8 ms whatever the sizes.  Here a step is two calls: activations go
// into one buffer of the caller's, the element-wise work rides in the products' epilogues (bias, GELU kept with its
// argument, residual sums, GELU's derivative) or in one kernel per norm, weight gradients are split over their long k
// where the output alone does not fill the chip, and all sums of partial results of a block are one launch.
#include "train_ops.cuh"

namespace tmw {
namespace {

int64_t align256(int64_t n) { return (n + 255) & ~(int64_t)255; }
bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

constexpr int64_t kPartBytes = 24ll << 20;  // what the ranges of one split product may take

struct Dims {
    int dtype, B, L, H, dh, D, F, np, window, block, taps;
    float scale, eps;
    int rows() const { return B * L; }
};

tmw_prefill_desc core_desc(const Dims& d) {
    tmw_prefill_desc c = {};
    c.dtype = d.dtype; c.algo = TMW_ALGO_AUTO; c.batch = d.B; c.heads = d.H; c.head_dim = d.dh;
    c.q_rows = c.k_rows = d.L; c.window = d.window; c.n_persistent = d.np;
    c.q_pos0 = 0; c.k_pos0 = d.np; c.scale = d.scale;
    const int64_t D = d.D, in[3] = {d.L * 3 * D, d.dh, 3 * D}, out[3] = {d.L * D, d.dh, D};
    for (int i = 0; i < 3; ++i) {
        c.q_stride[i] = c.k_stride[i] = c.v_stride[i] = in[i];
        c.o_stride[i] = out[i];
    }
    return c;
}

// Room for the ranges of the product whose output is [n, k] and whose sum runs over the rows: what launch_gemm_splitk can ask
// for at most, so that a small batch does not come with megabytes of scratch.
int64_t split_room(const Dims& d, int64_t n, int64_t k) {
    const int64_t splits = gemm_most_splits(d.rows()), bytes = splits * n * k * 4;
    return splits < 2 ? 0 : align256(bytes < kPartBytes ? bytes : kPartBytes);
}

// c[m, n] = a[m, k] w[n, k]^T
int product(const Dims& d, int m, int n, int k, const void* a, const void* w, const void* bias, void* c, int epilogue, void* aux,
            int chain, cudaStream_t s) {
    GemmCall g;
    g.dtype = d.dtype; g.m = m; g.n = n; g.k = k; g.a = a; g.lda = k; g.b = w; g.ldb = k; g.c = c; g.ldc = n;
    g.bias = bias; g.epilogue = epilogue; g.aux = aux; g.chain = chain;
    return launch_gemm_call(g, s);
}
// gradient of the input: c[m, n] = dy[m, k] w[k, n]
int input_grad(const Dims& d, int m, int n, int k, const void* dy, const void* w, void* c, int epilogue, void* aux, int chain,
               cudaStream_t s) {
    GemmCall g;
    g.dtype = d.dtype; g.m = m; g.n = n; g.k = k; g.a = dy; g.lda = k; g.b = w; g.ldb = n; g.b_mn = true; g.c = c; g.ldc = n;
    g.epilogue = epilogue; g.aux = aux; g.chain = chain;
    return launch_gemm_call(g, s);
}

// Partial results of one block, added up by one launch at its end.
struct Pending {
    SumParts sums;
    char* base;
    int64_t used = 0, room;
    float* take(int64_t floats) {
        float* p = reinterpret_cast<float*>(base + used);
        used += align256(floats * 4);
        return p;
    }
    // gradient of the weight [n, k] of y = x w^T: dw[n, k] = dy[rows, n]^T x[rows, k]
    int weight_grad(const Dims& d, int rows, int n, int k, const void* dy, const void* x, void* dw, int chain, cudaStream_t s) {
        GemmCall g;
        g.dtype = d.dtype; g.m = n; g.n = k; g.k = rows; g.a = dy; g.lda = n; g.a_mn = true; g.b = x; g.ldb = k; g.b_mn = true;
        g.c = dw; g.ldc = k; g.chain = chain;
        g.partial = reinterpret_cast<float*>(base + used);
        int splits = 1;
        const int64_t left = room - used, most = left < kPartBytes ? left : kPartBytes;
        const int rc = launch_gemm_splitk(g, (size_t)(most > 0 ? most : 0), &splits, s);
        if (rc == TMW_OK && splits > 1) sums.add(take((int64_t)splits * n * k), dw, (int64_t)n * k, splits);
        return rc;
    }
    int flush(const Dims& d, cudaStream_t s) {
        const int rc = launch_sum_parts(d.dtype, sums, s);
        sums.count = 0;
        used = 0;
        return rc;
    }
};

struct AttentionSaved {
    char *qkv, *conv, *o;
    float* lse;
};
struct AttentionWeights {
    const void *w_qkv, *w_out, *conv[3];
};
struct AttentionGrads {
    void *w_qkv, *w_out, *conv[3];
};

int64_t attention_saved_bytes(const Dims& d) {
    const int64_t row = (int64_t)d.rows() * d.D * 2;
    return align256(3 * row) * (d.taps > 0 ? 2 : 1) + align256(row) + align256((int64_t)d.rows() * d.H * 4);
}
AttentionSaved attention_saved(const Dims& d, char* p) {
    const int64_t row = (int64_t)d.rows() * d.D * 2;
    AttentionSaved a;
    a.qkv = p;
    p += align256(3 * row);
    a.conv = a.qkv;
    if (d.taps > 0) {
        a.conv = p;
        p += align256(3 * row);
    }
    a.o = p;
    a.lse = reinterpret_cast<float*>(p + align256(row));
    return a;
}

// y [rows, D] = attention(x); residual != nullptr: y = residual + attention(x)
int attention_forward(const Dims& d, const void* x, const AttentionWeights& w, const AttentionSaved& a, void* y, void* residual,
                      int first, cudaStream_t s) {
    const int R = d.rows(), D = d.D;
    int rc = product(d, R, 3 * D, D, x, w.w_qkv, nullptr, a.qkv, GEMM_NONE, nullptr, first ? 0 : kChainDependent, s);
    if (rc == TMW_OK && d.taps > 0) rc = launch_dwconv(d.dtype, d.B, d.L, 3 * D, d.taps, a.qkv, w.conv, 3, a.conv, s, true);
    if (rc != TMW_OK) return rc;
    const tmw_prefill_desc c = core_desc(d);
    const char *q = a.conv, *k = q + 2ll * D, *v = q + 4ll * D;
    const bool link = prefill_tc_supports(c, q, k, v, a.o);
    if (d.block > 0) rc = prefill_block_sparse(&c, d.block, q, k, v, a.o, a.lse, s, kChainLink);
    else if (link) rc = launch_prefill_tc(c, q, k, v, a.o, s, 0, a.lse, nullptr, kChainLink);
    else rc = tmw_prefill_lse(&c, q, k, v, a.o, a.lse, s);
    if (rc != TMW_OK) return rc;
    return product(d, R, D, D, a.o, w.w_out, nullptr, y, residual != nullptr ? GEMM_ADD : GEMM_NONE, residual,
                   link ? kChainDependent : 0, s);
}

struct AttentionScratch {
    char *d_o, *d_conv, *d_qkv;  // [rows, D], [rows, 3D] (only with convolutions), [rows, 3D]
    float* d_taps;               // [3D, taps]
};

// dx = gradient of x given dy; weight gradients through `pending`; none of what is not wanted (dx, g.*: nullptr)
int attention_backward(const Dims& d, const void* x, const AttentionWeights& w, const AttentionSaved& a, const void* dy, void* dx,
                       const AttentionGrads& g, const AttentionScratch& t, Pending& pending, bool first, cudaStream_t s) {
    const int R = d.rows(), D = d.D;
    const bool through = dx != nullptr || g.w_qkv != nullptr || g.conv[0] != nullptr || g.conv[1] != nullptr || g.conv[2] != nullptr;
    const int link = first ? 0 : kChainDependent;
    int rc = TMW_OK;
    if (through) rc = input_grad(d, R, D, D, dy, w.w_out, t.d_o, GEMM_NONE, nullptr, link, s);
    if (rc == TMW_OK && g.w_out != nullptr) rc = pending.weight_grad(d, R, D, D, dy, a.o, g.w_out, through ? kChainDependent : link, s);
    if (rc != TMW_OK || !through) return rc;
    const tmw_prefill_desc c = core_desc(d);
    const char *q = a.conv, *k = q + 2ll * D, *v = q + 4ll * D;
    char *dq = d.taps > 0 ? t.d_conv : t.d_qkv, *dk = dq + 2ll * D, *dv = dq + 4ll * D;
    rc = d.block > 0 ? tmw_prefill_block_sparse_backward(&c, d.block, q, k, v, a.o, t.d_o, a.lse, dq, dk, dv, s)
                     : tmw_prefill_backward(&c, q, k, v, a.o, t.d_o, a.lse, dq, dk, dv, s);
    if (rc == TMW_OK && d.taps > 0) {
        TMW_CUDA_TRY(cudaMemsetAsync(t.d_taps, 0, (size_t)3 * D * d.taps * sizeof(float), s));
        rc = launch_dwconv_backward(d.dtype, d.B, d.L, 3 * D, d.taps, a.qkv, w.conv, 3, dq, t.d_qkv, t.d_taps, s);
        for (int i = 0; i < 3; ++i)
            if (g.conv[i] != nullptr) pending.sums.add(t.d_taps + (int64_t)i * D * d.taps, g.conv[i], (int64_t)D * d.taps, 1);
    }
    // (the kernels in front take no part in chains: an ordinary launch behind them)
    if (rc == TMW_OK && dx != nullptr) rc = input_grad(d, R, D, 3 * D, t.d_qkv, w.w_qkv, dx, GEMM_NONE, nullptr, 0, s);
    if (rc == TMW_OK && g.w_qkv != nullptr)
        rc = pending.weight_grad(d, R, 3 * D, D, t.d_qkv, x, g.w_qkv, dx != nullptr ? kChainDependent : 0, s);
    return rc;
}

// ---- the whole model -----------------------------------------------------------------------------------------
struct LayerSaved {
    char *x, *y1, *x2, *y2, *pre, *f;
    AttentionSaved attn;
};
int64_t layer_saved_bytes(const Dims& d) {
    const int64_t row = (int64_t)d.rows() * 2;
    return 4 * align256(row * d.D) + 2 * align256(row * d.F) + attention_saved_bytes(d);
}
LayerSaved layer_saved(const Dims& d, char* p) {
    const int64_t row = (int64_t)d.rows() * 2;
    LayerSaved l;
    char** parts[] = {&l.x, &l.y1, &l.x2, &l.y2};
    for (char** q : parts) {
        *q = p;
        p += align256(row * d.D);
    }
    l.pre = p;
    l.f = p + align256(row * d.F);
    l.attn = attention_saved(d, p + 2 * align256(row * d.F));
    return l;
}
int64_t stack_saved_bytes(const Dims& d, int layers) {  // layers, then the last residual stream and its norm
    return layers * layer_saved_bytes(d) + 2 * align256((int64_t)d.rows() * 2 * d.D);
}

struct StackScratch {
    char *g, *g2, *dy, *pre;
    AttentionScratch attn;
    float *norm_parts[4];
    char* partial;
    int64_t room;  // of `partial` for the split products; behind it the column sums of fc1's bias
    int* owner;
    float* acc;
    int64_t total;
};
StackScratch stack_scratch(const Dims& d, int vocab, int tokens, char* base) {
    StackScratch t;
    int64_t at = 0;
    auto take = [&](int64_t bytes) {
        char* p = base + at;
        at += align256(bytes);
        return p;
    };
    const int64_t R = d.rows(), row = R * 2;
    t.g = take(row * d.D);
    t.g2 = take(row * d.D);
    t.dy = take(row * d.D);
    t.pre = take(row * d.F);
    t.attn.d_o = t.dy;  // (dy is used up when d_o is written, and d_o when dy is written again)
    t.attn.d_qkv = take(3 * row * d.D);
    t.attn.d_conv = d.taps > 0 ? take(3 * row * d.D) : nullptr;
    t.attn.d_taps = reinterpret_cast<float*>(take((int64_t)3 * d.D * (d.taps > 0 ? d.taps : 1) * 4));
    for (float*& p : t.norm_parts) p = reinterpret_cast<float*>(take((int64_t)norm_bwd_blocks(R) * d.D * 4));
    const int64_t layer = 2 * split_room(d, d.F, d.D) + split_room(d, d.D, d.D) + split_room(d, 3 * d.D, d.D);
    const int64_t head = split_room(d, vocab, d.D);
    t.room = layer > head ? layer : head;
    t.partial = take(t.room + (int64_t)colsum_strips((int)R) * d.F * 4);
    t.owner = reinterpret_cast<int*>(take((int64_t)vocab * 4));
    t.acc = reinterpret_cast<float*>(t.partial);  // (the partial results are used up by then)
    const int64_t acc = (int64_t)d.B * tokens * d.D * 4;
    if (acc > t.room) t.acc = reinterpret_cast<float*>(take(acc));
    t.total = at;
    return t;
}

Dims dims_of(const tmw_stack_desc& k, int tokens) {
    Dims d;
    d.dtype = k.dtype; d.B = k.batch; d.L = tokens + k.n_persistent; d.H = k.heads; d.dh = k.head_dim; d.D = k.d_model;
    d.F = k.d_ff; d.np = k.n_persistent; d.window = k.window; d.block = k.block_size; d.taps = k.conv_taps;
    d.scale = 0.f; d.eps = k.eps;
    return d;
}

int validate_train(const tmw_stack_desc* d, int tokens) {
    if (d == nullptr || tokens <= 0) return TMW_ERR_INVALID_ARGUMENT;
    if (d->dtype != TMW_BF16 && d->dtype != TMW_F16) return TMW_ERR_UNSUPPORTED;
    if (d->batch <= 0 || d->layers < 1 || d->heads <= 0 || d->head_dim <= 0 || d->head_dim % 8 != 0 || d->d_ff <= 0 ||
        d->d_ff % 8 != 0 || d->vocab <= 0 || d->vocab % 8 != 0 || tokens > d->max_positions || d->n_persistent < 0 ||
        d->window < 0 || d->block_size < 0 || d->conv_taps < 0 || d->conv_taps > 8 || !(d->eps >= 0.f) ||
        d->d_model != d->heads * d->head_dim)
        return TMW_ERR_INVALID_ARGUMENT;
    if (d->d_model > 2048) return TMW_ERR_UNSUPPORTED;
    if ((int64_t)d->batch * (tokens + d->n_persistent) >= 0x7fffffff / 8) return TMW_ERR_TOO_LARGE;
    return TMW_OK;
}

int validate_blocks(const tmw_stack_desc& d, const tmw_block* blocks) {
    if (blocks == nullptr) return TMW_ERR_INVALID_ARGUMENT;
    for (int l = 0; l < d.layers; ++l) {
        const tmw_block& b = blocks[l];
        const void* need[] = {b.norm_attn, b.w_qkv, b.w_out, b.norm_mlp, b.w_fc1, b.w_fc2};
        for (const void* q : need)
            if (q == nullptr || !aligned16(q)) return TMW_ERR_INVALID_ARGUMENT;
        if (d.conv_taps > 0 && (b.conv_q == nullptr || b.conv_k == nullptr || b.conv_v == nullptr)) return TMW_ERR_INVALID_ARGUMENT;
    }
    return TMW_OK;
}

AttentionWeights weights_of(const tmw_block& b) { return {b.w_qkv, b.w_out, {b.conv_q, b.conv_k, b.conv_v}}; }

}  // namespace
}  // namespace tmw

using namespace tmw;

extern "C" size_t tmw_stack_train_saved(const tmw_stack_desc* desc, int32_t tokens) {
    if (validate_train(desc, tokens) != TMW_OK) return 0;
    return (size_t)stack_saved_bytes(dims_of(*desc, tokens), desc->layers);
}
extern "C" size_t tmw_stack_train_scratch(const tmw_stack_desc* desc, int32_t tokens) {
    if (validate_train(desc, tokens) != TMW_OK) return 0;
    return (size_t)stack_scratch(dims_of(*desc, tokens), desc->vocab, tokens, nullptr).total;
}

extern "C" int tmw_stack_train_forward(const tmw_stack_desc* desc, const tmw_block* blocks, const int64_t* token_ids, int32_t tokens,
                                       void* logits, void* saved, size_t saved_bytes, void* stream) {
    int rc = validate_train(desc, tokens);
    if (rc == TMW_OK) rc = validate_blocks(*desc, blocks);
    if (rc != TMW_OK) return rc;
    const tmw_stack_desc& k = *desc;
    const void* need[] = {token_ids, logits, saved, k.embed_tokens, k.embed_positions, k.norm, k.head};
    for (const void* q : need)
        if (q == nullptr || !aligned16(q)) return TMW_ERR_INVALID_ARGUMENT;
    if (k.n_persistent > 0 && (k.persistent == nullptr || !aligned16(k.persistent))) return TMW_ERR_INVALID_ARGUMENT;
    const Dims d = dims_of(k, tokens);
    if (saved_bytes < (size_t)stack_saved_bytes(d, k.layers)) return TMW_ERR_TOO_LARGE;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int R = d.rows(), D = d.D, F = d.F;
    char* base = static_cast<char*>(saved);
    auto layer = [&](int l) { return layer_saved(d, base + l * layer_saved_bytes(d)); };
    char* x_last = base + k.layers * layer_saved_bytes(d);
    char* y_last = x_last + align256((int64_t)R * 2 * D);
    rc = launch_embed_seq(k, token_ids, tokens, blocks[0].norm_attn, layer(0).x, layer(0).y1, s);
    for (int l = 0; l < k.layers && rc == TMW_OK; ++l) {
        const tmw_block& b = blocks[l];
        const LayerSaved a = layer(l);
        rc = attention_forward(d, a.y1, weights_of(b), a.attn, a.x2, a.x, l == 0, s);
        if (rc == TMW_OK) rc = launch_add_rmsnorm(d.dtype, R, D, a.x2, nullptr, b.norm_mlp, d.eps, nullptr, a.y2, s, true);
        if (rc == TMW_OK) rc = product(d, R, F, D, a.y2, b.w_fc1, b.b_fc1, a.f, GEMM_GELU_KEEP, a.pre, kChainDependent, s);
        const bool more = l + 1 < k.layers;
        char* x = more ? layer(l + 1).x : x_last;
        if (rc == TMW_OK) rc = product(d, R, D, F, a.f, b.w_fc2, b.b_fc2, x, GEMM_ADD, a.x2, kChainDependent, s);
        if (rc == TMW_OK)
            rc = launch_add_rmsnorm(d.dtype, R, D, x, nullptr, more ? blocks[l + 1].norm_attn : k.norm, d.eps, nullptr,
                                    more ? layer(l + 1).y1 : y_last, s, true);
    }
    return rc != TMW_OK ? rc : product(d, R, k.vocab, D, y_last, k.head, nullptr, logits, GEMM_NONE, nullptr, kChainDependent, s);
}

extern "C" int tmw_stack_train_backward(const tmw_stack_desc* desc, const tmw_block* blocks, const tmw_stack_grads* grads,
                                        const tmw_block_grads* block_grads, const int64_t* token_ids, int32_t tokens,
                                        const void* d_logits, const void* saved, void* scratch, size_t scratch_bytes, void* stream) {
    int rc = validate_train(desc, tokens);
    if (rc == TMW_OK) rc = validate_blocks(*desc, blocks);
    if (rc != TMW_OK) return rc;
    if (grads == nullptr || block_grads == nullptr || token_ids == nullptr || d_logits == nullptr || saved == nullptr ||
        scratch == nullptr || !aligned16(d_logits) || !aligned16(scratch))
        return TMW_ERR_INVALID_ARGUMENT;
    const tmw_stack_desc& k = *desc;
    const Dims d = dims_of(k, tokens);
    const StackScratch t = stack_scratch(d, k.vocab, tokens, static_cast<char*>(scratch));
    if (scratch_bytes < (size_t)t.total) return TMW_ERR_TOO_LARGE;
    // Where gradients go, before anything is launched: products and the embedding's kernels write 16 bytes at a time, sums of
    // partial results 8.
    auto written = [](const void* q, uintptr_t bytes) { return q != nullptr && (reinterpret_cast<uintptr_t>(q) & (bytes - 1)) == 0; };
    auto optional = [&](const void* q) { return q == nullptr || written(q, 8); };
    bool ok = aligned16(saved) && written(grads->embed_tokens, 16) && written(grads->head, 16) && written(grads->embed_positions, 16) &&
              (k.n_persistent == 0 || written(grads->persistent, 16)) && written(grads->norm, 8);
    for (int l = 0; l < k.layers && ok; ++l) {
        const tmw_block_grads& q = block_grads[l];
        for (const void* w : {q.w_qkv, q.w_out, q.w_fc1, q.w_fc2}) ok = ok && written(w, 16);
        for (const void* n : {q.norm_attn, q.norm_mlp}) ok = ok && written(n, 8);
        for (const void* o : {q.b_fc1, q.b_fc2}) ok = ok && optional(o);
        for (const void* o : {q.conv_q, q.conv_k, q.conv_v}) ok = ok && (k.conv_taps == 0 || optional(o));
    }
    if (!ok) return TMW_ERR_INVALID_ARGUMENT;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int R = d.rows(), D = d.D, F = d.F, V = k.vocab;
    char* base = static_cast<char*>(const_cast<void*>(saved));
    char* x_last = base + k.layers * layer_saved_bytes(d);
    char* y_last = x_last + align256((int64_t)R * 2 * D);
    Pending pending;
    pending.base = t.partial;
    pending.room = t.room;
    const int blocks_n = norm_bwd_blocks(R), strips = colsum_strips(R);
    // colsum_parts: column sums of t.g, the gradient of fc2's bias in the layer below
    auto norm_bwd = [&](const void* dy, const void* x, const void* gain, const void* add, void* out, float* dgain_part, float* sum_part,
                        void* dgain) {
        NormBwd n;
        n.dy = dy; n.x = x; n.gain = gain; n.add = add; n.out = out; n.dgain_part = dgain_part; n.sum_part = sum_part;
        n.rows = R; n.dim = D; n.eps = d.eps;
        const int st = launch_rmsnorm_bwd(d.dtype, n, s);
        if (st == TMW_OK) pending.sums.add(dgain_part, dgain, D, blocks_n);
        return st;
    };

    rc = input_grad(d, R, D, V, d_logits, k.head, t.dy, GEMM_NONE, nullptr, 0, s);
    if (rc == TMW_OK) rc = pending.weight_grad(d, R, V, D, d_logits, y_last, grads->head, kChainDependent, s);
    if (rc == TMW_OK) rc = norm_bwd(t.dy, x_last, k.norm, nullptr, t.g, t.norm_parts[0], t.norm_parts[1], grads->norm);
    if (rc == TMW_OK) rc = pending.flush(d, s);
    for (int l = k.layers - 1; l >= 0 && rc == TMW_OK; --l) {
        const tmw_block& b = blocks[l];
        const tmw_block_grads& q = block_grads[l];
        const LayerSaved a = layer_saved(d, base + l * layer_saved_bytes(d));
        if (q.b_fc2 != nullptr) pending.sums.add(t.norm_parts[1], q.b_fc2, D, blocks_n);
        rc = input_grad(d, R, F, D, t.g, b.w_fc2, t.pre, GEMM_GELU_GRAD, a.pre, kChainDependent, s);
        if (rc == TMW_OK) rc = pending.weight_grad(d, R, D, F, t.g, a.f, q.w_fc2, kChainDependent, s);
        if (rc == TMW_OK) rc = input_grad(d, R, D, F, t.pre, b.w_fc1, t.dy, GEMM_NONE, nullptr, kChainDependent, s);
        if (rc == TMW_OK) rc = pending.weight_grad(d, R, F, D, t.pre, a.y2, q.w_fc1, kChainDependent, s);
        if (rc == TMW_OK && q.b_fc1 != nullptr) {
            float* part = reinterpret_cast<float*>(t.partial + t.room);
            rc = launch_colsum(d.dtype, t.pre, part, R, F, s);
            pending.sums.add(part, q.b_fc1, F, strips);
        }
        if (rc == TMW_OK) rc = norm_bwd(t.dy, a.x2, b.norm_mlp, t.g, t.g2, t.norm_parts[2], nullptr, q.norm_mlp);
        const AttentionGrads ag = {q.w_qkv, q.w_out, {q.conv_q, q.conv_k, q.conv_v}};
        if (rc == TMW_OK)
            rc = attention_backward(d, a.y1, weights_of(b), a.attn, t.g2, t.dy, ag, t.attn, pending, false, s);
        // norm_parts[1] is still waiting to be added up here: the new column sums go to a buffer of their own
        if (rc == TMW_OK) rc = pending.flush(d, s);
        if (rc == TMW_OK) rc = norm_bwd(t.dy, a.x, b.norm_attn, t.g2, t.g, t.norm_parts[3], t.norm_parts[1], q.norm_attn);
    }
    if (rc == TMW_OK) rc = pending.flush(d, s);
    if (rc != TMW_OK) return rc;
    EmbedBwd e;
    e.g = t.g; e.ids = token_ids;
    e.d_tokens = grads->embed_tokens; e.d_positions = grads->embed_positions; e.d_persistent = grads->persistent;
    e.owner = t.owner; e.acc = t.acc;
    e.batch = d.B; e.seq = tokens; e.np = d.np; e.dim = D; e.vocab = V;
    if (grads->embed_tokens != grads->head)
        TMW_CUDA_TRY(cudaMemsetAsync(grads->embed_tokens, 0, (size_t)V * D * 2, s));
    if (tokens < k.max_positions)
        TMW_CUDA_TRY(cudaMemsetAsync(static_cast<char*>(grads->embed_positions) + (size_t)tokens * D * 2, 0,
                                     (size_t)(k.max_positions - tokens) * D * 2, s));
    return launch_embed_bwd(d.dtype, e, s);
}

// ---- the attention module alone --------------------------------------------------------------------------------
namespace {
Dims dims_of(const tmw_attention_desc& a) {
    Dims d = {};
    d.dtype = a.dtype; d.B = a.batch; d.L = a.rows; d.H = a.heads; d.dh = a.head_dim; d.D = a.heads * a.head_dim;
    d.np = a.n_persistent; d.window = a.window; d.block = a.block_size; d.taps = a.conv_taps; d.scale = a.scale;
    return d;
}
int validate_module(const tmw_attention_desc* a) {
    if (a == nullptr) return TMW_ERR_INVALID_ARGUMENT;
    if (a->dtype != TMW_BF16 && a->dtype != TMW_F16) return TMW_ERR_UNSUPPORTED;
    if (a->batch <= 0 || a->rows <= 0 || a->heads <= 0 || a->head_dim <= 0 || a->head_dim % 8 != 0 || a->n_persistent < 0 ||
        a->window < 0 || a->block_size < 0 || a->conv_taps < 0 || a->conv_taps > 8 || !(a->scale >= 0.f))
        return TMW_ERR_INVALID_ARGUMENT;
    if (a->n_persistent >= a->rows) return TMW_ERR_PERSISTENT_GE_LEN;
    if ((int64_t)a->batch * a->rows >= 0x7fffffff / 8) return TMW_ERR_TOO_LARGE;
    return TMW_OK;
}
struct ModuleScratch {
    AttentionScratch attn;
    char* partial;
    int64_t room, total;
};
ModuleScratch module_scratch(const Dims& d, char* base) {
    const int64_t row = (int64_t)d.rows() * d.D * 2;
    ModuleScratch t;
    t.attn.d_o = base;
    t.attn.d_qkv = base + align256(row);
    t.attn.d_conv = t.attn.d_qkv + align256(3 * row);
    char* p = t.attn.d_conv + (d.taps > 0 ? align256(3 * row) : 0);
    t.attn.d_taps = reinterpret_cast<float*>(p);
    t.partial = p + align256((int64_t)3 * d.D * 8 * 4);
    t.room = split_room(d, d.D, d.D) + split_room(d, 3 * d.D, d.D);
    t.total = t.partial - base + t.room;
    return t;
}
}  // namespace

extern "C" size_t tmw_attention_train_saved(const tmw_attention_desc* desc) {
    return validate_module(desc) != TMW_OK ? 0 : (size_t)attention_saved_bytes(dims_of(*desc));
}
extern "C" size_t tmw_attention_train_scratch(const tmw_attention_desc* desc) {
    return validate_module(desc) != TMW_OK ? 0 : (size_t)module_scratch(dims_of(*desc), nullptr).total;
}

extern "C" int tmw_attention_train_forward(const tmw_attention_desc* desc, const void* x, const void* w_qkv, const void* conv_q,
                                           const void* conv_k, const void* conv_v, const void* w_out, void* y, void* saved,
                                           size_t saved_bytes, void* stream) {
    const int rc = validate_module(desc);
    if (rc != TMW_OK) return rc;
    const void* need[] = {x, w_qkv, w_out, y, saved};
    for (const void* q : need)
        if (q == nullptr || !aligned16(q)) return TMW_ERR_INVALID_ARGUMENT;
    if (desc->conv_taps > 0 && (conv_q == nullptr || conv_k == nullptr || conv_v == nullptr)) return TMW_ERR_INVALID_ARGUMENT;
    const Dims d = dims_of(*desc);
    if (saved_bytes < (size_t)attention_saved_bytes(d)) return TMW_ERR_TOO_LARGE;
    const AttentionWeights w = {w_qkv, w_out, {conv_q, conv_k, conv_v}};
    return attention_forward(d, x, w, attention_saved(d, static_cast<char*>(saved)), y, nullptr, true, static_cast<cudaStream_t>(stream));
}

extern "C" int tmw_attention_train_backward(const tmw_attention_desc* desc, const void* x, const void* w_qkv, const void* conv_q,
                                            const void* conv_k, const void* conv_v, const void* w_out, const void* dy, const void* saved,
                                            void* dx, const tmw_block_grads* grads, void* scratch, size_t scratch_bytes, void* stream) {
    int rc = validate_module(desc);
    if (rc != TMW_OK) return rc;
    if (grads == nullptr) return TMW_ERR_INVALID_ARGUMENT;
    const void* need[] = {x, w_qkv, w_out, dy, saved, scratch};
    for (const void* q : need)
        if (q == nullptr || !aligned16(q)) return TMW_ERR_INVALID_ARGUMENT;
    const void* wanted[] = {dx, grads->w_qkv, grads->w_out, grads->conv_q, grads->conv_k, grads->conv_v};
    for (const void* q : wanted)
        if (!aligned16(q)) return TMW_ERR_INVALID_ARGUMENT;
    if (desc->conv_taps > 0 && (conv_q == nullptr || conv_k == nullptr || conv_v == nullptr)) return TMW_ERR_INVALID_ARGUMENT;
    const Dims d = dims_of(*desc);
    const ModuleScratch t = module_scratch(d, static_cast<char*>(scratch));
    if (scratch_bytes < (size_t)t.total) return TMW_ERR_TOO_LARGE;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    Pending pending;
    pending.base = t.partial;
    pending.room = t.room;
    const AttentionWeights w = {w_qkv, w_out, {conv_q, conv_k, conv_v}};
    const bool conv = desc->conv_taps > 0;
    const AttentionGrads g = {grads->w_qkv, grads->w_out, {conv ? grads->conv_q : nullptr, conv ? grads->conv_k : nullptr,
                                                           conv ? grads->conv_v : nullptr}};
    rc = attention_backward(d, x, w, attention_saved(d, static_cast<char*>(const_cast<void*>(saved))), dy, dx, g, t.attn, pending, true, s);
    return rc != TMW_OK ? rc : pending.flush(d, s);
}

extern "C" int tmw_cross_entropy(int32_t dtype, int32_t batch, int32_t tokens, int32_t n_persistent, int32_t vocab,
                                 const void* logits, const int64_t* labels, void* loss, float* stats, const void* grad,
                                 void* d_logits, void* stream) {
    if (dtype != TMW_BF16 && dtype != TMW_F16) return TMW_ERR_UNSUPPORTED;
    if (batch <= 0 || tokens <= 0 || n_persistent < 0 || vocab <= 0 || vocab % 8 != 0 || logits == nullptr || labels == nullptr ||
        stats == nullptr || (d_logits == nullptr ? loss == nullptr : grad == nullptr))
        return TMW_ERR_INVALID_ARGUMENT;
    if (!aligned16(logits) || !aligned16(d_logits)) return TMW_ERR_INVALID_ARGUMENT;
    if ((int64_t)batch * (tokens + n_persistent) > 0x7fffffff) return TMW_ERR_TOO_LARGE;
    CrossEntropy p;
    p.rows = batch * (tokens + n_persistent);
    p.logits = logits; p.labels = labels; p.loss = loss; p.grad = grad; p.d_logits = d_logits;
    p.count = stats; p.lse = stats + 4; p.row_loss = p.lse + p.rows;
    p.seq = tokens; p.np = n_persistent; p.vocab = vocab;
    p.status = device_status_word();
    if (p.status == nullptr) return TMW_ERR_CUDA;
    return launch_cross_entropy(dtype, p, d_logits != nullptr, static_cast<cudaStream_t>(stream));
}
