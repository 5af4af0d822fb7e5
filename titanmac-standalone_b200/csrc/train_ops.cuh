// Kernels of the training step (internal header; see train_ops.cu).
#pragma once

#include "tmw_common.cuh"

namespace tmw {

struct NormBwd {
    const void *dy, *x, *gain, *add;  // add: gradient of the residual branch, or nullptr
    void* out;
    float *dgain_part, *sum_part;  // [norm_bwd_blocks(rows)][dim]; sum_part (column sums of out) optional
    long long rows;
    int dim;
    float eps;
};
int norm_bwd_blocks(long long rows);
int launch_rmsnorm_bwd(int dtype, const NormBwd& p, cudaStream_t stream);  // dim <= 2048

int colsum_strips(int rows);
int launch_colsum(int dtype, const void* src, float* part, int rows, int cols, cudaStream_t stream);  // part: [strips][cols]

struct SumParts {
    static constexpr int kMost = 12;
    struct Item {
        const float* src;  // [parts][n]
        void* dst;         // [n], n a multiple of 4
        long long n;
        int parts;
    } item[kMost];
    int count = 0;
    void add(const float* src, void* dst, long long n, int parts) { item[count++] = Item{src, dst, n, parts}; }
};
int launch_sum_parts(int dtype, const SumParts& p, cudaStream_t stream);

struct CrossEntropy {
    const void *logits, *grad;
    const int64_t* labels;
    void *loss, *d_logits;
    float *row_loss, *lse, *count;
    int* status;
    int rows, seq, np, vocab;
};
int launch_cross_entropy(int dtype, const CrossEntropy& p, bool backward, cudaStream_t stream);

struct EmbedBwd {
    const void* g;
    const int64_t* ids;
    void *d_tokens, *d_positions, *d_persistent;  // d_tokens is added to; the others are written
    int* owner;                                   // [vocab]
    float* acc;                                   // [batch * seq][dim]
    int batch, seq, np, dim, vocab;
};
int launch_embed_bwd(int dtype, const EmbedBwd& p, cudaStream_t stream);

}  // namespace tmw
