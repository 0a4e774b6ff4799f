// The float32 single track of a Pairformer block (single_attention.cu), as the block driver
// uses it: activations travel between the kernels as three bf16 pieces [3][rows][channels],
// products leave as float32 partial sums [splits][rows][channels] that the next row kernel adds.
#pragma once
#include <cuda_bf16.h>

#include "gemm.cuh"

namespace b200 {

constexpr int SINGLE_MAX_SPLITS = 8;

// x = (base + sum of partials); rows with row_mask == 0 become zero; x -> sum_out (may alias
// base); pieces of LN(x) (of x itself when scale is null) -> pieces. c <= 384.
struct RowArgs {
  const float* base;
  const float* partial;  // [splits][rows][c] or null
  int splits, rows, c;
  const float* row_mask;
  const void* scale;
  const void* bias;  // bf16
  float eps;
  float* sum_out;            // or null
  __nv_bfloat16* pieces;     // [3][rows][c] or null
};
int launch_row_norm(const RowArgs& a, cudaStream_t stream, bool pdl);

// How many ways K is split for a product of `tiles` output tiles and `kb` k steps.
int single_splits(int tiles, int kb);

// Bytes of scratch in which tma_weight may place a padded copy of a [k][n] weight.
size_t tma_weight_bytes(int k, int n);
// The weight itself when TMA can read it (16-byte aligned, n a multiple of 8), else a padded copy.
int tma_weight(const void* w, int k, int n, void* scratch, cudaStream_t stream, const void** out, long long* pitch);

// partial[split][rows][n] = pieces[3][rows][k] @ w[k][n]
int launch_linear_partial(const __nv_bfloat16* pieces, long long pitch, int rows, int k, const void* w, int n,
                          void* w_scratch, float* partial, int* splits, cudaStream_t stream, bool pdl);
// h pieces[3][rows][hidden] (row pitch `pitch`) = split(silu(x @ fc1) * (x @ fc2))
int launch_swiglu(const __nv_bfloat16* pieces, int rows, int k, const void* fc1, const void* fc2, int hidden,
                  void* w1_scratch, void* w2_scratch, __nv_bfloat16* h, long long pitch, cudaStream_t stream, bool pdl);

struct SingleAttentionWork {  // offsets inside the attention workspace
  size_t q, k, vt, g, bias, mask, ao, w[5], total;
};
SingleAttentionWork single_attention_work(int n, int c_s, int heads);
// The attention with pair bias in three steps, `work` carved by single_attention_work:
// q, k, v and the gate from the pieces of the query-side and key-side rows (does not read z);
int single_project(const b200tri_attention_pair_bias_args* a, const __nv_bfloat16* xq, const __nv_bfloat16* xk, uint8_t* work,
                   cudaStream_t stream);
// the projected pair bias and the mask row (reads z and the token mask only);
int single_pair_bias(const b200tri_attention_pair_bias_args* a, uint8_t* work, cudaStream_t stream, bool pdl);
// partial[splits][n][c_s] = (g * softmax(q k^T / sqrt(d) + bias + mask) v) @ Wo.
int single_attend(const b200tri_attention_pair_bias_args* a, uint8_t* work, float* partial, int* splits, cudaStream_t stream,
                  bool pdl);

}  // namespace b200
