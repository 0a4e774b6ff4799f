// Attention core of any head shape, with bf16 operands or float32 ones carried as bf16 pieces (att_split.cu).
#pragma once
#include <cuda_bf16.h>

#include "host.cuh"

namespace b200 {

// Mask-bias values stay finite: a row without a kept key is then still a uniform average. Dropped
// keys are clamped here, keys past the row's end lie below them.
constexpr float SPLIT_MASK_MIN = -1e30f, SPLIT_MASK_PAD = -3e30f;

struct AttSplitArgs {
  bool bf16;                           // q, k, vt, bias and o are bf16 (one piece); else float32
  int batch, n_i, n, heads, head_dim;  // batch items of n_i rows; n queries and keys per row
  const __nv_bfloat16* q;              // [pieces][batch * n_i][n][heads * head_dim]
  const __nv_bfloat16* k;
  const __nv_bfloat16* vt;             // [pieces][batch * n_i][heads * head_dim][v_ld], v_ld a multiple of 8
  long long v_ld;
  const void* bias;                    // [batch][heads][n][bias_ld], bias_ld a multiple of 8
  long long bias_ld;
  const float* mask_bias;              // [batch * n_i][mask_ld], mask_ld = n rounded up to 64
  long long mask_ld;
  float scale;                         // of q . k, in the one-row form
  void* o;                             // [batch * n_i][n][heads * head_dim]
  const float* gate;                   // one-row form: [n][heads * head_dim]
  __nv_bfloat16* pieces;               // one-row form: the output, o * gate as pieces [3][n][heads * head_dim]
  bool pdl;                            // the predecessor in the stream is a kernel of the library
};
int launch_att_split(const AttSplitArgs& a, cudaStream_t stream);

}  // namespace b200
