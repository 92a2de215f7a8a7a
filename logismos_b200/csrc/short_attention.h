// Attention over short texts from the fp32 sums of their q, k, v projection (short_attention.cu).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace lg {

constexpr int kShortText = 64;         // tokens of a text
constexpr int kShortBatchTokens = 128; // tokens of a batch: one row tile of the projections

// Heads of 128, halves rotated. sums fp32 [n_tokens][(n_heads + 2 n_kv) 128], without the bias; out bf16 [n_tokens][n_heads 128].
// zero: a buffer as large as sums that is left all zero.
struct ShortAttention {
  const float *sums, *bias, *cos, *sin;  // tables [max_pos][64]
  const int *positions, *cu;
  float* zero;
  __nv_bfloat16* out;
  int n_tokens, n_seqs, max_len, n_heads, n_kv, max_pos, causal;
  float scale;
  int* status;
};

uint32_t launch_short_attention(const ShortAttention& p, cudaStream_t stream);

}  // namespace lg
