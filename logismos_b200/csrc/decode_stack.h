// All layers of a decode step of one to four sequences in one launch, for the int4 decoder (decode_stack.cu).
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace lg {

namespace stack {
constexpr int kDim = 128, kMaxWarps = 12, kMaxChunks = 32, kTokens = 16 /* of a cache block */, kStage = 2 * kTokens * kDim * 2;
enum { kQkv, kOut, kGateUp, kDown, kMats };

__host__ __device__ constexpr int round_up(int v, int to) { return (v + to - 1) / to * to; }
// a row of codes in shared memory: rows lie 16 bytes apart modulo the banks, so that eight rows' words of a group meet no conflict
__host__ __device__ constexpr int code_stride(int k) { return round_up(k / 2, 128) + 16; }
__host__ __device__ constexpr int row_bytes(int k) { return code_stride(k) + k / 16; }
}  // namespace stack

struct StackMat {
  const uint8_t* codes;  // [n][k / 2]
  const __half* scales;  // [n][k / 32]
};
struct StackLayer {  // an array of these on the device
  const float *norm1, *norm2, *bias;  // bias: of q | k | v
  StackMat qkv, out, gate_up, down;   // gate_up: 32 gate rows, then the 32 matching up rows
  __nv_bfloat16 *k_pool, *v_pool;
};

struct StackDims { int hidden, inter, n_heads, n_kv, rows; };  // heads of 128

// How a launch is laid out: what each of the CTAs takes of every matrix, and the shared memory for it.
struct StackPlan {
  int ctas, warps;         // a warp per 128 values of the hidden size
  int qkv_tiles, gu_tiles; // tiles of 16 weight rows (8 pairs) per CTA
  int out_rows;            // rows of the output and down projections per CTA
  int att_warps;           // warps of a CTA that take cache blocks
  int max_chunks;          // chunks of a context at most
  // offsets of the parts of shared memory: rows of q, k, v | output | gate, up | down and their scales, activations, angles of q, k, v, sums of activations, the warps' sums (part_step bytes each)
  uint32_t at[4], at_scales[4], at_x, at_turn, at_sums, at_part, part_step, bytes;
};
bool stack_plan(const StackDims& d, int ctas, StackPlan* plan);
// tokens per chunk of the longest of `rows` contexts
int stack_chunk(const StackPlan& plan, const int32_t* ctx, int rows);
// Contexts that the one launch reads faster than a launch per projection with its split over all SMs: here a warp requests a cache block when it has done with the one before, 1.2 to 1.7 us
// a round, and a CTA has as many warps for it as its shared memory holds blocks. Steps of 8 layers of 256 to 1536 values, 1 to 12 key heads, one to four rows, up to 32000 tokens, time against
// the other route's: 0.5 to 0.99 at up to 10 rounds, 0.94 to 1.10 at 12 and 13, 0.91 to 1.19 at 14, 0.92 to 1.7 at 18 to 32, up to 3.8 at more.
constexpr int kMaxRounds = 10;
bool stack_contexts(const StackPlan& plan, const int32_t* ctx, int rows);
// No row's new token goes to a block that another row, or another place of its own table, holds: blocks without a new token may be read before it is stored.
bool stack_blocks_apart(const int32_t* tables, int max_blocks, const int32_t* ctx, int rows);
// 64-bit words by which the CTAs of launches of up to d.rows rows pass on results; all zero before the first launch and after a failed one
size_t stack_words(const StackDims& d);
// Launches whose numbers, one per layer from 1 on, fit 32 bits. A model's count starts 64 short of it, so that the words are cleared soon and not after weeks.
inline uint32_t stack_most_launches(int n_layers) { return 0xffffffffu / (uint32_t)(n_layers > 0 ? n_layers : 1); }
inline uint32_t stack_first_count(int n_layers) { return stack_most_launches(n_layers) > 64 ? stack_most_launches(n_layers) - 64 : 0; }

constexpr size_t kStackCounts = 2;  // words of 64 bits for the three counts behind the others

struct StackArgs {
  StackDims d;
  const StackLayer* layers;
  int n_layers;
  float eps;
  float* x;  // [rows][hidden], in place
  const float *cos, *sin;  // [max_pos][64]
  const int* positions;
  int max_pos;
  const int64_t* slots;
  const int *ctx, *tables;
  int max_blocks, n_pool_blocks, chunk;
  unsigned long long* words;  // n_words = stack_words of the most rows
  size_t n_words;
  uint32_t* launches;         // how many went before since the words were zero; then the CTAs that met to clear them; then those of this launch that have read the first count
  uint32_t most_launches;     // whose numbers fit 32 bits: the next one clears the words
  int* status;
};
uint32_t launch_decode_stack(const StackArgs& a, const StackPlan& plan, cudaStream_t stream);

}  // namespace lg
