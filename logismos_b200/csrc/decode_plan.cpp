// How the one launch of a decode step of few rows (decode_stack.cu) is laid out, and which steps it takes: arithmetic on the host.
#include <algorithm>

#include "decode_stack.h"
#include "int4_rows.h"

namespace lg {

using namespace stack;

bool stack_plan(const StackDims& d, int ctas, StackPlan* plan) {
  const int H = d.hidden, I = d.inter, R = d.rows;
  if (R < 1 || R > kFewRows || H % 256 || I % 256 || H / kDim > kMaxWarps || d.n_heads * kDim != H || d.n_kv < 1 || d.n_heads % d.n_kv || d.n_heads / d.n_kv > 8) return false;
  StackPlan p{};
  p.ctas = ctas;
  p.warps = H / kDim;
  auto share = [&](int n) { return (n + p.ctas - 1) / p.ctas; };
  p.qkv_tiles = share((d.n_heads + 2 * d.n_kv) * (kDim / 16));
  p.gu_tiles = share(I / 8);
  p.out_rows = share(H);
  p.max_chunks = std::max(1, std::min(kMaxChunks, p.ctas / (R * d.n_kv)));
  const int rp = R == 1 ? 1 : R == 2 ? 2 : 4, out_tiles = (p.out_rows + 15) / 16, rep = d.n_heads / d.n_kv;
  auto align = [](size_t v) { return (v + 127) & ~(size_t)127; };
  p.at[kGateUp] = 0;
  size_t at = align(std::max((size_t)16 * p.gu_tiles * row_bytes(H), (size_t)R * (I + 32) * 2 + (size_t)(I / 32) * 16));
  p.at[kDown] = (uint32_t)at;
  // cached blocks and the sums of their warps lie where the down projection's rows come next
  const size_t down = (size_t)p.out_rows * row_bytes(I), per_warp = std::max((size_t)kStage, (size_t)rep * (kDim + 6) * 4);
  p.att_warps = std::min(p.warps, std::max(2, (int)(down / per_warp)));
  at += align(std::max(down, p.att_warps * per_warp));
  p.at[kQkv] = (uint32_t)at;
  at += align((size_t)16 * p.qkv_tiles * row_bytes(H));
  p.at[kOut] = (uint32_t)at;
  at += align((size_t)p.out_rows * row_bytes(H));
  p.at_x = (uint32_t)at;
  at += align((size_t)R * (H + 32) * 2);
  p.at_turn = (uint32_t)at;
  at += align((size_t)8 * p.qkv_tiles * R * 16);
  p.at_sums = (uint32_t)at;
  at += align((size_t)(H / 32) * 16);
  p.at_part = (uint32_t)at;  // and the chunks that a CTA puts together
  p.part_step = (uint32_t)(16 * std::max({p.gu_tiles, p.qkv_tiles, out_tiles}) * rp * 4);
  at += align(std::max((size_t)round_up(p.warps, 4) * p.part_step, (size_t)p.warps * kDim * 4));
  p.bytes = (uint32_t)at;
  p.at_scales[kQkv] = p.at[kQkv] + 16 * p.qkv_tiles * code_stride(H);
  p.at_scales[kOut] = p.at[kOut] + p.out_rows * code_stride(H);
  p.at_scales[kGateUp] = 16 * p.gu_tiles * code_stride(H);
  p.at_scales[kDown] = p.at[kDown] + p.out_rows * code_stride(I);
  // tiles that end in rows which are not there read up to 15 rows on
  for (int m : {kOut, kDown}) {
    const int k = m == kOut ? H : I;
    p.bytes = std::max({p.bytes, p.at[m] + 16 * out_tiles * code_stride(k), p.at_scales[m] + 16 * out_tiles * (k / 16)});
  }
  const int threads = 32 * p.warps;  // one for each pair of q, k, v and for each value of the projections
  if (p.bytes > 226 * 1024 || 8 * p.qkv_tiles * R > threads || p.out_rows * R > threads || sizeof(StackLayer) / 8 > (size_t)threads) return false;
  *plan = p;
  return true;
}

int stack_chunk(const StackPlan& plan, const int32_t* ctx, int rows) {
  int longest = 1;
  for (int r = 0; r < rows; ++r) longest = std::max(longest, ctx[r]);
  const int least = (longest + plan.max_chunks - 1) / plan.max_chunks;
  return std::max(round_up(least, kTokens), kTokens * plan.att_warps);
}

bool stack_contexts(const StackPlan& plan, const int32_t* ctx, int rows) {
  return (stack_chunk(plan, ctx, rows) / kTokens + plan.att_warps - 1) / plan.att_warps <= kMaxRounds;
}

bool stack_blocks_apart(const int32_t* tables, int max_blocks, const int32_t* ctx, int rows) {
  for (int r = 0; r < rows; ++r) {
    const int last = (ctx[r] - 1) / kTokens;
    if (ctx[r] < 1 || last >= max_blocks) return false;
    for (int s = 0; s < rows; ++s)
      for (int b = 0; b < max_blocks && b * kTokens < ctx[s]; ++b)
        if (tables[(size_t)s * max_blocks + b] == tables[(size_t)r * max_blocks + last] && !(s == r && b == last)) return false;
  }
  return true;
}

size_t stack_words(const StackDims& d) {
  const size_t R = (size_t)d.rows, heads = (size_t)d.n_heads;
  return R * ((heads + 2 * d.n_kv) * (kDim / 2) + heads * kMaxChunks * (kDim + 2) + heads * (kDim / 2) + 2 * (size_t)d.hidden + d.inter / 2);
}

}  // namespace lg
