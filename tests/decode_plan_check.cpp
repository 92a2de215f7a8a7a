// The layout of the one launch of a decode step, over the widths that it takes: parts of shared memory that are in use at the same time do not overlap, copies
// are aligned, every row of a matrix has its CTA, and contexts of any length fit the chunks.
#include <algorithm>
#include <cstdio>
#include <vector>

#include "decode_stack.h"
#include "int4_rows.h"

using namespace lg;
using namespace lg::stack;

struct Part { const char* name; size_t at, size; };

static bool apart(const std::vector<Part>& parts, size_t bytes, const char* when, const StackDims& d) {
  for (size_t i = 0; i < parts.size(); ++i) {
    const Part& a = parts[i];
    if (a.at + a.size > bytes) return std::printf("%s: %s ends at %zu of %zu (%d %d %d %d, %d rows)\n", when, a.name, a.at + a.size, bytes, d.hidden, d.n_heads, d.n_kv, d.inter, d.rows), false;
    for (size_t j = 0; j < i; ++j) {
      const Part& b = parts[j];
      if (a.at < b.at + b.size && b.at < a.at + a.size)
        return std::printf("%s: %s overlaps %s (%d %d %d %d, %d rows)\n", when, a.name, b.name, d.hidden, d.n_heads, d.n_kv, d.inter, d.rows), false;
    }
  }
  return true;
}

static bool check(const StackDims& d, const StackPlan& p) {
  const int H = d.hidden, I = d.inter, R = d.rows, rep = d.n_heads / d.n_kv, rp = R == 3 ? 4 : R, out_tiles = (p.out_rows + 15) / 16;
  auto rows = [](int n, int k) { return (size_t)n * (code_stride(k) + k / 16); };
  const Part qkv{"q, k, v", p.at[kQkv], rows(16 * p.qkv_tiles, H)}, out{"output", p.at[kOut], rows(p.out_rows, H)}, gate_up{"gate, up", p.at[kGateUp], rows(16 * p.gu_tiles, H)},
      down{"down", p.at[kDown], rows(p.out_rows, I)}, x{"activations", p.at_x, (size_t)R * (H + 32) * 2}, turn{"angles", p.at_turn, (size_t)8 * p.qkv_tiles * R * 16},
      sums{"sums of activations", p.at_sums, (size_t)H / 32 * 16}, wide{"activations of down", 0, (size_t)R * (I + 32) * 2 + (size_t)I / 32 * 16},
      cached{"cached blocks", p.at[kDown], (size_t)p.att_warps * kStage}, heads{"sums of cached blocks", p.at[kDown], (size_t)p.att_warps * rep * (kDim + 4 + 2) * 4},
      // the warps' sums, of a multiple of four warps, and the rooms in which chunks are put together ahead of the next ones
      part{"products", p.at_part, (size_t)round_up(p.warps, 4) * p.part_step}, merge{"merge", p.at_part, (size_t)p.warps * kDim * 4};
  if (p.part_step < (size_t)16 * std::max({p.qkv_tiles, p.gu_tiles, out_tiles}) * rp * 4 || p.part_step % 8 || p.warps % 2) return std::puts("step of the sums"), false;
  for (const Part& sum : {part, merge})
    if (!apart({qkv, out, gate_up, down, x, turn, sums, sum}, p.bytes, "weights", d) || !apart({qkv, out, gate_up, cached, x, turn, sums, sum}, p.bytes, "attention", d) ||
        !apart({qkv, out, gate_up, heads, x, turn, sums, sum}, p.bytes, "sums of the attention", d) || !apart({qkv, out, wide, down, x, turn, sums, sum}, p.bytes, "down", d))
      return false;
  for (int m = 0; m < kMats; ++m)
    if (p.at[m] % 128 || p.at_scales[m] % 16) return std::puts("alignment of a matrix"), false;
  for (uint32_t at : {p.at_x, p.at_turn, p.at_sums, p.at_part})
    if (at % 128) return std::puts("alignment"), false;
  if (p.bytes > 227 * 1024 - 1024) return std::puts("more shared memory than a CTA has beside the launch's static part"), false;
  if ((size_t)p.ctas * p.qkv_tiles < (size_t)(d.n_heads + 2 * d.n_kv) * 8 || (size_t)p.ctas * p.gu_tiles < (size_t)I / 8 || p.ctas * p.out_rows < H) return std::puts("rows without a CTA"), false;
  for (int ctx : {1, 15, 16, 17, 100, 1000, 4097, 40960, 1 << 20}) {
    const int chunk = stack_chunk(p, &ctx, 1);
    if (chunk % kTokens || (ctx + chunk - 1) / chunk > p.max_chunks || p.max_chunks > kMaxChunks) return std::printf("chunks of %d tokens for %d\n", chunk, ctx), false;
  }
  int ctx = 1;
  while (stack_contexts(p, &ctx, 1)) ctx += kTokens;
  if (ctx <= kMaxRounds * kTokens || stack_chunk(p, &ctx, 1) <= kMaxRounds * kTokens * p.att_warps) return std::printf("contexts end at %d tokens\n", ctx), false;
  return true;
}

int main() {
  int taken = 0;
  for (int ctas : {132, 148, 160})
    for (int heads = 1; heads <= 16; ++heads)
      for (int kv = 1; kv <= heads; ++kv)
        for (int inter = 128; inter <= 20480; inter += 128)
          for (int rows = 1; rows <= 5; ++rows) {
            const StackDims d{128 * heads, inter, heads, kv, rows};
            StackPlan p;
            if (heads % kv || !stack_plan(d, ctas, &p)) continue;
            ++taken;
            if (rows > kFewRows || !check(d, p)) return 1;
          }
  const StackDims own{1536, 8960, 12, 2, 4};
  StackPlan p;
  if (!stack_plan(own, 148, &p)) return std::puts("the decoder's own widths are refused"), 1;
  std::printf("%d layouts\n", taken);
  return taken > 5000 ? 0 : 1;
}
