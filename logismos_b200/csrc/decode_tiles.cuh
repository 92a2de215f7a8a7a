// Building blocks of the mma.sync attention kernels: a 16-row query tile as fragments, keys and values of 16 or more tokens
// in shared memory, scores, running softmax, products with the values. Templates on the head dimension HD.
#pragma once
#include "common.cuh"

namespace lg {

constexpr int kBlock = 16;  // tokens per KV block

// shared-memory address of 16-byte chunk `chunk` of row `row` in a [rows][HD] bf16 tile
template <int HD>
LG_DEVINL uint32_t tile_addr(uint32_t base, int row, int chunk) {
  return base + (uint32_t)row * (HD * 2) + (uint32_t)((chunk ^ (row & 7)) << 4);
}

// A fragments (16 rows x HD) of a query tile staged at `qbase`: qf[ks] covers k = 16ks..16ks+15
template <int HD>
LG_DEVINL void load_q_frags(uint32_t qbase, int lane, uint32_t (&qf)[HD / 16][4]) {
  const int mat = lane >> 3, r = lane & 7;
  const int row = r + 8 * (mat & 1);
#pragma unroll
  for (int ks = 0; ks < HD / 16; ++ks) ldmatrix_x4(qf[ks], tile_addr<HD>(qbase, row, 2 * ks + (mat >> 1)));
}

// s[t][:] = Q(16xHD) . K(tokens tok0+8t .. +7)^T for NT 8-token tiles of the K tile at kbase
template <int NT, int HD>
LG_DEVINL void qk_tile(const uint32_t (&qf)[HD / 16][4], uint32_t kbase, int tok0, int lane, float (&s)[NT][4]) {
  const int mat = lane >> 3, r = lane & 7;
#pragma unroll
  for (int t = 0; t < NT; ++t)
#pragma unroll
    for (int i = 0; i < 4; ++i) s[t][i] = 0.0f;
#pragma unroll
  for (int ks = 0; ks < HD / 16; ++ks) {
#pragma unroll
    for (int t = 0; t < NT; t += 2) {
      uint32_t b[4];
      ldmatrix_x4(b, tile_addr<HD>(kbase, tok0 + 8 * (t + (mat >> 1)) + r, 2 * ks + (mat & 1)));
      const uint32_t b0[2] = {b[0], b[1]}, b1[2] = {b[2], b[3]};
      mma_bf16_16816(s[t], qf[ks], b0, s[t]);
      mma_bf16_16816(s[t + 1], qf[ks], b1, s[t + 1]);
    }
  }
}

// o(16xHD) += P(16 x 8NT tokens) . V(tokens tok0.. , HD)
template <int NT, int HD>
LG_DEVINL void pv_tile(const float (&p)[NT][4], uint32_t vbase, int tok0, int lane, float (&o)[HD / 8][4]) {
  const int mat = lane >> 3, r = lane & 7;
#pragma unroll
  for (int kt = 0; kt < NT / 2; ++kt) {
    uint32_t a[4];
    a[0] = pack_bf16x2(p[2 * kt][0], p[2 * kt][1]);
    a[1] = pack_bf16x2(p[2 * kt][2], p[2 * kt][3]);
    a[2] = pack_bf16x2(p[2 * kt + 1][0], p[2 * kt + 1][1]);
    a[3] = pack_bf16x2(p[2 * kt + 1][2], p[2 * kt + 1][3]);
#pragma unroll
    for (int j = 0; j < HD / 8; j += 2) {
      uint32_t b[4];
      ldmatrix_x4_trans(b, tile_addr<HD>(vbase, tok0 + 16 * kt + 8 * (mat & 1) + r, j + (mat >> 1)));
      const uint32_t b0[2] = {b[0], b[1]}, b1[2] = {b[2], b[3]};
      mma_bf16_16816(o[j], a, b0, o[j]);
      mma_bf16_16816(o[j + 1], a, b1, o[j + 1]);
    }
  }
}

// Online softmax step over s (raw scores, -inf where masked) for the two rows a lane owns
// (g and g+8). m/l are running max (raw domain) and running sum; o is rescaled in place and
// s is overwritten with the probabilities exp2((s - m) * sl2).
template <int NT, int DT>
LG_DEVINL void softmax_step(float (&s)[NT][4], float (&m)[2], float (&l)[2], float (&o)[DT][4], float sl2) {
  float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll
  for (int t = 0; t < NT; ++t) {
    mx0 = fmaxf(mx0, fmaxf(s[t][0], s[t][1]));
    mx1 = fmaxf(mx1, fmaxf(s[t][2], s[t][3]));
  }
  mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 1));
  mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 2));
  mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 1));
  mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 2));
  const float mn0 = fmaxf(m[0], mx0), mn1 = fmaxf(m[1], mx1);
  const float use0 = (mn0 == -INFINITY) ? 0.0f : mn0, use1 = (mn1 == -INFINITY) ? 0.0f : mn1;
  const float a0 = exp2f((m[0] - use0) * sl2), a1 = exp2f((m[1] - use1) * sl2);
  float rs0 = 0.0f, rs1 = 0.0f;
#pragma unroll
  for (int t = 0; t < NT; ++t) {
    s[t][0] = exp2f((s[t][0] - use0) * sl2);
    s[t][1] = exp2f((s[t][1] - use0) * sl2);
    s[t][2] = exp2f((s[t][2] - use1) * sl2);
    s[t][3] = exp2f((s[t][3] - use1) * sl2);
    rs0 += s[t][0] + s[t][1];
    rs1 += s[t][2] + s[t][3];
  }
  l[0] = l[0] * a0 + rs0;
  l[1] = l[1] * a1 + rs1;
  m[0] = mn0;
  m[1] = mn1;
#pragma unroll
  for (int j = 0; j < DT; ++j) {
    o[j][0] *= a0; o[j][1] *= a0;
    o[j][2] *= a1; o[j][3] *= a1;
  }
}

// issue the cp.async copies of one 16-token block (K then V) of kv head `kvh` into a warp's stage
template <int HD>
LG_DEVINL void stage_block(uint32_t sbase, const __nv_bfloat16* kpool, const __nv_bfloat16* vpool,
                           int64_t phys_block, int row_elems, int kvh, int lane) {
  constexpr int CH = HD / 8;
  const __nv_bfloat16* kb = kpool + (phys_block * kBlock) * (int64_t)row_elems + kvh * HD;
  const __nv_bfloat16* vb = vpool + (phys_block * kBlock) * (int64_t)row_elems + kvh * HD;
#pragma unroll
  for (int i = 0; i < (kBlock * CH) / 32; ++i) {
    const int u = lane + 32 * i;
    const int row = u / CH, chunk = u % CH;
    cp_async16(tile_addr<HD>(sbase, row, chunk), kb + (int64_t)row * row_elems + chunk * 8);
    cp_async16(tile_addr<HD>(sbase + kBlock * HD * 2, row, chunk), vb + (int64_t)row * row_elems + chunk * 8);
  }
}

}  // namespace lg
