// int4 group-32 projections of one to four rows, for decode steps of that many sequences: the hybrid decoder's, and the decoder's where
// decode_stack.cu does not take a step (its width, long contexts of many key heads, blocks that sequences share).
//
// What bounds them is not the 1 to 16 MB of a matrix (0.2 to 2.4 us from HBM) but the length of a launch: start, dependency,
// one round of latency to memory, a warp's own chain of instructions, the sum over k. The fused-dequant tcgen05 kernel takes 7.6 us
// for 1536 x 1536 and 11.6 for 17920 x 1536 at one row, with its ring of roles and fp32 reductions that a second launch has to finish.
// So: no roles and no second launch. A warp takes 16 weight rows and a slice of k and requests it ahead of the
// dependency wait. Products on mma.sync m16n8k16 from the exact integers 136 + q, 32 values of a group in two instructions whose
// accumulators start at -136 times the group's sum of activations, so that the fp16 scale is applied to the finished group in
// fp32. The slices of a row meet in shared memory in a fixed order. The RMS norm ahead of a projection is computed by every
// CTA for itself (one row is 6 KB, read from L2), which is shorter than a launch of its own; so is the rotation of q and k with the
// store into the cache in the epilogue, where a warp has both halves of a head's pairs.
// Measured at one row, us: 1536 x 1536 4.0, 2048 x 1536 with its norm 4.8, 17920 x 1536 with norm and SwiGLU 10.6 (on the FMA
// units, 7.9 instructions per weight, 13.7; word by word, each load touching eight lines, 14.5), 1536 x 8960 7.3. A step of the 28-layer decoder, one /
// two / four / eight rows: 1.18 / 1.25 / 1.51 / 1.91 ms against 1.58 / 1.60 / 1.63 / 1.63 on the general route (the copies of the activations
// into shared memory grow with the rows), the 48-layer hybrid 1.91 / 2.13 / 2.49 / 3.28 against 2.44 / 2.48 / 2.53 / 2.61: hence four rows.
#include "int4_rows.h"

#include <algorithm>

#include "common.cuh"
#include "logismos_kernels.h"

namespace {

using namespace lg;

constexpr int kTileRows = 16, kMaxWarps = 18;
constexpr int kEpiHeads = 100;  // q, k and v heads: rotated and stored (DecodeHeads)

struct Params {
  const float *x, *gain;
  float eps;
  const __nv_bfloat16* a;
  int lda;
  const uint8_t* codes;
  const __half* scales;
  const float* bias;
  void* out;
  int n, k, ldc, epi, slices, tiles, rows;  // slices of k per tile of 16 weight rows, tiles per CTA at a time, activation rows
  DecodeHeads heads;                   // with kEpiHeads
};

// Weight rows g and g + 8 of a tile: consecutive ones; gated, a gate row and the matching up row 32 further on; heads, a row of
// the first half of a head and the one it is rotated with.
LG_DEVINL bool is_paired(int epi) { return epi == LG_EPI_SWIGLU || epi == kEpiHeads; }
LG_DEVINL int2 rows_of(const Params& p, int tile, int g) {
  int2 r;
  if (is_paired(p.epi)) {
    const int half = p.epi == kEpiHeads ? p.heads.dim >> 1 : 32, o = 8 * tile;
    r.x = o / half * 2 * half + o % half + g;
    r.y = r.x + half;
  } else {
    r.x = kTileRows * tile + g;
    r.y = r.x + 8;
  }
  return make_int2(min(r.x, p.n - 1), min(r.y, p.n - 1));  // what lies beyond is computed and not stored
}

// eight activations, rounded, in the order 0 4 1 5 2 6 3 7 of the nibble pairs; their sum over the four lanes of a group of 32
LG_DEVINL void stage8(const float (&v)[8], __nv_bfloat16* dst, float* sum, int lane, bool in) {
  float r[8], s = 0.0f;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    r[i] = __bfloat162float(__float2bfloat16_rn(v[i]));
    s += r[i];
  }
  if (in) *reinterpret_cast<uint4*>(dst) = make_uint4(pack_bf16x2(r[0], r[4]), pack_bf16x2(r[1], r[5]), pack_bf16x2(r[2], r[6]), pack_bf16x2(r[3], r[7]));
  s += __shfl_xor_sync(0xffffffffu, s, 1);
  s += __shfl_xor_sync(0xffffffffu, s, 2);
  if (in && (lane & 3) == 0) *sum = -136.0f * s;
}

// w[i] of lane t (of four) <-> w[t] of lane i
LG_DEVINL void transpose4(uint4& w, int t) {
  uint32_t a = __shfl_xor_sync(0xffffffffu, t & 1 ? w.x : w.y, 1), b = __shfl_xor_sync(0xffffffffu, t & 1 ? w.z : w.w, 1);
  if (t & 1) { w.x = a; w.z = b; } else { w.y = a; w.w = b; }
  a = __shfl_xor_sync(0xffffffffu, t & 2 ? w.x : w.z, 2);
  b = __shfl_xor_sync(0xffffffffu, t & 2 ? w.y : w.w, 2);
  if (t & 2) { w.x = a; w.y = b; } else { w.z = a; w.w = b; }
}

// CHUNK: blocks of four groups (128 values of k) whose weights a warp has in flight. Two where that leaves k to at most eight
// warps: 24 warps fit an SM then, and each waits on its own chain of products most of the time (17920 x 1536: 13.1 us with four, 10.6 with two).
template <int CHUNK>
__global__ void __launch_bounds__(CHUNK == 2 ? 256 : 32 * kMaxWarps, CHUNK == 2 ? 3 : 1)
int4_rows_kernel(const Params p) {
  lg::pdl_trigger();
  extern __shared__ __align__(16) uint8_t smem[];
  const int n_groups = p.k >> 5, ld = p.k + 32;  // rows lie 64 bytes apart modulo the banks
  float* sums = reinterpret_cast<float*>(smem);                                          // [n_groups][8]: -136 sum of x
  __nv_bfloat16* xs = reinterpret_cast<__nv_bfloat16*>(smem + (size_t)n_groups * 8 * 4);  // [rows][ld]
  __shared__ float part[kMaxWarps][kTileRows][8];
  __shared__ float red[kMaxWarps][kFewRows];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, n_warps = blockDim.x >> 5, g = lane >> 2, t = lane & 3;
  const int slice = warp % p.slices, blocks = n_groups >> 2, q0 = slice * blocks / p.slices, q1 = (slice + 1) * blocks / p.slices;
  const int n_sets = (p.n + kTileRows * p.tiles - 1) / (kTileRows * p.tiles);  // sets of `tiles` tiles
  // a lane reads whole groups, 16 bytes at a time, of rows g and g + 8: group t of each block of four; the transposition
  // then leaves it word t of all four, since the products of one instruction have to lie in one group
  uint4 lo[CHUNK], hi[CHUNK];
  uint2 slo[CHUNK], shi[CHUNK];  // scales of a block's four groups
  int2 at_row;  // groups ahead of rows g and g + 8
  auto aim = [&](int set) {
    at_row = rows_of(p, set * p.tiles + warp / p.slices, g);
    at_row.x *= n_groups;
    at_row.y *= n_groups;
  };
  auto request = [&](int i, int q) {  // block q to place i
    if (q >= q1) return;
    const uint4* codes = reinterpret_cast<const uint4*>(p.codes);
    const uint2* scales = reinterpret_cast<const uint2*>(p.scales);
    lo[i] = __ldg(codes + (at_row.x + 4 * q + t));
    hi[i] = __ldg(codes + (at_row.y + 4 * q + t));
    slo[i] = __ldg(scales + ((at_row.x >> 2) + q));
    shi[i] = __ldg(scales + ((at_row.y >> 2) + q));
  };
  aim(blockIdx.x);
#pragma unroll
  for (int i = 0; i < CHUNK; ++i) request(i, q0 + i);  // the weights are static
  if (p.x)
    for (int j = threadIdx.x * 32; j < p.k; j += blockDim.x * 32) asm volatile("prefetch.global.L1 [%0];\n" ::"l"(p.gain + j));
  lg::pdl_wait();

  // activations as bf16 in shared memory, four threads per group of 32, all rows at a time
  const int per_row = p.k >> 3, items = p.rows * per_row;
  if (p.x) {
    const int team = max(1, n_warps / p.rows), teams = n_warps / team, member = warp % team;  // warps of a row
    for (int r = warp / team; r < p.rows && warp / team < teams; r += teams) {
      const float* src = p.x + (size_t)r * p.k;
      float ss = 0.0f;
#pragma unroll 4
      for (int j = (member * 32 + lane) * 4; j < p.k; j += team * 128) {
        const float4 v = *reinterpret_cast<const float4*>(src + j);
        ss += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
      }
      ss = warp_sum(ss);
      if (lane == 0) red[member][r] = ss;
    }
    __syncthreads();
#pragma unroll 2
    for (int e0 = 0; e0 < items; e0 += blockDim.x) {
      const int e = e0 + threadIdx.x;
      if (e0 + (int)(threadIdx.x & ~31u) >= items) break;  // whole warps
      const bool in = e < items;  // a group's four lanes agree
      const int r = in ? e / per_row : 0, j = in ? (e - r * per_row) * 8 : 0;
      const float4* src = reinterpret_cast<const float4*>(p.x + (size_t)r * p.k + j);
      const float4* gain = reinterpret_cast<const float4*>(p.gain + j);
      const float4 a = src[0], b = src[1], ga = __ldg(gain), gb = __ldg(gain + 1);
      float sum = 0.0f;
      for (int w = 0; w < team; ++w) sum += red[w][r];
      const float inv = 1.0f / sqrtf(sum / (float)p.k + p.eps);
      const float v[8] = {a.x * inv * ga.x, a.y * inv * ga.y, a.z * inv * ga.z, a.w * inv * ga.w, b.x * inv * gb.x, b.y * inv * gb.y, b.z * inv * gb.z, b.w * inv * gb.w};
      stage8(v, xs + (size_t)r * ld + j, sums + (size_t)(j >> 5) * 8 + r, lane, in);
    }
  } else {
#pragma unroll 4
    for (int e0 = 0; e0 < items; e0 += blockDim.x) {
      const int e = e0 + threadIdx.x;
      if (e0 + (int)(threadIdx.x & ~31u) >= items) break;
      const bool in = e < items;
      const int r = in ? e / per_row : 0, j = in ? (e - r * per_row) * 8 : 0;
      const uint4 w = *reinterpret_cast<const uint4*>(p.a + (size_t)r * p.lda + j);
      const float2 e0v = unpack_bf16x2(w.x), e1 = unpack_bf16x2(w.y), e2 = unpack_bf16x2(w.z), e3 = unpack_bf16x2(w.w);
      const float v[8] = {e0v.x, e0v.y, e1.x, e1.y, e2.x, e2.y, e3.x, e3.y};
      stage8(v, xs + (size_t)r * ld + j, sums + (size_t)(j >> 5) * 8 + r, lane, in);
    }
  }
  __syncthreads();

  const uint32_t mask = opaque(0x000f000fu), flip = opaque(0x43084308u);
  const bool col = g < p.rows;  // the activation row of this lane's B values
  const __nv_bfloat16* xg = xs + (size_t)(col ? g : 0) * ld + 8 * t;
  for (int set = blockIdx.x; set < n_sets; set += gridDim.x) {
    float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};  // rows g, g + 8; columns 2 t, 2 t + 1: as mma leaves them
    for (int q = q0; q < q1; q += CHUNK) {
      if (q != q0) {
#pragma unroll
        for (int i = 0; i < CHUNK; ++i) request(i, q + i);
      }
#pragma unroll
      for (int i = 0; i < CHUNK; ++i) {
        if (q + i >= q1) break;
        transpose4(lo[i], t);
        transpose4(hi[i], t);
        const uint32_t wl[4] = {lo[i].x, lo[i].y, lo[i].z, lo[i].w}, wh[4] = {hi[i].x, hi[i].y, hi[i].z, hi[i].w};
        auto pair = [=](uint32_t w, int n) { return and_xor(w >> (4 * n), mask, flip); };  // nibbles n, n + 4 as 136 + q
        uint4 x[4];
        float d[4][4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {  // four groups side by side: an instruction's result is the next one's accumulator
          const int group = 4 * (q + i) + j;
          x[j] = make_uint4(0u, 0u, 0u, 0u);
          if (col) x[j] = *reinterpret_cast<const uint4*>(xg + (size_t)group * 32);
          const float2 c = *reinterpret_cast<const float2*>(sums + (size_t)group * 8 + 2 * t);  // columns beyond the rows hold anything and are not stored
          d[j][0] = d[j][2] = c.x;
          d[j][1] = d[j][3] = c.y;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint32_t a[4] = {pair(wl[j], 0), pair(wh[j], 0), pair(wl[j], 1), pair(wh[j], 1)}, b[2] = {x[j].x, x[j].y};
          mma_bf16_16816(d[j], a, b, d[j]);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint32_t a[4] = {pair(wl[j], 2), pair(wh[j], 2), pair(wl[j], 3), pair(wh[j], 3)}, b[2] = {x[j].z, x[j].w};
          mma_bf16_16816(d[j], a, b, d[j]);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint32_t sl2 = j < 2 ? slo[i].x : slo[i].y, sh2 = j < 2 ? shi[i].x : shi[i].y;
          const float sl = __half2float(__ushort_as_half((unsigned short)(j & 1 ? sl2 >> 16 : sl2 & 0xffffu))), sh = __half2float(__ushort_as_half((unsigned short)(j & 1 ? sh2 >> 16 : sh2 & 0xffffu)));
          acc[0] = fmaf(sl, d[j][0], acc[0]);
          acc[1] = fmaf(sl, d[j][1], acc[1]);
          acc[2] = fmaf(sh, d[j][2], acc[2]);
          acc[3] = fmaf(sh, d[j][3], acc[3]);
        }
      }
    }
    if (set + (int)gridDim.x < n_sets) {  // on the way while the slices are added
      aim(set + gridDim.x);
#pragma unroll
      for (int i = 0; i < CHUNK; ++i) request(i, q0 + i);
    }
    if (set != blockIdx.x) __syncthreads();                        // the last set's sums have been read
    *reinterpret_cast<float2*>(&part[warp][g][2 * t]) = make_float2(acc[0], acc[1]);
    *reinterpret_cast<float2*>(&part[warp][g + 8][2 * t]) = make_float2(acc[2], acc[3]);
    __syncthreads();
    const bool paired = is_paired(p.epi);
    const int per = paired ? 8 : kTileRows;  // outputs (or pairs of them) of a tile and activation row
    for (int e = threadIdx.x; e < p.tiles * per * p.rows; e += blockDim.x) {
      const int i = e % per, r = e / per % p.rows, m = e / (per * p.rows), at = (set * p.tiles + m) * per + i;  // output column
      if (at >= (paired ? p.n >> 1 : p.n)) continue;
      float v = 0.0f, u = 0.0f;
      for (int w = 0; w < p.slices; ++w) {
        v += part[m * p.slices + w][i][r];
        if (paired) u += part[m * p.slices + w][i + 8][r];
      }
      if (p.epi == kEpiHeads) {
        const DecodeHeads& h = p.heads;
        const int half = h.dim >> 1, head = at / half, o = at - head * half, pos = h.positions[r];
        const int64_t slot = h.slots[r];
        if (pos < 0 || pos >= h.max_pos || slot < 0 || slot >= h.n_slots) {
          if (h.status) atomicExch(h.status, 1);
          continue;
        }
        // as the projection leaves them everywhere else: one rounding ahead of the rotation
        const int c = head * h.dim + o;
        v = __bfloat162float(__float2bfloat16_rn(v + (p.bias ? __ldg(p.bias + c) : 0.0f)));
        u = __bfloat162float(__float2bfloat16_rn(u + (p.bias ? __ldg(p.bias + c + half) : 0.0f)));
        __nv_bfloat16* dst;
        if (head < h.n_heads) dst = h.q_out + ((size_t)r * h.n_heads + head) * h.dim;
        else if (head < h.n_heads + h.n_kv) dst = h.k_pool + (slot * h.n_kv + head - h.n_heads) * h.dim;
        else if (head < h.n_heads + 2 * h.n_kv) dst = h.v_pool + (slot * h.n_kv + head - h.n_heads - h.n_kv) * h.dim;
        else dst = h.rest + (size_t)r * h.ld_rest + (size_t)(head - h.n_heads - 2 * h.n_kv) * h.dim;
        if (head < h.n_heads + h.n_kv) {
          const float cs = __ldg(h.cos + (size_t)pos * half + o), sn = __ldg(h.sin + (size_t)pos * half + o), a = v * cs - u * sn;
          u = v * sn + u * cs;
          v = a;
        }
        dst[o] = __float2bfloat16_rn(v);
        dst[o + half] = __float2bfloat16_rn(u);
        continue;
      }
      const size_t o = (size_t)r * p.ldc + at;
      if (p.bias) v += __ldg(p.bias + at);  // not with SwiGLU
      if (paired) reinterpret_cast<__nv_bfloat16*>(p.out)[o] = __float2bfloat16_rn(v / (1.0f + __expf(-v)) * u);
      else if (p.epi == LG_EPI_BF16) reinterpret_cast<__nv_bfloat16*>(p.out)[o] = __float2bfloat16_rn(v);
      else if (p.epi == LG_EPI_RESID_F32) reinterpret_cast<float*>(p.out)[o] += v;
      else reinterpret_cast<float*>(p.out)[o] = v;
    }
  }
}

}  // namespace

namespace lg {

bool int4_rows_takes(const Int4Rows& p) {
  const bool paired = p.heads.dim > 0 || p.epi == LG_EPI_SWIGLU;
  return int4_rows_fit(p.rows, p.k) && p.n >= 1 && (int64_t)p.n * (p.k / 32) <= 0x7fffffff &&
         (!paired || p.n % (p.heads.dim ? p.heads.dim : 64) == 0) && p.heads.dim % 16 == 0 && (p.heads.dim || p.epi != LG_EPI_SWIGLU || !p.bias) &&
         (p.x ? p.gain && (((uintptr_t)p.x | (uintptr_t)p.gain) & 15) == 0 : p.a && p.lda % 8 == 0 && p.lda >= p.k && ((uintptr_t)p.a & 15) == 0) &&
         ((uintptr_t)p.codes & 15) == 0 && ((uintptr_t)p.scales & 7) == 0;
}

uint32_t launch_int4_rows(const Int4Rows& a, cudaStream_t stream) {
  if (!int4_rows_takes(a)) return kInvalidValue;
  const int n_tiles = (a.n + kTileRows - 1) / kTileRows, groups = a.k / 32;
  // slices of k: no more than a warp has in flight, and four warps per SM as long as each keeps a block; tiles of up to eight
  // warps; and no more CTAs than run at once, evenly filled, since each brings the activations to shared memory for itself
  const int sms = lg::sm_count(), blocks = groups / 4, chunk = blocks <= 16 ? 2 : 4, max_warps = chunk == 2 ? 8 : kMaxWarps;
  int slices = std::max((blocks + chunk - 1) / chunk, std::min(blocks, (4 * sms + n_tiles - 1) / n_tiles));
  slices = std::max(1, std::min(slices, max_warps));
  const int tiles = std::max(1, std::min(8 / slices, n_tiles / (2 * sms))), sets = (n_tiles + tiles - 1) / tiles;
  const int at_once = sms * std::max(1, (chunk == 2 ? 24 : 18) / (tiles * slices)), rounds = (sets + at_once - 1) / at_once, ctas = (sets + rounds - 1) / rounds;
  auto kern = chunk == 2 ? int4_rows_kernel<2> : int4_rows_kernel<4>;
  const size_t smem = int4_rows_shared(a.rows, a.k);
  // the attribute belongs to the kernel, not to the call: always the same value, or a model in another thread could take it back before the launch
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFewShared);
  if (e != cudaSuccess) return (uint32_t)e;
  const Params p{(const float*)a.x, (const float*)a.gain, a.eps, (const __nv_bfloat16*)a.a, a.lda, (const uint8_t*)a.codes, (const __half*)a.scales, (const float*)a.bias, a.out,
                 a.n, a.k, a.ldc, a.heads.dim ? kEpiHeads : a.epi, slices, tiles, a.rows, a.heads};
  lg::launch(kern, dim3((unsigned)ctas), dim3((unsigned)(32 * tiles * slices)), smem, stream, p);
  return launch_status();
}

}  // namespace lg
