// Attention over short texts (up to 64 tokens) straight from the fp32 sums of the q, k, v projection: bias, rotation and
// attention in one launch, everything in fp32.
//
// A text of 17 tokens has 2 MFLOP of attention per layer; what it takes is launches. On the general route the projection runs on
// 16 tiles without slices of k (its bf16 output cannot be accumulated: 12.6 us), a launch rotates q and k and transposes V (4.4)
// and the tensor-core kernel computes a whole 128 x 128 tile (8.0). Here the projection accumulates slices of k into a zeroed
// buffer (6.6 us) and one launch of 9.4 us does the rest (a forward of 17 tokens through 28 layers 1.99 -> 1.49 ms). CTA = (head, text): q, k, v in shared memory, a warp takes a query at a time,
// a lane one or two keys for the scores and four columns for the result.
#include "short_attention.h"

#include "common.cuh"

namespace {

using namespace lg;

constexpr int kDim = 128, kRow = kDim + 4;  // rows four banks apart: a lane per row reads 16 bytes without conflicts
constexpr int kWarps = 16;

template <int KEYS>  // keys per lane
__global__ void __launch_bounds__(32 * kWarps)
short_attention_kernel(const ShortAttention p) {
  lg::pdl_prologue();
  extern __shared__ float smem[];
  const int head = blockIdx.x, seq = blockIdx.y, kv = head / (p.n_heads / p.n_kv);
  const int t0 = p.cu[seq], len = min(p.cu[seq + 1] - t0, p.max_len);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, width = (p.n_heads + 2 * p.n_kv) * kDim;
  float *qs = smem, *ks = qs + p.max_len * kRow, *vs = ks + p.max_len * kRow;
  // the buffer that the next layer accumulates into
  const int n_zero = p.n_tokens * width / 4, at = (blockIdx.y * gridDim.x + blockIdx.x) * blockDim.x + threadIdx.x;
  for (int i = at; i < n_zero; i += gridDim.x * gridDim.y * blockDim.x) reinterpret_cast<float4*>(p.zero)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  // thread = four pairs (i, i + 64) of a row of q or k, or eight values of v
  for (int e = threadIdx.x; e < len * 48; e += blockDim.x) {
    const int r = e / 48, c = e - r * 48, part = c >> 4, o = 4 * (c & 15);
    const int col = (part == 0 ? head : p.n_heads + (part == 2 ? p.n_kv : 0) + kv) * kDim + o;
    const float* src = p.sums + (size_t)(t0 + r) * width + col;
    float4 a = *reinterpret_cast<const float4*>(src), b = *reinterpret_cast<const float4*>(src + 64);
    const float4 ba = __ldg(reinterpret_cast<const float4*>(p.bias + col)), bb = __ldg(reinterpret_cast<const float4*>(p.bias + col + 64));
    a.x += ba.x; a.y += ba.y; a.z += ba.z; a.w += ba.w;
    b.x += bb.x; b.y += bb.y; b.z += bb.z; b.w += bb.w;
    float* dst = (part == 0 ? qs : part == 1 ? ks : vs) + r * kRow + o;
    if (part < 2) {
      const int pos = p.positions[t0 + r];
      if (pos < 0 || pos >= p.max_pos) {
        if (p.status) atomicExch(p.status, 1);
      } else {
        const float4 c4 = __ldg(reinterpret_cast<const float4*>(p.cos + (size_t)pos * 64 + o)), s4 = __ldg(reinterpret_cast<const float4*>(p.sin + (size_t)pos * 64 + o));
        const float4 x = a, y = b;
        a = make_float4(x.x * c4.x - y.x * s4.x, x.y * c4.y - y.y * s4.y, x.z * c4.z - y.z * s4.z, x.w * c4.w - y.w * s4.w);
        b = make_float4(x.x * s4.x + y.x * c4.x, x.y * s4.y + y.y * c4.y, x.z * s4.z + y.z * c4.z, x.w * s4.w + y.w * c4.w);
      }
    }
    *reinterpret_cast<float4*>(dst) = a;
    *reinterpret_cast<float4*>(dst + 64) = b;
  }
  __syncthreads();
  const float sl2 = p.scale * 1.4426950408889634f;
  for (int i = warp; i < len; i += kWarps) {
    const int seen = p.causal ? i + 1 : len;
    float s[KEYS];
#pragma unroll
    for (int n = 0; n < KEYS; ++n) s[n] = 0.0f;
    const float4* q = reinterpret_cast<const float4*>(qs + i * kRow);
#pragma unroll 8
    for (int c = 0; c < kDim / 4; ++c) {
      const float4 a = q[c];
#pragma unroll
      for (int n = 0; n < KEYS; ++n) {
        const float4 b = reinterpret_cast<const float4*>(ks + min(lane + 32 * n, len - 1) * kRow)[c];
        s[n] = fmaf(a.x, b.x, fmaf(a.y, b.y, fmaf(a.z, b.z, fmaf(a.w, b.w, s[n]))));
      }
    }
    float m = -INFINITY, sum = 0.0f;
#pragma unroll
    for (int n = 0; n < KEYS; ++n) {
      s[n] = lane + 32 * n < seen ? s[n] * sl2 : -INFINITY;
      m = fmaxf(m, s[n]);
    }
    m = warp_max(m);
#pragma unroll
    for (int n = 0; n < KEYS; ++n) {
      s[n] = exp2f(s[n] - m);
      sum += s[n];
    }
    const float inv = 1.0f / warp_sum(sum);
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int n = 0; n < KEYS; ++n) {
#pragma unroll 4
      for (int j = 32 * n; j < min(seen, 32 * n + 32); ++j) {
        const float w = __shfl_sync(0xffffffffu, s[n], j & 31);
        const float4 v = reinterpret_cast<const float4*>(vs + j * kRow)[lane];
        o.x = fmaf(w, v.x, o.x); o.y = fmaf(w, v.y, o.y); o.z = fmaf(w, v.z, o.z); o.w = fmaf(w, v.w, o.w);
      }
    }
    *reinterpret_cast<uint2*>(p.out + ((size_t)(t0 + i) * p.n_heads + head) * kDim + 4 * lane) = make_uint2(pack_bf16x2(o.x * inv, o.y * inv), pack_bf16x2(o.z * inv, o.w * inv));
  }
}

}  // namespace

namespace lg {

uint32_t launch_short_attention(const ShortAttention& p, cudaStream_t stream) {
  if (p.max_len < 1 || p.max_len > kShortText || p.n_seqs < 1 || p.n_seqs > 65535 || p.n_heads < 1 || p.n_kv < 1 || p.n_heads % p.n_kv) return kInvalidValue;
  const size_t smem = (size_t)3 * p.max_len * kRow * 4;
  auto kern = p.max_len <= 32 ? short_attention_kernel<1> : short_attention_kernel<2>;
  if (smem > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (uint32_t)e;
  }
  lg::launch(kern, dim3((unsigned)p.n_heads, (unsigned)p.n_seqs), dim3(32 * kWarps), smem, stream, p);
  return launch_status();
}

}  // namespace lg
