// The layers of a decode step of one to four sequences over int4 group-32 weights as ONE launch.
//
// Such a step is 28 layers x 26 MB of weights, 4 us a layer from HBM; as six launches a layer it took 42 us, nearly all of it starts of launches,
// dependencies and first loads (int4_rows.cu has the launches); here 24. Device time of a step at contexts of 1200, one / two / three / four rows: 0.68 / 0.78 /
// 0.86 / 0.93 ms against 1.20 / 1.28 / 1.45 / 1.55; at 300 and at 8000 the ratio is the same (1.5 to 1.8). What is left of a layer, one row at 1200 tokens, by clock stamps of
// thread 0 of every CTA (which cost 5 %; 45 thousand cycles a layer with them): q, k, v 7100 (2500 until the stream's words are there, norm 1400, products 1900, sums and rotation 1300);
// 12900 from there until the merged heads are (3600 the attention of a CTA that has a chunk, the rest two exchanges and the merge); output 3600; gate and up 12700 (2700 until the words are there,
// norm and products 7800, sums and SwiGLU 2200); down 8800 (2200, 5300, 1300). So an exchange between all SMs takes 2100 to 2700 cycles, and there are six; the products of
// gate, up and down are bound by the unpacking of int4 on the ALU pipe. The step holds every SM: what other streams have for the GPU waits until it is over.
//
// One CTA per SM stays for the whole step. What an SM needs of a layer's weights (190 KB) fits its shared memory, so each matrix has a place there and the next
// layer's copy (cp.async.bulk, a row at a time, rows 16 bytes apart modulo the banks, issued by a warp of its own) starts as soon as the products have used
// it: weights arrive a layer ahead and nothing waits for memory.
//
// A layer is norm, q, k, v, rotation, cache store | attention over chunks of the contexts | merge of the chunks | output
// projection, residual | norm, gate, up, SwiGLU | down projection, residual. Between these every CTA needs what the others have made. A barrier of the grid costs
// 2450 cycles here (an atomic, polls, a fence) and the loads behind it 1300 more, so there is none: a value travels as one 64-bit word with
// the number of its layer beside it, and who needs it reads the word until the number is right (as NCCL's LL protocol does). A word
// is written again a layer later, by a CTA that has by then seen results of everyone who reads it. Nothing else is passed
// between CTAs within a launch: the new token's keys and values travel this way too, and the stores into the cache are for later steps.
// Registers matter: shared memory leaves an L1 of 28 KB, and spilled values that do not fit it come from L2 (352 bytes of stack a thread:
// 56 thousand cycles a layer). Two places in shared memory are shared: the activations of the down projection lie where gate and up lay, cached keys and values where
// the down projection's weights come next.
//
// A warp takes 128 values of the hidden size in every phase (in the output projection: one head) and all of the CTA's weight rows. Products as in
// int4_rows.cu: mma.sync m16n8k16 on the exact integers 136 + q with accumulators that start at -136 times the group's sum of activations, scales in
// fp32 on the finished group; the sums of the warps are added in shared memory in order. Nothing is added without an order, so results repeat.
#include "decode_stack.h"

#include "common.cuh"
#include "decode_tiles.cuh"
#include "int4_rows.h"
#include "tcgen05.cuh"

namespace lg {
namespace {

using namespace tc;
using namespace stack;

constexpr int kBringers = 1;
static_assert(kTokens == kBlock, "cache blocks");
constexpr uint32_t kPolls = 1u << 20;  // of a word: about a second

struct Kernel {
  StackArgs a;
  StackPlan p;
};

LG_DEVINL void bulk_copy(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}

extern __shared__ __align__(128) uint8_t smem[];  // places in it are offsets
template <typename T>
LG_DEVINL T lds(uint32_t at) { return *reinterpret_cast<const T*>(smem + at); }
LG_DEVINL float load_now(const float* p) {  // not moved to where the value is used
  float v;
  asm volatile("ld.global.nc.f32 %0, [%1];\n" : "=f"(v) : "l"(p));
  return v;
}
LG_DEVINL float4 load4_now(const float* p) {
  float4 v;
  asm volatile("ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];\n" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}
template <typename T>
LG_DEVINL void sts(uint32_t at, T v) { *reinterpret_cast<T*>(smem + at) = v; }

// the warps that compute meet; the others bring the weights
LG_DEVINL void meet(int threads) { asm volatile("bar.sync 1, %0;\n" ::"r"(threads) : "memory"); }
LG_DEVINL bool meet_any(int threads, bool v) {
  uint32_t any;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %2, 0;\n\t"
      "bar.red.or.pred q, 1, %1, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}\n"
      : "=r"(any)
      : "r"(threads), "r"((uint32_t)v)
      : "memory");
  return any != 0;
}

// ---- words that travel: 32 bits of payload and the number of their layer -------------------------------------------

using Word = unsigned long long;

LG_DEVINL Word word(uint32_t payload, uint32_t number) { return (Word)number << 32 | payload; }
LG_DEVINL void send(Word* to, uint32_t payload, uint32_t number) { asm volatile("st.relaxed.gpu.global.u64 [%0], %1;\n" ::"l"(to), "l"(word(payload, number)) : "memory"); }
LG_DEVINL void send2(Word* to, uint32_t a, uint32_t b, uint32_t number) {
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};\n" ::"l"(to), "l"(word(a, number)), "l"(word(b, number)) : "memory");
}
// N pairs of neighbouring words, at(i) the i-th pair, where(i) false: not wanted. Whole warps.
template <int N, typename At, typename Where>
LG_DEVINL void receive(uint2 (&out)[N], uint32_t number, volatile int* abort_flag, At&& at, Where&& where) {
#pragma unroll 1
  for (uint32_t i = 0;; ++i) {
    Word w[N][2];
#pragma unroll
    for (int j = 0; j < N; ++j) {
      w[j][0] = w[j][1] = word(0u, number);
      if (where(j)) asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];\n" : "=l"(w[j][0]), "=l"(w[j][1]) : "l"(at(j)) : "memory");
    }
    bool all = true;
#pragma unroll
    for (int j = 0; j < N; ++j) {
      all = all && (uint32_t)(w[j][0] >> 32) == number && (uint32_t)(w[j][1] >> 32) == number;
      out[j] = make_uint2((uint32_t)w[j][0], (uint32_t)w[j][1]);
    }
    if (__all_sync(0xffffffffu, all)) return;
    if (i >= kPolls || *abort_flag) {
      *abort_flag = 1;
      return;
    }
  }
}

// The numbers have been through 32 bits: every word is zero again, as before the first launch. All CTAs meet, once in 2^32 layers.
__device__ __noinline__ bool clear_words(Word* words, size_t n, uint32_t* met) {
  __shared__ int s_ok;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) words[i] = 0;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    const uint32_t until = (atomicAdd(met, 1u) / gridDim.x + 1) * gridDim.x;
    s_ok = 0;
#pragma unroll 1
    for (uint32_t i = 0; i < kPolls && !s_ok; ++i) {
      uint32_t v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];\n" : "=r"(v) : "l"(met) : "memory");
      s_ok = (int)(v - until) >= 0;
    }
  }
  __syncthreads();
  return s_ok;
}

// what the CTA's weight slot stands for
LG_DEVINL int weight_row(const StackPlan& p, int m, int cta, int slot) {
  if (m == kOut || m == kDown) return cta * p.out_rows + slot;
  const int half = m == kQkv ? kDim / 2 : 32, o = 8 * (cta * (m == kQkv ? p.qkv_tiles : p.gu_tiles) + (slot >> 4)) + (slot & 7);
  return o / half * 2 * half + o % half + (slot & 8 ? half : 0);
}

// This warp's share of the CTA's n rows of a matrix: a copy per row of codes (a warp issues one in about 110 cycles, whatever its size), one per run of rows for the
// scales.
LG_DEVINL void bring(const Kernel& k, int m, uint32_t bar, const StackMat& w, int n, int who) {
  const int kk = m == kDown ? k.a.d.inter : k.a.d.hidden, lane = threadIdx.x & 31, at = lane * kBringers + who, run = m == kOut || m == kDown ? n : 8;
  const uint32_t to = smem_u32(smem) + k.p.at[m], to_scales = smem_u32(smem) + k.p.at_scales[m];
  if (at == 0) mbar_expect_tx(bar, (uint32_t)n * (uint32_t)(kk / 2 + kk / 16));
#pragma unroll 1
  for (int s = at; s < n; s += 32 * kBringers) {
    const size_t row = (size_t)weight_row(k.p, m, blockIdx.x, s);
    bulk_copy(to + (uint32_t)(s * code_stride(kk)), w.codes + row * (kk / 2), (uint32_t)(kk / 2), bar);
    if (s % run == 0)
      bulk_copy(to_scales + (uint32_t)(s * (kk / 16)), reinterpret_cast<const uint8_t*>(w.scales) + row * (kk / 16), (uint32_t)(run * (kk / 16)), bar);
  }
}

LG_DEVINL bool wait_for(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
#pragma unroll 1
  for (uint32_t i = 0; i < kSpinLimit; ++i) {
    if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
    if (*abort_flag) return false;
  }
  *abort_flag = 1;
  return false;
}

// four consecutive activations per lane of 128 of a row: rounded, in the order 0 4 1 5 2 6 3 7 of the nibble pairs, to xs + 8 lane, and -136
// times the sums of their groups to sums + 16 group
LG_DEVINL void stage4(float4 v, uint32_t xs, uint32_t sums, int lane) {
  const float x0 = __bfloat162float(__float2bfloat16_rn(v.x)), x1 = __bfloat162float(__float2bfloat16_rn(v.y)), x2 = __bfloat162float(__float2bfloat16_rn(v.z)),
              x3 = __bfloat162float(__float2bfloat16_rn(v.w));
  const bool odd = lane & 1;
  const float s0 = __shfl_xor_sync(0xffffffffu, odd ? x0 : x2, 1), s1 = __shfl_xor_sync(0xffffffffu, odd ? x1 : x3, 1);
  sts(xs + 8u * lane, odd ? make_uint2(pack_bf16x2(s0, x2), pack_bf16x2(s1, x3)) : make_uint2(pack_bf16x2(x0, s0), pack_bf16x2(x1, s1)));
  float s = (x0 + x1) + (x2 + x3);
  s += __shfl_xor_sync(0xffffffffu, s, 1);
  s += __shfl_xor_sync(0xffffffffu, s, 2);
  s += __shfl_xor_sync(0xffffffffu, s, 4);
  if ((lane & 7) == 0) sts(sums + 16u * (lane >> 3), -136.0f * s);
}

// mma_bf16_16816 that may be moved among other instructions
LG_DEVINL void mma_free(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2], const float (&c)[4]) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};\n"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "f"(c[0]), "f"(c[1]), "f"(c[2]), "f"(c[3]));
}

// Products of a block of 128 values of k with a tile of 16 weight rows, onto acc (rows g, g + 8; columns 2 t, 2 t + 1). lo, sc: this lane's word and the scales in row g.
struct Block {
  uint4 x[4];
  float c[4][4];  // the accumulators' start
  uint32_t mask, flip;
};
template <int R>
LG_DEVINL void load_block(Block& b, uint32_t xs, uint32_t ld, uint32_t sums, int g, int t) {
  b.mask = opaque(0x000f000fu);
  b.flip = opaque(0x43084308u);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    b.x[j] = make_uint4(0u, 0u, 0u, 0u);
    if (g < R) b.x[j] = lds<uint4>(xs + (uint32_t)g * ld + 16u * t + 64u * j);
    float2 s = make_float2(0.0f, 0.0f);
    if (t < 2) s = lds<float2>(sums + 16u * j + 8u * t);  // columns beyond the rows hold anything and are not used
    b.c[j][0] = b.c[j][2] = s.x;
    b.c[j][1] = b.c[j][3] = s.y;
  }
}
template <int R>
LG_DEVINL void tile_products(float (&acc)[4], const Block& b, uint32_t lo, uint32_t stride, uint32_t sc, uint32_t scale_stride) {
  uint32_t wl[4], wh[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    wl[j] = lds<uint32_t>(lo + 16u * j);
    wh[j] = lds<uint32_t>(lo + 8u * stride + 16u * j);
  }
  const uint2 scl = lds<uint2>(sc), sch = lds<uint2>(sc + 8u * scale_stride);
  const uint32_t mask = b.mask, flip = b.flip;
  auto pair = [=](uint32_t w, int at) { return and_xor(w >> (4 * at), mask, flip); };  // nibbles at, at + 4 as 136 + q
  float d[4][4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint32_t a[4] = {pair(wl[j], 0), pair(wh[j], 0), pair(wl[j], 1), pair(wh[j], 1)}, x[2] = {b.x[j].x, b.x[j].y};
    mma_free(d[j], a, x, b.c[j]);
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint32_t a[4] = {pair(wl[j], 2), pair(wh[j], 2), pair(wl[j], 3), pair(wh[j], 3)}, x[2] = {b.x[j].z, b.x[j].w};
    mma_free(d[j], a, x, d[j]);
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint32_t l2 = j < 2 ? scl.x : scl.y, h2 = j < 2 ? sch.x : sch.y;
    const float2 sl = __half22float2(*reinterpret_cast<const __half2*>(&l2)), sh = __half22float2(*reinterpret_cast<const __half2*>(&h2));
    acc[0] = fmaf(j & 1 ? sl.y : sl.x, d[j][0], acc[0]);
    if (R > 1) acc[1] = fmaf(j & 1 ? sl.y : sl.x, d[j][1], acc[1]);
    acc[2] = fmaf(j & 1 ? sh.y : sh.x, d[j][2], acc[2]);
    if (R > 1) acc[3] = fmaf(j & 1 ? sh.y : sh.x, d[j][3], acc[3]);
  }
}
// a tile's sums to the warp's part
template <int R>
LG_DEVINL void store_tile(const float (&acc)[4], uint32_t part, int g, int t) {
  constexpr int RP = R == 3 ? 4 : R;
  if (2 * t >= R) return;
  const uint32_t at = part + (uint32_t)(g * RP + 2 * t) * 4u, hi = at + 8u * RP * 4u;
  if (R == 1) {
    sts(at, acc[0]);
    sts(hi, acc[2]);
  } else {
    sts(at, make_float2(acc[0], acc[1]));
    sts(hi, make_float2(acc[2], acc[3]));
  }
}

// A warp's products of one block with all tiles of a matrix. Addresses: codes and scales of the block in the first row, activations of the block
// (rows ld bytes apart), their sums, the warp's part. Tiles that end in rows which are not there read what lies behind them, and
// nothing looks at the result.
template <int R>
LG_DEVINL void products(uint32_t codes, uint32_t stride, uint32_t scales, uint32_t scale_stride, int tiles, uint32_t xs, uint32_t ld, uint32_t sums, uint32_t part) {
  constexpr int RP = R == 3 ? 4 : R;
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  Block b;
  load_block<R>(b, xs, ld, sums, g, t);
  uint32_t lo = codes + (uint32_t)g * stride + 4u * t, sc = scales + (uint32_t)g * scale_stride;
#pragma unroll 2
  for (int i = 0; i < tiles; ++i) {
    float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    tile_products<R>(acc, b, lo, stride, sc, scale_stride);
    store_tile<R>(acc, part, g, t);
    lo += 16u * stride;
    sc += 16u * scale_stride;
    part += 16u * RP * 4u;
  }
}
// The same of every step-th block from `first` on, block by block for each tile.
template <int R>
LG_DEVINL void products_blocks(uint32_t codes, uint32_t stride, uint32_t scales, uint32_t scale_stride, int tiles, uint32_t xs, uint32_t ld, uint32_t sums, uint32_t part,
                                             int first, int blocks, int step) {
  constexpr int RP = R == 3 ? 4 : R;
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const uint32_t lo = codes + (uint32_t)g * stride + 4u * t, sc = scales + (uint32_t)g * scale_stride;
#pragma unroll 1
  for (int i = 0; i < tiles; ++i) {
    float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 2
    for (int n = first; n < blocks; n += step) {
      Block b;
      load_block<R>(b, xs + 256u * n, ld, sums + 64u * n, g, t);
      tile_products<R>(acc, b, lo + 64u * n + 16u * i * stride, stride, sc + 8u * n + 16u * i * scale_stride, scale_stride);
    }
    store_tile<R>(acc, part + 16u * i * RP * 4u, g, t);
  }
}

// RMS norm of the rows of the residual stream into shared memory: a warp takes 128 values of every row, a lane four. words: the stream
// as it travels, or x as it lies in memory ahead of the first layer.
template <int R>
LG_DEVINL void norm_rows(int warps, const float* x, const Word* words, uint32_t number, int hidden, float eps, float4 gain, float* red, uint32_t xs, uint32_t ld, uint32_t sums,
                                       volatile int* abort_flag) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float4 v[R];
  if (words) {
    uint2 w[2 * R];
    receive<2 * R>(w, number, abort_flag, [&](int j) { return words + (size_t)(j >> 1) * hidden + 4 * threadIdx.x + 2 * (j & 1); }, [](int) { return true; });
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = make_float4(__uint_as_float(w[2 * r].x), __uint_as_float(w[2 * r].y), __uint_as_float(w[2 * r + 1].x), __uint_as_float(w[2 * r + 1].y));
  } else {
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = __ldcg(reinterpret_cast<const float4*>(x + (size_t)r * hidden) + threadIdx.x);
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const float ss = warp_sum(v[r].x * v[r].x + v[r].y * v[r].y + v[r].z * v[r].z + v[r].w * v[r].w);
    if (lane == 0) red[r * kMaxWarps + warp] = ss;
  }
  meet(32 * warps);
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const float sum = warp_sum(lane < warps ? red[r * kMaxWarps + lane] : 0.0f);
    const float inv = 1.0f / sqrtf(sum / (float)hidden + eps);
    stage4(make_float4(v[r].x * inv * gain.x, v[r].y * inv * gain.y, v[r].z * inv * gain.z, v[r].w * inv * gain.w), xs + (uint32_t)r * ld + 256u * warp, sums + 64u * warp + 4u * r, lane);
  }
  __syncwarp();
}

// sum over the warps, in order; step: bytes of a warp's part. The parts are there for a multiple of four warps.
LG_DEVINL float total(uint32_t at, uint32_t step, int warps) {
  float v = 0.0f;
#pragma unroll 1
  for (int w = 0; w < warps; w += 4, at += 4 * step) {
    const float a = lds<float>(at), b = lds<float>(at + step), c = lds<float>(at + 2 * step), d = lds<float>(at + 3 * step);
    v = (((v + a) + b) + c) + d;
  }
  return v;
}

// a warp requests one cache block of a key head: keys, then values
LG_DEVINL void stage_kv(uint32_t stage, const __nv_bfloat16* k_pool, const __nv_bfloat16* v_pool, int block, int row_elems, int kvh) {
  const int lane = threadIdx.x & 31, ch = lane & 15;
  const size_t from = ((size_t)block * kBlock + (lane >> 4)) * row_elems + kvh * kDim + ch * 8;
#pragma unroll 2
  for (int i = 0; i < kBlock; i += 2) {
    const uint32_t to = tile_addr<kDim>(stage, i + (lane >> 4), ch);
    cp_async16(to, k_pool + from + (size_t)i * row_elems);
    cp_async16(to + kStage / 2, v_pool + from + (size_t)i * row_elems);
  }
}

// a chunk of a row's context for one key head; a warp takes every att_warps-th of its cache blocks
struct Item { int r, kvh, chunk, ctx, first, count; };
LG_DEVINL Item item_of(const Kernel& k, int it) {
  Item i;
  i.chunk = it % k.p.max_chunks;
  i.kvh = it / k.p.max_chunks % k.a.d.n_kv;
  i.r = it / (k.p.max_chunks * k.a.d.n_kv);
  i.ctx = __ldg(k.a.ctx + i.r);
  const int tok0 = i.chunk * k.a.chunk, tok1 = min(i.ctx, tok0 + k.a.chunk);
  i.first = tok0 / kBlock;
  i.count = tok1 > tok0 ? (tok1 - tok0 + kBlock - 1) / kBlock : 0;
  return i;
}
LG_DEVINL int block_of(const Kernel& k, const Item& i, int n) {  // -1: not a block of the pool
  const int pb = i.first + n < k.a.max_blocks ? __ldg(k.a.tables + (size_t)i.r * k.a.max_blocks + i.first + n) : -1;
  if (pb >= 0 && pb < k.a.n_pool_blocks) return pb;
  if ((threadIdx.x & 31) == 0) atomicExch(k.a.status, 1);
  return -1;
}

// scores of 16 cached keys (rows) for eight heads (columns); a lane's channels are 4 t + 16 ks .. + 3 of keys g and g + 8
LG_DEVINL void scores16(const uint2 (&q)[kDim / 16], uint32_t keys, int lane, float (&s)[4]) {
  const int g = lane >> 2, t = lane & 3;
  float odd[4] = {0.0f, 0.0f, 0.0f, 0.0f};  // two chains
  s[0] = s[1] = s[2] = s[3] = 0.0f;
#pragma unroll
  for (int ks = 0; ks < kDim / 16; ++ks) {
    const uint32_t at = tile_addr<kDim>(keys, g, 2 * ks + (t >> 1)) + 8u * (t & 1);
    const uint2 k0 = lds<uint2>(at), k1 = lds<uint2>(at + 8u * kDim * 2u);  // (row g + 8 has the same swizzle)
    const uint32_t a[4] = {k0.x, k1.x, k0.y, k1.y}, b[2] = {q[ks].x, q[ks].y};
    mma_free(ks & 1 ? odd : s, a, b, ks & 1 ? odd : s);
  }
#pragma unroll
  for (int e = 0; e < 4; ++e) s[e] += odd[e];
}
LG_DEVINL uint32_t transpose8x8(uint32_t v) {
  uint32_t d;
  asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;\n" : "=r"(d) : "r"(v));
  return d;
}

struct Turn {  // of a pair of q, k, v: angle and cache slot (-1: none)
  float cs, sn;
  int64_t cache;
};
struct Mail {  // places of the words
  Word *heads;   // [rows][n_heads + 2 n_kv][64]: q, k, v of the new tokens, two channels a word
  Word *o, *ml;  // [rows][n_heads][max_chunks][128], [..][2]: unnormalised outputs of the chunks, their maxima and sums
  Word *attn;    // [rows][n_heads][64]
  Word *mid, *x; // [rows][hidden]: the residual stream behind the attention and behind the layer
  Word *act;     // [rows][inter / 2]
};

// The attention of an item for the (up to eight) query heads of its key head, scores and outputs transposed: keys and channels are the rows of a product and
// heads its columns, so nothing is computed for heads that are not there. The warps meet in shared memory. block0: this warp's first block,
// -2: to be looked up; ahead: it has been requested.
constexpr int kOutRow = kDim + 4;  // floats of a head in shared memory: heads lie 8 banks apart
LG_DEVINL void attend(const Kernel& k, const Mail& mail, uint32_t number, volatile int* abort_flag, const __nv_bfloat16* k_pool, const __nv_bfloat16* v_pool, const Item& i, int block0,
                      bool ahead) {
  const StackPlan& p = k.p;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3, threads = 32 * p.warps, n_heads = k.a.d.n_heads, n_kv = k.a.d.n_kv, n_rep = n_heads / n_kv,
            all_heads = n_heads + 2 * n_kv;
  const uint32_t room = p.at[kDown] + (uint32_t)(warp * kStage), stage = smem_u32(smem) + room;
  const float sl2 = 1.4426950408889634f / sqrtf((float)kDim);
  const bool works = warp < p.att_warps && warp < i.count;
  const uint32_t so = p.at[kDown], sml = so + (uint32_t)(p.att_warps * n_rep * kOutRow) * 4u;  // [warp][n_rep][kOutRow], [warp][n_rep][2]
  float o[kDim / 16][4], m[2] = {-INFINITY, -INFINITY}, sum[2] = {0.0f, 0.0f};  // of heads 2 t, 2 t + 1
  if (works) {
    uint2 q[kDim / 16];  // head g
    receive<kDim / 16>(q, number, abort_flag, [&](int ks) { return mail.heads + ((size_t)i.r * all_heads + i.kvh * n_rep + g) * (kDim / 2) + 2 * t + 8 * ks; }, [&](int) { return g < n_rep; });
#pragma unroll
    for (int j = 0; j < kDim / 16; ++j) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.0f;
    int pb = block0;
#pragma unroll 1
    for (int n = warp; n < i.count; n += p.att_warps) {
      const int tok = (i.first + n) * kBlock;
      if (n != warp || pb == -2) pb = block_of(k, i, n);
      if (pb >= 0 && !(ahead && n == warp)) stage_kv(stage, k_pool, v_pool, pb, n_kv * kDim, i.kvh);
      cp_async_commit();
      cp_async_wait<0>();
      __syncwarp();
      if (pb < 0) continue;
      if (tok + kBlock >= i.ctx) {  // the block of the new token, whose row has come as words; what lies behind it is cleared: 0 * NaN is NaN
        uint2 w[2];
        receive<2>(w, number, abort_flag, [&](int j) { return mail.heads + ((size_t)i.r * all_heads + n_heads + j * n_kv + i.kvh) * (kDim / 2) + 2 * lane; }, [](int) { return true; });
        const int at = i.ctx - 1 - tok;
#pragma unroll
        for (int j = 0; j < 2; ++j) sts(tile_addr<kDim>(room + j * (kStage / 2), at, lane >> 1) + 8u * (lane & 1), w[j]);
#pragma unroll 1
        for (int row = at + 1; row < kBlock; ++row)
#pragma unroll
          for (int j = 0; j < 2; ++j) sts(tile_addr<kDim>(room + j * (kStage / 2), row, lane >> 1) + 8u * (lane & 1), make_uint2(0u, 0u));
        __syncwarp();
      }
      float s[4];  // keys g, g + 8; heads 2 t, 2 t + 1
      scores16(q, room, lane, s);
      if (tok + g >= i.ctx) s[0] = s[1] = -INFINITY;
      if (tok + g + 8 >= i.ctx) s[2] = s[3] = -INFINITY;
      float alpha[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {  // a block holds at least one key, so the maximum is a score
        float mx = fmaxf(s[e], s[2 + e]);
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
        mx = fmaxf(mx, m[e]);
        alpha[e] = exp2f((m[e] - mx) * sl2);
        m[e] = mx;
        s[e] = exp2f((s[e] - mx) * sl2);
        s[2 + e] = exp2f((s[2 + e] - mx) * sl2);
        sum[e] = sum[e] * alpha[e] + (s[e] + s[2 + e]);
      }
      const uint32_t w[2] = {transpose8x8(pack_bf16x2(s[0], s[1])), transpose8x8(pack_bf16x2(s[2], s[3]))};
#pragma unroll
      for (int j = 0; j < kDim / 16; ++j) {  // channels 16 j + g, + 8; heads 2 t, 2 t + 1
        uint32_t v[4];
        ldmatrix_x4_trans(v, tile_addr<kDim>(stage + kStage / 2, (lane & 7) + 8 * (lane >> 4), 2 * j + ((lane >> 3) & 1)));
        const float c[4] = {o[j][0] * alpha[0], o[j][1] * alpha[1], o[j][2] * alpha[0], o[j][3] * alpha[1]};
        mma_free(o[j], v, w, c);
      }
      __syncwarp();
    }
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      sum[e] += __shfl_xor_sync(0xffffffffu, sum[e], 4);
      sum[e] += __shfl_xor_sync(0xffffffffu, sum[e], 8);
      sum[e] += __shfl_xor_sync(0xffffffffu, sum[e], 16);
    }
  }
  meet(threads);  // the blocks have been read
  if (works) {
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      if (2 * t + e >= n_rep) continue;
      const uint32_t to = so + (uint32_t)((warp * n_rep + 2 * t + e) * kOutRow + g) * 4u;
#pragma unroll
      for (int j = 0; j < kDim / 16; ++j) {
        sts(to + 64u * j, o[j][e]);
        sts(to + 64u * j + 32u, o[j][2 + e]);
      }
      if (g == 0) sts(sml + (uint32_t)(warp * n_rep + 2 * t + e) * 8u, make_float2(m[e], sum[e]));
    }
  }
  meet(threads);
  const int used = min(p.att_warps, i.count);
#pragma unroll 1
  for (int u = tid; u < n_rep * (kDim / 2); u += threads) {  // two channels of a head
    const int row = u / (kDim / 2), dd = u % (kDim / 2);
    float M = -INFINITY, Lsum = 0.0f;
    float2 acc = make_float2(0.0f, 0.0f);
#pragma unroll 2
    for (int w = 0; w < used; ++w) M = fmaxf(M, lds<float>(sml + (uint32_t)(w * n_rep + row) * 8u));
#pragma unroll 2
    for (int w = 0; w < used; ++w) {
      const float2 ml = lds<float2>(sml + (uint32_t)(w * n_rep + row) * 8u);
      const float f = ml.x == -INFINITY ? 0.0f : exp2f((ml.x - M) * sl2);
      const float2 v = lds<float2>(so + (uint32_t)((w * n_rep + row) * kOutRow + 2 * dd) * 4u);
      Lsum += ml.y * f;
      acc.x += v.x * f;
      acc.y += v.y * f;
    }
    const size_t at = ((size_t)i.r * n_heads + i.kvh * n_rep + row) * p.max_chunks + i.chunk;
    send2(mail.o + at * kDim + 2 * dd, __float_as_uint(acc.x), __float_as_uint(acc.y), number);
    if (dd == 0) send2(mail.ml + at * 2, __float_as_uint(M), __float_as_uint(Lsum), number);
  }
  meet(threads);  // read before the next item's blocks
}

// The chunks of one head of one row put together: warp w takes chunks w, w + warps, ..; the warps meet at `room` (512 bytes each).
LG_DEVINL void merge(const Kernel& k, const Mail& mail, uint32_t number, volatile int* abort_flag, int r, int head, uint32_t room) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, warps = k.p.warps, chunks = (__ldg(k.a.ctx + r) + k.a.chunk - 1) / k.a.chunk;
  const float sl2 = 1.4426950408889634f / sqrtf((float)kDim);
  const size_t at = ((size_t)r * k.a.d.n_heads + head) * k.p.max_chunks;
  float f = 0.0f, L = 0.0f;
  float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 1
  for (int c = warp; c == warp || c < chunks; c += warps) {
    uint2 w[3];
    receive<3>(w, number, abort_flag, [&](int j) { return j < 2 ? mail.o + (at + c) * kDim + 4 * lane + 2 * j : mail.ml + (at + lane) * 2; },
               [&](int j) { return j < 2 ? c < chunks : c == warp && lane < chunks; });
    if (c == warp) {
      const bool in = lane < chunks;
      const float m = in ? __uint_as_float(w[2].x) : -INFINITY, M = warp_max(m);
      f = m == -INFINITY ? 0.0f : exp2f((m - M) * sl2);
      L = warp_sum(in ? __uint_as_float(w[2].y) * f : 0.0f);
    }
    const float s = __shfl_sync(0xffffffffu, f, c & 31);
    if (c < chunks) {
      acc.x = fmaf(__uint_as_float(w[0].x), s, acc.x); acc.y = fmaf(__uint_as_float(w[0].y), s, acc.y);
      acc.z = fmaf(__uint_as_float(w[1].x), s, acc.z); acc.w = fmaf(__uint_as_float(w[1].y), s, acc.w);
    }
  }
  sts(room + (uint32_t)(warp * kDim + 4 * lane) * 4u, acc);
  meet(32 * warps);
  if (tid < kDim / 2) {
    float2 v = make_float2(0.0f, 0.0f);
#pragma unroll 4
    for (int w = 0; w < warps; ++w) {
      const float2 a = lds<float2>(room + (uint32_t)(w * kDim + 2 * tid) * 4u);
      v.x += a.x;
      v.y += a.y;
    }
    send(mail.attn + ((size_t)r * k.a.d.n_heads + head) * (kDim / 2) + tid, L > 0.0f ? pack_bf16x2(v.x / L, v.y / L) : 0u, number);
  }
  meet(32 * warps);
}

template <int R>
__global__ void __launch_bounds__(32 * (kMaxWarps + kBringers), 1) decode_stack_kernel(const __grid_constant__ Kernel kern) {
  __shared__ __align__(8) uint64_t s_bars[2 * kMats];
  __shared__ int s_abort;
  __shared__ uint32_t s_before;  // launches before this one since the words were zero
  __shared__ float s_red[R * kMaxWarps];
  __shared__ StackLayer s_layer[2];  // this layer's and the next one's addresses
  __shared__ Mail s_mail;
  __shared__ Item s_item;  // the first one
  constexpr int RP = R == 3 ? 4 : R, kLayerWords = sizeof(StackLayer) / 8;
  const StackArgs& a = kern.a;
  const StackPlan& p = kern.p;
  const uint32_t bars = smem_u32(s_bars), frees = smem_u32(s_bars + kMats);  // a matrix is there; its place is free
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, cta = blockIdx.x, warps = p.warps, threads = 32 * warps;  // that compute
  const int H = a.d.hidden, I = a.d.inter, n_heads = a.d.n_heads, n_kv = a.d.n_kv, all_heads = n_heads + 2 * n_kv;
  auto layer_word = [&](int l) { return reinterpret_cast<const uint64_t*>(a.layers + l)[tid]; };
  if (tid == 0) {
    for (int m = 0; m < kMats; ++m) {
      mbar_init(bars + 8u * m, 1);
      mbar_init(frees + 8u * m, (uint32_t)warps);
    }
    s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    fence_proxy_async();
    s_item = item_of(kern, min(cta, R * n_kv * p.max_chunks - 1));
    Word* at = a.words;
    auto take = [&](size_t n) { Word* w = at; at += n; return w; };
    s_mail.heads = take((size_t)R * all_heads * (kDim / 2));
    s_mail.o = take((size_t)R * n_heads * p.max_chunks * kDim);
    s_mail.ml = take((size_t)R * n_heads * p.max_chunks * 2);
    s_mail.attn = take((size_t)R * n_heads * (kDim / 2));
    s_mail.mid = take((size_t)R * H);
    s_mail.x = take((size_t)R * H);
    s_mail.act = take((size_t)R * I / 2);
  }
  if (tid < kLayerWords) reinterpret_cast<uint64_t*>(s_layer)[tid] = layer_word(0);
  if (tid == 0) s_before = *a.launches;
  const uint32_t parts = p.at_part;
  // the parts of warps that are not there are zero whenever sums are taken: what else goes to their place is cleared again
  auto clear_tail = [&](int n) {
    for (uint32_t i = 4u * tid; i < (uint32_t)(round_up(warps, 4) - warps) * p.part_step; i += 4u * n) sts(parts + warps * p.part_step + i, 0.0f);
  };
  clear_tail(blockDim.x);
  __syncthreads();
  if (s_before >= a.most_launches) {
    const bool ok = clear_words(a.words, a.n_words, a.launches + 1);
    if (tid == 0) {
      s_before = 0;
      if (!ok) s_abort = 1;
    }
    __syncthreads();
  }

  // rows of this CTA and what they are, the same in every layer
  const int n_qkv = 16 * max(0, min(p.qkv_tiles, all_heads * (kDim / 16) - cta * p.qkv_tiles)), n_gu = 16 * max(0, min(p.gu_tiles, I / 8 - cta * p.gu_tiles)),
            n_out = max(0, min(p.out_rows, H - cta * p.out_rows)), t_out = (n_out + 15) >> 4;
  if (warp >= warps) {
    // ---- the warps that bring the weights
    // (none for a CTA without rows of a matrix: there nothing would keep the warps that give its place back from running phases ahead)
    auto rows = [&](int m) { return m == kQkv ? n_qkv : m == kGateUp ? n_gu : n_out; };
    auto go = [&](int m, int l) {
      const StackLayer& L = a.layers[l];
      bring(kern, m, bars + 8u * m, m == kQkv ? L.qkv : m == kOut ? L.out : m == kGateUp ? L.gate_up : L.down, rows(m), warp - warps);
    };
#pragma unroll 1
    for (int i = -3; i < 4 * a.n_layers; ++i) {  // in the order in which places become free; the first three are
      const int l = i >> 2, m = (i & 3) == 0 ? kQkv : (i & 3) == 1 ? kDown : (i & 3) == 2 ? kOut : kGateUp, next = m == kDown ? l : l + 1, first = i == -3 ? kQkv : m;
      if (next >= a.n_layers || !rows(first)) continue;
      if (i >= 0 && !mbar_wait_sleep_warp(frees + 8u * m, (uint32_t)(l & 1), &s_abort)) break;
      go(first, i < 0 ? 0 : next);
    }
    // The last CTA that comes here writes the count that the next launch finds: all have read this one's. (A CTA without a part in the step, at narrow widths, is
    // waited for by nobody else. It would take a count that changed under it for a reason to clear the words.)
    if (warp == warps && lane == 0) {
      __threadfence();
      if (atomicInc(a.launches + 2, gridDim.x - 1) == gridDim.x - 1) *a.launches = s_before + 1;
    }
    __syncthreads();
    return;
  }
  auto give_back = [&](int m) {  // this warp has done with what lies in a matrix's place
    __syncwarp();
    if (lane == 0) mbar_arrive(frees + 8u * m);
  };
  const uint32_t xs = p.at_x, ld = (uint32_t)(H + 32) * 2u, sums = p.at_sums, xs5 = 0u, ld5 = (uint32_t)(I + 32) * 2u, sums5 = R * ld5;
  const uint32_t own_part = parts + (uint32_t)warp * p.part_step;
  // q, k, v: a thread finishes one pair of one row
  const int qn = n_qkv >> 1;
  auto pair_of = [&](int& r, int& j, int& head, int& o) {
    int id = tid;
    asm volatile("" : "+r"(id));  // worked out where it is needed: registers that hold it over the layers end in local memory, which has no room in L1 here
    r = qn ? id / qn : R;
    j = id - r * qn;
    const int pair = 8 * cta * p.qkv_tiles + j;
    head = pair / (kDim / 2);
    o = pair % (kDim / 2);
    return r < R;
  };
  {
    int r, j, head, o;
    if (pair_of(r, j, head, o)) {
      Turn t{1.0f, 0.0f, a.slots[r]};
      const int pos = a.positions[r];
      if (pos < 0 || pos >= a.max_pos || t.cache < 0 || t.cache >= (int64_t)a.n_pool_blocks * kBlock) {
        atomicExch(a.status, 1);
        t.cache = -1;
      } else if (head < n_heads + n_kv) {
        t.cs = __ldg(a.cos + (size_t)pos * (kDim / 2) + o);
        t.sn = __ldg(a.sin + (size_t)pos * (kDim / 2) + o);
      }
      sts(p.at_turn + 16u * tid, t);
    }
  }
  // output and down: one value, whose residual the thread keeps
  const int on = n_out * R;
  auto value_of = [&](uint32_t& x_at, uint32_t& part) {
    int id = tid;
    asm volatile("" : "+r"(id));
    const int row = n_out ? id % n_out : 0, r = n_out ? id / n_out : 0;
    x_at = (uint32_t)(r * H + cta * p.out_rows + row);
    part = parts + (uint32_t)(row * RP + r) * 4u;
  };
  uint32_t x_at, o_part;
  value_of(x_at, o_part);
  float x_own = tid < on ? __ldcg(a.x + x_at) : 0.0f;
  const int items = R * n_kv * p.max_chunks, merges = R * n_heads;
  const uint32_t stage = smem_u32(smem) + p.at[kDown] + (uint32_t)(warp * kStage);
  const int block0 = cta < items && warp < p.att_warps && warp < s_item.count ? block_of(kern, s_item, warp) : -1;
  float4 gain = load4_now(s_layer[0].norm1 + 4 * tid);
  uint32_t number = s_before * (uint32_t)a.n_layers;
#pragma unroll 1
  for (int l = 0; l < a.n_layers; ++l) {
    const StackLayer& L = s_layer[l & 1];
    const StackLayer& N = s_layer[(l + 1) & 1];
    const bool more = l + 1 < a.n_layers;
    const uint32_t parity = (uint32_t)(l & 1);
    ++number;  // of this layer

    // ---- norm, q, k, v: rotated and stored
    if (meet_any(threads, s_abort)) break;
    uint64_t next_word = 0;
    if (more && tid >= threads - 32 && lane < kLayerWords) asm volatile("ld.global.nc.u64 %0, [%1];\n" : "=l"(next_word) : "l"(reinterpret_cast<const uint64_t*>(a.layers + l + 1) + lane));
    if (block0 >= 0) stage_kv(stage, L.k_pool, L.v_pool, block0, n_kv * kDim, s_item.kvh);
    cp_async_commit();
    if (n_qkv > 0) {
      float b0 = 0.0f, b1 = 0.0f;
      {
        int r, j, head, o;
        if (pair_of(r, j, head, o)) {
          b0 = load_now(L.bias + head * kDim + o);
          b1 = load_now(L.bias + head * kDim + o + kDim / 2);
        }
      }
      norm_rows<R>(warps, a.x, l ? s_mail.x : nullptr, number - 1, H, a.eps, gain, s_red, xs, ld, sums, &s_abort);
      if (wait_for(bars + 8u * kQkv, parity, &s_abort))
        products<R>(p.at[kQkv] + 64u * warp, code_stride(H), p.at_scales[kQkv] + 8u * warp, H / 16, n_qkv >> 4, xs + 256u * warp, ld, sums + 64u * warp, own_part);
      give_back(kQkv);
      meet(threads);
      if (warp * 32 < qn * R) {
        // as the projection leaves them everywhere else: one rounding ahead of the rotation
        int r, j, head, o;
        const bool in = pair_of(r, j, head, o);
        float v = 0.0f, u = 0.0f;
        Turn t{1.0f, 0.0f, -1};
        if (in) {
          const uint32_t part = parts + (uint32_t)(((j >> 3) * 16 + (j & 7)) * RP + r) * 4u;
          t = lds<Turn>(p.at_turn + 16u * tid);
          v = __bfloat162float(__float2bfloat16_rn(total(part, p.part_step, warps) + b0));
          u = __bfloat162float(__float2bfloat16_rn(total(part + 8u * RP * 4u, p.part_step, warps) + b1));
        }
        if (head < n_heads + n_kv) {
          const float w = v * t.cs - u * t.sn;
          u = v * t.sn + u * t.cs;
          v = w;
        }
        // an even thread takes the pair's first channels, the odd one beside it the second ones
        const bool odd = tid & 1;
        const float got = __shfl_xor_sync(0xffffffffu, odd ? v : u, 1);
        const uint32_t two = odd ? pack_bf16x2(got, u) : pack_bf16x2(v, got);
        const int first = (o & ~1) + (odd ? kDim / 2 : 0), kh = head - n_heads;
        if (in) {
          send(s_mail.heads + ((size_t)r * all_heads + head) * (kDim / 2) + (first >> 1), two, number);
          if (kh >= 0 && t.cache >= 0) *reinterpret_cast<uint32_t*>((kh < n_kv ? L.k_pool + (t.cache * n_kv + kh) * kDim : L.v_pool + (t.cache * n_kv + kh - n_kv) * kDim) + first) = two;
        }
      }
    }

    // ---- attention over chunks, merge of the chunks
#pragma unroll 1
    for (int it = cta; it < items; it += p.ctas) {
      const Item i = it == cta ? s_item : item_of(kern, it);
      if (i.count == 0) continue;  // the same for the whole CTA
      attend(kern, s_mail, number, &s_abort, L.k_pool, L.v_pool, i, it == cta ? block0 : -2, it == cta && block0 >= 0);
    }
    if (more && tid >= threads - 32 && lane < kLayerWords) reinterpret_cast<uint64_t*>(&s_layer[(l + 1) & 1])[lane] = next_word;
    fence_proxy_async();  // keys and values have been where the down projection's rows come now
    if (n_out > 0) give_back(kDown);
    if (meet_any(threads, s_abort)) break;
#pragma unroll 1
    for (int t = p.ctas - 1 - cta; t < merges; t += p.ctas) merge(kern, s_mail, number, &s_abort, t / n_heads, t % n_heads, parts);
    if (p.ctas - 1 - cta < merges) clear_tail(threads);  // where a warp's part is smaller than its room, the rooms reach there

    gain = load4_now(L.norm2 + 4 * tid);

    // ---- output projection (a warp has a head), residual
    if (n_out > 0) {
      uint2 w[R];
      receive<R>(w, number, &s_abort, [&](int r) { return s_mail.attn + ((size_t)r * n_heads + warp) * (kDim / 2) + 2 * lane; }, [](int) { return true; });
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const float2 lo = unpack_bf16x2(w[r].x), hi = unpack_bf16x2(w[r].y);
        stage4(make_float4(lo.x, lo.y, hi.x, hi.y), xs + (uint32_t)r * ld + 256u * warp, sums + 64u * warp + 4u * r, lane);
      }
      __syncwarp();
      if (wait_for(bars + 8u * kOut, parity, &s_abort))
        products<R>(p.at[kOut] + 64u * warp, code_stride(H), p.at_scales[kOut] + 8u * warp, H / 16, t_out, xs + 256u * warp, ld, sums + 64u * warp, own_part);
      give_back(kOut);
      meet(threads);
      if (tid < on) {
        value_of(x_at, o_part);
        x_own += total(o_part, p.part_step, warps);
        send(s_mail.mid + x_at, __float_as_uint(x_own), number);
      }
    }

    // ---- norm, gate and up, SwiGLU
    if (n_gu > 0) {
      norm_rows<R>(warps, nullptr, s_mail.mid, number, H, a.eps, gain, s_red, xs, ld, sums, &s_abort);
      if (wait_for(bars + 8u * kGateUp, parity, &s_abort))
        products<R>(p.at[kGateUp] + 64u * warp, code_stride(H), p.at_scales[kGateUp] + 8u * warp, H / 16, n_gu >> 4, xs + 256u * warp, ld, sums + 64u * warp, own_part);
      meet(threads);
      const int gn = n_gu >> 1;
#pragma unroll 1
      for (int e0 = warp * 32; e0 < gn * R; e0 += threads) {
        const int e = e0 + lane, r = R == 1 ? 0 : e / gn, j = e - r * gn;
        const uint32_t at = parts + (uint32_t)(((j >> 3) * 16 + (j & 7)) * RP + r) * 4u;
        float y = 0.0f;
        if (e < gn * R) {
          const float v = total(at, p.part_step, warps), u = total(at + 8u * RP * 4u, p.part_step, warps);
          y = v / (1.0f + __expf(-v)) * u;
        }
        const float next = __shfl_down_sync(0xffffffffu, y, 1);
        if (e < gn * R && !(lane & 1)) send(s_mail.act + ((size_t)r * I + 8 * (cta * p.gu_tiles) + j) / 2, pack_bf16x2(y, next), number);
      }
    }
    if (more) gain = load4_now(N.norm1 + 4 * tid);

    // ---- down projection, residual
    if (n_out > 0) {
      // (the products of gate and up, where the activations go now, are behind every warp)
      const int blocks5 = I / kDim, pieces = (blocks5 - warp + warps - 1) / warps * R * 16;  // of eight values; a block and row are half a warp
      constexpr int kBatch = 3;
#pragma unroll 1
      for (int e0 = 0; e0 < pieces; e0 += 32 * kBatch) {
        uint2 w[2 * kBatch];
        auto piece = [&](int j, int& ch, int& r, int& b) {
          const int e = e0 + 32 * j + lane;
          ch = e & 15; r = (e >> 4) % R; b = warp + (e >> 4) / R * warps;
          return e < pieces;
        };
        int ch, r, b;
        receive<2 * kBatch>(w, number, &s_abort,
                            [&](int j) {
                              piece(j >> 1, ch, r, b);
                              return s_mail.act + ((size_t)r * I + b * kDim + 8 * ch) / 2 + 2 * (j & 1);
                            },
                            [&](int j) { return e0 + 32 * (j >> 1) + lane < pieces; });
#pragma unroll
        for (int j = 0; j < kBatch; ++j) {
          const uint2 lo = w[2 * j], hi = w[2 * j + 1];
          const float2 f0 = unpack_bf16x2(lo.x), f1 = unpack_bf16x2(lo.y), f2 = unpack_bf16x2(hi.x), f3 = unpack_bf16x2(hi.y);
          float s = ((f0.x + f0.y) + (f1.x + f1.y)) + ((f2.x + f2.y) + (f3.x + f3.y));
          s += __shfl_xor_sync(0xffffffffu, s, 1);
          s += __shfl_xor_sync(0xffffffffu, s, 2);
          if (!piece(j, ch, r, b)) continue;
          sts(xs5 + (uint32_t)r * ld5 + 256u * b + 16u * ch,
              make_uint4(__byte_perm(lo.x, hi.x, 0x5410), __byte_perm(lo.x, hi.x, 0x7632), __byte_perm(lo.y, hi.y, 0x5410), __byte_perm(lo.y, hi.y, 0x7632)));
          if ((ch & 3) == 0) sts(sums5 + (uint32_t)(4 * b + (ch >> 2)) * 16u + 4u * r, -136.0f * s);
        }
      }
      meet(threads);  // the sums of gate and up have been read from where the next ones go
      if (wait_for(bars + 8u * kDown, parity, &s_abort))
        products_blocks<R>(p.at[kDown], code_stride(I), p.at_scales[kDown], I / 16, t_out, xs5, ld5, sums5, own_part, warp, blocks5, warps);
      fence_proxy_async();  // activations have been where gate and up come now
      if (n_gu > 0) give_back(kGateUp);
      meet(threads);
      if (tid < on) {
        value_of(x_at, o_part);
        x_own += total(o_part, p.part_step, warps);
        if (more) send(s_mail.x + x_at, __float_as_uint(x_own), number);
        else a.x[x_at] = x_own;
      }
    } else if (n_gu > 0) {
      give_back(kGateUp);
    }
  }
  __syncthreads();
  if (s_abort) {
    // a wait expired: copies that may still be in flight land before the shared memory is released
#pragma unroll 1
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);
    if (tid == 0) atomicExch(a.status, 2 | (5 << 8));
  }
}

}  // namespace

uint32_t launch_decode_stack(const StackArgs& a, const StackPlan& plan, cudaStream_t stream) {
  if (a.n_layers <= 0) return 0;
  auto kern = a.d.rows == 1 ? decode_stack_kernel<1> : a.d.rows == 2 ? decode_stack_kernel<2> : a.d.rows == 3 ? decode_stack_kernel<3> : decode_stack_kernel<4>;
  const cudaError_t e = allow_shared((const void*)kern, plan.bytes);
  if (e != cudaSuccess) return (uint32_t)e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)plan.ctas);
  cfg.blockDim = dim3((unsigned)(32 * (plan.warps + kBringers)));
  cfg.dynamicSmemBytes = plan.bytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeCooperative;  // its CTAs wait for one another
  attr.val.cooperative = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  (void)cudaLaunchKernelEx(&cfg, kern, Kernel{a, plan});
  return launch_status();
}

}  // namespace lg
