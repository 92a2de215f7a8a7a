// The sampling chain on the device: the logit processors and the multinomial sampler of the
// reference's decode crate over fp32 logits [rows, n] (n = 151936 for the decoder configurations),
// in place, one launch per processor so that a chain keeps the reference's free ordering
// (crates/decode/src/chain.rs:33-76), or one launch for the usual order with a small k (few_survivors_kernel):
//   TemperatureScale    crates/decode/src/processors.rs:18-28
//   TopK                :50-82     (k-th largest by radix select on the float bits: exact)
//   TopP                :89-122    (smallest prefix by descending probability whose mass reaches p)
//   MinP                :130-146
//   RepetitionPenalty   :160-181
//   MultinomialSampler  crates/decode/src/sampler.rs:31-58  (the uniform draw is an input)
// The reference sorts the whole vocabulary per step for TopK / TopP; here the cut is found by a radix select over an
// order-preserving integer key of the logit, 11 bits per pass (three passes of 2048 bins). One CTA per row left most of the
// chip idle; a row is a cluster of eight CTAs that meet through each other's shared memory (rows below kClusterFrom
// values: one CTA). What bounds them is the work that does not shrink with the slice, barriers and the reduction of the
// bins, so a CTA has 256 threads (64 x 151936, TopK by radix select: 49 us; 512 threads 57, 1024 threads with the slice held in
// shared memory 75) and goes over its slice as rarely as it can: values that can still hold the cut, or all that TopK has left,
// are listed in shared memory, and later passes go over the list. Bins hold integers, counts and probabilities in units of
// 2^-40 (2^-56 in rows above 262 thousand values: one below half a unit has no mass), so shared-memory atomics give the same sums in any order and results do not change between runs. Ties
// at the cut are kept in index order, as the reference's stable sort does.
#include <cooperative_groups.h>

#include <algorithm>

#include "common.cuh"
#include "logismos_kernels.h"

namespace {

using namespace lg;

namespace cg = cooperative_groups;

constexpr int kThreads = 256;
constexpr int kBins = 2048;       // 11 bits of the key
constexpr int kMaxCluster = 8;    // portable cluster size
constexpr int kSegment = kBins / kMaxCluster;
static_assert(kSegment == kThreads, "a thread per bin of a segment");
// Below this a CTA's share of a row is one load per thread and the cluster's barriers cost more than they save (top-p of 64
// rows: 2500 values 24 us either way, 4001 28 as one CTA and 27 as a cluster, 8000 42 and 31).
constexpr int kClusterFrom = 2048;
constexpr int kListed = 1024;     // values that a CTA can list
// few_survivors_kernel: the largest k, and the most values that it may find above its bound. Of 2048 shares, k = 256 of them hold the
// 273 largest values on average, so twice k leaves room for values that lie together. (Which calls take it: few_survivors below.)
constexpr int kFewK = 256, kFound = 512;
static_assert(2 * kFound <= kListed && kMaxCluster * kThreads <= 2 * kBins, "found values twice in the list, a key per thread in the bins");

// Masses are counted in units of 2^-(24 + bits): 2^-40 as long as the sums of a slice's low words fit 32 bits (262 thousand values); longer rows, whose
// probabilities are smaller, in units of 2^-56 with carries.
LG_DEVINL int mass_bits(int n, int size) { return (n + size - 1) / size + 4 < 32768 ? 16 : 32; }

// larger float <-> larger key; NaN is ordered like -inf (TopK folds NaN to -inf before its sort)
LG_DEVINL uint32_t order_key(float v) {
  if (v != v) v = -INFINITY;
  const uint32_t b = __float_as_uint(v);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

// a true division, as the reference does (not a reciprocal multiply); four values per thread where the pointer is aligned
__global__ void temperature_kernel(float* __restrict__ logits, int64_t total, float t, int vec) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (!vec) {
    if (i < total) logits[i] = logits[i] / t;
    return;
  }
  if (4 * i + 4 <= total) {
    float4 v = reinterpret_cast<float4*>(logits)[i];
    v.x /= t; v.y /= t; v.z /= t; v.w /= t;
    reinterpret_cast<float4*>(logits)[i] = v;
  } else {
    for (int64_t j = 4 * i; j < total; ++j) logits[j] = logits[j] / t;
  }
}

// one thread per row walks the row's list in order: a token listed twice is penalised twice
__global__ void repetition_penalty_rows_kernel(float* __restrict__ logits, int rows, int n, const uint32_t* __restrict__ tokens,
                                               const int* __restrict__ counts, int max_tokens, float penalty) {
  const int row = blockIdx.x * blockDim.x + threadIdx.x;
  if (row >= rows) return;
  float* l = logits + (size_t)row * n;
  const int c = min(max(counts[row], 0), max_tokens);
  for (int j = 0; j < c; ++j) {
    const uint32_t t = tokens[(size_t)row * max_tokens + j];
    if (t >= (uint32_t)n) continue;
    const float v = l[t];
    l[t] = v > 0.0f ? v / penalty : v * penalty;
  }
}

// What the CTAs of a row tell each other, and the values [begin, end) of the row that this CTA owns.
struct Shared {
  float max[kMaxCluster], sum[kMaxCluster];
  unsigned long long seg[kMaxCluster], above;  // above: of the last radix pass, as are bin and none
  uint32_t bin, none;
  uint32_t tie_counts[kMaxCluster];
  uint32_t best, count;
  float red[32];
  unsigned long long red64[kThreads / 32];
};

struct Row {
  float* l;
  int n, begin, end, rank, size;
  bool vec;  // the row is 16-byte aligned
  const int2* list = nullptr;  // (index, value) of the values that `each` and `mask` go over instead of the slice
  int listed = 0;

  LG_DEVINL Row(float* logits, int n_, const cg::cluster_group& c) : n(n_) {
    rank = (int)c.block_rank();
    size = (int)c.num_blocks();
    l = logits + (size_t)(blockIdx.x / size) * n;
    const int per = ((n + size - 1) / size + 3) & ~3;
    begin = min(rank * per, n);
    end = min(begin + per, n);
    vec = (reinterpret_cast<uintptr_t>(l) & 15) == 0;
  }

  // f(index, value) for every value of the slice, whichever thread it falls to
  template <typename F>
  LG_DEVINL void stream(F&& f) const {
    if (vec) {
      const int full = begin + ((end - begin) & ~3);
#pragma unroll 4
      for (int i = begin + 4 * (int)threadIdx.x; i < full; i += 4 * kThreads) {
        const float4 v = *reinterpret_cast<const float4*>(l + i);
        f(i, v.x); f(i + 1, v.y); f(i + 2, v.z); f(i + 3, v.w);
      }
      for (int i = full + (int)threadIdx.x; i < end; i += kThreads) f(i, l[i]);
    } else {
#pragma unroll 4
      for (int i = begin + (int)threadIdx.x; i < end; i += kThreads) f(i, l[i]);
    }
  }

  template <typename F>
  LG_DEVINL void each(F&& f) const {
    if (!list) { stream(f); return; }
    for (int j = threadIdx.x; j < listed; j += kThreads) {
      const int2 e = list[j];
      f(e.x, __int_as_float(e.y));
    }
  }

  // f(i, v) for the whole slice; the values for which it holds are listed, unless there are more than `room` holds
  template <typename F>
  LG_DEVINL void collect(int2* room, uint32_t* count, F&& f) {
    if (threadIdx.x == 0) *count = 0;
    __syncthreads();
    bool open = true;  // until this thread has seen more than the room holds
    stream([&](int i, float v) {
      if (!f(i, v) || !open) return;
      open = *reinterpret_cast<volatile uint32_t*>(count) <= (uint32_t)kListed;
      if (!open) return;
      const uint32_t lanes = __activemask(), lane = threadIdx.x & 31;
      uint32_t at = 0;
      if (lane == (uint32_t)(__ffs(lanes) - 1)) at = atomicAdd(count, (uint32_t)__popc(lanes));
      at = __shfl_sync(lanes, at, __ffs(lanes) - 1) + __popc(lanes & ((1u << lane) - 1u));
      if (at < (uint32_t)kListed) room[at] = make_int2(i, __float_as_int(v));
    });
    __syncthreads();
    if (*count <= (uint32_t)kListed) { list = room; listed = (int)*count; }
  }

  // the values for which drop(value) holds become -inf; what is -inf already is not written again
  template <typename F>
  LG_DEVINL void mask(F&& drop) const {
    auto one = [&](float& v) {
      const bool d = v != -INFINITY && drop(v);
      if (d) v = -INFINITY;
      return d;
    };
    if (!list && vec) {
      const int full = begin + ((end - begin) & ~3);
#pragma unroll 4
      for (int i = begin + 4 * (int)threadIdx.x; i < full; i += 4 * kThreads) {
        float4 v = *reinterpret_cast<const float4*>(l + i);
        const bool a = one(v.x), b = one(v.y), c = one(v.z), d = one(v.w);
        if (a || b || c || d) *reinterpret_cast<float4*>(l + i) = v;
      }
      for (int i = full + (int)threadIdx.x; i < end; i += kThreads) {
        float v = l[i];
        if (one(v)) l[i] = v;
      }
    } else {
      each([&](int i, float v) { if (one(v)) l[i] = v; });
    }
  }
};

LG_DEVINL void row_sync(const cg::cluster_group& c, const Row& row) {
  if (row.size == 1) __syncthreads();
  else c.sync();
}

// every CTA of the row gets value[r] of each CTA r in its own sh.field[r]; a barrier of the cluster makes it visible
template <typename T>
LG_DEVINL void tell(const cg::cluster_group& c, const Row& row, T* field, T value) {
  if ((int)threadIdx.x < row.size) c.map_shared_rank(field, (int)threadIdx.x)[row.rank] = value;
}

LG_DEVINL unsigned long long block_sum64(unsigned long long v, unsigned long long* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  v = 0;
#pragma unroll
  for (int w = 0; w < kThreads / 32; ++w) v += red[w];
  __syncthreads();
  return v;
}

// The row's maximum and the sum of exp(l - max); finite_only: non-finite logits carry no mass (the sampler). What is
// above -inf is listed where it fits, unless room is null.
LG_DEVINL void row_max_sum(const cg::cluster_group& c, Row& row, bool finite_only, int2* room, Shared& sh, float& mx, float& sum) {
  float m = -INFINITY;
  if (room) {
    row.collect(room, &sh.count, [&](int, float v) {
      m = fmaxf(m, v);  // fmaxf ignores NaN, as f32::max does
      return !(v == -INFINITY);
    });
  } else {
    row.stream([&](int, float v) { m = fmaxf(m, v); });
  }
  tell(c, row, sh.max, block_max(m, sh.red));
  row_sync(c, row);
  mx = sh.max[0];
  for (int r = 1; r < row.size; ++r) mx = fmaxf(mx, sh.max[r]);
  float s = 0.0f;
  auto mass = [&](float v) {
    const bool fin = fabsf(v) <= 3.402823466e38f;  // false for inf and NaN
    return !(finite_only && !fin) && v != -INFINITY ? expf(v - mx) : 0.0f;
  };
  if (row.list) {
    // The list has no order that repeats: a sum of integers, in units of 2^-50 (at most kListed values of at most one).
    unsigned long long q = 0;
    bool nan = false;
    row.each([&](int, float v) {
      const float e = mass(v);
      nan = nan || e != e;
      q += __float2ull_rn(e * 1125899906842624.0f);
    });
    s = (float)block_sum64(q, sh.red64) * (1.0f / 1125899906842624.0f);
    if (__syncthreads_or(nan)) s = NAN;
    if (!finite_only && mx == -INFINITY) s = NAN;  // exp(-inf + inf)
    tell(c, row, sh.sum, s);
  } else {
    row.stream([&](int, float v) { s += mass(v); });
    if (!finite_only && mx == -INFINITY) s = NAN;
    tell(c, row, sh.sum, block_sum(s, sh.red));
  }
  row_sync(c, row);
  sum = 0.0f;
  for (int r = 0; r < row.size; ++r) sum += sh.sum[r];
}

// Radix select shared by TopK (by count) and TopP (by probability mass). Returns the key at which the cut falls and
// leaves in `sh` what lies strictly above it, and `none` when the target was never reached (everything is kept).
template <bool BY_MASS>
LG_DEVINL uint32_t radix_select(const cg::cluster_group& c, Row& row, float mx, float inv_sum, unsigned long long target_mass, uint32_t target_count, int lo_bits,
                                uint32_t* bins, int2* room, Shared& sh) {
  uint32_t* cnt = bins;         // BY_MASS: the leading 24 bits of probabilities, and the lo_bits below them
  uint32_t* lo = bins + kBins;  // (bins without mass cannot hold the cut, so counts of them are not needed)
  const float unit = ldexpf(1.0f, 24 + lo_bits);
  const uint32_t lo_mask = lo_bits ? 0xffffffffu >> (32 - lo_bits) : 0u;
  const bool carries = lo_bits == 32;  // the low words may wrap
  uint32_t prefix = 0, cnt_above = 0;
  unsigned long long mass_above = 0;
#pragma unroll 1
  for (int pass = 0; pass < 3; ++pass) {
    const int shift = pass == 0 ? 21 : pass == 1 ? 10 : 0;
    const uint32_t pmask = pass == 0 ? 0u : pass == 1 ? 0xffe00000u : 0xfffffc00u;
    const uint32_t bmask = pass == 2 ? 1023u : 2047u;
    for (int i = threadIdx.x; i < (BY_MASS ? 2 : 1) * kBins; i += kThreads) bins[i] = 0;
    if (threadIdx.x == 0) sh.none = 1;
    if (pass == 1 && !row.list) row.collect(room, &sh.count, [&](int, float v) { return (order_key(v) & pmask) == prefix; });
    __syncthreads();
    row.each([&](int, float v) {
      const uint32_t key = order_key(v);
      if ((key & pmask) != prefix) return;
      const uint32_t d = (key >> shift) & bmask;
      if (!BY_MASS) {
        atomicAdd(cnt + d, 1u);
        return;
      }
      if (!(v > -INFINITY)) return;
      const unsigned long long m = __float2ull_rn(expf(v - mx) * inv_sum * unit);
      if (m >> lo_bits) atomicAdd(cnt + d, (uint32_t)(m >> lo_bits));
      const uint32_t low = (uint32_t)m & lo_mask;
      if (!low) return;
      if (!carries) atomicAdd(lo + d, low);
      else if (atomicAdd(lo + d, low) + low < low) atomicAdd(cnt + d, 1u);
    });
    row_sync(c, row);
    // the bins are summed over the cluster in kMaxCluster segments, one per CTA (or all by the one CTA), and every CTA
    // gets every segment's total
    const int own_segs = kMaxCluster / row.size;
    __shared__ unsigned long long w_seg[kMaxCluster][kThreads / 32];
    for (int i = 0; i < own_segs; ++i) {
      const int j = (row.rank + i) * kSegment + threadIdx.x;
      unsigned long long m = 0;  // count or mass
      for (int r = 0; r < row.size; ++r) {
        const uint32_t a = c.map_shared_rank(cnt, r)[j];
        m += BY_MASS ? ((unsigned long long)a << lo_bits) + c.map_shared_rank(lo, r)[j] : (unsigned long long)a;
      }
      // the CTA's own segment, which only it reads from here on: the sums stay where its own addends were
      cnt[j] = (uint32_t)(BY_MASS ? m >> lo_bits : m);
      if (BY_MASS) lo[j] = (uint32_t)m & lo_mask;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) m += __shfl_xor_sync(0xffffffffu, m, o);
      if ((threadIdx.x & 31) == 0) w_seg[i][threadIdx.x >> 5] = m;
    }
    __syncthreads();
    if (threadIdx.x < kMaxCluster) {
      const int i = row.size == 1 ? (int)threadIdx.x : 0;
      unsigned long long m = 0;
      for (int w = 0; w < kThreads / 32; ++w) m += w_seg[i][w];
      c.map_shared_rank(sh.seg, row.size == 1 ? 0 : (int)threadIdx.x)[row.rank + i] = m;
    }
    row_sync(c, row);
    // the segment in which the target is reached, from the top (a later pass lies inside a bin that reached it)
    const unsigned long long target = BY_MASS ? target_mass : target_count;
    unsigned long long above = BY_MASS ? mass_above : cnt_above;
    int sel = -1;
    for (int r = kMaxCluster - 1; r >= 0; --r) {
      if (sh.seg[r] == 0) continue;
      if (above + sh.seg[r] >= target) { sel = r; break; }
      above += sh.seg[r];
    }
    if (sel >= 0 && row.rank == (row.size == 1 ? 0 : sel) && threadIdx.x < 32) {  // 32 bins at a time from the top
      const int lane = threadIdx.x, first = sel * kSegment;
      for (int b = kSegment - 32; b >= 0; b -= 32) {
        const int j = first + b + 31 - lane;  // lane 0 holds the highest
        const unsigned long long own = BY_MASS ? ((unsigned long long)cnt[j] << lo_bits) + lo[j] : cnt[j];
        unsigned long long m = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const unsigned long long t = __shfl_up_sync(0xffffffffu, m, o);
          if (lane >= o) m += t;
        }
        const uint32_t hit = __ballot_sync(0xffffffffu, own > 0 && above + m >= target);
        if (hit) {
          const int at = __ffs(hit) - 1;
          const uint32_t bin = (uint32_t)(first + b + 31 - at);
          const unsigned long long over = above + __shfl_sync(0xffffffffu, m - own, at);
          if (lane < row.size) {
            Shared* o = c.map_shared_rank(&sh, lane);
            o->bin = bin; o->above = over; o->none = 0;
          }
          break;
        }
        above += __shfl_sync(0xffffffffu, m, 31);
      }
    }
    row_sync(c, row);
    if (sh.none) return 0;
    prefix |= sh.bin << shift;
    if (BY_MASS) mass_above = sh.above;
    else cnt_above = (uint32_t)sh.above;
    __syncthreads();  // read by all before the next pass sets it again
  }
  return prefix;
}

// Values below the cut become -inf, and of those with key == cut all but the first `keep` in index order.
LG_DEVINL void mask_below_cut(const cg::cluster_group& c, const Row& row, uint32_t cut, unsigned long long keep, bool mask_nan, Shared& sh) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __shared__ uint32_t s_warp[kThreads / 32];
  uint32_t base = 0, ties = 0;  // ties in the slices before this one, and in the row
  if (keep != ~0ull) {
    uint32_t own = 0;
    row.each([&](int, float v) { own += order_key(v) == cut ? 1u : 0u; });
    own = __reduce_add_sync(0xffffffffu, own);
    if (lane == 0) s_warp[warp] = own;
    __syncthreads();
    uint32_t total = 0;
    for (int w = 0; w < kThreads / 32; ++w) total += s_warp[w];
    tell(c, row, sh.tie_counts, total);
    row_sync(c, row);
    for (int r = 0; r < row.size; ++r) {
      if (r < row.rank) base += sh.tie_counts[r];
      ties += sh.tie_counts[r];
    }
  }
  if (keep >= ties) {
    row.mask([&](float v) { return order_key(v) < cut || (mask_nan && v != v); });
    return;
  }
  for (int i0 = row.begin; i0 < row.end; i0 += kThreads) {
    const int i = i0 + threadIdx.x;
    const float v = i < row.end ? row.l[i] : 0.0f;
    const uint32_t key = i < row.end ? order_key(v) : 0u;
    const bool tie = i < row.end && key == cut;
    const uint32_t bal = __ballot_sync(0xffffffffu, tie);
    __syncthreads();
    if (lane == 0) s_warp[warp] = __popc(bal);
    __syncthreads();
    uint32_t before = base;
    for (int w = 0; w < kThreads / 32; ++w) {
      if (w < warp) before += s_warp[w];
      base += s_warp[w];
    }
    const uint32_t rank = before + __popc(bal & ((1u << lane) - 1u));
    if (i < row.end && (key < cut || (tie && rank >= keep) || (mask_nan && v != v))) row.l[i] = -INFINITY;
  }
}

// A CTA may not leave while another still reads its shared memory: every kernel ends with a barrier of the cluster.

__device__ __noinline__ void top_k_row(const cg::cluster_group& c, Row row, int k, uint32_t* bins, int2* room, Shared& sh) {
  row_sync(c, row);  // every CTA of the row runs, so its shared memory may be written
  const uint32_t cut = radix_select<false>(c, row, 0.0f, 0.0f, 0ull, (uint32_t)k, 0, bins, room, sh);
  row.list = nullptr;
  // every element tied with the k-th largest survives (the reference masks only `l < threshold`)
  mask_below_cut(c, row, cut, ~0ull, true, sh);
  row_sync(c, row);
}

__device__ __noinline__ void top_p_row(const cg::cluster_group& c, Row row, float p, uint32_t* bins, int2* room, Shared& sh) {
  row_sync(c, row);  // every CTA of the row runs, so its shared memory may be written
  float mx, sum;
  row_max_sum(c, row, false, room, sh, mx, sum);
  const bool whole = row.list != nullptr;  // the list has all that is above -inf: nothing else is to be masked
  const float inv = sum > 0.0f ? 1.0f / sum : 1.0f;
  const int lo_bits = mass_bits(row.n, row.size);
  const float unit = ldexpf(1.0f, 24 + lo_bits);
  const unsigned long long target = (unsigned long long)ceil((double)p * (double)unit);
  const bool finite = fabsf(mx) <= 3.402823466e38f;
  if (finite && !(sum > 0.0f)) {
    // a NaN took the sum: probabilities stay unnormalised, and the first maximum alone has mass one
    row.list = nullptr;
    mask_below_cut(c, row, order_key(mx), 1ull, false, sh);
  } else if (finite) {  // an infinite maximum leaves no probability that is a number: the mass never reaches p
    const uint32_t cut = radix_select<true>(c, row, mx, inv, target, 0u, lo_bits, bins, room, sh);
    if (!sh.none) {  // otherwise the mass never reaches p: the reference keeps everything
      // the tied elements share one probability; they are taken one by one until the mass reaches p
      const uint32_t b = (cut & 0x80000000u) ? (cut & 0x7fffffffu) : ~cut;
      const unsigned long long q = __float2ull_rn(expf(__uint_as_float(b) - mx) * inv * unit);
      const unsigned long long missing = target > sh.above ? target - sh.above : 0ull;
      if (!whole) row.list = nullptr;
      mask_below_cut(c, row, cut, max((missing + q - 1) / q, 1ull), false, sh);
    }
  }
  row_sync(c, row);
}

__device__ __noinline__ void min_p_row(const cg::cluster_group& c, Row row, float p, int2* room, Shared& sh) {
  row_sync(c, row);  // every CTA of the row runs, so its shared memory may be written
  float mx, sum;
  row_max_sum(c, row, false, room, sh, mx, sum);
  const bool norm = sum > 0.0f;
  const float max_p = norm ? 1.0f / sum : 1.0f;  // exp(0) over the sum
  const float threshold = p * max_p;
  row.mask([&](float v) {
    float pr = expf(v - mx);
    if (norm) pr /= sum;
    return pr < threshold;
  });
  row_sync(c, row);
}

// MultinomialSampler::sample for a given uniform draw. The reference walks the row (u < p_i returns i, else u -= p_i);
// here a CTA owns a contiguous slice, each warp a part of it and each chunk of at least 128 values a part of that. Masses are
// summed per chunk; the warp whose part holds the draw finds its chunk and walks on from there 32 values at a time
// (whole parts walked: one load's latency per 32 values). A value without mass is never drawn.
__device__ __noinline__ void multinomial_row(const cg::cluster_group& c, Row row, const float* uniforms, uint32_t* out, int2* room, Shared& sh) {
  constexpr int kWarps = kThreads / 32;
  __shared__ float s_chunk[kWarps][32], s_mass[kWarps];
  const int n = row.n, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, out_row = blockIdx.x / row.size;
  if (threadIdx.x == 0) sh.best = 0xffffffffu;
  row_sync(c, row);  // every CTA of the row runs, so its shared memory may be written
  float mx, sum;
  row_max_sum(c, row, true, room, sh, mx, sum);
  uint32_t* best = c.map_shared_rank(&sh.best, 0);
  if (!(sum > 0.0f)) {  // no mass anywhere: greedy (first strict maximum from -inf, index 0 if none)
    uint32_t bi = 0xffffffffu;
    row.each([&](int i, float v) { if (v == mx && v > -INFINITY) bi = min(bi, (uint32_t)i); });
    if (bi != 0xffffffffu) atomicMin(best, bi);
    row_sync(c, row);
    if (row.rank == 0 && threadIdx.x == 0) out[out_row] = sh.best == 0xffffffffu ? 0u : sh.best;
    return;
  }
  const float u = uniforms[out_row];
  auto prob = [&](int i) {
    const float v = row.l[i];
    return v != -INFINITY && fabsf(v) <= 3.402823466e38f ? expf(v - mx) / sum : 0.0f;
  };
  const int per = (row.end - row.begin + kWarps - 1) / kWarps;
  const int i0 = min(row.begin + warp * per, row.end), i1 = min(i0 + per, row.end);
  const int chunk = 128 * ((per + 128 * 32 - 1) / (128 * 32)), n_chunks = (i1 - i0 + chunk - 1) / max(chunk, 1);  // up to 32 chunks
  for (int k = 0; k < n_chunks; ++k) {
    const int c0 = i0 + k * chunk, c1 = min(c0 + chunk, i1);
    float m = 0.0f;
#pragma unroll 4
    for (int i = c0 + lane; i < c1; i += 32) m += prob(i);
    m = warp_sum(m);
    if (lane == 0) s_chunk[warp][k] = m;
  }
  __syncwarp();
  float upto = lane < n_chunks ? s_chunk[warp][lane] : 0.0f;  // of the chunks up to and with this one
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float t = __shfl_up_sync(0xffffffffu, upto, o);
    if (lane >= o) upto += t;
  }
  const float mine = __shfl_sync(0xffffffffu, upto, 31);
  if (lane == 0) s_mass[warp] = mine;
  __syncthreads();
  // The parts' bounds: each is the next one's beginning to the bit (sums from the left over warps, then over CTAs), so every draw
  // below the total falls into exactly one part, and that part has mass.
  float before = 0.0f, up_to = 0.0f, cta = 0.0f;
  for (int w = 0; w < kWarps; ++w) {
    if (w == warp) before = cta;
    cta += s_mass[w];
    if (w == warp) up_to = cta;
  }
  tell(c, row, sh.max, cta);  // the maxima were read by every CTA ahead of the last barrier
  row_sync(c, row);
  float base = 0.0f, total = 0.0f;
  for (int r = 0; r < row.size; ++r) {
    if (r == row.rank) base = total;
    total += sh.max[r];
  }
  if (u < total) {
    if (u >= base + before && u < base + up_to) {
      float r = u - (base + before);
      // the first chunk that reaches the draw; where rounding leaves none, the last that has mass
      const uint32_t reach = __ballot_sync(0xffffffffu, lane < n_chunks && r < upto), full = __ballot_sync(0xffffffffu, lane < n_chunks && s_chunk[warp][min(lane, n_chunks - 1)] > 0.0f);
      const int from = reach ? __ffs(reach) - 1 : 31 - __clz(full);
      const float ahead = __shfl_sync(0xffffffffu, upto, max(from - 1, 0));
      if (from > 0) r = fmaxf(r - ahead, 0.0f);
      int last = -1;  // the last value with mass: what the draw comes to where rounding carries it past the part
      for (int i = i0 + from * chunk; i < i1; i += 32) {
        const float pr = i + lane < i1 ? prob(i + lane) : 0.0f;
        float incl = pr;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const float t = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += t;
        }
        const uint32_t has = __ballot_sync(0xffffffffu, pr > 0.0f), hit = __ballot_sync(0xffffffffu, pr > 0.0f && r < incl);
        if (has) last = i + (hit ? __ffs(hit) - 1 : 31 - __clz(has));
        if (hit) break;
        r -= __shfl_sync(0xffffffffu, incl, 31);
      }
      if (lane == 0 && last >= 0) atomicMin(best, (uint32_t)last);
    }
  } else if (mine > 0.0f) {  // a draw that rounding leaves above the total: the last value with mass
    int last = -1;
    for (int i = i0; i < i1; i += 32) {
      const uint32_t has = __ballot_sync(0xffffffffu, i + lane < i1 && prob(i + lane) > 0.0f);
      if (has) last = i + 31 - __clz(has);
    }
    if (lane == 0 && last >= 0) atomicMin(best, (uint32_t)(n - 1 - last));  // the largest index
  }
  row_sync(c, row);
  if (row.rank == 0 && threadIdx.x == 0) out[out_row] = sh.best == 0xffffffffu ? (uint32_t)(n - 1) : u < total ? sh.best : (uint32_t)(n - 1) - sh.best;
}


// 215 -> 100 us on 64 x 151936, 36 after a top-k of 50
__global__ void __launch_bounds__(kThreads, 4)
top_p_kernel(float* __restrict__ logits, int n, float p) {
  __shared__ uint32_t bins[2 * kBins];
  __shared__ int2 room[kListed];
  __shared__ Shared sh;
  const cg::cluster_group c = cg::this_cluster();
  top_p_row(c, Row(logits, n, c), p, bins, room, sh);
}

// 53 -> 39 us on 64 x 151936
__global__ void __launch_bounds__(kThreads, 4)
min_p_kernel(float* __restrict__ logits, int n, float p) {
  __shared__ int2 room[kListed];
  __shared__ Shared sh;
  const cg::cluster_group c = cg::this_cluster();
  min_p_row(c, Row(logits, n, c), p, room, sh);
}

// 88 -> 35 us on 64 x 151936 after top-k 50
__global__ void __launch_bounds__(kThreads, 4)
multinomial_kernel(const float* __restrict__ logits, int n, const float* __restrict__ uniforms, uint32_t* __restrict__ out) {
  __shared__ int2 room[kListed];
  __shared__ Shared sh;
  const cg::cluster_group c = cg::this_cluster();
  multinomial_row(c, Row(const_cast<float*>(logits), n, c), uniforms, out, room, sh);
}

// where few_survivors does not hold
__global__ void __launch_bounds__(kThreads, 4)
top_k_kernel(float* __restrict__ logits, int n, int k) {
  __shared__ uint32_t bins[kBins];
  __shared__ int2 room[kListed];
  __shared__ Shared sh;
  const cg::cluster_group c = cg::this_cluster();
  top_k_row(c, Row(logits, n, c), k, bins, room, sh);
}

// Temperature, top-k with few survivors and what a chain does with these.
struct Chain {
  float temperature;      // 1: none
  int k;                  // 1 .. kFewK, below n
  float p, min_p;         // p >= 1, min_p <= 0: none
  const float* uniforms;  // null: no draw
  uint32_t* out;
};

// Sums of the masses of list[0 .. m) as row_max_sum leaves them: integers per slice, fp32 over the slices. Every thread gets the sum.
LG_DEVINL float survivor_sum(const int2* list, int m, int n, int size, float mx, bool finite_only, unsigned long long* seg, uint32_t* nan) {
  const int per = ((n + size - 1) / size + 3) & ~3;
  __syncthreads();
  if (threadIdx.x < kMaxCluster) { seg[threadIdx.x] = 0; nan[threadIdx.x] = 0; }
  __syncthreads();
  for (int j = threadIdx.x; j < m; j += kThreads) {
    const float v = __int_as_float(list[j].y), e = finite_only && !(fabsf(v) <= 3.402823466e38f) ? 0.0f : expf(v - mx);
    if (e != e) nan[list[j].x / per] = 1;
    else atomicAdd(seg + list[j].x / per, __float2ull_rn(e * 1125899906842624.0f));
  }
  __syncthreads();
  float sum = 0.0f;
  for (int r = 0; r < size; ++r) sum += nan[r] ? NAN : (float)seg[r] * (1.0f / 1125899906842624.0f);
  return sum;
}

// One launch for temperature, top-k, top-p, min-p and the draw, where k is small: after top-k the rest of the chain has k values to look at
// and no row. What bounds it is one read and one write of the rows. The read leaves each thread the maximum of its
// share; the k-th largest of the row's 2048 maxima is a lower bound of its k-th largest value (k shares hold a value that
// large), few values lie above it, and only the threads whose maximum does go over their share again. The values found
// go to the first CTA of the row, which orders them by value (ties by index) and finishes the chain while all CTAs set the row to -inf; then it
// puts the survivors back. Division by the temperature keeps the order, so only maxima, bounds and the values found are divided.
// A row with more values above the bound than kFound (many ties) goes through the general functions. Masses and sums are
// formed as these form them, so the survivors are the same. 64 x 151936, temperature, k = 50, p = 0.95 and the draw: 25 us on rows that lie in L2, 31
// from HBM (39 MB read and written, 12 us at the copy rate) against 136 in four launches; top-k alone 53 before.
__global__ void __launch_bounds__(kThreads, 4)
few_survivors_kernel(float* __restrict__ logits, int n, const Chain ch) {
  __shared__ __align__(16) uint32_t bins[2 * kBins];
  __shared__ int2 room[kListed];
  __shared__ Shared sh;
  __shared__ uint32_t s_count[32], s_found, s_nan[kMaxCluster];
  const cg::cluster_group c = cg::this_cluster();
  const Row row(logits, n, c);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool divide = ch.temperature != 1.0f;
  auto scaled = [&](float v) { return divide ? v / ch.temperature : v; };
  // 16-byte pieces of the row, the first and the last one perhaps in part; piece q holds values 4 q - lead ..
  const int lead = (int)((reinterpret_cast<uintptr_t>(row.l) >> 2) & 3), pieces = (lead + n + 3) >> 2, per = (pieces + row.size - 1) / row.size;
  const int q0 = min(row.rank * per, pieces), q1 = min(q0 + per, pieces);
  float* const first = row.l - lead;
  auto whole = [&](int q) { return 4 * q >= lead && 4 * q + 4 <= lead + n; };
  auto load = [&](int q) {  // a partial one
    const int i = 4 * q - lead;
    auto at = [&](int j) { return j >= 0 && j < n ? row.l[j] : -INFINITY; };
    return make_float4(at(i), at(i + 1), at(i + 2), at(i + 3));
  };
  // the pieces of this slice that are whole; what is left of it is the row's first or last piece
  const int w0 = q0 == 0 && lead && q1 > q0 ? 1 : q0, w1 = q1 == pieces && q1 > q0 && !whole(pieces - 1) ? max(q1 - 1, w0) : q1;
  if (tid < 32) s_count[tid] = 0;
  if (tid == 0) s_found = 0;
  c.barrier_arrive();  // every CTA of the row runs once this is passed, so its shared memory may be written
  float m = -INFINITY;
  auto larger = [&](float4 v) { m = fmaxf(m, fmaxf(fmaxf(v.x, v.y), fmaxf(v.z, v.w))); };  // fmaxf drops NaN, which top-k takes for -inf
#pragma unroll 8
  for (int q = w0 + tid; q < w1; q += kThreads) larger(*reinterpret_cast<const float4*>(first + 4 * (size_t)q));
  // the partial pieces belong to the last two threads
  const int part = tid == kThreads - 1 && w0 > q0 ? q0 : tid == kThreads - 2 && w1 < q1 ? q1 - 1 : -1;
  if (part >= 0) larger(load(part));
  c.barrier_wait();
  uint32_t* const keys = bins;  // [size][kThreads]
  const uint32_t own_key = order_key(m);
  for (int r = 0; r < row.size; ++r) c.map_shared_rank(keys, r)[row.rank * kThreads + tid] = own_key;
  row_sync(c, row);
  uint32_t held[kMaxCluster];
  for (int r = 0; r < kMaxCluster; ++r) held[r] = r < row.size ? keys[r * kThreads + tid] : 0u;
  uint32_t bound = 0;  // the leading 16 bits of the k-th largest maximum, two at a time
#pragma unroll 1
  for (int bit = 30; bit >= 16; bit -= 2) {
    const uint32_t step = 1u << bit;
    uint32_t c12 = 0, c3 = 0;
#pragma unroll
    for (int r = 0; r < kMaxCluster; ++r) {
      c12 += (held[r] >= bound + step ? 1u : 0u) + (held[r] >= bound + 2 * step ? 0x10000u : 0u);
      c3 += held[r] >= bound + 3 * step ? 1u : 0u;
    }
    c12 = __reduce_add_sync(0xffffffffu, c12);
    c3 = __reduce_add_sync(0xffffffffu, c3);
    if (lane == 0) {
      if (c12) atomicAdd(s_count + bit, c12);
      if (c3) atomicAdd(s_count + bit + 1, c3);
    }
    __syncthreads();
    const uint32_t n12 = s_count[bit], n3 = s_count[bit + 1], k = (uint32_t)ch.k;
    bound += n3 >= k ? 3 * step : (n12 >> 16) >= k ? 2 * step : (n12 & 0xffffu) >= k ? step : 0u;
  }
  // at and below -inf (whose truncated key would be a NaN) every number counts
  const float low = bound <= 0x007fffffu ? -INFINITY : scaled(__uint_as_float(bound & 0x80000000u ? bound & 0x7fffffffu : ~bound));
  uint32_t* const found = c.map_shared_rank(&s_found, 0);
  int2* const list = c.map_shared_rank(room, 0);
  auto above = [&](float v) { return v >= low && v > -INFINITY; };
  auto look = [&](int q, float4 v) {
    const float w[4] = {scaled(v.x), scaled(v.y), scaled(v.z), scaled(v.w)};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (!above(w[j])) continue;
      const uint32_t at = atomicAdd(found, 1u);
      if (at < (uint32_t)kFound) list[at] = make_int2(4 * q + j - lead, __float_as_int(w[j]));
    }
  };
  const bool has = above(scaled(m));
  if (has && part >= 0) look(part, load(part));
  // the lanes of a warp go over the share of each of them that has something, one round of loads for 32 pieces
  for (uint32_t lanes = __ballot_sync(0xffffffffu, has); lanes; lanes &= lanes - 1) {
    const int whose = w0 + (tid & ~31) + __ffs(lanes) - 1;
    for (int q = whose + lane * kThreads; q < w1; q += 32 * kThreads) look(q, *reinterpret_cast<const float4*>(first + 4 * (size_t)q));
  }
  row_sync(c, row);
  const uint32_t total = *found;
  if (total > (uint32_t)kFound) {
    if (divide) {
      for (int i = row.begin + tid; i < row.end; i += kThreads) row.l[i] = row.l[i] / ch.temperature;
    }
    top_k_row(c, row, ch.k, bins, room, sh);
    if (ch.p < 1.0f) top_p_row(c, row, ch.p, bins, room, sh);
    if (ch.min_p > 0.0f) min_p_row(c, row, ch.min_p, room, sh);
    if (ch.uniforms) multinomial_row(c, row, ch.uniforms, ch.out, room, sh);
    return;
  }
  const float4 none = make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
#pragma unroll 4
  for (int q = w0 + tid; q < w1; q += kThreads) *reinterpret_cast<float4*>(first + 4 * (size_t)q) = none;
  if (part >= 0)
    for (int i = max(4 * part - lead, 0); i < min(4 * part + 4 - lead, n); ++i) row.l[i] = -INFINITY;
  int kept = 0;
  int2* const sorted = room + kFound;  // by value, ties by index
  if (row.rank == 0) {
    const int count = (int)total;
    for (int j = tid; j < count; j += kThreads) {
      const int2 e = room[j];
      const uint32_t key = order_key(__int_as_float(e.y));
      int rank = 0;
      for (int i = 0; i < count; ++i) {
        const int2 o = room[i];
        const uint32_t other = order_key(__int_as_float(o.y));
        rank += other > key || (other == key && o.x < e.x) ? 1 : 0;
      }
      sorted[rank] = e;
    }
    __syncthreads();
    auto value = [&](int j) { return __int_as_float(sorted[j].y); };
    auto leading = [&](auto&& keep) {  // how many of the kFound first hold
      int k = 0;
#pragma unroll
      for (int j0 = 0; j0 < kFound; j0 += kThreads) k += __syncthreads_count(j0 + tid < kept && keep(j0 + tid));
      return k;
    };
    unsigned long long* const seg = sh.seg;
    kept = count;
    if (count > ch.k) {
      const uint32_t cut = order_key(value(ch.k - 1));  // what ties with the k-th largest survives
      kept = leading([&](int j) { return order_key(value(j)) >= cut; });
    }
    const float mx = kept ? value(0) : -INFINITY;
    if (ch.p < 1.0f && fabsf(mx) <= 3.402823466e38f) {
      const float sum = survivor_sum(sorted, kept, n, row.size, mx, false, seg, s_nan), inv = 1.0f / sum;
      const int bits = mass_bits(n, row.size);
      const float unit = ldexpf(1.0f, 24 + bits);
      const unsigned long long target = max((unsigned long long)ceil((double)ch.p * (double)unit), 1ull);
      unsigned long long* const mass = reinterpret_cast<unsigned long long*>(bins);
      for (int j = tid; j < kept; j += kThreads) mass[j] = __float2ull_rn(expf(value(j) - mx) * inv * unit);
      __syncthreads();
      kept = leading([&](int j) {
        unsigned long long ahead = 0;
        for (int i = 0; i < j; ++i) ahead += mass[i];
        return ahead < target;
      });
    }
    if (ch.min_p > 0.0f && kept) {
      const float sum = survivor_sum(sorted, kept, n, row.size, mx, false, seg, s_nan);
      const bool norm = sum > 0.0f;
      const float threshold = ch.min_p * (norm ? 1.0f / sum : 1.0f);
      kept = leading([&](int j) {
        float pr = expf(value(j) - mx);
        if (norm) pr /= sum;
        return !(pr < threshold);
      });
    }
    if (ch.uniforms) {
      const float sum = survivor_sum(sorted, kept, n, row.size, mx, true, seg, s_nan);
      int2* const by_index = room;  // (index, probability)
      for (int j = tid; j < kept; j += kThreads) {
        const int own = sorted[j].x;
        const float v = value(j);
        int rank = 0;
        for (int i = 0; i < kept; ++i) rank += sorted[i].x < own ? 1 : 0;
        // without mass anywhere the first maximum is taken
        const float pr = !(sum > 0.0f) ? (v == mx ? 1.0f : 0.0f) : fabsf(v) <= 3.402823466e38f ? expf(v - mx) / sum : 0.0f;
        by_index[rank] = make_int2(own, __float_as_int(pr));
      }
      __syncthreads();
      if (warp == 0) {
        const int out_row = blockIdx.x / row.size;
        float r = sum > 0.0f ? ch.uniforms[out_row] : 0.0f;
        int token = 0;  // the last value with mass where rounding carries the draw past all of them
        for (int j0 = 0; j0 < kept; j0 += 32) {
          const int j = j0 + lane;
          const float pr = j < kept ? __int_as_float(by_index[j].y) : 0.0f;
          float incl = pr;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const float t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
          }
          const uint32_t has = __ballot_sync(0xffffffffu, pr > 0.0f), hit = __ballot_sync(0xffffffffu, pr > 0.0f && r < incl);
          if (has) token = by_index[j0 + (hit ? __ffs(hit) - 1 : 31 - __clz(has))].x;
          if (hit) break;
          r -= __shfl_sync(0xffffffffu, incl, 31);
        }
        if (lane == 0) ch.out[out_row] = (uint32_t)token;
      }
    }
  }
  row_sync(c, row);  // the row is -inf
  if (row.rank == 0)
    for (int j = tid; j < kept; j += kThreads) row.l[sorted[j].x] = __int_as_float(sorted[j].y);
}

// Calls that few_survivors_kernel takes. Its time grows with k (each found value is an atomic, a further look at a share and a row of the ranking), and where k comes near the number of
// shares that hold anything, most of a row is found and the general functions follow behind. What it saves are the launches of the chain, top-p's first, and reading long rows again. The
// lines lie below the crossings measured at 1 and 64 rows of 300 to 151936 random values, its time against the launches', just within | at the next size beyond:
// top-k alone: k = 24 | 48 at 300 values 0.85 | 1.2, 64 | 96 at 2048 1.0 | 1.17, 64 | 112 at 8192 0.87 | 1.03, 192 | 256 at 151936 0.80 | 1.12;
// with the draw: 24 | 48 at 300 0.73 | 1.06, 80 | 112 at 1500 0.94 | 1.15, 80 | 112 at 2048 0.88 | 1.06, 96 | 160 at 8192 0.78 | 1.11, 192 | 256 at 65536 0.80 | 1.16;
// with top-p as well: 32 | 80 at 300 0.51 | 1.21, 128 | 160 at 1500 0.84 | 1.10, 160 | 224 at 2048 0.78 | 1.17, 192 | 256 at 8192 0.76 | 1.04.
bool few_survivors(int n, int k, float p, bool draw) {
  const int shares = std::min((n + 3) / 4, (n < kClusterFrom ? 1 : kMaxCluster) * kThreads);
  const int most = p < 1.0f ? std::min(9 * shares / 16, 160 + n / 256) : draw ? std::min(3 * shares / 8, 80 + n / 512) : std::min(3 * shares / 8, 64 + n / 1024);
  return k > 0 && k < n && k <= std::min(most, kFewK);
}

// a row is a cluster of eight CTAs, or one CTA
template <typename... P, typename... A>
uint32_t launch_rows(void (*kern)(P...), int rows, int n, void* stream, A... args) {
  const unsigned size = n >= kClusterFrom ? kMaxCluster : 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)rows * size);
  cfg.blockDim = dim3(kThreads);
  cfg.stream = (cudaStream_t)stream;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = size;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  (void)cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
  return launch_status();
}

}  // namespace

extern "C" {

uint32_t logismos_launch_temperature_f32(void* logits, int32_t rows, int32_t n, float temperature, void* stream) {
  lg::LaunchScope launch_scope_;
  if (rows < 0 || n < 0 || !logits) return lg::kInvalidValue;
  const float t = fmaxf(temperature, 1e-6f);
  if (fabsf(t - 1.0f) < 1e-9f || rows == 0 || n == 0) return 0;
  const int64_t total = (int64_t)rows * n;
  const int vec = ((uintptr_t)logits & 15) == 0;
  const int64_t threads = vec ? (total + 3) / 4 : total;
  temperature_kernel<<<(unsigned)((threads + 255) / 256), 256, 0, (cudaStream_t)stream>>>((float*)logits, total, t, vec);
  return lg::launch_status();
}

uint32_t logismos_launch_top_k_f32(void* logits, int32_t rows, int32_t n, int32_t k, void* stream) {
  lg::LaunchScope launch_scope_;
  if (rows < 0 || n < 0 || k < 0 || !logits) return lg::kInvalidValue;
  if (k == 0 || k >= n || rows == 0) return 0;
  if (few_survivors(n, k, 1.0f, false)) return launch_rows(few_survivors_kernel, rows, n, stream, (float*)logits, n, Chain{1.0f, k, 1.0f, 0.0f, nullptr, nullptr});
  return launch_rows(top_k_kernel, rows, n, stream, (float*)logits, n, k);
}

uint32_t logismos_launch_top_p_f32(void* logits, int32_t rows, int32_t n, float p, void* stream) {
  lg::LaunchScope launch_scope_;
  if (rows < 0 || n < 0 || !logits) return lg::kInvalidValue;
  const float pc = fminf(fmaxf(p, 0.0f), 1.0f);
  if (pc >= 1.0f || rows == 0 || n == 0) return 0;
  return launch_rows(top_p_kernel, rows, n, stream, (float*)logits, n, pc);
}

uint32_t logismos_launch_min_p_f32(void* logits, int32_t rows, int32_t n, float p, void* stream) {
  lg::LaunchScope launch_scope_;
  if (rows < 0 || n < 0 || !logits) return lg::kInvalidValue;
  const float pc = fminf(fmaxf(p, 0.0f), 1.0f);
  if (pc <= 0.0f || rows == 0 || n == 0) return 0;
  return launch_rows(min_p_kernel, rows, n, stream, (float*)logits, n, pc);
}

uint32_t logismos_launch_repetition_penalty_f32(void* logits, int32_t rows, int32_t n, const void* tokens_u32,
                                                const void* counts_i32, int32_t max_tokens, float penalty, void* stream) {
  lg::LaunchScope launch_scope_;
  if (rows < 0 || n < 0 || max_tokens < 0 || !logits || (max_tokens > 0 && (!tokens_u32 || !counts_i32))) return lg::kInvalidValue;
  if (fabsf(penalty - 1.0f) < 1e-9f || rows == 0 || n == 0 || max_tokens == 0) return 0;
  repetition_penalty_rows_kernel<<<(rows + 63) / 64, 64, 0, (cudaStream_t)stream>>>((float*)logits, rows, n, (const uint32_t*)tokens_u32,
                                                                                     (const int*)counts_i32, max_tokens, penalty);
  return lg::launch_status();
}

uint32_t logismos_launch_multinomial_f32(const void* logits, int32_t rows, int32_t n, const void* uniforms_f32, void* out_u32,
                                         void* stream) {
  lg::LaunchScope launch_scope_;
  if (rows < 0 || n < 0 || !out_u32 || (rows > 0 && n > 0 && (!logits || !uniforms_f32))) return lg::kInvalidValue;
  if (rows == 0) return 0;
  if (n == 0) return (uint32_t)cudaMemsetAsync(out_u32, 0, (size_t)rows * 4, (cudaStream_t)stream);  // an empty slice samples 0
  return launch_rows(multinomial_kernel, rows, n, stream, (const float*)logits, n, (const float*)uniforms_f32, (uint32_t*)out_u32);
}

uint32_t logismos_launch_sample_chain_f32(void* logits, int32_t rows, int32_t n, float temperature, int32_t k, float p, float min_p, const void* uniforms_f32,
                                          void* out_u32, void* stream) {
  lg::LaunchScope launch_scope_;
  if (rows < 0 || n < 0 || k < 0 || !logits || !out_u32 || (rows > 0 && n > 0 && !uniforms_f32)) return lg::kInvalidValue;
  if (rows == 0) return 0;
  if (few_survivors(n, k, p, true)) {
    const float t = fmaxf(temperature, 1e-6f);
    return launch_rows(few_survivors_kernel, rows, n, stream, (float*)logits, n,
                       Chain{fabsf(t - 1.0f) < 1e-9f ? 1.0f : t, k, fminf(fmaxf(p, 0.0f), 1.0f), fminf(fmaxf(min_p, 0.0f), 1.0f), (const float*)uniforms_f32, (uint32_t*)out_u32});
  }
  uint32_t rc = logismos_launch_temperature_f32(logits, rows, n, temperature, stream);
  if (!rc) rc = logismos_launch_top_k_f32(logits, rows, n, k, stream);
  if (!rc) rc = logismos_launch_top_p_f32(logits, rows, n, p, stream);
  if (!rc) rc = logismos_launch_min_p_f32(logits, rows, n, min_p, stream);
  return rc ? rc : logismos_launch_multinomial_f32(logits, rows, n, uniforms_f32, out_u32, stream);
}

}  // extern "C"
