// Helpers shared by the model executors: device buffers, int4 matrices on the device, error macro.
#pragma once
#include <cuda_runtime.h>
#include <sys/mman.h>

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <string>
#include <thread>
#include <vector>

#include "int4_rows.h"
#include "logismos_kernels.h"
#include "logismos_model.h"

namespace lg {
int sm_count();  // cudacore.cu
}

namespace lgm {

void set_error(const std::string& s);

inline uint16_t f32_to_bf16(float f) {
  uint32_t u;
  std::memcpy(&u, &f, 4);
  if ((u & 0x7fffffffu) > 0x7f800000u) return (uint16_t)((u >> 16) | 0x0040u);
  u += 0x7fffu + ((u >> 16) & 1u);
  return (uint16_t)(u >> 16);
}

struct Buf {
  void* p = nullptr;
  bool alloc(size_t n) { return cudaMalloc(&p, n ? n : 1) == cudaSuccess; }
  bool upload(const void* src, size_t n) { return alloc(n) && cudaMemcpy(p, src, n, cudaMemcpyHostToDevice) == cudaSuccess; }
  void release() { if (p) cudaFree(p); p = nullptr; }
};

// Rows of fp32 from the device to pageable host memory, each to a place of its own. A copy into pageable memory goes through
// the driver's staging at a few GB/s, and a temporary of the same size costs its page faults besides: 64 rows of 32768
// took 1.8 ms that way. Here the rows land in a pinned buffer of at most kCap bytes, part by part, and several threads move each
// part on, every one a range of the columns. They take the destination's page faults while the first part is on its way, so that
// what is left behind the last part is an eighth of it for each: 0.73 -> 0.41 ms, of which the transfer takes 0.31.
// Eight processes at once on 16 cores, 310 us of transfer, pages of 4 KB / 2 MB: 1.00 / 0.57 ms, with parts handed to three threads as before 1.06 / 0.52 (one process: 0.75 / 0.54 against 1.11 / 0.73).
struct HostRows {
  static constexpr size_t kCap = (size_t)16 << 20, kParts = 8, kAlone = (size_t)1 << 20, kMovers = 8, kPage = 4096;
  uint8_t* pinned = nullptr;
  size_t capacity = 0;
  cudaEvent_t landed[kParts] = {};

  void release() {
    if (pinned) cudaFreeHost(pinned);
    pinned = nullptr;
    capacity = 0;
    for (cudaEvent_t& e : landed) {
      if (e) cudaEventDestroy(e);
      e = nullptr;
    }
  }

  // whether the destination of some of the rows has pages
  static bool there(const float* host_out, size_t width, const int* order, int n) {
    for (int i = 0; i < 4; ++i) {
      const uintptr_t at = (uintptr_t)(host_out + (size_t)order[(size_t)(n - 1) * i / 3] * width + width / 2);
      unsigned char in = 0;
      if (mincore((void*)(at & ~(uintptr_t)(kPage - 1)), 1, &in) != 0 || !(in & 1)) return false;
    }
    return true;
  }

  // row k of dev [rows][width] to host_out + order[k] * width; nothing on the device writes the rows meanwhile
  cudaError_t copy(const void* dev, int rows, size_t width, const int* order, float* host_out, cudaStream_t s) {
    const size_t row = width * 4, want = std::max(row, std::min(kCap, row * (size_t)rows));
    if (rows <= 0 || row == 0) return cudaSuccess;
    if (capacity < want) {
      release();
      if (cudaMallocHost((void**)&pinned, want) != cudaSuccess) {
        pinned = nullptr;
        (void)cudaGetLastError();
      } else {
        capacity = want;
      }
    }
    for (cudaEvent_t& e : landed)
      if (pinned && !e && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) return cudaGetLastError();
    if (!pinned) {  // no pinned memory to be had: straight to the destination
      for (int k = 0; k < rows; ++k) {
        const cudaError_t e = cudaMemcpy(host_out + (size_t)order[k] * width, (const uint8_t*)dev + (size_t)k * row, row, cudaMemcpyDeviceToHost);
        if (e != cudaSuccess) return e;
      }
      return cudaSuccess;
    }
    const int room = (int)std::min<size_t>(capacity / row, (size_t)rows);
    for (int r0 = 0; r0 < rows; r0 += room) {
      const int n = std::min(room, rows - r0), parts = (size_t)n * row <= kAlone ? 1 : std::min<int>((int)kParts, n);
      for (int i = 0; i < parts; ++i) {
        const int a = n * i / parts, b = n * (i + 1) / parts;
        cudaError_t e = cudaMemcpyAsync(pinned + (size_t)a * row, (const uint8_t*)dev + (size_t)(r0 + a) * row, (size_t)(b - a) * row, cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaEventRecord(landed[i], s);
        if (e != cudaSuccess) {
          (void)cudaStreamSynchronize(s);  // nothing is on its way to the buffer when it is given up
          return e;
        }
      }
      // A quarter of a MB each; below 2 MB one alone where the destination's pages are there already, as in memory that a program has freed and gets again (9 / 12 / 15 rows of 32768,
      // pages there: 47 / 62 / 77 us alone, 120 / 144 / 175 by threads; not there: 274 / 370 / 466 against 190 / 222 / 290).
      const bool alone = parts == 1 || ((size_t)n * row < 2 * kAlone && there(host_out, width, order + r0, n));
      const int movers = alone ? 1 : (int)std::max(1u, std::min({(unsigned)kMovers, std::thread::hardware_concurrency(), (unsigned)(4 * (size_t)n * row / kAlone)}));
      std::atomic<int> arrived{0};  // parts in the pinned buffer; negative: no more will come
      auto move_on = [&](int i, int w) {
        const size_t c0 = width * w / movers, c1 = width * (w + 1) / movers;
        for (int k = n * i / parts; k < n * (i + 1) / parts; ++k)
          std::memcpy(host_out + (size_t)order[r0 + k] * width + c0, pinned + (size_t)k * row + c0 * 4, (c1 - c0) * 4);
      };
      // The page faults of a range. An exchange of zero for zero asks for the page as a write does and leaves what it finds (rows that do not arrive stay as they were); reading the byte first
      // maps the page twice, and the second time with a flush on every core: 8 MB in pages of 4 KB then took 9 ms in place of 0.75.
      auto touch = [&](int w) {
        const size_t c0 = width * w / movers, c1 = width * (w + 1) / movers;
        for (int k = 0; k < n; ++k) {
          uint8_t* dst = reinterpret_cast<uint8_t*>(host_out + (size_t)order[r0 + k] * width + c0);
          for (size_t at = 0; at < (c1 - c0) * 4; at += kPage) {
            uint8_t zero = 0;
            __atomic_compare_exchange_n(dst + at, &zero, (uint8_t)0, false, __ATOMIC_RELAXED, __ATOMIC_RELAXED);
          }
        }
      };
      // A thread of its own for a range of columns. Only the calling one calls CUDA: a new thread stands on device 0 until it chooses another.
      auto mover = [&](int w) {
        touch(w);
        for (int i = 0; i < parts; ++i) {
          int there;
          while ((there = arrived.load(std::memory_order_acquire)) >= 0 && there <= i) std::this_thread::yield();
          if (there < 0) return;
          move_on(i, w);
        }
      };
      std::thread helpers[kMovers];
      for (int w = 1; w < movers; ++w) {
        try {
          helpers[w] = std::thread(mover, w);
        } catch (...) {
        }  // no thread to be had: this one does the range
      }
      if (movers > 1) touch(0);
      cudaError_t err = cudaSuccess;
      for (int i = 0; i < parts; ++i) {
        err = cudaEventSynchronize(landed[i]);
        arrived.store(err == cudaSuccess ? i + 1 : -1, std::memory_order_release);
        if (err != cudaSuccess) break;
        for (int w = 0; w < movers; ++w)
          if (!helpers[w].joinable()) move_on(i, w);
      }
      for (std::thread& t : helpers)
        if (t.joinable()) t.join();
      if (err != cudaSuccess) return err;
    }
    return cudaSuccess;
  }
};

// an int4 matrix on the device; `dense` is its optional bf16 expansion [n, k], made once at load for
// the steps that are bound by tensor throughput rather than by the weight stream
struct QMat { Buf codes, scales, dense; int n = 0, k = 0; };

// expands q into q.dense (blocking); false on allocation or launch failure
inline bool make_dense_copy(QMat& q) {
  if (!q.dense.alloc((size_t)q.n * q.k * 2)) return false;
  if (logismos_launch_dequant_int4_g32_bf16(q.codes.p, q.scales.p, q.dense.p, q.n, q.k, nullptr) != 0) return false;
  return cudaDeviceSynchronize() == cudaSuccess;
}

// gate and up rows interleaved in blocks of 32 (32 gate rows, then the 32 matching up rows), the
// row order the fused SwiGLU epilogue of the GEMM expects
inline bool upload_q_gate_up(QMat& q, const lg_int4_matrix_t& gate, const lg_int4_matrix_t& up, int inter, int k) {
  const size_t cb = (size_t)32 * (k / 2), sb = (size_t)32 * (k / 32);
  std::vector<uint8_t> codes((size_t)2 * inter * (k / 2));
  std::vector<uint16_t> scales((size_t)2 * inter * (k / 32));
  for (int b = 0; b < inter / 32; ++b) {
    std::memcpy(codes.data() + (size_t)(2 * b) * cb, gate.codes + (size_t)b * cb, cb);
    std::memcpy(codes.data() + (size_t)(2 * b + 1) * cb, up.codes + (size_t)b * cb, cb);
    std::memcpy(scales.data() + (size_t)(2 * b) * sb, gate.scales + (size_t)b * sb, sb * 2);
    std::memcpy(scales.data() + (size_t)(2 * b + 1) * sb, up.scales + (size_t)b * sb, sb * 2);
  }
  q.n = 2 * inter;
  q.k = k;
  return q.codes.upload(codes.data(), codes.size()) && q.scales.upload(scales.data(), scales.size() * 2);
}

inline bool upload_q(QMat& q, const std::vector<const lg_int4_matrix_t*>& parts, const std::vector<int>& rows, int k) {
  size_t n = 0;
  for (int r : rows) n += (size_t)r;
  std::vector<uint8_t> codes(n * (k / 2));
  std::vector<uint16_t> scales(n * (k / 32));
  size_t o = 0;
  for (size_t i = 0; i < parts.size(); ++i) {
    std::memcpy(codes.data() + o * (k / 2), parts[i]->codes, (size_t)rows[i] * (k / 2));
    std::memcpy(scales.data() + o * (k / 32), parts[i]->scales, (size_t)rows[i] * (k / 32) * 2);
    o += (size_t)rows[i];
  }
  q.n = (int)n;
  q.k = k;
  return q.codes.upload(codes.data(), codes.size()) && q.scales.upload(scales.data(), scales.size() * 2);
}

// C = A W^T with int4 weights, epilogue as for logismos_launch_linear_t_bf16. Up to 128 rows the
// dequantisation is fused into the tensor-core kernel (fp32 accumulation into the residual stream
// itself, or into the zeroed workspace `accws` finished to bf16); above that the weights are
// expanded to bf16 (the matrix's persistent copy when it has one, else into `wscratch` on every
// call) and the dense GEMM runs with its fused epilogues. The
// crossover is measured: the fused kernel's fp32 reductions grow with rows x columns, and the kernel
// that reads the accumulation target next waits for them to drain (a finishing kernel of 4 us alone
// took 21 us behind a 256-row accumulation).
constexpr int kFusedDequantMaxRows = 128;
inline uint32_t qlinear_any(const void* a, const QMat& w, const void* bias, void* out, int T, int lda, int ldc, int epi,
                            void* wscratch, void* accws, void* status, int* launches, cudaStream_t s) {
  uint32_t rc;
  // with a persistent bf16 copy at hand the dense GEMM (split over k for the narrow output projections)
  // is as fast or faster above 32 rows (measured at 64 / 128 rows: 6.5 / 6.7 us against 6.7 / 8.2 us for
  // 2048 x 2048, 9.5 / 9.8 against 10.7 / 14.6 us for 2048 x 6144, 14-18 against 19-24 us for the wide
  // projections with their finishing pass); below that the int4 stream wins
  const bool fused_ok = T <= kFusedDequantMaxRows && w.k % 256 == 0 && (!w.dense.p || T <= 32);
  if (fused_ok) {
    if (epi == LG_EPI_RESID_F32 && !bias) {
      *launches += 1;
      return logismos_launch_qlinear_int4_g32_acc_f32_static(a, w.codes.p, w.scales.p, out, T, w.n, w.k, lda, ldc, status, s);
    }
    if (epi != LG_EPI_RESID_F32) {
      rc = logismos_launch_qlinear_int4_g32_acc_f32_static(a, w.codes.p, w.scales.p, accws, T, w.n, w.k, lda, w.n, status, s);
      if (rc) return rc;
      *launches += 2;
      return logismos_launch_qlinear_finish_bf16(accws, bias, out, T, w.n, w.n, ldc, epi == LG_EPI_SWIGLU ? 1 : 0, s);
    }
  }
  if (w.dense.p) {
    *launches += 1;
    return logismos_launch_linear_t_bf16(a, w.dense.p, bias, out, T, w.n, w.k, lda, ldc, epi | LG_EPI_STATIC_W, status, s);  // the copy is made once at load
  }
  rc = logismos_launch_dequant_int4_g32_bf16(w.codes.p, w.scales.p, wscratch, w.n, w.k, s);
  if (rc) return rc;
  *launches += 2;
  return logismos_launch_linear_t_bf16(a, wscratch, bias, out, T, w.n, w.k, lda, ldc, epi, status, s);
}

// The projections of a pure decode step of one to four rows (int4_rows.cu). norm: x is the fp32 residual stream and goes
// through its RMS norm on the way; otherwise a is bf16 activations with row stride lda.
inline lg::Int4Rows few_rows(const QMat& w, const void* bias, void* out, int rows, int ldc, int epi) {
  lg::Int4Rows p{};
  p.codes = w.codes.p; p.scales = w.scales.p; p.bias = bias; p.out = out;
  p.rows = rows; p.n = w.n; p.k = w.k; p.ldc = ldc; p.epi = epi;
  return p;
}
inline uint32_t few_norm(const Buf& x, const Buf& gain, float eps, const QMat& w, const void* bias, void* out, int rows, int ldc, int epi, int* launches, cudaStream_t s) {
  lg::Int4Rows p = few_rows(w, bias, out, rows, ldc, epi);
  p.x = x.p; p.gain = gain.p; p.eps = eps;
  *launches += 1;
  return lg::launch_int4_rows(p, s);
}
inline uint32_t few_heads(const Buf& x, const Buf& gain, float eps, const QMat& w, const void* bias, const lg::DecodeHeads& heads, int rows, int* launches, cudaStream_t s) {
  lg::Int4Rows p = few_rows(w, bias, nullptr, rows, 0, LG_EPI_BF16);
  p.x = x.p; p.gain = gain.p; p.eps = eps; p.heads = heads;
  *launches += 1;
  return lg::launch_int4_rows(p, s);
}
inline uint32_t few_act(const void* a, int lda, const QMat& w, void* out, int rows, int ldc, int epi, int* launches, cudaStream_t s) {
  lg::Int4Rows p = few_rows(w, nullptr, out, rows, ldc, epi);
  p.a = a; p.lda = lda;
  *launches += 1;
  return lg::launch_int4_rows(p, s);
}

// Tokens per decode chunk of a step: logismos_pick_decode_chunk's, and shorter where that leaves most SMs without a CTA
// (one sequence of 1200 tokens, two key heads of 128: 6 CTAs of 512 tokens 14.5 us, 20 of 128 8.8 us), as far as the
// scratch holds the partial results.
inline int step_decode_chunk(const int32_t* ctx, int n_dec, int n_kv_heads, int head_dim, size_t max_chunks) {
  int chunk = logismos_pick_decode_chunk(ctx, n_dec, n_kv_heads, head_dim);
  if (chunk > 512 || logismos_get_deterministic()) return chunk;  // the order of a sequence's sums follows the chunks
  auto count = [&](int c) {
    int64_t n = 0;
    for (int i = 0; i < n_dec; ++i) n += (std::max(ctx[i], 1) + c - 1) / c;
    return n;
  };
  while (chunk > 128 && count(chunk) * n_kv_heads < lg::sm_count() && count(chunk / 2) <= (int64_t)max_chunks) chunk /= 2;
  return chunk;
}
constexpr size_t kMinDecodeChunks = 1024;  // partial results that a model's scratch holds at least

// logits = hidden W^T over the vocabulary and decode::greedy (crates/decode/src/lib.rs:73-83) on
// them. The logits stay fp32 up to the argmax on every route, as in the reference (greedy takes the
// first strict maximum of fp32 logits), so the emitted token does not depend on how many rows the
// step had: up to 16 rows the streaming int4 GEMV stores its fp32 accumulators; above that the
// fused-dequant tensor-core kernel accumulates into the zeroed buffer. `logits` must hold rows * vocab
// floats. *logits_f32 is always 1 (kept for the readers of the buffer).
inline uint32_t lm_head_and_greedy(const QMat& lm_head, const void* hidden_bf16, void* logits, void* tokens, int rows, int hidden,
                                   void* status, int* logits_f32, int* launches, cudaStream_t s) {
  uint32_t rc;
  const int vocab = lm_head.n;
  *logits_f32 = 1;
  if (rows > 16 && hidden % 256 == 0) {
    for (int b0 = 0; b0 < rows; b0 += kFusedDequantMaxRows) {
      const int nb = rows - b0 < kFusedDequantMaxRows ? rows - b0 : kFusedDequantMaxRows;
      float* dst = (float*)logits + (size_t)b0 * vocab;
      if (cudaMemsetAsync(dst, 0, (size_t)nb * vocab * 4, s) != cudaSuccess) return (uint32_t)cudaGetLastError();
      rc = logismos_launch_qlinear_int4_g32_acc_f32_static((const uint16_t*)hidden_bf16 + (size_t)b0 * hidden, lm_head.codes.p,
                                                    lm_head.scales.p, dst, nb, vocab, hidden, hidden, vocab, status, s);
      if (rc) return rc;
      *launches += 1;
    }
  } else {
    for (int b0 = 0; b0 < rows; b0 += 64) {  // the GEMV takes up to 64 rows per launch
      const int nb = rows - b0 < 64 ? rows - b0 : 64;
      rc = logismos_launch_gemv_int4_g32_f32(lm_head.codes.p, lm_head.scales.p, (const uint16_t*)hidden_bf16 + (size_t)b0 * hidden,
                                             (float*)logits + (size_t)b0 * vocab, nb, vocab, hidden, s);
      if (rc) return rc;
      *launches += 1;
    }
  }
  *launches += 1;
  return logismos_launch_greedy_argmax(logits, 1, tokens, rows, vocab, s);
}

}  // namespace lgm

#define LG_TRY(expr, what)                                                                         \
  do {                                                                                             \
    uint32_t rc_ = (uint32_t)(expr);                                                               \
    if (rc_ != 0) {                                                                                \
      char buf_[192];                                                                              \
      std::snprintf(buf_, sizeof(buf_), "%s failed: %s (code %u)", what, cudaGetErrorString((cudaError_t)rc_), rc_); \
      lgm::set_error(buf_);                                                                             \
      return LG_EMB_COMPUTE;                                                                       \
    }                                                                                              \
  } while (0)

