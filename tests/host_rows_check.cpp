// HostRows of the model executors over a CUDA runtime that is a few lines of host code: which threads call it, and where rows end.
#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <thread>
#include <vector>

#include <sys/mman.h>
#include <sys/resource.h>

#include "model_util.h"

static std::thread::id g_caller;
static std::atomic<int> g_foreign{0}, g_calls{0};
static bool g_no_pinned = false;
static int g_fail_event = -1, g_events = 0;  // the wait with this number fails

static cudaError_t called(cudaError_t e = cudaSuccess) {
  ++g_calls;
  if (std::this_thread::get_id() != g_caller) ++g_foreign;
  return e;
}

extern "C" {
cudaError_t cudaMallocHost(void** p, size_t n) { *p = g_no_pinned ? nullptr : std::malloc(n); return called(g_no_pinned ? cudaErrorMemoryAllocation : cudaSuccess); }
cudaError_t cudaFreeHost(void* p) { std::free(p); return called(); }
cudaError_t cudaGetLastError() { return called(); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = (cudaEvent_t)std::malloc(1); return called(); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { std::free((void*)e); return called(); }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return called(); }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return called(g_events++ == g_fail_event ? cudaErrorLaunchFailure : cudaSuccess); }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return called(); }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { std::memcpy(d, s, n); return called(); }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { std::memcpy(d, s, n); return called(); }
}

int main() {
  g_caller = std::this_thread::get_id();
  lgm::HostRows rows;
  struct Case { int rows; size_t width; } cases[] = {{1, 7}, {3, 1000}, {64, 32768}, {5, 151936}, {40, 151936}, {1, 5000000}};
  for (int no_pinned = 0; no_pinned < 2; ++no_pinned) {
    for (const Case& c : cases) {
      g_no_pinned = no_pinned != 0;
      if (no_pinned) rows.release();
      std::vector<float> dev(c.rows * c.width), out(c.rows * c.width, -1.0f);
      std::vector<int> order(c.rows);
      for (size_t i = 0; i < dev.size(); ++i) dev[i] = (float)(i % 16777213);
      for (int i = 0; i < c.rows; ++i) order[i] = (i * 7 + 3) % c.rows;
      if (c.rows % 7 == 0) std::reverse(order.begin(), order.end());
      if (rows.copy(dev.data(), c.rows, c.width, order.data(), out.data(), nullptr) != cudaSuccess) return std::puts("copy failed"), 1;
      for (int i = 0; i < c.rows; ++i)
        if (std::memcmp(&out[order[i] * c.width], &dev[i * c.width], c.width * 4)) return std::printf("row %d of %d x %zu\n", i, c.rows, c.width), 1;
      if (rows.capacity > ((size_t)16 << 20) && rows.capacity > c.width * 4) return std::puts("pinned buffer above its cap"), 1;
    }
  }
  g_no_pinned = false;
  g_fail_event = g_events + 2;  // a wait in the middle fails: the error comes back, no thread is left behind
  std::vector<float> dev(64 * 32768), out(dev.size());
  std::vector<int> order(64);
  for (int i = 0; i < 64; ++i) order[i] = i;
  if (rows.copy(dev.data(), 64, 32768, order.data(), out.data(), nullptr) != cudaErrorLaunchFailure) return std::puts("a failed wait went unseen"), 1;
  // the same from an address that is no multiple of a page, nor are its rows' ranges: what does not arrive stays as it was
  g_fail_event = g_events + 2;
  out.assign(dev.size() + 1, 0.1f);
  for (size_t i = 0; i < dev.size(); ++i) dev[i] = (float)(i % 16777213) + 1.0f;
  if (rows.copy(dev.data(), 64, 32768, order.data(), out.data() + 1, nullptr) != cudaErrorLaunchFailure) return std::puts("a failed wait went unseen"), 1;
  for (size_t i = 0; i < dev.size(); ++i)
    if (out[i + 1] != dev[i] && out[i + 1] != 0.1f) return std::printf("value %zu is neither what it was nor what was sent\n", i), 1;
  if (out.back() != 0.1f) return std::puts("the last row came although its part did not"), 1;
  for (int n : {8, 9, 10, 12, 15, 16, 17, 33}) {  // one to several threads, rows off a page
    std::fill(out.begin(), out.end(), 0.1f);
    if (rows.copy(dev.data(), n, 32767, order.data(), out.data() + 1, nullptr) != cudaSuccess) return std::puts("copy failed"), 1;
    if (std::memcmp(out.data() + 1, dev.data(), (size_t)n * 32767 * 4) || out[0] != 0.1f || out[(size_t)n * 32767 + 1] != 0.1f) return std::printf("%d rows\n", n), 1;
  }
  for (int n : {9, 15, 16}) {  // a destination that is fresh, and the same one again
    const size_t bytes = (size_t)n * 32768 * 4;
    float* fresh = (float*)mmap(nullptr, bytes, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    if (fresh == MAP_FAILED) return std::puts("no memory"), 1;
    for (int again = 0; again < 2; ++again) {
      if (lgm::HostRows::there(fresh, 32768, order.data(), n) != (again == 1)) return std::puts("pages"), 1;
      for (float& v : dev) v += 1.0f;
      if (rows.copy(dev.data(), n, 32768, order.data(), fresh, nullptr) != cudaSuccess || std::memcmp(fresh, dev.data(), bytes)) return std::printf("%d rows, %d\n", n, again), 1;
    }
    munmap(fresh, bytes);
  }
  {  // a fresh destination costs one fault a page: reading a page ahead of the first write to it makes two of it, the second one with a flush on every core
    const size_t bytes = dev.size() * 4, pages = bytes / 4096;
    float* fresh = (float*)mmap(nullptr, bytes, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    if (fresh == MAP_FAILED) return std::puts("no memory"), 1;
    madvise(fresh, bytes, MADV_NOHUGEPAGE);
    rusage before, after;
    getrusage(RUSAGE_SELF, &before);
    if (rows.copy(dev.data(), 64, 32768, order.data(), fresh, nullptr) != cudaSuccess) return std::puts("copy failed"), 1;
    getrusage(RUSAGE_SELF, &after);
    if (std::memcmp(fresh, dev.data(), bytes)) return std::puts("rows of a fresh destination"), 1;
    munmap(fresh, bytes);
    if ((size_t)(after.ru_minflt - before.ru_minflt) > pages + pages / 2) return std::printf("%ld faults for %zu pages\n", after.ru_minflt - before.ru_minflt, pages), 1;
  }
  rows.release();
  if (g_foreign) return std::printf("%d of %d CUDA calls from other threads\n", g_foreign.load(), g_calls.load()), 1;
  return 0;
}
