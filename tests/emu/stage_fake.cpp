// csrc/host_stage.cpp with a CUDA runtime made of host memory: allocations
// that fail, streams that are busy.  One scenario per run; exit code 0 when
// the copies arrived and nothing was left behind.
#include "host_stage.h"

#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

static int g_host_alloc_fails = 0, g_stream_fails_at = 0, g_streams = 0, g_host_bufs = 0, g_made = 0;
static cudaError_t g_last = cudaSuccess;
static std::mutex g_mu;
static std::condition_variable g_cv;
static std::map<cudaStream_t, bool> g_busy;  // a stream whose work does not end yet
static cudaStream_t const kA = (cudaStream_t)1, kB = (cudaStream_t)2;
static bool g_block_stage = false;  // the first staged chunk's DMA does not end yet
static std::atomic<int> g_waiting(0);

static cudaError_t fail(cudaError_t e) {
  g_last = e;
  return e;
}
extern "C" {
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
  if (g_host_alloc_fails) return fail(cudaErrorMemoryAllocation);
  *p = malloc(n);
  g_host_bufs++;
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
  free(p);
  g_host_bufs--;
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  if (g_stream_fails_at && g_streams + 1 >= g_stream_fails_at) return fail(cudaErrorMemoryAllocation);
  g_streams++;
  *s = (cudaStream_t)(uintptr_t)(100 + g_made++);
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) {
  g_streams--;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() {
  cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) {
  std::memset(a, 0, sizeof(*a));
  a->type = cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  std::unique_lock<std::mutex> lk(g_mu);
  const bool stage = (uintptr_t)s >= 100;
  if (!stage && !g_busy[s]) return cudaSuccess;
  if (stage && !g_block_stage) return cudaSuccess;
  g_waiting++;
  g_cv.wait(lk, [&] { return stage ? !g_block_stage : !g_busy[s]; });
  g_waiting--;
  return cudaSuccess;
}
}

using namespace b200fem;

struct Copy {
  std::vector<double> host, dev;
  std::shared_ptr<HostStage> hold;
  explicit Copy(size_t n) : host(n), dev(n) {
    for (size_t i = 0; i < n; i++) dev[i] = 1.0 + (double)i;
  }
  cudaError_t get(cudaStream_t s) {
    return stage_copy(0, s, hold, {{host.data(), dev.data(), host.size() * sizeof(double)}}, true);
  }
  bool same() const { return host == dev; }
};

static int check(bool ok, const char* what) {
  if (!ok) printf("%s\n", what);
  return ok ? 0 : 1;
}

int main(int argc, char** argv) {
  const std::string s = argc > 1 ? argv[1] : "";
  int bad = 0;
  if (s == "no_host_memory" || s == "no_stream") {
    // the stage cannot be made: plain copies, no error left for a later launch
    // to report; it is made once it can be
    g_host_alloc_fails = s == "no_host_memory";
    g_stream_fails_at = s == "no_stream" ? 3 : 0;
    Copy c((size_t)1 << 20);
    bad += check(c.get(kA) == cudaSuccess, "refused");
    bad += check(c.same(), "wrong values");
    bad += check(cudaGetLastError() == cudaSuccess, "error left behind");
    bad += check(g_host_bufs == 0 && g_streams == 0, "part of a stage kept");
    g_host_alloc_fails = g_stream_fails_at = 0;
    std::fill(c.host.begin(), c.host.end(), 0.0);
    bad += check(c.get(kA) == cudaSuccess && c.same() && g_host_bufs == 1, "no stage later");
    return bad;
  }
  if (s == "stage_in_use" || s == "stream_busy") {
    // another engine's copy or earlier work does not end: this one's copy does
    Copy a((size_t)1 << 20), b((size_t)1 << 20);
    a.get(kA);
    std::fill(a.host.begin(), a.host.end(), 0.0);
    (s == "stage_in_use" ? g_block_stage : g_busy[kA]) = true;
    std::thread ta([&] { a.get(kA); });
    while (g_waiting == 0) std::this_thread::yield();
    std::atomic<bool> done(false);
    std::thread tb([&] {
      b.get(kB);
      done = true;
    });
    for (int i = 0; i < 500 && !done; i++) std::this_thread::sleep_for(std::chrono::milliseconds(10));
    bad += check(done, "waits for the other engine");
    {
      std::lock_guard<std::mutex> lk(g_mu);
      g_block_stage = g_busy[kA] = false;
    }
    g_cv.notify_all();
    ta.join();
    tb.join();
    bad += check(a.same() && b.same(), "wrong values");
    return bad;
  }
  return 2;
}
