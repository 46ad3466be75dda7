// host_stage.cpp -- copies between the caller's arrays and the device through
// page-locked chunks, several host threads at a time.
#include "host_stage.h"

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstring>
#include <map>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>

namespace b200fem {

// A double is finite iff its exponent field is not all ones: adding one to
// the masked exponent carries into bit 63 exactly for all-ones fields.  The
// OR-reduction vectorises (the host-state step checks 2 x 3N values per
// call: 9 us for the 40x10x10 hex beam's x or v with a per-element fabs
// compare, 3 us this way).
__attribute__((optimize("O3"))) bool all_finite(const double* a, size_t n) {
  const uint64_t kExp = 0x7ff0000000000000ull, kOne = 0x0010000000000000ull;
  uint64_t acc = 0;
  for (size_t i = 0; i < n; i++) {
    uint64_t b;
    std::memcpy(&b, a + i, sizeof b);
    acc |= (b & kExp) + kOne;
  }
  return (acc >> 63) == 0;
}

// Page-locked chunks and a stream for each worker of a staged copy.  The
// engines of a device share one: page-locking 4 MB takes 5 ms, more than the
// copies it serves.  It is made on the first staged copy and goes with the
// last engine that has made one.  A copy holds its mutex; another engine's
// copy takes the plain way meanwhile, so engines in several threads do not
// wait for one another.
struct HostStage {
  static constexpr int kWorkers = 4;
  static constexpr size_t kChunk = 1 << 20;
  int device = 0;
  std::mutex busy;
  unsigned char* buf = nullptr;
  cudaStream_t stream[kWorkers] = {};
  ~HostStage() {
    cudaSetDevice(device);
    for (auto& st : stream)
      if (st) cudaStreamDestroy(st);
    if (buf) cudaFreeHost(buf);
  }
};

namespace {
// The device's stage, or null where its memory or streams cannot be had (or
// another thread is making one).
std::shared_ptr<HostStage> host_stage(int device) {
  static std::mutex mu;
  static std::map<int, std::weak_ptr<HostStage>> stages;
  std::unique_lock<std::mutex> lk(mu, std::try_to_lock);
  if (!lk) return nullptr;
  std::shared_ptr<HostStage> s = stages[device].lock();
  if (s) return s;
  s = std::make_shared<HostStage>();
  s->device = device;
  cudaError_t e = cudaHostAlloc((void**)&s->buf, HostStage::kWorkers * HostStage::kChunk, cudaHostAllocDefault);
  for (auto& st : s->stream)
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
  if (e != cudaSuccess) {
    cudaGetLastError();  // (no later launch is to report it)
    return nullptr;
  }
  stages[device] = s;
  return s;
}

// f(worker) on the stage's number of threads, the caller's among them.
template <typename F>
void on_stage_workers(F&& f) {
  std::vector<std::thread> pool;
  try {
    for (int w = 1; w < HostStage::kWorkers; w++) pool.emplace_back(f, w);
  } catch (const std::system_error&) {  // no more threads: those there are share the work
  }
  f(0);
  for (auto& t : pool) t.join();
}

}  // namespace

bool all_finite_arrays(std::initializer_list<std::pair<const double*, size_t>> arrays) {
  size_t total = 0;
  for (auto& a : arrays) total += a.first ? a.second : 0;
  constexpr size_t kPart = 1 << 17;
  if (total < 2 * kPart) {
    for (auto& a : arrays)
      if (a.first && !all_finite(a.first, a.second)) return false;
    return true;
  }
  std::atomic<size_t> next(0);
  std::atomic<bool> ok(true);
  on_stage_workers([&](int) {
    for (size_t q; ok && (q = next++ * kPart) < total;) {
      // part [q, q + kPart) of the arrays laid end to end
      size_t off = q, left = std::min(kPart, total - q);
      for (auto& a : arrays) {
        const size_t n = a.first ? a.second : 0;
        if (off >= n) {
          off -= n;
          continue;
        }
        const size_t m = std::min(left, n - off);
        if (!all_finite(a.first + off, m)) ok = false;
        left -= m;
        off = 0;
        if (left == 0) break;
      }
    }
  });
  return ok;
}

// Copies between host arrays and the device.  Large pageable arrays go
// through page-locked chunks, several host threads copying while the DMA
// engine moves the other chunks: the driver's own staging is one thread, and
// a destination the caller has just allocated takes its page faults in it
// (256 beams of 331,000 nodes, set, step and get: 11.6 ms, 8.5 this way and with
// the velocity history copied on the device).
// Small or page-locked arrays take plain asynchronous copies on the engine's
// stream, and so do all where the stage cannot be had or another engine uses
// it.
// (kStageMin: an update's 16 MB take 2.2 ms staged and 3.6 plain, 4 MB 1.4 and
// 1.2: below it the threads cost more than they save)
constexpr size_t kStageMin = 6 << 20;
cudaError_t stage_copy(int device, cudaStream_t stream, std::shared_ptr<HostStage>& hold,
                       std::initializer_list<HostCopy> list, bool to_host) {
  const cudaMemcpyKind kind = to_host ? cudaMemcpyDeviceToHost : cudaMemcpyHostToDevice;
  auto plain = [&](const HostCopy& c) {
    return cudaMemcpyAsync(to_host ? c.host : c.dev, to_host ? c.dev : c.host, c.bytes, kind, stream);
  };
  std::vector<HostCopy> large, chunks;
  cudaError_t e = cudaSuccess;
  size_t total = 0;
  for (const HostCopy& c : list) total += c.host ? c.bytes : 0;
  for (const HostCopy& c : list) {
    if (!c.host || c.bytes == 0) continue;
    bool pageable = total >= kStageMin && c.bytes >= HostStage::kChunk;
    if (pageable) {
      cudaPointerAttributes at{};
      if (cudaPointerGetAttributes(&at, c.host) != cudaSuccess) cudaGetLastError();
      else pageable = at.type == cudaMemoryTypeUnregistered;
    }
    if (pageable) large.push_back(c);
    else if ((e = plain(c)) != cudaSuccess) return e;
  }
  if (large.empty()) return cudaSuccess;
  if (!hold) hold = host_stage(device);
  std::unique_lock<std::mutex> lk;
  if (hold) {
    // earlier work on the engine's stream writes the source or reads the
    // target; it is awaited before the stage is taken from the others
    if ((e = cudaStreamSynchronize(stream)) != cudaSuccess) return e;
    lk = std::unique_lock<std::mutex>(hold->busy, std::try_to_lock);
  }
  if (!lk.owns_lock()) {
    for (const HostCopy& c : large)
      if ((e = plain(c)) != cudaSuccess) return e;
    return cudaSuccess;
  }
  HostStage& stage = *hold;
  for (const HostCopy& c : large)
    for (size_t o = 0; o < c.bytes; o += HostStage::kChunk)
      chunks.push_back({(char*)c.host + o, (char*)c.dev + o, std::min(HostStage::kChunk, c.bytes - o)});
  std::atomic<size_t> next(0);
  std::atomic<int> err((int)cudaSuccess);
  on_stage_workers([&](int w) {
    cudaError_t r = cudaSetDevice(device);
    unsigned char* buf = stage.buf + (size_t)w * HostStage::kChunk;
    for (size_t q; r == cudaSuccess && err == (int)cudaSuccess && (q = next++) < chunks.size();) {
      const HostCopy& c = chunks[q];
      if (!to_host) std::memcpy(buf, c.host, c.bytes);
      r = cudaMemcpyAsync(to_host ? (void*)buf : c.dev, to_host ? c.dev : (void*)buf, c.bytes, kind, stage.stream[w]);
      if (r == cudaSuccess) r = cudaStreamSynchronize(stage.stream[w]);
      if (r == cudaSuccess && to_host) std::memcpy(c.host, buf, c.bytes);
    }
    if (r != cudaSuccess) err = (int)r;
  });
  return (cudaError_t)(int)err;
}

}  // namespace b200fem
