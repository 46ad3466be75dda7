// CTAs of a kernel on one host thread: every CUDA thread is a fiber, a fiber
// runs until it waits (warp shuffle, barrier) or polls memory, and the next
// one is chosen by a rule of the test.  So an interleaving that a GPU takes
// once in a million launches is the one that runs, and a wait that nothing
// ends is reported instead of hanging.
//
// Semantics kept: a shuffle or vote waits for the 32 lanes of the warp; barrier
// 0 waits for every thread of the CTA that has not left the kernel; a named
// barrier with a count waits for that many arrivals, whoever has left.
#pragma once

#include <setjmp.h>
#include <ucontext.h>

#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <functional>
#include <map>
#include <memory>
#include <string>
#include <vector>

namespace emu {

constexpr size_t kStack = 96 << 10;

struct Dim {
  int x = 0, y = 0, z = 0;
};
struct Cta;
struct Fiber {
  ucontext_t ctx;  // of its first run; later switches leave the signal mask alone
  jmp_buf at;
  Cta* cta = nullptr;
  int tid = 0;
  enum { kReady, kBlocked, kDone } state = kReady;
  bool started = false, polled = false;
  std::unique_ptr<char[]> stack;
  int warp() const { return tid >> 5; }
};
struct Warp {
  int arrived = 0;
  unsigned gen = 0;
  uint64_t val[2][32] = {};
};
struct Cta {
  int block = 0, alive = 0;
  int bar0 = 0, bar1 = 0;
  std::vector<Fiber> fibers;
  std::vector<Warp> warps;
  std::vector<unsigned char> dyn;
  std::map<std::string, std::vector<unsigned char>> shared;
};

struct Machine {
  std::vector<std::unique_ptr<Cta>> ctas;
  std::deque<Fiber*> ready;
  jmp_buf scheduler;
  Fiber* cur = nullptr;
  std::function<void()> body;
  int grid = 0;
  uint64_t clock_ns = 0, resumes = 0, clock_step = 10;
  // the test's hooks: before a fiber runs; fibers that run only when no other
  // can (0), by choice (1: default)
  std::function<void(Fiber&)> before;
  std::function<int(const Fiber&)> rank = [](const Fiber&) { return 1; };
  // which of n ready fibers runs next (default: the one that has waited longest)
  std::function<size_t(size_t n)> choose;
};
inline Machine* M = nullptr;

inline void to_scheduler() {
  if (_setjmp(M->cur->at) == 0) _longjmp(M->scheduler, 1);
}
inline void wake(Fiber& f) {
  if (f.state != Fiber::kBlocked) return;
  f.state = Fiber::kReady;
  M->ready.push_back(&f);
}
// a poll that found nothing: let the others run
inline void yield() {
  Fiber& f = *M->cur;
  f.polled = true;
  M->ready.push_back(&f);
  to_scheduler();
}
inline void block() {
  M->cur->state = Fiber::kBlocked;
  to_scheduler();
}
// the fibers blocked at each barrier
struct Waiters {
  std::vector<Fiber*> at0, at1;
};
inline std::map<Cta*, Waiters>& waiters() {
  static std::map<Cta*, Waiters> w;
  return w;
}
inline void release(std::vector<Fiber*>& v) {
  std::vector<Fiber*> go;
  go.swap(v);
  for (Fiber* f : go) wake(*f);
}
inline void sync_threads() {
  Cta& c = *M->cur->cta;
  Waiters& w = waiters()[&c];
  if (++c.bar0 >= c.alive) {
    c.bar0 = 0;
    release(w.at0);
    return;
  }
  w.at0.push_back(M->cur);
  block();
}
inline void sync_named(int count) {
  Cta& c = *M->cur->cta;
  Waiters& w = waiters()[&c];
  if (++c.bar1 >= count) {
    c.bar1 = 0;
    release(w.at1);
    return;
  }
  w.at1.push_back(M->cur);
  block();
}
// every lane's value, once the warp's 32 lanes are there
inline const uint64_t* exchange(uint64_t mine) {
  Fiber& f = *M->cur;
  Cta& c = *f.cta;
  Warp& w = c.warps[f.warp()];
  const unsigned g = w.gen;
  w.val[g & 1][f.tid & 31] = mine;
  if (++w.arrived == 32) {
    w.arrived = 0;
    w.gen++;
    for (int l = 0; l < 32; l++) {
      Fiber& o = c.fibers[(f.warp() << 5) + l];
      if (&o != &f) wake(o);
    }
  } else {
    block();
  }
  return w.val[g & 1];
}
template <typename T>
uint64_t bits(T v) {
  uint64_t b = 0;
  static_assert(sizeof(T) <= 8, "");
  std::memcpy(&b, &v, sizeof(T));
  return b;
}
template <typename T>
T shfl(T v, int src) {
  const uint64_t b = exchange(bits(v))[src & 31];
  T o;
  std::memcpy(&o, &b, sizeof(T));
  return o;
}
template <typename T>
T& shared(const char* name) {
  auto& v = M->cur->cta->shared[name];
  if (v.empty()) v.assign(sizeof(T) + 16, 0);
  return *(T*)(((uintptr_t)v.data() + 15) & ~(uintptr_t)15);
}
inline unsigned char* dyn() { return (unsigned char*)(((uintptr_t)M->cur->cta->dyn.data() + 15) & ~(uintptr_t)15); }

inline void fiber_main() {
  M->body();
  Fiber& f = *M->cur;
  Cta& c = *f.cta;
  f.state = Fiber::kDone;
  c.alive--;
  // barrier 0 no longer waits for this thread
  if (c.alive > 0 && c.bar0 >= c.alive) {
    c.bar0 = 0;
    release(waiters()[&c].at0);
  }
  to_scheduler();
}

// Runs `body` on grid x threads; empty when every thread ended, else where
// they hang.
inline std::string run(Machine& m, int grid, int threads, size_t dyn_bytes, std::function<void()> body,
                       uint64_t max_resumes = 20000000ull) {
  M = &m;
  m.body = std::move(body);
  m.grid = grid;
  waiters().clear();
  for (int b = 0; b < grid; b++) {
    m.ctas.emplace_back(new Cta);
    Cta& c = *m.ctas.back();
    c.block = b;
    c.alive = threads;
    c.dyn.assign(dyn_bytes + 16, 0);
    c.warps.resize(threads / 32);
    c.fibers = std::vector<Fiber>(threads);
    for (int t = 0; t < threads; t++) {
      Fiber& f = c.fibers[t];
      f.cta = &c;
      f.tid = t;
      f.stack.reset(new char[kStack]);
      m.ready.push_back(&f);
    }
  }
  while (!m.ready.empty()) {
    // first come first served; a fiber of rank 0 waits while another can run
    // (a fiber that polls counts as running)
    auto pick = m.ready.begin();
    if (m.choose) std::swap(*pick, m.ready[m.choose(m.ready.size())]);
    while (pick != m.ready.end() && m.rank(**pick) == 0) ++pick;
    if (pick == m.ready.end()) pick = m.ready.begin();
    Fiber* f = *pick;
    m.ready.erase(pick);
    f->polled = false;
    m.cur = f;
    m.clock_ns += m.clock_step;
    if (++m.resumes > max_resumes) return "no end";
    if (m.before) m.before(*f);
    if (_setjmp(m.scheduler) != 0) continue;
    if (f->started) _longjmp(f->at, 1);  // (across stacks: built without the fortified longjmp)
    f->started = true;
    getcontext(&f->ctx);
    f->ctx.uc_stack.ss_sp = f->stack.get();
    f->ctx.uc_stack.ss_size = kStack;
    f->ctx.uc_link = nullptr;
    makecontext(&f->ctx, (void (*)())fiber_main, 0);
    setcontext(&f->ctx);
  }
  for (auto& c : m.ctas)
    if (c->alive > 0) {
      int at[3] = {0, (int)waiters()[c.get()].at0.size(), (int)waiters()[c.get()].at1.size()};
      at[0] = c->alive - at[1] - at[2];
      char buf[160];
      snprintf(buf, sizeof(buf), "hang: CTA %d, %d of %d threads left: %d at a barrier, %d at the row barrier, %d in a warp",
               c->block, c->alive, (int)c->fibers.size(), at[1], at[2], at[0]);
      return buf;
    }
  return "";
}

}  // namespace emu

// ---- what kernel source names
#undef __global__
#undef __device__
#undef __host__
#undef __launch_bounds__
#undef __forceinline__
#define __global__
#define __device__
#define __host__
#define __launch_bounds__(...)
#define __forceinline__ inline
#define threadIdx (emu::Dim{emu::M->cur->tid, 0, 0})
#define blockIdx (emu::Dim{emu::M->cur->cta->block, 0, 0})
#define blockDim (emu::Dim{(int)emu::M->cur->cta->fibers.size(), 1, 1})
#define gridDim (emu::Dim{emu::M->grid, 1, 1})
#define __syncthreads emu::sync_threads

template <typename T>
T __shfl_xor_sync(unsigned, T v, int m) { return emu::shfl(v, (emu::M->cur->tid & 31) ^ m); }
template <typename T>
T __shfl_sync(unsigned, T v, int src) { return emu::shfl(v, src); }
inline bool __all_sync(unsigned, bool p) {
  const uint64_t* v = emu::exchange(p);
  bool r = true;
  for (int l = 0; l < 32; l++) r &= v[l] != 0;
  return r;
}
inline bool __any_sync(unsigned, bool p) {
  const uint64_t* v = emu::exchange(p);
  bool r = false;
  for (int l = 0; l < 32; l++) r |= v[l] != 0;
  return r;
}
inline long long __double_as_longlong(double v) { return (long long)emu::bits(v); }
inline double __longlong_as_double(long long b) {
  double v;
  std::memcpy(&v, &b, 8);
  return v;
}
inline int __double2hiint(double v) { return (int)(emu::bits(v) >> 32); }
inline int __double2loint(double v) { return (int)(unsigned)emu::bits(v); }
inline double __hiloint2double(int hi, int lo) {
  return __longlong_as_double((long long)(((uint64_t)(unsigned)hi << 32) | (unsigned)lo));
}
template <typename T>
T atomicAdd(T* p, T v) { T o = *p; *p = o + v; return o; }
inline int atomicExch(int* p, int v) { int o = *p; *p = v; return o; }
