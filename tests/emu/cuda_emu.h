// CUDA kernels on the host, for tests of their ordering: every CTA is an OS thread, every CUDA thread of
// it a fiber that runs until a barrier or a warp exchange stops it.  One fiber runs at a time, and the
// order is the test's: which CTA of a cluster goes first, which warp, which lane.  A kernel whose barriers
// order everything it shares gives the same bits under every order; one that relies on timing does not.
// A barrier that can no longer complete, and a warp exchange that an exited lane should have joined, end
// the run with an error.
#pragma once
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <ucontext.h>

#include <algorithm>
#include <condition_variable>
#include <functional>
#include <map>
#include <mutex>
#include <random>
#include <thread>
#include <type_traits>
#include <vector>

#define __global__
#define __device__
#define __host__
#define __forceinline__ inline
#define __noinline__
#define __shared__ static thread_local
#define __align__(n) __attribute__((aligned(n)))
#define __launch_bounds__(...)
#define __cluster_dims__(...)
#define __builtin_assume(x) ((void)0)
#define __isShared(x) true

struct alignas(16) double2 {
  double x, y;
};
inline double2 make_double2(double x, double y) { return double2{x, y}; }
struct dim3 {
  unsigned x, y, z;
  dim3(unsigned a = 1, unsigned b = 1, unsigned c = 1) : x(a), y(b), z(c) {}
};
using cudaStream_t = void*;
using cudaError_t = int;
constexpr int cudaErrorInvalidValue = 1, cudaFuncAttributeMaxDynamicSharedMemorySize = 0;
inline int cudaGetLastError() { return 0; }
template <class F>
int cudaFuncSetAttribute(F, int, int) { return 0; }
template <class T>
T min(T a, T b) { return b < a ? b : a; }
template <class T>
T max(T a, T b) { return a < b ? b : a; }

namespace emu {

enum Order { kAscending, kDescending, kRandom };
// flip: once that many fibers have started, *flip_word = flip_value (another kernel's write)
struct Config {
  Order cta = kAscending, thread = kAscending;
  unsigned seed = 1;
  int flip_after = -1, flip_value = 0;
  int* flip_word = nullptr;
};

struct Barrier {
  int arrived = 0;
  long gen = 0;
};
struct Cta;
struct Fiber {
  ucontext_t ctx;
  char* stack = nullptr;
  Cta* cta = nullptr;
  dim3 tid;
  int flat = 0;
  bool started = false, done = false;
  Barrier* on = nullptr;  // blocked until on->gen != seen
  long seen = 0, cluster_seen = 0;
};
struct Grid;
struct Cta {
  Grid* grid = nullptr;
  dim3 idx;
  int flat = 0, rank = 0, live = 0;
  bool finished = false;
  std::vector<Fiber> fibers;
  std::vector<Barrier> warp, named;
  std::vector<double> slot;  // one exchange word per thread
  std::vector<double> dyn;
  char* anchor = nullptr;  // of the CTA's shared variables
  ucontext_t sched;
};
struct Grid {
  dim3 grid, block;
  int cluster = 1;
  Config cfg;
  std::vector<Cta> ctas;
  std::vector<Barrier> cluster_bar;
  std::function<void()> body;
  std::mutex m;
  std::condition_variable cv;
  int baton = -1, started = 0;
  std::string error;
};

inline thread_local Fiber* cur = nullptr;
inline thread_local char tls_anchor = 0;

inline void fail(const char* what) {
  Cta* c = cur->cta;
  if (c->grid->error.empty()) {
    char buf[200];
    snprintf(buf, sizeof(buf), "%s (CTA %d, thread %d)", what, c->flat, cur->flat);
    c->grid->error = buf;
  }
  setcontext(&c->sched);  // the run is over: back to the scheduler for good
}
inline void block_on(Barrier* b, long seen) {
  cur->on = b;
  cur->seen = seen;
  Fiber* self = cur;
  swapcontext(&self->ctx, &self->cta->sched);
}
inline void release(Barrier& b) {
  b.arrived = 0;
  ++b.gen;
}
inline void arrive_wait(Barrier& b, int expect, bool wait) {
  const long g = b.gen;
  if (++b.arrived >= expect) release(b);
  else if (wait) block_on(&b, g);
}
inline void warp_sync() {
  Cta* c = cur->cta;
  const int w = cur->flat / 32, lanes = std::min<int>(32, (int)c->fibers.size() - 32 * w);
  for (int l = 0; l < lanes; ++l)
    if (c->fibers[32 * w + l].done) fail("warp exchange with a lane that has exited");
  arrive_wait(c->warp[w], lanes, true);
}
inline void cta_sync() { arrive_wait(cur->cta->named[0], cur->cta->live, true); }
inline void named(int id, int n, bool wait) { arrive_wait(cur->cta->named[id], n, wait); }

inline int cluster_live(Grid* g, int base) {
  int n = 0;
  for (int q = 0; q < g->cluster; ++q) n += g->ctas[base + q].live;
  return n;
}
inline void cluster_arrive() {
  Cta* c = cur->cta;
  Grid* g = c->grid;
  Barrier& b = g->cluster_bar[c->flat / g->cluster];
  cur->cluster_seen = b.gen;
  if (++b.arrived >= cluster_live(g, c->flat / g->cluster * g->cluster)) release(b);
}
inline void cluster_wait() {
  Cta* c = cur->cta;
  Barrier& b = c->grid->cluster_bar[c->flat / c->grid->cluster];
  if (b.gen == cur->cluster_seen) block_on(&b, cur->cluster_seen);
}

inline void fiber_main() {
  cur->cta->grid->body();
  Fiber* f = cur;
  Cta* c = f->cta;
  f->done = true;
  --c->live;
  // a thread that exits no longer counts for the barriers of the whole CTA or cluster (a counted named
  // barrier still waits for it)
  if (c->live > 0 && c->named[0].arrived > 0 && c->named[0].arrived >= c->live) release(c->named[0]);
  Grid* g = c->grid;
  const int base = c->flat / g->cluster * g->cluster, all = cluster_live(g, base);
  Barrier& b = g->cluster_bar[c->flat / g->cluster];
  if (all > 0 && b.arrived > 0 && b.arrived >= all) release(b);
  setcontext(&c->sched);
}

inline bool runnable(const Fiber& f) { return !f.done && (!f.on || f.on->gen != f.seen); }

// Runs the CTA's fibers until none can go on.  Returns whether any ran.
inline bool run_cta(Cta& c, std::mt19937& rng) {
  Grid* g = c.grid;
  bool any = false;
  const int n = (int)c.fibers.size();
  for (;;) {
    int pick = -1;
    if (g->cfg.thread == kRandom) {
      std::vector<int> can;
      const int nw = (n + 31) / 32, w0 = (int)(rng() % nw);  // a random warp, then a random lane of it
      for (int q = 0; q < nw && can.empty(); ++q) {
        const int w = (w0 + q) % nw;
        for (int i = 32 * w; i < std::min(n, 32 * w + 32); ++i)
          if (runnable(c.fibers[i])) can.push_back(i);
      }
      if (!can.empty()) pick = can[rng() % can.size()];
    } else {
      for (int i = 0; i < n && pick < 0; ++i) {
        const int q = g->cfg.thread == kAscending ? i : n - 1 - i;
        if (runnable(c.fibers[q])) pick = q;
      }
    }
    if (pick < 0 || !g->error.empty()) return any;
    any = true;
    Fiber& f = c.fibers[pick];
    f.on = nullptr;
    cur = &f;
    if (!f.started) {
      f.started = true;
      if (g->started++ == g->cfg.flip_after) *g->cfg.flip_word = g->cfg.flip_value;
    }
    swapcontext(&c.sched, &f.ctx);
  }
}

// Runs body() once per thread of the grid.  Returns "" or what went wrong.
inline std::string run(dim3 grid, dim3 block, int cluster, size_t smem, const Config& cfg, std::function<void()> body) {
  Grid g;
  g.grid = grid;
  g.block = block;
  g.cluster = cluster;
  g.cfg = cfg;
  g.body = body;
  const int ncta = (int)(grid.x * grid.y * grid.z), nt = (int)(block.x * block.y * block.z);
  constexpr size_t kStack = 96 * 1024;
  g.ctas.resize(ncta);
  g.cluster_bar.resize((ncta + cluster - 1) / cluster);
  for (int q = 0; q < ncta; ++q) {
    Cta& c = g.ctas[q];
    c.grid = &g;
    c.flat = q;
    c.idx = dim3(q % grid.x, q / grid.x % grid.y, q / grid.x / grid.y);
    c.rank = q % cluster;
    c.live = nt;
    c.fibers.resize(nt);
    c.warp.resize((nt + 31) / 32);
    c.named.resize(16);
    c.slot.resize(nt);
    c.dyn.assign((smem + 15) / 8 + 2, NAN);  // shared memory holds nothing at the start
  }
  std::mt19937 rng(cfg.seed);
  std::vector<std::thread> threads;
  for (int q = 0; q < ncta; ++q)
    threads.emplace_back([&g, &rng, q, nt] {
      Cta& c = g.ctas[q];
      std::unique_lock<std::mutex> lk(g.m);
      c.anchor = &tls_anchor;
      g.cv.wait(lk, [&] { return g.baton == q || g.baton == -2; });
      std::vector<char> stacks(kStack * nt);
      for (int t = 0; t < nt; ++t) {
        Fiber& f = c.fibers[t];
        f.cta = &c;
        f.flat = t;
        f.tid = dim3(t % g.block.x, t / g.block.x % g.block.y, t / g.block.x / g.block.y);
        getcontext(&f.ctx);
        f.ctx.uc_stack.ss_sp = stacks.data() + kStack * t;
        f.ctx.uc_stack.ss_size = kStack;
        f.ctx.uc_link = nullptr;
        makecontext(&f.ctx, fiber_main, 0);
      }
      for (;;) {
        if (g.baton == -2) return;
        const bool any = run_cta(c, rng);
        c.finished = c.live == 0;
        // hand over: to the first CTA in order that can go on
        std::vector<int> order(g.ctas.size());
        for (size_t i = 0; i < order.size(); ++i) order[i] = g.cfg.cta == kDescending ? (int)(order.size() - 1 - i) : (int)i;
        if (g.cfg.cta == kRandom) std::shuffle(order.begin(), order.end(), rng);
        int next = -1;
        bool left = false;
        for (int o : order) {
          Cta& d = g.ctas[o];
          if (d.finished) continue;
          left = true;
          if (o == q && !any) continue;
          const bool fresh = d.fibers[0].cta == nullptr;
          bool can = fresh;
          for (size_t i = 0; i < d.fibers.size() && !can; ++i) can = runnable(d.fibers[i]);
          if (can && next < 0) next = o;
        }
        if (!g.error.empty() || !left || next < 0) {
          if (g.error.empty() && left) g.error = "a barrier that cannot complete";
          g.baton = -2;
          g.cv.notify_all();
          return;
        }
        g.baton = next;
        g.cv.notify_all();
        const bool fin = c.finished;
        if (fin) return;
        g.cv.wait(lk, [&] { return g.baton == q || g.baton == -2; });
      }
    });
  {
    std::unique_lock<std::mutex> lk(g.m);
    g.baton = cfg.cta == kDescending ? ncta - 1 : cfg.cta == kRandom ? (int)(rng() % ncta) : 0;
    g.cv.notify_all();
  }
  for (auto& t : threads) t.join();
  return g.error;
}

inline double exchange(double v, int src, bool valid) {
  Cta* c = cur->cta;
  const int w = cur->flat / 32 * 32;
  c->slot[cur->flat] = v;
  warp_sync();
  const double r = valid ? c->slot[w + src] : v;
  warp_sync();
  return r;
}
template <class T>
T shuffle(T v, int src) {
  static_assert(sizeof(T) <= 8, "one word");
  double d = 0.0;
  memcpy(&d, &v, sizeof(T));
  d = exchange(d, src & 31, src >= 0 && src < 32);
  memcpy(&v, &d, sizeof(T));
  return v;
}
inline int lane() { return cur->flat & 31; }
inline double* dyn_smem() {
  double* p = cur->cta->dyn.data();
  return reinterpret_cast<double*>((reinterpret_cast<uintptr_t>(p) + 15) & ~(uintptr_t)15);
}

}  // namespace emu

#define threadIdx (emu::cur->tid)
#define blockIdx (emu::cur->cta->idx)
#define blockDim (emu::cur->cta->grid->block)
#define gridDim (emu::cur->cta->grid->grid)

inline void __syncthreads() { emu::cta_sync(); }
inline void __syncwarp(unsigned = 0xffffffffu) { emu::warp_sync(); }
template <class T>
T __shfl_sync(unsigned, T v, int src) { return emu::shuffle(v, src); }
template <class T>
T __shfl_xor_sync(unsigned, T v, int o) { return emu::shuffle(v, emu::lane() ^ o); }
template <class T>
T __shfl_up_sync(unsigned, T v, int o) { return emu::shuffle(v, emu::lane() - o); }
template <class T>
T __shfl_down_sync(unsigned, T v, int o) { return emu::shuffle(v, emu::lane() + o); }
inline unsigned __ballot_sync(unsigned, int p) {
  emu::Cta* c = emu::cur->cta;
  const int w = emu::cur->flat / 32 * 32;
  c->slot[emu::cur->flat] = p ? 1.0 : 0.0;
  emu::warp_sync();
  unsigned r = 0;
  for (int l = 0; l < 32; ++l) r |= c->slot[w + l] != 0.0 ? 1u << l : 0u;
  emu::warp_sync();
  return r;
}
inline int __any_sync(unsigned m, int p) { return __ballot_sync(m, p) != 0; }
inline int __reduce_add_sync(unsigned, int v) {
  int s = 0;
  for (int o = 0; o < 32; ++o) s += __shfl_sync(0xffffffffu, v, o);
  return s;
}
inline int __syncthreads_or(int p) {
  emu::Cta* c = emu::cur->cta;
  c->slot[emu::cur->flat] = p ? 1.0 : 0.0;
  emu::cta_sync();
  int r = 0;
  for (size_t l = 0; l < c->fibers.size(); ++l) r |= !c->fibers[l].done && c->slot[l] != 0.0;
  emu::cta_sync();
  return r;
}
inline int __ffs(unsigned v) { return __builtin_ffs((int)v); }
inline double __ldcg(const double* p) { return *p; }
inline double2 __ldcg(const double2* p) { return *p; }
inline void __stcg(double* p, double v) { *p = v; }
inline void __stcg(double2* p, double2 v) { *p = v; }
inline double rsqrt(double x) { return 1.0 / sqrt(x); }
inline long long __double_as_longlong(double x) {
  long long r;
  memcpy(&r, &x, 8);
  return r;
}
inline int __double2hiint(double x) { return (int)(__double_as_longlong(x) >> 32); }
inline double __longlong_as_double(long long x) {
  double r;
  memcpy(&r, &x, 8);
  return r;
}
template <class T, class U>
T atomicAdd(T* p, U v) {
  const T old = *p;
  *p = old + (T)v;
  return old;
}
template <class T>
T atomicMax(T* p, T v) {
  const T old = *p;
  if (v > old) *p = v;
  return old;
}
inline int atomicCAS(int* p, int cmp, int v) {
  const int old = *p;
  if (old == cmp) *p = v;
  return old;
}
inline double __double2float_rn(double x) { return (double)(float)x; }
inline double __double2half(double x) { return x; }  // the storage rule 'mixed' is not run here
inline double __half2float(double x) { return x; }

// what the kernels write in PTX
namespace tlr {
inline void dmma884(double& d0, double& d1, double a, double b) {
  emu::Cta* c = emu::cur->cta;
  const int w = emu::cur->flat / 32 * 32, g = emu::lane() >> 2, t = emu::lane() & 3;
  double av[4], b0[4], b1[4];
  c->slot[emu::cur->flat] = a;
  emu::warp_sync();
  for (int k = 0; k < 4; ++k) av[k] = c->slot[w + 4 * g + k];
  emu::warp_sync();
  c->slot[emu::cur->flat] = b;
  emu::warp_sync();
  for (int k = 0; k < 4; ++k) {
    b0[k] = c->slot[w + 4 * (2 * t) + k];
    b1[k] = c->slot[w + 4 * (2 * t + 1) + k];
  }
  emu::warp_sync();
  for (int k = 0; k < 4; ++k) {
    d0 = fma(av[k], b0[k], d0);
    d1 = fma(av[k], b1[k], d1);
  }
}
inline void cp_async16(void* s, const void* g, int bytes) {
  memset(s, 0, 16);
  memcpy(s, g, (size_t)bytes);
}
inline void cp_async8(void* s, const void* g, int bytes) {
  memset(s, 0, 8);
  memcpy(s, g, (size_t)bytes);
}
inline void cp_async_commit() {}
inline void cp_async_wait_all() {}
inline double rcp_approx(double x) { return (double)(float)1.0 / x; }
inline double rsqrt_approx(double x) { return 1.0 / sqrt(x); }
template <int N>
void bar_sync(int id) { emu::named(id, N, true); }
template <int N>
void bar_arrive(int id) { emu::named(id, N, false); }
}  // namespace tlr

namespace cooperative_groups {
struct cluster_group {
  unsigned block_rank() const { return (unsigned)emu::cur->cta->rank; }
  void sync() const {
    emu::cluster_arrive();
    emu::cluster_wait();
  }
  void barrier_arrive() const { emu::cluster_arrive(); }
  void barrier_wait() const { emu::cluster_wait(); }
  template <class T>
  T* map_shared_rank(T* p, int rank) const {
    emu::Cta* c = emu::cur->cta;
    emu::Cta* d = &c->grid->ctas[c->flat - c->rank + rank];
    return reinterpret_cast<T*>(d->anchor + (reinterpret_cast<char*>(p) - c->anchor));
  }
};
inline cluster_group this_cluster() { return cluster_group{}; }
}  // namespace cooperative_groups
