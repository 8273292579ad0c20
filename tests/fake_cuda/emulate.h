// CUDA threads as fibers on the CPU, for running the LU panel kernels without a GPU: one OS thread per
// CTA, `__shared__` variables as thread-local ones, a warp's collectives, named barriers, cluster barriers, mbarriers
// and st.async as the PTX ISA describes them.  The functions of the kernels' headers that are inline assembly are
// taken out of the source and defined here instead.
// Faults are counted, not suffered: stores outside the buffers show in their guard zones (Guarded), an
// mbarrier that gets more arrivals than it waits for, and a remote store into a CTA that has left, in
// emu::faults.  Messages (st.async) can be dropped, which makes a wait run out.
#pragma once
#include <math.h>
#include <sched.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <sys/mman.h>
#include <ucontext.h>

#include <algorithm>
#include <atomic>
#include <functional>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

#define __host__
#define __device__
#define __global__
#define __forceinline__ inline
#define __launch_bounds__(...)
#define __align__(n) __attribute__((aligned(n)))
#define __shared__ thread_local

struct alignas(8) float2 { float x, y; };
struct alignas(16) double2 { double x, y; };
struct alignas(8) uint2 { unsigned x, y; };
struct alignas(16) float4 { float x, y, z, w; };
struct alignas(16) uint4 { unsigned x, y, z, w; };
struct dim3 { unsigned x = 1, y = 1, z = 1; };
inline float2 make_float2(float x, float y) { return {x, y}; }
inline double2 make_double2(double x, double y) { return {x, y}; }
inline uint2 make_uint2(unsigned x, unsigned y) { return {x, y}; }
inline uint4 make_uint4(unsigned x, unsigned y, unsigned z, unsigned w) { return {x, y, z, w}; }
using cudaError_t = int;
template <typename T, typename U> T bits_as(U u) {
  static_assert(sizeof(T) == sizeof(U), "same size");
  T t;
  memcpy(&t, &u, sizeof(t));
  return t;
}
inline unsigned __float_as_uint(float v) { return bits_as<unsigned>(v); }
inline float __uint_as_float(unsigned v) { return bits_as<float>(v); }
inline long long __double_as_longlong(double v) { return bits_as<long long>(v); }
inline int __double2hiint(double v) { return (int)(bits_as<uint64_t>(v) >> 32); }
inline int __double2loint(double v) { return (int)bits_as<uint64_t>(v); }
inline double __hiloint2double(int h, int l) { return bits_as<double>(((uint64_t)(unsigned)h << 32) | (unsigned)l); }
inline int __ffs(unsigned v) { return __builtin_ffs((int)v); }
template <typename T> T __ldg(const T* p) { return *p; }
template <typename T> T __ldcg(const T* p) { return *p; }
template <typename T> void __stcg(T* p, T v) { *p = v; }
inline int max(int a, int b) { return a > b ? a : b; }
inline int min(int a, int b) { return a < b ? a : b; }
inline unsigned max(unsigned a, unsigned b) { return a > b ? a : b; }

namespace emu {

struct Barrier { int n = 0; unsigned gen = 0; };
struct Warp { int n = 0; unsigned gen = 0; uint64_t in[32], out[2][32]; };
struct Fiber { ucontext_t ctx; dim3 tid; bool done = false; unsigned cluster_gen = 0; unsigned sends[16] = {}; };
struct Cluster {
  std::atomic<int> arrived{0};
  std::atomic<unsigned> gen{0};
  int threads = 0;
  char* base[16] = {};            // a thread-local address of every CTA's OS thread
  std::atomic<bool> left[16] = {};
};
struct Cta {
  dim3 bid, bdim, gdim;
  int rank = 0, live = 0, cur = 0;
  Cluster* cluster = nullptr;
  Barrier bar[16];
  std::vector<Warp> warps;
  std::vector<Fiber> fibers;
  ucontext_t home;
  const std::function<void()>* body = nullptr;
};
inline thread_local Cta* cta = nullptr;
inline thread_local __attribute__((aligned(64))) char tls_mark[64];
inline thread_local __attribute__((aligned(64))) unsigned char dynamic_smem[200 * 1024];
inline std::mutex mu;
inline std::atomic<int> faults{0};
inline unsigned wait_limit = 1u << 30;
// messages from CTA drop_src (-1: any) to CTA drop_dst, from a thread's drop_from-th send on, are lost
inline int drop_src = -1, drop_dst = -1;
inline unsigned drop_from = 0;

inline void fault(const char* what) {
  if (faults++ < 8) fprintf(stderr, "emulator: %s\n", what);
}
inline Fiber& me() { return cta->fibers[cta->cur]; }
inline int lane() { return cta->cur & 31; }
inline void yield() {
  Cta& c = *cta;
  const int from = c.cur, n = (int)c.fibers.size();
  int to = from;
  do to = to + 1 == n ? 0 : to + 1; while (c.fibers[to].done);
  if (to <= from) sched_yield();
  if (to == from) return;
  c.cur = to;
  swapcontext(&c.fibers[from].ctx, &c.fibers[to].ctx);
}
inline void entry() {
  Cta& c = *cta;
  (*c.body)();
  c.fibers[c.cur].done = true;
  if (--c.live == 0) setcontext(&c.home);
  int to = c.cur;
  do to = to + 1 == (int)c.fibers.size() ? 0 : to + 1; while (c.fibers[to].done);
  c.cur = to;
  setcontext(&c.fibers[to].ctx);
}
inline void barrier(int id, int threads) {
  Barrier& b = cta->bar[id];
  const unsigned g = b.gen;
  if (++b.n == threads) {
    b.n = 0;
    ++b.gen;
  } else {
    while (b.gen == g) yield();
  }
}
inline const uint64_t* exchange(uint64_t v) {  // every lane's value
  Warp& w = cta->warps[cta->cur >> 5];
  const unsigned g = w.gen;
  w.in[lane()] = v;
  if (++w.n == 32) {
    w.n = 0;
    memcpy(w.out[g & 1], w.in, sizeof(w.in));
    ++w.gen;
  } else {
    while (w.gen == g) yield();
  }
  return w.out[g & 1];
}

// kernel body on grid CTAs; concurrent: one cluster (or a cooperative grid), else one CTA after the other
inline void launch(int grid, int threads, bool concurrent, const std::function<void()>& body) {
  Cluster cl;
  cl.threads = grid * threads;
  std::atomic<int> up{0};
  auto run = [&](int b) {
    Cta c;
    cta = &c;
    c.rank = b & 15;
    c.cluster = &cl;
    c.bid.x = b;
    c.bdim.x = threads;
    c.gdim.x = grid;
    c.live = threads;
    c.body = &body;
    c.warps.resize(threads / 32);
    c.fibers.resize(threads);
    constexpr size_t kStack = 64 * 1024;
    char* st = (char*)mmap(nullptr, kStack * threads, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
    for (int t = 0; t < threads; ++t) {
      Fiber& f = c.fibers[t];
      f.tid.x = t;
      getcontext(&f.ctx);
      f.ctx.uc_stack.ss_sp = st + kStack * t;
      f.ctx.uc_stack.ss_size = kStack;
      f.ctx.uc_link = nullptr;
      makecontext(&f.ctx, entry, 0);
    }
    cl.base[c.rank] = tls_mark;
    ++up;
    while (concurrent && up.load() < grid) sched_yield();
    swapcontext(&c.home, &c.fibers[0].ctx);
    cl.left[c.rank] = true;
    ++up;
    while (concurrent && up.load() < 2 * grid) sched_yield();  // the thread-local memory stays until all CTAs have left
    munmap(st, kStack * threads);
    cta = nullptr;
  };
  std::vector<std::thread> th;
  for (int b = 0; b < grid; ++b) {
    th.emplace_back(run, b);
    if (!concurrent) th.back().join();
  }
  if (concurrent)
    for (auto& t : th) t.join();
}

// shared-memory addresses: rank << 27 | offset from the CTA's tls_mark + 2^26
inline uint32_t address(const void* p) {
  return ((uint32_t)cta->rank << 27) | (uint32_t)((const char*)p - tls_mark + (1 << 26));
}
inline char* resolve(uint32_t a) { return cta->cluster->base[a >> 27] + (int)(a & ((1u << 27) - 1)) - (1 << 26); }

struct Mbar { int16_t pending; uint16_t phase; int32_t tx; };
inline void mbar_step(Mbar* b, int arrive, int tx) {  // under mu
  b->pending = (int16_t)(b->pending - arrive);
  b->tx += tx;
  if (b->pending < 0) fault("more arrivals than the mbarrier waits for");
  if (b->pending <= 0 && b->tx == 0) {
    b->phase ^= 1;
    b->pending = 1;
  }
}

// memory of n elements between guard zones
template <typename T> struct Guarded {
  static constexpr size_t kGuard = 1 << 25;
  size_t n;
  std::vector<unsigned char> mem;
  T* p;
  explicit Guarded(size_t n_) : n(n_), mem(2 * kGuard + n_ * sizeof(T), 0xA7), p((T*)(mem.data() + kGuard)) { memset((void*)p, 0, n * sizeof(T)); }
  size_t hits() const {
    size_t h = 0;
    for (size_t i = 0; i < kGuard; ++i) h += (mem[i] != 0xA7) + (mem[mem.size() - 1 - i] != 0xA7);
    return h;
  }
};
}  // namespace emu

#define threadIdx (emu::me().tid)
#define blockIdx (emu::cta->bid)
#define blockDim (emu::cta->bdim)
#define gridDim (emu::cta->gdim)
inline void __syncthreads() { emu::barrier(0, (int)blockDim.x); }
inline void __syncwarp(unsigned = 0xffffffffu) { emu::exchange(0); }
inline unsigned __ballot_sync(unsigned, bool v) {
  const uint64_t* a = emu::exchange(v);
  unsigned m = 0;
  for (int i = 0; i < 32; ++i) m |= (unsigned)(a[i] != 0) << i;
  return m;
}
inline bool __any_sync(unsigned m, bool v) { return __ballot_sync(m, v) != 0; }
inline unsigned __reduce_max_sync(unsigned, unsigned v) {
  const uint64_t* a = emu::exchange(v);
  return (unsigned)*std::max_element(a, a + 32);
}
template <typename T> T __shfl_down_sync(unsigned, T v, int o) {
  static_assert(sizeof(T) <= 8, "one word");
  uint64_t w = 0;
  memcpy(&w, &v, sizeof(v));
  const int src = emu::lane() + o;
  const uint64_t r = emu::exchange(w)[src < 32 ? src : emu::lane()];
  memcpy(&v, &r, sizeof(v));
  return v;
}
template <typename T, typename F> T emu_atomic(T* p, F f) {
  std::lock_guard<std::mutex> lk(emu::mu);
  const T old = *p;
  *p = f(old);
  return old;
}
template <typename T> T atomicAdd(T* p, T v) { return emu_atomic(p, [&](T o) { return (T)(o + v); }); }
template <typename T> T atomicMax(T* p, T v) { return emu_atomic(p, [&](T o) { return o > v ? o : v; }); }
template <typename T> T atomicMin(T* p, T v) { return emu_atomic(p, [&](T o) { return o < v ? o : v; }); }
inline int atomicExch(int* p, int v) { return emu_atomic(p, [&](int) { return v; }); }
inline int atomicCAS(int* p, int c, int v) { return emu_atomic(p, [&](int o) { return o == c ? v : o; }); }
inline void __nanosleep(unsigned) { emu::yield(); }
inline int emu_load(const int* p) { return emu_atomic(const_cast<int*>(p), [](int o) { return o; }); }

namespace hprmat {
inline void cp_async_elem(float2* d, const float2* s) { *d = *s; }
inline void cp_async_elem(double2* d, const double2* s) { *d = *s; }
inline void cp_async_wait_all() {}
inline long long device_ns() { return 0; }
inline void cluster_arrive() {
  emu::Cluster& c = *emu::cta->cluster;
  emu::me().cluster_gen = c.gen.load();
  if (c.arrived.fetch_add(1) + 1 == c.threads) {
    c.arrived = 0;
    ++c.gen;
  }
}
inline void cluster_wait() {
  while (emu::cta->cluster->gen.load() == emu::me().cluster_gen) emu::yield();
}
inline void grid_arrive(int* counter) { atomicAdd(counter, 1); }
inline bool grid_wait(int* counter, int* timeout_flag, unsigned target, int site, unsigned = 0) {
  static thread_local int ok_w;  // as in the kernel: thread 0 waits, the CTA learns of it
  if (threadIdx.x == 0) {
    int ok = 1;
    for (unsigned spins = 1; (unsigned)emu_load(counter) < target; ++spins) {
      if (emu_load(timeout_flag) != 0 || spins >= emu::wait_limit) {
        if (spins >= emu::wait_limit) atomicExch(timeout_flag, site);
        ok = 0;
        break;
      }
      emu::yield();
    }
    ok_w = ok;
  }
  __syncthreads();
  return ok_w != 0;
}
inline uint32_t mapa_u32(uint32_t a, uint32_t rank) { return (a & ((1u << 27) - 1)) | (rank << 27); }
inline void st_async16(uint32_t dst, uint4 v, uint32_t bar) {
  const int d = (int)(dst >> 27);
  const unsigned k = emu::me().sends[d]++;
  if (d == emu::drop_dst && (emu::drop_src < 0 || emu::drop_src == emu::cta->rank) && k >= emu::drop_from) return;
  std::lock_guard<std::mutex> lk(emu::mu);
  if (emu::cta->cluster->left[d]) return emu::fault("remote store into a CTA that has left");
  memcpy(emu::resolve(dst), &v, 16);
  emu::mbar_step((emu::Mbar*)emu::resolve(bar), 0, -16);
}
inline void st_cluster_u32(uint32_t dst, unsigned v) {
  std::lock_guard<std::mutex> lk(emu::mu);
  if (emu::cta->cluster->left[dst >> 27]) return emu::fault("remote store into a CTA that has left");
  memcpy(emu::resolve(dst), &v, 4);
}
namespace tc {
inline uint32_t smem_u32(const void* p) { return emu::address(p); }
inline void mbar_init(uint64_t* b, uint32_t n) {
  const emu::Mbar m{(int16_t)n, 0, 0};
  memcpy(b, &m, sizeof(m));
}
inline bool mbar_try_wait(uint64_t* b, uint32_t parity) {
  emu::yield();
  std::lock_guard<std::mutex> lk(emu::mu);
  return ((emu::Mbar*)b)->phase != parity;
}
inline void mbar_expect_tx(uint64_t* b, uint32_t bytes) {
  std::lock_guard<std::mutex> lk(emu::mu);
  emu::mbar_step((emu::Mbar*)b, 1, (int)bytes);
}
}  // namespace tc
}  // namespace hprmat
