// cuda_host.h -- enough of CUDA C++ to compile the solve kernel for host threads: one std::thread per CUDA thread,
// one process per block (static variables stand in for shared memory, a shared mapping for global memory).
//
// Lanes run freely, which CUDA allows, so code that needs a warp to reconverge by itself shows up: a lane that waits
// in a warp-wide operation for a lane that waits at a block barrier, or threads of a block that wait at different
// block barriers, end the process with status 3.
#pragma once
#include <cuda_runtime.h>
#include <execinfo.h>
#include <sched.h>
#include <sys/mman.h>
#include <sys/wait.h>
#include <unistd.h>

#include <atomic>
#include <chrono>
#include <climits>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <thread>
#include <type_traits>
#include <vector>

#undef __device__
#undef __host__
#undef __global__
#undef __shared__
#undef __forceinline__
#undef __launch_bounds__
#define __device__
#define __host__
#define __global__
#define __shared__ static
#define __forceinline__ inline __attribute__((always_inline))
#define __launch_bounds__(...)

struct Dim {
  unsigned x = 1;
};
inline thread_local Dim threadIdx;
inline Dim blockIdx, blockDim, gridDim;

namespace emu {

constexpr int kMaxThreads = 256;
constexpr int kWaitSeconds = 60;

[[noreturn]] inline void broken(const char *what) {
  std::fprintf(stderr, "block %u thread %u: %s\n", blockIdx.x, threadIdx.x, what);
  std::fflush(stderr);
  _exit(3);
}

// the block barrier: where each thread waits, and the barrier's generation
inline std::atomic<unsigned> bar_gen{0};
inline std::atomic<int> bar_count{0};
inline std::atomic<void *> bar_site{nullptr};
inline std::atomic<unsigned> parked[kMaxThreads];  // 1 + the generation the thread waits in
inline int bar_or[2];

struct Wait {
  std::chrono::steady_clock::time_point t0 = std::chrono::steady_clock::now();
  unsigned n = 0;
  void step(const char *what) {
    sched_yield();
    if (++n % 1024 == 0 && std::chrono::steady_clock::now() - t0 > std::chrono::seconds(kWaitSeconds)) broken(what);
  }
};

// `site` is the return address, so that one barrier inlined at two places counts as two barriers.
__attribute__((noinline)) inline int block_barrier(int v = 0) {
  void *site = __builtin_return_address(0), *none = nullptr;
  const unsigned gen = bar_gen.load();
  if (!bar_site.compare_exchange_strong(none, site) && none != site) {
    void *both[2] = {none, site};
    backtrace_symbols_fd(both, 2, 2);
    broken("block barrier reached at two places");
  }
  if (v) __atomic_store_n(&bar_or[gen & 1], 1, __ATOMIC_SEQ_CST);
  parked[threadIdx.x] = 1 + gen;
  if (bar_count.fetch_add(1) + 1 == (int)blockDim.x) {
    bar_count = 0;
    bar_site = nullptr;
    __atomic_store_n(&bar_or[(gen + 1) & 1], 0, __ATOMIC_SEQ_CST);
    bar_gen.fetch_add(1);
  } else {
    for (Wait w; bar_gen.load() == gen;) w.step("block barrier never completes");
  }
  return __atomic_load_n(&bar_or[gen & 1], __ATOMIC_SEQ_CST);
}

// A collective of the lanes first .. first + size - 1 of a warp: everybody's value, twice buffered.
struct Coll {
  std::atomic<int> count{0};
  std::atomic<unsigned> gen{0};
  unsigned long long val[2][32];
};
inline Coll colls[kMaxThreads / 32][64];  // per warp: tiles of 32, 16, 8, 4 lanes

inline const unsigned long long *exchange(int size, unsigned long long x) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  Coll &c = colls[warp][32 / size - 1 + lane / size];  // 0, 1-2, 3-6, 7-14
  const unsigned gen = c.gen.load();
  c.val[gen & 1][lane] = x;
  if (c.count.fetch_add(1) + 1 == size) {
    c.count = 0;
    c.gen.fetch_add(1);
  } else {
    for (Wait w; c.gen.load() == gen;) {
      for (int i = lane / size * size; i < (lane / size + 1) * size; i++)
        if (parked[warp * 32 + i] == 1 + bar_gen.load() && c.gen.load() == gen)
          broken("a lane left for a block barrier while its warp waits for it");
      w.step("warp collective never completes");
    }
  }
  return c.val[gen & 1];
}

template <class T>
inline unsigned long long bits(T x) {
  static_assert(sizeof(T) <= 8, "");
  unsigned long long b = 0;
  std::memcpy(&b, &x, sizeof x);
  return b;
}
template <class T>
inline T value(unsigned long long b) {
  T x;
  std::memcpy(&x, &b, sizeof x);
  return x;
}

// The whole warp, or (a lane on its own, as __activemask() below says) just this lane.
inline bool whole(unsigned mask) {
  if (mask == 0xffffffffu) return true;
  if (mask != 1u << (threadIdx.x & 31)) broken("partial mask");
  return false;
}
template <class T, class F>
inline T reduce(unsigned mask, T x, F f) {
  if (!whole(mask)) return x;
  const unsigned long long *v = exchange(32, bits(x));
  T r = value<T>(v[0]);
  for (int i = 1; i < 32; i++) r = f(r, value<T>(v[i]));
  return r;
}

inline int skip_barrier = 0;  // the grid barrier (1: the first) that the last block never arrives at
inline unsigned long long fake_tick = 0;  // 0: real time; else ns that every look at the clock takes
inline std::atomic<unsigned long long> *fake_now = nullptr;

}  // namespace emu

#define __syncthreads() ((void)emu::block_barrier())
#define __syncthreads_or(x) emu::block_barrier((x) != 0)
inline void __syncwarp(unsigned mask = 0xffffffffu) {
  if (emu::whole(mask)) emu::exchange(32, 0);
}
inline unsigned __activemask() { return 1u << (threadIdx.x & 31); }
inline unsigned __ballot_sync(unsigned mask, int p) {
  const int lane = threadIdx.x & 31;
  if (!emu::whole(mask)) return p ? 1u << lane : 0;
  const unsigned long long *v = emu::exchange(32, p != 0);
  unsigned b = 0;
  for (int i = 0; i < 32; i++) b |= (unsigned)v[i] << i;
  return b;
}
inline int __any_sync(unsigned mask, int p) { return __ballot_sync(mask, p) != 0; }
inline int __all_sync(unsigned mask, int p) { return __ballot_sync(mask, !p) == 0; }
template <class T>
inline T __shfl_sync(unsigned mask, T x, int src) {
  return emu::whole(mask) ? emu::value<T>(emu::exchange(32, emu::bits(x))[src & 31]) : x;
}
inline unsigned __reduce_add_sync(unsigned mask, unsigned x) {
  return emu::reduce(mask, x, [](unsigned a, unsigned b) { return a + b; });
}
inline int __reduce_min_sync(unsigned mask, int x) {
  return emu::reduce(mask, x, [](int a, int b) { return a < b ? a : b; });
}
inline int __reduce_max_sync(unsigned mask, int x) {
  return emu::reduce(mask, x, [](int a, int b) { return a > b ? a : b; });
}

template <class T>
inline T emu_load(const T *p) {
  if constexpr (std::is_scalar<T>::value) return __atomic_load_n(p, __ATOMIC_RELAXED);
  else return *p;
}
template <class T>
inline T __ldg(const T *p) { return emu_load(p); }
template <class T>
inline T __ldcg(const T *p) { return emu_load(p); }
template <class T>
inline T __ldcs(const T *p) { return emu_load(p); }

template <class T, class U>
inline T atomicAdd(T *p, U v) { return __atomic_fetch_add(p, (T)v, __ATOMIC_SEQ_CST); }
template <class T, class U>
inline T atomicSub(T *p, U v) { return __atomic_fetch_sub(p, (T)v, __ATOMIC_SEQ_CST); }
template <class T, class U>
inline T atomicOr(T *p, U v) { return __atomic_fetch_or(p, (T)v, __ATOMIC_SEQ_CST); }
template <class T, class U>
inline T atomicExch(T *p, U v) { return __atomic_exchange_n(p, (T)v, __ATOMIC_SEQ_CST); }
template <class T, class U, class V>
inline T atomicCAS(T *p, U cmp, V v) {
  T want = (T)cmp;
  __atomic_compare_exchange_n(p, &want, (T)v, false, __ATOMIC_SEQ_CST, __ATOMIC_SEQ_CST);
  return want;
}
template <class T, class U>
inline T atomicMin(T *p, U v) {
  T old = __atomic_load_n(p, __ATOMIC_SEQ_CST);
  while ((T)v < old && !__atomic_compare_exchange_n(p, &old, (T)v, false, __ATOMIC_SEQ_CST, __ATOMIC_SEQ_CST)) {
  }
  return old;
}
template <class T, class U>
inline T atomicMax(T *p, U v) {
  T old = __atomic_load_n(p, __ATOMIC_SEQ_CST);
  while ((T)v > old && !__atomic_compare_exchange_n(p, &old, (T)v, false, __ATOMIC_SEQ_CST, __ATOMIC_SEQ_CST)) {
  }
  return old;
}

inline int min(int a, int b) { return a < b ? a : b; }
inline int max(int a, int b) { return a > b ? a : b; }
inline int __ffs(unsigned x) { return __builtin_ffs((int)x); }
inline int __popc(unsigned x) { return __builtin_popcount(x); }
inline unsigned long long __umul64hi(unsigned long long a, unsigned long long b) {
  return (unsigned long long)(((unsigned __int128)a * b) >> 64);
}
inline void __nanosleep(unsigned) { sched_yield(); }
inline void __threadfence_system() { __atomic_thread_fence(__ATOMIC_SEQ_CST); }

// ---- the kernel's inline PTX (dmf_ptx.cuh) -------------------------------------------------------------------------
#define DMF_PTX_CUH
namespace dmfd {
inline unsigned ld_acquire_u32(const unsigned *p) { sched_yield(); return __atomic_load_n(p, __ATOMIC_ACQUIRE); }
inline unsigned atom_add_release_u32(unsigned *p, unsigned x) {  // only grid barriers use it
  static int count = 0;
  if (blockIdx.x == gridDim.x - 1 && ++count == emu::skip_barrier) return __atomic_load_n(p, __ATOMIC_SEQ_CST);
  return __atomic_fetch_add(p, x, __ATOMIC_SEQ_CST);
}
inline unsigned atom_add_acqrel_u32(unsigned *p, unsigned x) { return __atomic_fetch_add(p, x, __ATOMIC_SEQ_CST); }
inline void st_release_sys_u32(unsigned *p, unsigned x) { __atomic_store_n(p, x, __ATOMIC_RELEASE); }
inline int ld_rlx(const int *p) { return __atomic_load_n(p, __ATOMIC_RELAXED); }
inline long long ld_rlx(const long long *p) { return __atomic_load_n(p, __ATOMIC_RELAXED); }
inline unsigned long long ld_rlx(const unsigned long long *p) { return __atomic_load_n(p, __ATOMIC_RELAXED); }
inline unsigned long long globaltimer() {
  if (emu::fake_tick) return emu::fake_now->fetch_add(emu::fake_tick);
  return (unsigned long long)std::chrono::steady_clock::now().time_since_epoch().count();
}
inline unsigned lanemask_lt() { return (1u << (threadIdx.x & 31)) - 1; }
inline void keep_u64(unsigned long long) {}
}  // namespace dmfd

namespace emu {

// Global memory: one mapping that every block's process shares.
inline char *heap = nullptr, *heap_end = nullptr;
template <class T>
T *global(size_t count) {
  if (!heap) {
    constexpr size_t kHeap = 64 << 20;
    heap = (char *)mmap(nullptr, kHeap, PROT_READ | PROT_WRITE, MAP_SHARED | MAP_ANONYMOUS, -1, 0);
    if (heap == MAP_FAILED) std::abort();
    heap_end = heap + kHeap;
  }
  T *p = (T *)heap;
  heap += (sizeof(T) * count + 255) / 256 * 256;
  if (heap > heap_end) std::abort();
  return p;
}

// Runs f on `blocks` blocks of `threads` threads; 0, or the status of a block that failed.
template <class F>
int launch(int blocks, int threads, F f) {
  if (threads > kMaxThreads || threads % 32) std::abort();
  gridDim.x = blocks;
  blockDim.x = threads;
  fake_now = global<std::atomic<unsigned long long>>(1);
  std::fflush(stdout);
  std::vector<pid_t> kids;
  for (int b = 0; b < blocks; b++) {
    const pid_t pid = fork();
    if (pid == 0) {
      blockIdx.x = b;
      std::vector<std::thread> th;
      for (int i = 0; i < threads; i++)
        th.emplace_back([&f, i] {
          threadIdx.x = i;
          f();
        });
      for (auto &t : th) t.join();
      _exit(0);
    }
    kids.push_back(pid);
  }
  int rc = 0;
  for (size_t left = kids.size(); left > 0; left--) {  // the first failure ends the others
    int st = 0;
    const pid_t pid = wait(&st);
    const int code = WIFEXITED(st) ? WEXITSTATUS(st) : 4;
    for (pid_t &k : kids)
      if (k == pid) k = 0;
    if (code && !rc) {
      rc = code;
      for (pid_t k : kids)
        if (k > 0) kill(k, SIGKILL);
    }
  }
  return rc;
}

}  // namespace emu
