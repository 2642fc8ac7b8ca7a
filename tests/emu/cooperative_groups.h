// cooperative_groups.h -- the tiles the solve kernel uses, on cuda_host.h's collectives.
#pragma once

namespace cooperative_groups {

struct thread_block {};
inline thread_block this_thread_block() { return {}; }

template <unsigned T>
struct thread_block_tile {
  unsigned thread_rank() const { return threadIdx.x % T; }
  template <class X>
  X shfl(X x, int src) const {
    return emu::value<X>(emu::exchange(T, emu::bits(x))[(threadIdx.x & 31) / T * T + src % T]);
  }
  unsigned ballot(bool p) const {
    const unsigned long long *v = emu::exchange(T, p);
    unsigned b = 0;
    for (unsigned i = 0; i < T; i++) b |= (unsigned)v[(threadIdx.x & 31) / T * T + i] << i;
    return b;
  }
  bool any(bool p) const { return ballot(p) != 0; }
};

template <unsigned T>
thread_block_tile<T> tiled_partition(thread_block) { return {}; }

template <class X>
struct plus {
  X operator()(X a, X b) const { return a + b; }
};
template <class X>
struct less {
  X operator()(X a, X b) const { return b < a ? b : a; }
};
template <class X>
struct greater {
  X operator()(X a, X b) const { return b > a ? b : a; }
};

template <unsigned T, class X, class F>
X reduce(thread_block_tile<T>, X x, F f) {
  const unsigned long long *v = emu::exchange(T, emu::bits(x)) + (threadIdx.x & 31) / T * T;
  X r = emu::value<X>(v[0]);
  for (unsigned i = 1; i < T; i++) r = f(r, emu::value<X>(v[i]));
  return r;
}
template <unsigned T, class X, class F>
X exclusive_scan(thread_block_tile<T>, X x, F f) {
  const unsigned long long *v = emu::exchange(T, emu::bits(x)) + (threadIdx.x & 31) / T * T;
  X r = X(0);
  for (unsigned i = 0; i < threadIdx.x % T; i++) r = f(r, emu::value<X>(v[i]));
  return r;
}

}  // namespace cooperative_groups
