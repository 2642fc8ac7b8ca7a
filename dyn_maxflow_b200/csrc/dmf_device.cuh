// dmf_device.cuh -- device-side building blocks of the sm_100a solver:
// memory-order helpers, the bounded grid barrier, queue appends and the group
// abstractions (a warp tile or a whole block working on one vertex).
#pragma once

#include <climits>
#include <cstdint>
#include <cooperative_groups.h>
#include <cooperative_groups/reduce.h>
#include <cooperative_groups/scan.h>

#include "dmf_ptx.cuh"

namespace dmfd {

namespace cg = cooperative_groups;

// ---- error bits (Ctrl::err) ------------------------------------------------
enum : int {
  ERR_TIMEOUT = 1,       // a grid-barrier wait ran out of time
  ERR_NO_CONV = 2,       // outer-iteration bound reached
  ERR_UNKNOWN_ARC = 4,   // update names an absent arc
  ERR_DUP_ARC = 8,       // arc twice in one batch
  ERR_BAD_UPDATE = 16,   // vertex id out of range or capacity out of bounds
};

// Barrier wait limit: 4 s of %globaltimer.  Any single phase of a solve is
// orders of magnitude shorter; hitting it means a block never arrived.
constexpr unsigned long long kBarrierTimeoutNs = 4000000000ull;
// The limit under the failure-injection test hook (DMF_FLAG_TEST_BARRIER_TIMEOUT).
constexpr unsigned long long kTestBarrierTimeoutNs = 20000000ull;

// Per-phase counters, triple-buffered: phase k appends into slot k%3, reads
// slot (k-1)%3, and block 0 clears slot (k+1)%3.
struct Slot {
  int q;             // normal-queue tail
  int hq;            // hub-queue tail
  long long arcs;    // sum of degrees of appended vertices
  int cnt;           // generic counter (BFS: active vertices labelled; topo push: active seen)
  int pad;
};

// Control block of one solver (device memory, zero between launches: the last
// block of a launch clears it).
struct Ctrl {
  unsigned int bar_count;     // grid barrier: arrivals (low bits) and generation (top bit)
  unsigned int bar_gen;       // unused
  int err;
  int err_info;
  Slot slot[3];
  // per global relabel
  int act_q, act_hq;          // active list tails built by the BFS
  int pos_count;              // vertices with excess > 0 (not s, t, dead)
  int pad0;
  long long unexplored;       // arcs of not-yet-labelled candidate vertices
  long long flow;             // result
  // statistics
  unsigned long long st_outer, st_levels, st_rounds, st_pushes, st_relabels, st_arcs, st_visits, st_dead;
  unsigned int rounds_used;
  int trace_len;              // entries written to the optional timeline
  // push-round worklist tails and topology-driven active counts, round r uses [r % 3]
  int wtail[3], whtail[3], seen[3];
  int pad1;
  unsigned long long probe[2];  // longest work item of a phase, (ns << 32) | vertex
  unsigned long long blk[2];    // longest block work of a phase (ns), barrier exit to arrival
  // kept dead set (dynamic batches): vertices of the dead set whose excess a batch
  // lowered or that a pull moved a deficit to (candidates for deficits), the
  // deficits found among them, and those left after the local repair
  int dcand;
  int dseeds;
  int dleft;
  int dkept;                    // 1: the dead set was kept for the global relabels
  unsigned long long st_barcs;  // adjacency entries read by global-relabel BFS levels
  unsigned long long st_dseeds; // deficits inside the kept dead set (first local pass)
  unsigned long long st_revived; // dead vertices revived because they reach a deficit left over
  int dup_at;                   // 1 + an update whose arc an earlier update of the batch names (0: none)
  int berr, berr_info;          // error bits of a batch's lookup, and the update
  int nreopen;                  // updates queued for saturation: source arcs, reopened arcs
  int nrepair;                  // updates queued for the over-capacity repair
  // barrier-free phases (dmf_async.cuh): when the push phase ends (0: not set
  // yet), blocks idle in the relabel [0] and in the push phase [1], vertices whose
  // label is not settled, active vertices and greatest distance of the last
  // relabel
  unsigned long long adeadline;
  int aidle[2];
  int aunsettled;
  int aact;
  int adepth;
  unsigned done;                // blocks that have ended
};

// Where a launch leaves its result in pinned host memory: the control block,
// then the launch's number.
struct HostResult {
  Ctrl c;
  unsigned seq;
};

// ---- memory helpers ---------------------------------------------------------
__device__ __forceinline__ int ld_vol(const int *p) { return *(const volatile int *)p; }
__device__ __forceinline__ long long ld_vol(const long long *p) { return *(const volatile long long *)p; }
__device__ __forceinline__ long long atomic_add_ll(long long *p, long long v) {
  return (long long)atomicAdd((unsigned long long *)p, (unsigned long long)v);
}

// ---- warp-wide sums and prefixes ----------------------------------------------
// Written out with ballots and redux.sync instead of cooperative_groups'
// coalesced groups: those find a lane of a partial warp by a software search in
// every step of a scan, and partial warps are the rule here (a BFS level or a
// push round of a few hundred vertices).  A phase is bound by the instructions
// of its slowest warp, so these lengths matter more than the arithmetic.

// Sum of v over the lanes of `mask` (every one of them must call it), modulo
// 2^64: three redux.sync over 24-, 24- and 16-bit pieces, whose 32-lane sums
// cannot overflow.
__device__ __forceinline__ unsigned long long warp_sum_u64(unsigned mask, unsigned long long v) {
  const unsigned s0 = __reduce_add_sync(mask, (unsigned)v & 0xffffffu);
  const unsigned s1 = __reduce_add_sync(mask, (unsigned)(v >> 24) & 0xffffffu);
  const unsigned s2 = __reduce_add_sync(mask, (unsigned)(v >> 48));
  return (unsigned long long)s0 + ((unsigned long long)s1 << 24) + ((unsigned long long)s2 << 48);
}

// ---- block accumulators ---------------------------------------------------------
// Sums that every warp of the grid contributes to in a phase (thousands of
// same-address atomics would serialise at one L2 slice): warps add into shared
// memory, and the grid barrier that ends the phase adds a block's totals to
// global memory before it arrives.  Slot i of a phase has one destination.
constexpr int kAccSlots = 6;
struct BlockAcc {
  unsigned long long v[kAccSlots];
  unsigned long long *to[kAccSlots];  // bit 0 set: a 32-bit counter
};

__device__ __forceinline__ BlockAcc &block_acc() {
  __shared__ BlockAcc acc;
  return acc;
}

__device__ __forceinline__ void acc_init() {
  if (threadIdx.x < kAccSlots) block_acc().v[threadIdx.x] = 0;
  __syncthreads();
}

// Whole warps call it (any subset of the block's warps).
__device__ __forceinline__ void block_add_ll(int slot, long long *p, long long v) {
  BlockAcc &acc = block_acc();
  const unsigned long long s = warp_sum_u64(0xffffffffu, (unsigned long long)v);
  if ((threadIdx.x & 31) == 0 && s) {
    acc.to[slot] = (unsigned long long *)p;
    atomicAdd(&acc.v[slot], s);
  }
}

__device__ __forceinline__ void block_add_int(int slot, int *p, int v) {
  BlockAcc &acc = block_acc();
  const int s = (int)__reduce_add_sync(0xffffffffu, (unsigned)v);
  if ((threadIdx.x & 31) == 0 && s) {
    acc.to[slot] = (unsigned long long *)((unsigned long long)p | 1);
    atomicAdd(&acc.v[slot], (unsigned long long)(long long)s);
  }
}

// By lanes of one warp, after a block barrier: adds the totals to their
// destinations and clears them.
__device__ __forceinline__ void acc_flush() {
  BlockAcc &acc = block_acc();
  const int i = threadIdx.x;
  if (i < kAccSlots) {
    const unsigned long long x = acc.v[i];
    if (x) {
      const unsigned long long to = (unsigned long long)acc.to[i];
      // with the old value read back: in a grid of one block the same warp reads
      // the control block next, without a fence
      unsigned long long old;
      if (to & 1) old = (unsigned long long)atomicAdd((int *)(to & ~1ull), (int)x);
      else old = atomicAdd((unsigned long long *)to, x);
      keep_u64(old);
      acc.v[i] = 0;
    }
  }
}

// ---- bounded grid barrier ---------------------------------------------------
// All blocks of a cooperative launch call it the same number of times.  Thread
// 0 of each block arrives with ONE atomic on bar_count: block 0 adds
// 2^31 - (G - 1), every other block adds 1, so the counter's top bit flips
// exactly when the last of the G blocks arrives (and the low bits return to
// where they were: nothing has to be reset between barriers).  A waiter polls
// until the top bit differs from the value its own arrival saw; a block that
// is already in the next barrier cannot flip it back, because that flip needs
// every block, the waiter included.  Polls check the error word and the
// %globaltimer limit (`limit_ns`, normally kBarrierTimeoutNs) every 64 iterations.
//
// The arrival is a release (it orders the block's writes, which the block
// barrier before it collected), the poll an acquire: no further fence, and no
// sleep between polls.  With full fences around both and a 32 ns sleep an empty
// barrier of 296 blocks took 3.1 us; it takes 1.9 us, 0.6 of it the copy below.
//
// After the wait, warp 0 copies the whole control block into `snap` (shared
// memory): the phase that follows reads the counters the previous phase
// produced from there, so a phase costs G control-block reads instead of one
// per warp on a single L2 line.  Returns false (uniformly per block) when an
// error is set.
__device__ __forceinline__ bool grid_barrier(Ctrl *c, Ctrl *snap, unsigned long long limit_ns) {
  __shared__ int s_err;
  __syncthreads();
  if (threadIdx.x < 32) {
    acc_flush();
    __syncwarp();
    if (threadIdx.x == 0 && gridDim.x > 1) {  // one block: the block barriers are enough
      const unsigned nb = blockIdx.x == 0 ? 0x80000000u - (gridDim.x - 1) : 1u;
      const unsigned old = atom_add_release_u32(&c->bar_count, nb);
      unsigned long long t0 = 0;
      int spins = 0;
      while (((ld_acquire_u32(&c->bar_count) ^ old) & 0x80000000u) == 0) {
        if ((++spins & 63) == 0) {
          if (ld_vol(&c->err)) break;
          const unsigned long long now = globaltimer();
          if (!t0) {
            t0 = now;
          } else if (now - t0 > limit_ns) {
            atomicOr(&c->err, ERR_TIMEOUT);
            break;
          }
        }
      }
    }
    __syncwarp();
    const int *src = (const int *)c;
    int *dst = (int *)snap;
    constexpr int kWords = (int)(sizeof(Ctrl) / 4);
#pragma unroll
    for (int i = 0; i < (kWords + 31) / 32; i++) {
      const int w = threadIdx.x + 32 * i;
      if (w < kWords) dst[w] = __ldcg(src + w);
    }
    __syncwarp();
    if (threadIdx.x == 0) s_err = snap->err;
  }
  __syncthreads();
  return s_err == 0;
}

// ---- work-item numbering ----------------------------------------------------
// Worklist items are numbered blocks first: thread t of block b is worker
// t * G + b (G blocks), so items 0 .. G-1 go to G different blocks -- every SM
// -- before any block takes a second one.  A short list (a BFS level on a
// grid, a push round late in a solve) is then worked on by all SMs at once
// instead of filling the first blocks, whose load/store units would serialise
// its scattered accesses.  Loops over every vertex keep the contiguous
// numbering, which keeps their per-vertex array accesses coalesced.
// `rot` rotates the order inside a block so that thread `rot` takes a block's
// first item: the kinds of work of one phase (hub chunks, one-thread items,
// tile items) start on different warps and run side by side when the lists are
// short, instead of queueing on warp 0.
__device__ __forceinline__ int spread_thread(int rot = 0) {
  const int t = (int)threadIdx.x - rot;
  return (t < 0 ? t + (int)blockDim.x : t) * gridDim.x + blockIdx.x;
}
// The same for groups of T consecutive threads (T divides the block size and
// `rot`).
template <int T>
__device__ __forceinline__ int spread_group(int rot = 0) {
  const int t = (int)threadIdx.x - rot;
  return ((t < 0 ? t + (int)blockDim.x : t) / T) * gridDim.x + blockIdx.x;
}
// Threads numbered warps first over the blocks: lanes keep consecutive numbers
// (coalesced reads of a batch's arrays), warps 0 .. G-1 sit in G blocks.
__device__ __forceinline__ int spread_lane() { return spread_group<32>() * 32 + (int)(threadIdx.x & 31); }
// Rotations used by the phases: hub chunks from warp 0, tile items from the
// first warp of the second quarter of the block, one-thread items from the
// middle.
__device__ __forceinline__ int rot_tiles() { return (int)blockDim.x / 4; }
__device__ __forceinline__ int rot_threads() { return (int)blockDim.x / 2; }

// ---- queue append (warp-aggregated) -----------------------------------------
// Position of this thread's entry behind *tail, one atomic for the threads of
// the warp that call it together.
__device__ __forceinline__ int reserve_one(int *tail) {
  const unsigned mask = __activemask(), lt = lanemask_lt();
  const int leader = __ffs(mask) - 1;
  int base = 0;
  if ((mask & lt) == 0) base = atomicAdd(tail, __popc(mask));
  return __shfl_sync(mask, base, leader) + __popc(mask & lt);
}

// Reserves `cnt` (0 to 15) consecutive slots behind *tail for this thread, one
// atomic for the threads that call it together: the prefix over the lanes is
// summed bit by bit of the counts.
__device__ __forceinline__ int reserve(int *tail, int cnt) {
  const unsigned mask = __activemask(), lt = lanemask_lt();
  const int leader = __ffs(mask) - 1;
  int pre = 0, tot = 0;
#pragma unroll
  for (int b = 0; b < 4; b++) {
    const unsigned m = __ballot_sync(mask, (cnt >> b) & 1);
    pre += __popc(m & lt) << b;
    tot += __popc(m) << b;
  }
  int base = 0;
  if ((mask & lt) == 0) base = atomicAdd(tail, tot);
  return __shfl_sync(mask, base, leader) + pre;
}

__device__ __forceinline__ void append(int *q, int *tail, int v) { q[reserve_one(tail)] = v; }

// append() into a queue of `cap` entries: *tail still counts every append, so
// *tail > cap afterwards tells that entries were dropped.
__device__ __forceinline__ void append_bounded(int *q, int *tail, int v, int cap) {
  const int at = reserve_one(tail);
  if (at < cap) q[at] = v;
}

// ---- groups: one thread, T lanes of a warp, or the whole block ----------------
struct ThreadGroup {
  __device__ __forceinline__ int rank() const { return 0; }
  __host__ __device__ static constexpr int size() { return 1; }
  __device__ __forceinline__ long long scan(long long x, long long &tot) {
    tot = x;
    return 0;
  }
  __device__ __forceinline__ int min_all(int x) { return x; }
  __device__ __forceinline__ long long sum_all(long long x) { return x; }
  __device__ __forceinline__ bool any(bool x) { return x; }
};

template <int T>
struct TileGroup {
  cg::thread_block_tile<T> g;
  __device__ TileGroup() : g(cg::tiled_partition<T>(cg::this_thread_block())) {}
  __device__ __forceinline__ int rank() const { return (int)g.thread_rank(); }
  __host__ __device__ static constexpr int size() { return T; }
  // exclusive prefix sum and total
  __device__ __forceinline__ long long scan(long long x, long long &tot) {
    long long pre = cg::exclusive_scan(g, x, cg::plus<long long>());
    tot = g.shfl(pre + x, T - 1);
    return pre;
  }
  __device__ __forceinline__ int min_all(int x) {
    if constexpr (T == 32) return __reduce_min_sync(0xffffffffu, x);
    return cg::reduce(g, x, cg::less<int>());
  }
  __device__ __forceinline__ long long sum_all(long long x) {
    if constexpr (T == 32) return (long long)warp_sum_u64(0xffffffffu, (unsigned long long)x);
    return cg::reduce(g, x, cg::plus<long long>());
  }
  __device__ __forceinline__ bool any(bool x) { return g.any(x); }
};

// ---- arc table: (tail, head) -> arc ------------------------------------------
// Open addressing with linear probing over `nslots` 16-byte slots.  An empty
// slot has tail == kEmptyTail (the table is cleared with 0xFF bytes, which also
// sets arc = -1).  The table is only read after it is built: a lookup does not
// write the slot line, so the line is never written back.
struct __align__(16) ArcSlot {
  int tail, head, arc, unused;
};
constexpr int kEmptyTail = -1;

// Slots per arc count: load factor at most 0.5, so a found key takes 1.5
// probes on average, most of them in the first slot's DRAM sector (at R-MAT
// 24 the lookup phase measured 291 us at load 0.5, 340 us at 0.62, 540 us at
// 0.8, for 2.6 M updates).
__host__ __device__ constexpr long long arc_table_slots(long long m) { return 2 * m + 64; }

// The 64-bit key as it lies in the slot's first two words (tail low, head high).
__device__ __forceinline__ unsigned long long arc_key(int u, int v) {
  return ((unsigned long long)(unsigned)v << 32) | (unsigned)u;
}

// First slot of a key: the SplitMix64 finaliser (Steele, Lea and Flood,
// "Fast splittable pseudorandom number generators", OOPSLA 2014) mixes the
// key, and the high half of its product with nslots maps it onto [0, nslots)
// (Lemire's multiply-shift range reduction) without a division.
__device__ __forceinline__ long long arc_slot0(int u, int v, long long nslots) {
  unsigned long long x = arc_key(u, v);
  x ^= x >> 30;
  x *= 0xbf58476d1ce4e5b9ull;
  x ^= x >> 27;
  x *= 0x94d049bb133111ebull;
  x ^= x >> 31;
  return (long long)__umul64hi(x, (unsigned long long)nslots);
}

// One slot as one 16-byte load through L2, bypassing L1: a random slot is
// seldom read twice by one SM, and tail, head and arc never change after the
// build.
__device__ __forceinline__ ArcSlot load_slot(const ArcSlot *s) {
  const int4 x = __ldcg(reinterpret_cast<const int4 *>(s));
  return ArcSlot{x.x, x.y, x.z, x.w};
}

// Arc u->v, or -1 (read-only probe).
__device__ __forceinline__ int find_arc_table(const ArcSlot *tab, long long nslots, int u, int v) {
  long long sl = arc_slot0(u, v, nslots);
  for (long long probe = 0; probe < nslots; probe++) {
    const ArcSlot s = load_slot(tab + sl);
    if (s.tail == u && s.head == v) return s.arc;
    if (s.tail == kEmptyTail) return -1;
    sl = sl + 1 == nslots ? 0 : sl + 1;
  }
  return -1;
}

}  // namespace dmfd
