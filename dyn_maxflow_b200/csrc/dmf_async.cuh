// dmf_async.cuh -- barrier-free relabel and push phases for deep graphs, part
// of the solve kernel (included by dmf_kernel.cuh inside namespace dmfk).
//
// A grid-like graph of diameter D costs the level-synchronous phases about D
// grid barriers per global relabel and as many per run of push rounds, each
// with a few hundred vertices of work: 8.1 us a BFS level and 13 us a push
// round on the 256 x 256 grid, nearly all of it barrier and dependent loads.
// Here every vertex belongs to one lane for the whole phase (a warp owns
// windows of 32 consecutive vertices), the lane polls the vertex's word in L2
// and acts when it changes, and the grid meets at a barrier only when the phase
// ends.  A hop then costs one poll and one fire-and-forget atomic: 0.7 us a BFS
// level, about 0.3 of it L2 and the rest instructions.  256 x 256 grid, one B200:
// static solve 145 -> 16 ms, 1% batch 105 -> 10.6 ms.
#pragma once

// BFS levels after which a global relabel (and then the rest of the solve)
// goes over to the barrier-free phases.  R-MAT graphs end within 10 levels:
// there a level is real work and the worklists save polling every vertex.  A
// graph that needs 16 levels (9 us each) will need hundreds of short phases.
constexpr int kDeepLevels = 16;
// Levels after which the partial revival of a batch gives up on such a graph.
constexpr int kReviveLevels = 8;
// Windows of 32 vertices per warp at most: bounds the vertices a graph may
// have (kAsyncWin * 32 * resident warps) and the per-vertex shared memory.
constexpr int kAsyncWin = 4;
// Polls without work after which a warp counts as idle: longer than an atomic
// takes to become visible, so that a wave crossing from one block to another
// does not find every block idle.
constexpr int kQuietPolls = 8;
// A sink's row longer than this is relaxed by a level-synchronous level at the
// start of every relabel, over the whole grid, before the barrier-free phase: one
// warp takes about 1 ms for 65,536 arcs (from the totals below; the push phase gets
// as long again), the seeds with their frontier and the level tens of us for any
// length.  Segmentation graphs (every vertex of a grid joined to s and t), static
// solve with the level / without / barriers throughout:
// 1,024 arcs 0.96 / 0.98 / 1.9 ms, 2,304 arcs 0.65 / 0.75 / 1.5, 65,536 arcs 1.05 /
// 6.6 / 3.4, 262,144 arcs 3.0 / 16 / 7.2.  Other long rows stay with one warp: a
// hub of 100,000 arcs on a ladder, 43 ms against 220 with barriers throughout.
constexpr int kWideSink = 2048;
// Polls of a block's first warp in a phase at most (bounds the loop, whatever
// the polls find; a phase is far shorter).
constexpr int kMaxPolls = 1 << 20;

struct AsyncShared {
  int scan[kAsyncWin * kBlock];  // label the vertex's arcs were last relaxed from
  int idle_warps;
  int stop;
};

// The windows of a warp: block b owns `per` consecutive windows, warp i of it
// windows i, i + warps, ...
struct AsyncOwn {
  int first, count;  // this warp's first vertex and its windows
  int step;          // vertices from one window of the warp to the next
};

__device__ __forceinline__ AsyncOwn async_own(int n) {
  const int nw = blockDim.x >> 5, wid = threadIdx.x >> 5;
  const int nwin = (n + 31) >> 5, per = (nwin + (int)gridDim.x - 1) / (int)gridDim.x;
  const int lo = blockIdx.x * per + wid, hi = min(nwin, (int)(blockIdx.x + 1) * per);
  AsyncOwn o;
  o.first = lo * 32;
  o.step = nw * 32;
  o.count = lo < hi ? (hi - lo + nw - 1) / nw : 0;
  return o;
}

// Whether the grid's warps can own every vertex.
__device__ __forceinline__ bool async_fits(int n) {
  const int nwin = (n + 31) >> 5, per = (nwin + (int)gridDim.x - 1) / (int)gridDim.x;
  return per <= kAsyncWin * (int)(blockDim.x >> 5);
}

// Quiescence: a warp is idle after kQuietPolls polls without work, a block when
// all its warps are, and the phase ends once every block is idle (or a limit of
// async_look is reached).  This may end a phase too early (work in flight to an
// idle block); the relabel checks its labels after a barrier, and a push phase
// may end at any time.
struct AsyncIdle {
  int quiet = 0;
  bool idle = false;
};

__device__ __forceinline__ void async_begin(AsyncShared &sh) {
  if (threadIdx.x == 0) {
    sh.idle_warps = 0;
    sh.stop = 0;
  }
  __syncthreads();
}

// The block's look at the limits of the phase, every 8th poll whatever the polls
// find: a warp that finds work at every other poll (excess that goes to and fro
// between two windows until its labels reach n) would else never look.  Every
// block looks for itself: the block that set the deadline may have left already.
__device__ __forceinline__ void async_look(const Params &p, AsyncShared &sh, int poll, bool timed) {
  if (threadIdx.x != 0 || (poll & 7) != 7) return;
  const unsigned long long end = timed ? ld_rlx(&p.ctrl->adeadline) : 0;
  if (ld_rlx(&p.ctrl->err) || poll >= kMaxPolls || (end && globaltimer() > end)) *(volatile int *)&sh.stop = 1;
}

// A warp that found work; called before it does it, so that a long piece of work
// does not look like quiet.
__device__ __forceinline__ void async_wake(AsyncShared &sh, AsyncIdle &st, int *idle_blocks) {
  st.quiet = 0;
  if (st.idle) {
    st.idle = false;
    if ((threadIdx.x & 31) == 0 && atomicSub(&sh.idle_warps, 1) == (int)(blockDim.x >> 5)) atomicSub(idle_blocks, 1);
  }
}
// Whether the warp leaves the phase.  Every lane calls it, and the answer is the
// warp's: another warp (or thread 0 of this one, just before) may set the word
// between two lanes' reads, and a lane that left by itself would wait at
// async_end's block barrier for lanes that wait for it in the next poll's vote.
__device__ __forceinline__ bool async_stopped(const AsyncShared &sh) {
  return __any_sync(0xffffffffu, *(const volatile int *)&sh.stop != 0);
}

// Every warp has left: a block that stopped while one of its warps had just woken
// is counted as idle again, or the others would wait for it.
__device__ __forceinline__ void async_end(AsyncShared &sh, int *idle_blocks) {
  __syncthreads();
  if (threadIdx.x == 0 && sh.idle_warps < (int)(blockDim.x >> 5)) atomicAdd(idle_blocks, 1);
}

// A warp whose last poll found nothing; true: leave the phase.  The block's
// first warp looks at the number of idle blocks.  The SM's warps share its issue
// slots, so a poll is kept short and a warp without vertices sleeps.
__device__ __forceinline__ bool async_quiet(AsyncShared &sh, AsyncIdle &st, bool owner, int *idle_blocks) {
  if (++st.quiet < kQuietPolls && owner) return false;
  if (!st.idle) {
    st.idle = true;
    if ((threadIdx.x & 31) == 0 && atomicAdd(&sh.idle_warps, 1) == (int)(blockDim.x >> 5) - 1)
      atomicAdd(idle_blocks, 1);
  }
  if (threadIdx.x == 0 && (st.quiet & 3) == 0 && ld_rlx(idle_blocks) >= (int)gridDim.x)
    *(volatile int *)&sh.stop = 1;
  if (!owner) __nanosleep(200);
  return async_stopped(sh);
}

// Global relabel from the labels a level-synchronous BFS left after its level
// L0 (seeds only: L0 = 0): label-correcting, every vertex relaxes the tails of
// its residual in-arcs with an atomic minimum whenever its own label fell.
// Labels only fall and every fall is seen by its owner, so once no vertex has a
// label below the one it last relaxed from (ph_async_settled, between two
// barriers) the labels are the exact distances.

// Relaxes the tails of a long row's residual in-arcs, by a whole warp, kRelaxBatch
// arcs a lane with their loads in flight together.  No other warp helps with the
// row, so everything behind it waits: static solve of a 256 x 256 segmentation
// graph, its sink's row of 65,536 arcs taken this way, 8.4 ms with one arc a lane,
// 6.3 with 4, 6.3 with 8.
constexpr int kRelaxBatch = 4;

__device__ __forceinline__ void async_relax_row(const Params &p, int v, int h, LStats &ls) {
  const int b = __ldg(p.off + v), e = __ldg(p.off + v + 1);
  for (int a0 = b + (int)(threadIdx.x & 31); a0 < e; a0 += 32 * kRelaxBatch) {
    int w[kRelaxBatch], r[kRelaxBatch];
#pragma unroll
    for (int k = 0; k < kRelaxBatch; k++) {
      const int a = a0 + 32 * k;
      w[k] = a < e ? __ldg(p.adj + a) : -1;
      r[k] = a < e ? __ldg(p.par + a) : 0;
    }
#pragma unroll
    for (int k = 0; k < kRelaxBatch; k++) {
      if (w[k] < 0) continue;
      ls.barcs++;
      const int cur = __ldcg(p.height + w[k]);
      r[k] = __ldcg(p.res + r[k]);
      if (cur <= h + 1 || cur == p.n) r[k] = 0;
    }
#pragma unroll
    for (int k = 0; k < kRelaxBatch; k++)
      if (w[k] >= 0 && r[k] > 0) atomicMin(p.height + w[k], h + 1);
  }
  __syncwarp();
}

// One window per warp: the heads that can be labelled over the vertex's arcs sit
// in registers, so a hop is a poll, a vote and the atomics.
__device__ __forceinline__ void async_bfs_one(const Params &p, AsyncShared &sh, const AsyncOwn &own, int L0, bool first,
                                              LStats &ls) {
  Ctrl *c = p.ctrl;
  const int lane = threadIdx.x & 31, v = own.first + lane;
  const bool mine = own.count > 0 && v < p.n;
  int scan = INT_MIN, beg = 0, deg = 0, nh = 0;
  int hd[kSmallMax];
#pragma unroll
  for (int k = 0; k < kSmallMax; k++) hd[k] = 0;
  if (mine) {
    const int h = __ldcg(p.height + v);
    scan = first ? h : sh.scan[threadIdx.x];
    if (h != p.n && inst_on(p, v)) {  // neither a source nor dead
      // the frontier, and what a warp that began earlier has labelled already
      if (first && h >= L0) scan = UNV;
      beg = __ldg(p.off + v);
      deg = __ldg(p.off + v + 1) - beg;
      if (deg <= kSmallMax) {
        int w[kSmallMax];
        bool ok[kSmallMax];
#pragma unroll
        for (int k = 0; k < kSmallMax; k++) {
          ok[k] = false;
          w[k] = 0;
          if (k >= deg) continue;
          w[k] = __ldg(p.adj + beg + k);
          ok[k] = __ldcg(p.res + __ldg(p.par + beg + k)) > 0 && __ldcg(p.height + w[k]) != p.n;
        }
#pragma unroll
        for (int k = 0; k < kSmallMax; k++) {
          if (!ok[k]) continue;
#pragma unroll
          for (int j = 0; j < kSmallMax; j++)
            if (j == nh) hd[j] = w[k];
          nh++;
        }
      }
    }
  }
  const bool wide = deg > kSmallMax;
  const bool any_wide = __any_sync(0xffffffffu, wide), many = __any_sync(0xffffffffu, nh > 4);
  AsyncIdle st;
  for (int poll = 0;; poll++) {
    const int h = mine ? ld_rlx(p.height + v) : INT_MAX;
    const bool need = h < scan;
    async_look(p, sh, poll, false);
    if (!__any_sync(0xffffffffu, need)) {
      if (async_quiet(sh, st, own.count > 0, &c->aidle[0])) break;
      continue;
    }
    async_wake(sh, st, &c->aidle[0]);
    if (need) {
      scan = h;
#pragma unroll
      for (int k = 0; k < 4; k++)
        if (k < nh) atomicMin(p.height + hd[k], h + 1);
      if (many) {
#pragma unroll
        for (int k = 4; k < kSmallMax; k++)
          if (k < nh) atomicMin(p.height + hd[k], h + 1);
      }
      ls.barcs += (unsigned)nh;
    }
    if (any_wide) {
      unsigned todo = __ballot_sync(0xffffffffu, need && wide);
      while (todo) {  // longer rows by the whole warp
        const int src = __ffs(todo) - 1;
        todo &= todo - 1;
        async_relax_row(p, own.first + src, __shfl_sync(0xffffffffu, h, src), ls);
      }
    }
    if (async_stopped(sh)) break;
  }
  sh.scan[threadIdx.x] = scan;
}

template <int W>
__device__ __forceinline__ void async_bfs_loop(const Params &p, AsyncShared &sh, const AsyncOwn &own, int L0, bool first,
                                               LStats &ls) {
  Ctrl *c = p.ctrl;
  const int lane = threadIdx.x & 31;
  int scan[W], beg[W];
  unsigned mask[W];  // arcs (of degree <= 8) whose head can be labelled over them, and the degree << 8
#pragma unroll
  for (int j = 0; j < W; j++) {
    const int v = own.first + j * own.step + lane;
    scan[j] = INT_MIN;
    beg[j] = 0;
    mask[j] = 0;
    if (j < own.count && v < p.n) {
      const int h = __ldcg(p.height + v);
      scan[j] = first ? h : sh.scan[j * kBlock + (int)threadIdx.x];
      if (h != p.n && inst_on(p, v)) {        // neither a source nor dead
        // the frontier, and what a warp that began earlier has labelled already
        if (first && h >= L0) scan[j] = UNV;
        beg[j] = __ldg(p.off + v);
        const int deg = __ldg(p.off + v + 1) - beg[j];
        mask[j] = (unsigned)min(deg, 255) << 8;
        if (deg <= kSmallMax) {
#pragma unroll
          for (int k = 0; k < kSmallMax; k++)
            if (k < deg && __ldcg(p.res + __ldg(p.par + beg[j] + k)) > 0 &&
                __ldcg(p.height + __ldg(p.adj + beg[j] + k)) != p.n)
              mask[j] |= 1u << k;
        }
      }
    }
  }
  AsyncIdle st;
  for (int poll = 0;; poll++) {
    int h[W];
#pragma unroll
    for (int j = 0; j < W; j++) {
      const int v = own.first + j * own.step + lane;
      h[j] = j < own.count && v < p.n ? ld_rlx(p.height + v) : INT_MAX;
    }
    bool need_any = false;
#pragma unroll
    for (int j = 0; j < W; j++) need_any |= h[j] < scan[j];
    async_look(p, sh, poll, false);
    if (!__any_sync(0xffffffffu, need_any)) {
      if (async_quiet(sh, st, own.count > 0, &c->aidle[0])) break;
      continue;
    }
    async_wake(sh, st, &c->aidle[0]);
#pragma unroll
    for (int j = 0; j < W; j++) {
      const bool need = h[j] < scan[j];
      const unsigned deg = mask[j] >> 8;
      if (need) {
        scan[j] = h[j];
        if (deg <= kSmallMax) {
#pragma unroll
          for (int k = 0; k < kSmallMax; k++)
            if ((mask[j] >> k) & 1) atomicMin(p.height + __ldg(p.adj + beg[j] + k), h[j] + 1);
          ls.barcs += deg;
        }
      }
      unsigned wide = __ballot_sync(0xffffffffu, need && deg > kSmallMax);
      while (wide) {  // longer rows by the whole warp
        const int src = __ffs(wide) - 1;
        wide &= wide - 1;
        async_relax_row(p, own.first + j * own.step + src, __shfl_sync(0xffffffffu, h[j], src), ls);
      }
    }
    if (async_stopped(sh)) break;
  }
#pragma unroll
  for (int j = 0; j < W; j++) sh.scan[j * kBlock + (int)threadIdx.x] = scan[j];
}

__device__ __forceinline__ void ph_async_bfs(const Params &p, AsyncShared &sh, int L0, bool first, LStats &ls) {
  Ctrl *c = p.ctrl;
  const AsyncOwn own = async_own(p.n);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    c->aidle[1] = 0;  // the push phase's words
    c->adeadline = 0;
    c->aunsettled = 0;
    c->aact = 0;
    c->adepth = 0;
  }
  async_begin(sh);
  if (own.count <= 1) async_bfs_one(p, sh, own, L0, first, ls);
  else async_bfs_loop<kAsyncWin>(p, sh, own, L0, first, ls);
  async_end(sh, &c->aidle[0]);
}

// The seeds of a relabel of a deep solve: labels only (the frontier and active
// lists of ph_bfs_init are not used there; 3.5 us instead of 17 at 65,536
// vertices).
__device__ __forceinline__ void ph_deep_init(const Params &p) {
  const int nt = gridDim.x * blockDim.x;
  int pos = 0;
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < p.n; v += nt) {
    const bool is_dead = __ldcg(p.dead + v) != 0;
    const long long ex = __ldcg(p.excess + v);
    if (is_dead || !inst_on(p, v)) continue;
    const bool src = is_src(p, v), snk = is_snk(p, v);
    p.height[v] = src ? p.n : (snk || ex < 0) ? 0 : UNV;
    if (!src && !snk && ex > 0) pos++;
  }
  block_add_int(0, &p.ctrl->pos_count, pos);
}

// After a barrier: counts the vertices whose label fell since they last relaxed
// their arcs (0: the labels are exact).
__device__ __forceinline__ void ph_async_settled(const Params &p, AsyncShared &sh) {
  const AsyncOwn own = async_own(p.n);
  const int lane = threadIdx.x & 31;
  if (blockIdx.x == 0 && threadIdx.x == 0) p.ctrl->aidle[0] = 0;
  bool open = false;
  for (int j = 0; j < own.count; j++) {
    const int v = own.first + j * own.step + lane;
    if (v < p.n) open |= __ldcg(p.height + v) < sh.scan[j * kBlock + (int)threadIdx.x];
  }
  if (__syncthreads_or(open) && threadIdx.x == 0) atomicAdd(&p.ctrl->aunsettled, 1);
}

// ph_bfs_finalize of a complete relabel, which also counts the active vertices
// and finds the greatest distance.
__device__ __forceinline__ void ph_async_finalize(const Params &p, bool write_side, bool listed) {
  int nd = 0, act = 0, depth = 0;
  for_live<4>(p, listed, [&](int v) {
    const int h = __ldcg(p.height + v);
    if (h == UNV) {
      p.dead[v] = 1;
      p.height[v] = p.n;
      nd++;
    } else if (h < p.n) {
      depth = max(depth, h);
      if (__ldcg(p.excess + v) > 0 && !is_term(p, v)) act++;
    }
    if (write_side) p.side[v] = h < p.n ? 1 : 0;
  });
  block_add_ll(0, (long long *)&p.ctrl->st_dead, nd);
  block_add_int(1, &p.ctrl->aact, act);
  depth = __reduce_max_sync(0xffffffffu, depth);
  if ((threadIdx.x & 31) == 0 && depth > 0) atomicMax(&p.ctrl->adepth, depth);
}

// Push phase without rounds: every lane polls its vertices' excess and
// discharges the active ones (the push / relabel rule of discharge()); a vertex
// of more than 8 arcs is discharged by its whole warp.  As in the rounds, a
// vertex is only ever discharged by one thread or warp at a time, only its own
// discharges lower its residuals and excess, and heights only rise, so the
// races are those of the rounds.  Ends when no vertex is active, or budget_ns
// after its start (a deadline that the grid's first thread sets and every block
// keeps): the next relabel then gives exact distances again.
// One window per warp, every narrow vertex of it with at most D arcs: heads,
// partners and the label (only the owner changes it) sit in registers, and a
// discharge is one round of loads, up to `cycles` pushes and relabels on what
// they gave, and the atomics.
template <int D>
__device__ __forceinline__ void async_push_one(const Params &p, AsyncShared &sh, const AsyncOwn &own, bool live,
                                               LStats &ls) {
  Ctrl *c = p.ctrl;
  const int lane = threadIdx.x & 31, v = own.first + lane;
  int beg = 0, deg = 0, h = p.n;
  int hd[D], pa[D];
  if (live) {
    beg = __ldg(p.off + v);
    deg = __ldg(p.off + v + 1) - beg;
    h = __ldcg(p.height + v);
  }
  const bool wide = deg > kSmallMax;
#pragma unroll
  for (int k = 0; k < D; k++) {
    hd[k] = !wide && k < deg ? __ldg(p.adj + beg + k) : 0;
    pa[k] = !wide && k < deg ? __ldg(p.par + beg + k) : 0;
  }
  const bool any_wide = __any_sync(0xffffffffu, wide);
  TileGroup<32> wg;
  AsyncIdle st;
  for (int poll = 0;; poll++) {
    const long long ex = live ? ld_rlx(p.excess + v) : 0;
    const bool act = ex > 0 && h < p.n;
    async_look(p, sh, poll, true);
    if (!__any_sync(0xffffffffu, act)) {
      if (async_quiet(sh, st, own.count > 0, &c->aidle[1])) break;
      continue;
    }
    async_wake(sh, st, &c->aidle[1]);
    if (act && !wide) {
      int rr[D], hw[D], dd[D];
#pragma unroll
      for (int k = 0; k < D; k++) {
        rr[k] = k < deg ? __ldcg(p.res + beg + k) : 0;
        hw[k] = k < deg ? __ldcg(p.height + hd[k]) : INT_MAX;
        dd[k] = 0;
      }
      ls.visits++;
      ls.arcs += (unsigned)deg;
      long long left = ex;
      const int h0 = h;
      for (int cyc = 0; cyc < p.cycles && left > 0 && h < p.n; cyc++) {
#pragma unroll
        for (int k = 0; k < D; k++) {
          if (rr[k] > 0 && hw[k] < h) {
            const int d = (int)(rr[k] < left ? rr[k] : left);
            dd[k] += d;
            rr[k] -= d;
            left -= d;
          }
        }
        if (left > 0) {  // every admissible arc is saturated: relabel
          int mh = INT_MAX;
#pragma unroll
          for (int k = 0; k < D; k++)
            if (rr[k] > 0) mh = min(mh, hw[k]);
          h = mh >= p.n ? p.n : mh + 1;
          ls.relabels++;
        }
      }
#pragma unroll
      for (int k = 0; k < D; k++) {
        if (dd[k] > 0) {
          atomicSub(p.res + beg + k, dd[k]);
          push_excess(p, hd[k], dd[k], ls);
          atomicAdd(p.res + pa[k], dd[k]);
          ls.pushes++;
        }
      }
      if (h != h0) *(volatile int *)(p.height + v) = h;
      if (left != ex) atomic_add_ll(p.excess + v, left - ex);
    }
    if (any_wide) {
      unsigned todo = __ballot_sync(0xffffffffu, act && wide);
      while (todo) {
        const int src = __ffs(todo) - 1;
        todo &= todo - 1;
        discharge(wg, p, own.first + src, 0, false, ls, nullptr);
        __syncwarp();
        if (lane == src) h = __ldcg(p.height + v);
      }
    }
    if (async_stopped(sh)) break;
  }
}

// The same for a warp of several windows.
__device__ __forceinline__ void async_push_loop(const Params &p, AsyncShared &sh, const AsyncOwn &own, unsigned live,
                                                LStats &ls) {
  Ctrl *c = p.ctrl;
  const int lane = threadIdx.x & 31;
  TileGroup<32> wg;
  AsyncIdle st;
  for (int poll = 0;; poll++) {
    unsigned have = 0;  // windows in which this lane's vertex holds excess
    long long ex[kAsyncWin];
#pragma unroll
    for (int j = 0; j < kAsyncWin; j++)
      ex[j] = (live >> j) & 1 ? ld_rlx(p.excess + own.first + j * own.step + lane) : 0;
#pragma unroll
    for (int j = 0; j < kAsyncWin; j++)
      if (ex[j] > 0) have |= 1u << j;
    bool any = false;
    if (__any_sync(0xffffffffu, have)) {
#pragma unroll 1
      for (int j = 0; j < own.count; j++) {
        if (!__any_sync(0xffffffffu, (have >> j) & 1)) continue;
        const int v = own.first + j * own.step + lane;
        long long x = 0;
        int h = p.n, beg = 0, deg = 0;
        if ((have >> j) & 1) {
          x = __ldcg(p.excess + v);
          h = __ldcg(p.height + v);
          beg = __ldg(p.off + v);
          deg = __ldg(p.off + v + 1) - beg;
        }
        const bool act = x > 0 && h < p.n;
        if (__any_sync(0xffffffffu, act)) async_wake(sh, st, &c->aidle[1]);
        any |= act;
        if (act && deg <= kSmallMax) {
          ls.visits++;
          discharge_small(p, v, beg, deg, x, h, 0, false, ls);
        }
        unsigned wide = __ballot_sync(0xffffffffu, act && deg > kSmallMax);
        while (wide) {
          const int src = __ffs(wide) - 1;
          wide &= wide - 1;
          discharge(wg, p, __shfl_sync(0xffffffffu, v, src), 0, false, ls, nullptr);
          __syncwarp();
        }
      }
      any = __any_sync(0xffffffffu, any);
    }
    async_look(p, sh, poll, true);
    if (any) {
      if (async_stopped(sh)) break;
    } else if (async_quiet(sh, st, own.count > 0, &c->aidle[1])) {
      break;
    }
  }
}

__device__ __forceinline__ void ph_async_push(const Params &p, AsyncShared &sh, unsigned long long budget_ns,
                                              LStats &ls) {
  Ctrl *c = p.ctrl;
  const AsyncOwn own = async_own(p.n);
  const int lane = threadIdx.x & 31;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    *(volatile unsigned long long *)&c->adeadline = globaltimer() + budget_ns;
    c->pos_count = 0;
    c->unexplored = 0;
  }
  async_begin(sh);
  // a dead vertex's parked excess is not polled
  unsigned live = 0;
  for (int j = 0; j < own.count; j++) {
    const int v = own.first + j * own.step + lane;
    if (v < p.n && !__ldcg(p.dead + v) && !is_term(p, v) && inst_on(p, v)) live |= 1u << j;
  }
  // The warps of a block may own different numbers of windows: they part here and
  // meet again before the block barrier.
  if (own.count <= 1) {
    const int v = own.first + lane;
    const int deg = live & 1 ? deg_of(p, v) : 0;
    if (__any_sync(0xffffffffu, deg > 4 && deg <= kSmallMax))
      async_push_one<kSmallMax>(p, sh, own, live & 1, ls);
    else
      async_push_one<4>(p, sh, own, live & 1, ls);
  } else {
    async_push_loop(p, sh, own, live, ls);
  }
  async_end(sh, &c->aidle[1]);
  sink_flush(p, ls);
}
