// kernel_main.cpp -- the solve kernel on host threads (cuda_host.h).
//   kernel_main solve FILE BLOCKS THREADS SINK_DEG  flow of a solve from scratch, then of the file's batch, each with
//                                                   the number of barrier-free relabels and push phases it had
//                                                   (SINK_DEG: the sink's degree the kernel is told, 0: the true one)
//   kernel_main timeout FILE BLOCKS THREADS BARRIER  the batch with a grid barrier that a block never arrives at:
//                                                   the error word, and what differs in capacities and residuals
//   kernel_main push BLOCKS N                       a push phase past its time limit: does every block stop?
// FILE: int32 n, m, s, t, k, then index[n+1], adj[m], cap[m], par[m], src[k], dst[k], w[k].
#include "cuda_host.h"

#include "dmf_kernel.cuh"

using namespace dmfk;

namespace {

constexpr unsigned long long kSecond = 1000000000ull;

struct Device {
  Params p{};
  HostResult *res = nullptr;
  int *cap = nullptr;

  Device(int n, int m, int s, int t, int k) {
    const size_t N = (size_t)n + 1, M = (size_t)m, K = (size_t)k + 1;
    p.n = n, p.m = m, p.s = s, p.t = t, p.k = k;
    p.capx = emu::global<unsigned long long>(M);
    p.res = emu::global<int>(M);
    p.height = emu::global<int>(N);
    p.stamp = emu::global<int>(N);
    p.excess = emu::global<long long>(N);
    p.dead = emu::global<unsigned char>(N);
    p.side = emu::global<unsigned char>(N);
    for (int i = 0; i < 2; i++) {
      p.fq[i] = emu::global<int>(N);
      p.wq[i] = emu::global<int>(N);
      p.fh[i] = p.wh[i] = p.ah = emu::global<int2>(1);
    }
    p.aq = emu::global<int>(N);
    p.dq = emu::global<int>(N);
    p.dlab = emu::global<int>(N);
    p.pcur = emu::global<int>(N);
    p.lq = emu::global<int>(N);
    p.lst = emu::global<int>(1);
    p.inl = emu::global<unsigned char>(N);
    p.uarc = emu::global<int>(K);
    p.uold = emu::global<int>(K);
    p.nact = n;
    p.nslots = arc_table_slots(m);
    p.atab = emu::global<ArcSlot>((size_t)p.nslots);
    std::memset((void *)p.atab, 0xFF, sizeof(ArcSlot) * (size_t)p.nslots);
    p.nsrc = 1;
    p.hres = res = emu::global<HostResult>(1);
    p.ctrl = emu::global<Ctrl>(1);
    p.ninst = 1;
    p.cycles = 2;
    p.interval = 6;
    p.max_iters = 100000;
    p.hub_deg = INT_MAX;
    p.small_deg = 8;
    p.bu_alpha = 2;
    p.adaptive = 1;
    p.round_base = p.relabel_base = 1;
    p.barrier_ns = 30 * kSecond;
    p.absent_block = -1;
    p.trace_cap = 1 << 14;
    p.trace = emu::global<unsigned long long>(4 * (size_t)p.trace_cap);
  }

  int phases(int kind) const {
    int count = 0;
    for (int i = 0; i < res->c.trace_len; i++) count += (int)(p.trace[4 * i] & 0xff) == kind;
    return count;
  }

  const int *ints(FILE *f, size_t count) {
    int *a = emu::global<int>(count + 1);
    if (fread(a, 4, count, f) != count) std::abort();
    return a;
  }

  void graph(FILE *f) {
    p.off = ints(f, p.n + 1);
    p.adj = ints(f, p.m);
    const int *cap = ints(f, p.m);
    p.par = ints(f, p.m);
    p.sink_deg = p.off[p.t + 1] - p.off[p.t];
    p.usrc = p.xsrc = ints(f, p.k);
    p.udst = p.xdst = ints(f, p.k);
    p.uw = p.xw = ints(f, p.k);
    p.caps_bounded = 1;
    for (int e = 0; e < p.m; e++) {
      p.capx[e] = (unsigned)cap[e];
      if (cap[e] > kMaxUpdateCap) p.caps_bounded = 0;
    }
    for (int u = 0; u < p.n; u++)
      for (int a = p.off[u]; a < p.off[u + 1]; a++) {
        long long sl = arc_slot0(u, p.adj[a], p.nslots);
        while (p.atab[sl].tail != kEmptyTail) sl = sl + 1 == p.nslots ? 0 : sl + 1;
        p.atab[sl] = ArcSlot{u, p.adj[a], a, 0};
      }
  }

  // One launch; the error word, or -1 when a block ended badly.
  int run(int mode, int blocks, int threads) {
    p.mode = mode;
    p.epoch++;
    p.seq++;
    p.keep_dead = mode == MODE_DYNAMIC;
    if (emu::launch(blocks, threads, [&] { k_solve<4, kBlock, 2>(p); })) return -1;
    p.round_base += res->c.rounds_used + 2;
    p.relabel_base += (unsigned)res->c.st_outer + 2;
    return res->c.err;
  }
};

Device load(const char *path) {
  FILE *f = std::fopen(path, "rb");
  int h[5];
  if (!f || fread(h, 4, 5, f) != 5) std::abort();
  Device d(h[0], h[1], h[2], h[3], h[4]);
  d.graph(f);
  std::fclose(f);
  return d;
}

int solve(char **a) {
  Device d = load(a[0]);
  const int blocks = std::atoi(a[1]), threads = std::atoi(a[2]);
  if (std::atoi(a[3])) d.p.sink_deg = std::atoi(a[3]);
  for (int mode : {MODE_STATIC, MODE_DYNAMIC}) {
    const int err = d.run(mode, blocks, threads);
    if (err) return err < 0 ? 3 : 5;
    std::printf("%lld %d %d\n", d.res->c.flow, d.phases(TR_BFS_ASYNC), d.phases(TR_PUSH_ASYNC));
  }
  return 0;
}

int timeout(char **a) {
  Device d = load(a[0]);
  const int blocks = std::atoi(a[1]), threads = std::atoi(a[2]);
  if (d.run(MODE_STATIC, blocks, threads)) return 3;
  std::vector<unsigned> cap(d.p.m);
  for (int e = 0; e < d.p.m; e++) cap[e] = (unsigned)d.p.capx[e];
  const std::vector<int> res(d.p.res, d.p.res + d.p.m);
  emu::skip_barrier = std::atoi(a[3]);
  d.p.barrier_ns = kSecond / 5;
  const int err = d.run(MODE_DYNAMIC, blocks, threads);
  int diff = 0;
  for (int e = 0; e < d.p.m; e++) diff += cap[e] != (unsigned)d.p.capx[e] || res[e] != d.p.res[e];
  std::printf("%d %d\n", err, diff);
  return 0;
}

// Two neighbours in the last block's vertices hand one unit to and fro until their labels reach n; every other block
// is idle and counted so, as after a wave that crossed blocks late.  The clock passes the limit in a few looks.
int push(char **a) {
  const int blocks = std::atoi(a[0]), n = std::atoi(a[1]);
  Device d(n, 2, 0, 1, 0);
  int *off = emu::global<int>(n + 1), *adj = emu::global<int>(2), *par = emu::global<int>(2);
  const int u = n - 2, v = n - 1;
  for (int i = 0; i <= n; i++) off[i] = i <= u ? 0 : i == v ? 1 : 2;
  adj[0] = v, adj[1] = u, par[0] = 1, par[1] = 0;
  d.p.off = off, d.p.adj = adj, d.p.par = par;
  d.p.res[0] = d.p.res[1] = 1;
  d.p.excess[u] = 1;
  d.p.cycles = 1;
  d.p.ctrl->aidle[1] = blocks - 1;
  emu::fake_tick = 1000000;
  const int rc = emu::launch(blocks, 32, [&] {
    static AsyncShared ash;
    LStats ls;
    acc_init();
    ph_async_push(d.p, ash, 2 * emu::fake_tick, ls);
  });
  if (rc) return rc;
  std::printf("%d\n", std::max(d.p.height[u], d.p.height[v]));
  return 0;
}

}  // namespace

int main(int argc, char **argv) {
  if (argc == 6 && !std::strcmp(argv[1], "solve")) return solve(argv + 2);
  if (argc == 6 && !std::strcmp(argv[1], "timeout")) return timeout(argv + 2);
  if (argc == 4 && !std::strcmp(argv[1], "push")) return push(argv + 2);
  return 2;
}
