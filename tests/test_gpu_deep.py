"""Deep graphs: the barrier-free relabel and push phases, at the sizes where the
ownership of vertices changes (one window of 32 per warp, the edges of a window,
the most windows a grid can own, one vertex more), with long rows among short
ones, for each variant, and batched with instances that a call leaves alone."""
import ctypes

import numpy as np
import pytest

from test_gpu_parity import apply_host, certify

pytestmark = pytest.mark.gpu


def ladder(dmf, n, width, seed, hubs=0):
    """About n/width columns of `width` vertices, neighbours both ways, s before the first column and t after the
    last; `hubs` vertices are joined to every 7th vertex as well (rows far longer than 8 arcs)."""
    rng = np.random.default_rng(seed)
    inner = n - 2
    u = np.arange(inner)
    step = u[u + width < inner]
    up = u[(u + 1 < inner) & ((u + 1) % width != 0)]
    a = np.concatenate([step, step + width, up, up + 1])
    b = np.concatenate([step + width, step, up + 1, up])
    for h in rng.choice(inner, hubs, replace=False):
        far = np.arange(h % 7, inner, 7)
        far = far[far != h]
        a, b = np.concatenate([a, np.full(len(far), h)]), np.concatenate([b, far])
    s, t = inner, inner + 1
    first, last = u[:width], u[-width:]
    a = np.concatenate([a, np.full(len(first), s), last])
    b = np.concatenate([b, first, np.full(len(last), t)])
    return dmf.Graph.from_edges(a, b, rng.integers(1, 50, len(a))), s, t


def solve_and_check(dmf, oracle, g, s, t, sv, batches):
    off, adj, w, par = g.arrays()
    n, cur = g.num_nodes(), w.copy()
    want = oracle.dinic(n, off, adj, cur, par, s, t)
    assert sv.static_maxflow() == want
    certify(oracle, g, sv, s, t, want)
    for b in batches:
        apply_host(g, cur, b)
        want = oracle.dinic(n, off, adj, cur, par, s, t)
        assert sv.apply_updates(*b) == want
        certify(oracle, g, sv, s, t, want)
    # the sink side is what can reach t over arcs the maximum flow left residual: its boundary is a minimum cut
    side = sv.cut()
    tail = np.repeat(np.arange(n), np.diff(off))
    assert side[t] == 1 and side[s] == 0
    assert int(cur[(side[tail] == 0) & (side[adj] == 1)].sum()) == want


@pytest.mark.parametrize("variant", ("data", "topo", "pp"))
@pytest.mark.parametrize("n,width,hubs", [(33, 1, 0), (64, 1, 0), (65, 2, 0), (1000, 3, 0), (4097, 16, 0),
                                          (2000, 20, 3), (9001, 60, 5)])
def test_ladders(dmf, oracle, variant, n, width, hubs):
    g, s, t = ladder(dmf, n, width, n, hubs)
    batches = dmf.gen_batches(g, 3, frac=0.05, p_inc=0.5, p_dec=0.4, p_ins=0.0, delta_hi=30, seed=n)
    with dmf.Solver(g, s, t, variant=variant) as sv:
        solve_and_check(dmf, oracle, g, s, t, sv, batches)


# one block owns at most 4 windows of 32 vertices for each of its 16 warps
@pytest.mark.parametrize("blocks,n", [(1, 512), (1, 513), (1, 2048), (1, 2049), (3, 6144), (3, 6145), (2, 1025)])
def test_window_limits(dmf, oracle, blocks, n):
    g, s, t = ladder(dmf, n, 8, n)
    batches = dmf.gen_batches(g, 2, frac=0.05, p_inc=0.5, p_dec=0.5, p_ins=0.0, delta_hi=30, seed=n)
    with dmf.Solver(g, s, t) as sv:
        o = dmf.Opts()
        dmf._L.dmf_opts_default(ctypes.byref(o))
        o.grid_blocks = blocks
        dmf._check(dmf._L.dmf_solver_set_opts(sv._h, ctypes.byref(o)))
        solve_and_check(dmf, oracle, g, s, t, sv, batches)
        assert sv.stats()["grid_blocks"] == blocks


def test_masked_instances(dmf, oracle):
    made = [ladder(dmf, n, w, n, h) for n, w, h in ((700, 2, 0), (90, 1, 0), (1500, 12, 2), (31, 4, 0))]
    with dmf.MultiSolver([x[0] for x in made], [x[1] for x in made], [x[2] for x in made]) as ms:
        caps = [x[0].arrays()[2] for x in made]

        def want(i):
            off, adj, _, par = made[i][0].arrays()
            return oracle.dinic(made[i][0].num_nodes(), off, adj, caps[i], par, made[i][1], made[i][2])

        assert ms.static_maxflow_all().tolist() == [want(i) for i in range(4)]
        for touched in ((0,), (2, 3), (1, 2), (0, 1, 2, 3)):
            parts = []
            for i in touched:
                (b,) = dmf.gen_batches(made[i][0], 1, frac=0.1, p_inc=0.5, p_dec=0.5, p_ins=0.0, delta_hi=30,
                                       seed=10 * i + len(touched))
                apply_host(made[i][0], caps[i], b)
                parts.append((np.full(len(b[0]), i), *b))
            got = ms.apply_updates_all(*(np.concatenate(x) for x in zip(*parts)))
            assert got.tolist() == [want(i) for i in range(4)]


# a sink joined to every vertex of a grid: at, just above and far above the arcs from which its row gets a level of its
# own at the start of a barrier-free relabel
@pytest.mark.parametrize("variant", ("data", "pp"))
@pytest.mark.parametrize("side", (45, 46, 150))
def test_wide_sink(dmf, oracle, variant, side):
    rng = np.random.default_rng(side)
    v = np.arange(side * side).reshape(side, side)
    right, down = v[:, :-1].ravel(), v[:-1].ravel()
    a = np.concatenate([right, right + 1, down, down + side, np.full(side, v.size), v.ravel()])
    b = np.concatenate([right + 1, right, down + side, down, v[0], np.full(v.size, v.size + 1)])
    w = np.concatenate([rng.integers(20, 60, len(a) - side - v.size), np.full(side, 500), rng.integers(0, 4, v.size)])
    g, s, t = dmf.Graph.from_edges(a, b, w), v.size, v.size + 1
    index = g.arrays()[0]
    assert index[t + 1] - index[t] == v.size
    batches = dmf.gen_batches(g, 3, frac=0.05, p_inc=0.5, p_dec=0.4, p_ins=0.0, delta_hi=30, seed=side)
    with dmf.Solver(g, s, t, variant=variant, trace=True) as sv:
        assert sv.static_maxflow() > 0
        assert "bfs_async" in [x[0] for x in sv.trace()]
        solve_and_check(dmf, oracle, g, s, t, sv, batches)
