"""The one-pass lookup and claim of a batch, and the phases it lets a batch skip: rejected batches leave no trace
(with and without the bound on capacities that allows the one pass), source arcs are the only ones a batch has to
saturate, both arcs of a pair in one batch, the live list over batches that kill and revive vertices, the ways to sweep
it, and the sizes at which the staging of a host batch changes."""
import ctypes

import numpy as np
import pytest

from test_gpu_parity import apply_host, certify

pytestmark = pytest.mark.gpu


def rmat(dmf, scale, big=False):
    g, s, t = dmf.gen_rmat(scale, 8 << scale, seed=scale, cap_lo=1, cap_hi=1000)
    if big:  # one arc above 2^30 - 1: the claim waits for a barrier of its own
        index, adj, w, par = g.arrays()
        a = int(np.flatnonzero((w > 0) & (w[par] == 0))[0])
        w[a] = 2**30 + 5
        g = dmf.Graph.from_csr(index, adj, w, par)
    return g, s, t


def arcs_of(g, pick):
    index, adj, _, _ = g.arrays()
    return (np.searchsorted(index, pick, side="right") - 1).astype(np.int32), adj[pick]


# 1, one warp, the threads of a full grid and one more, and a few per thread of it
@pytest.mark.parametrize("big", (False, True))
@pytest.mark.parametrize("scale,k", [(8, 1), (8, 33), (12, 3000), (16, 151552), (16, 151553), (16, 400001)])
def test_rejected_batch_leaves_no_trace(dmf, oracle, scale, k, big):
    g, s, t = rmat(dmf, scale, big)
    index, adj, w, par = g.arrays()
    rng = np.random.default_rng(k)
    pick = rng.permutation(len(adj))[:k]
    src, dst = arcs_of(g, pick)
    to = rng.integers(0, 2000, len(pick)).astype(np.int32)
    with dmf.Solver(g, s, t) as sv:
        flow = sv.static_maxflow()
        before = sv.state()
        bad = []
        for at in sorted({0, len(src) // 2, len(src) - 1}):
            x = dst.copy()  # a head that is no neighbour of the tail
            near = set(adj[index[src[at]]:index[src[at] + 1]].tolist()) | {int(src[at])}
            x[at] = next(v for v in range(g.num_nodes()) if v not in near)
            bad.append((src, x, to))
            x = to.copy()
            x[at] = -1
            bad.append((src, dst, x))
        bad.append((np.append(src, src[:1]), np.append(dst, dst[:1]), np.append(to, np.int32(7))))
        for b in bad:
            with pytest.raises(dmf.DmfError):
                sv.apply_updates(*b)
            after = sv.state()
            assert all(np.array_equal(x, y) for x, y in zip(before[:3], after[:3]))
        assert sv.flow == flow
        cur = w.copy()
        cur[pick] = to
        want = oracle.dinic(g.num_nodes(), index, adj, cur, par, s, t)
        assert sv.apply_updates(src, dst, to) == want
        certify(oracle, g, sv, s, t, want)


@pytest.mark.parametrize("variant", ("data", "topo", "pp"))
def test_source_arcs_and_pairs(dmf, oracle, variant):
    g, s, t = rmat(dmf, 10)
    index, adj, w, par = g.arrays()
    rng = np.random.default_rng(3)
    cur = w.copy()
    out = np.arange(index[s], index[s + 1])
    pairs = rng.permutation(len(adj))[:300]
    pairs = np.unique(np.concatenate([pairs, par[pairs]]))
    with dmf.Solver(g, s, t, variant=variant) as sv:
        sv.static_maxflow()
        for pick, hi in ((out, 3000), (out[::3], 1), (par[out], 50), (pairs, 2000), (pairs, 5), (out, 1000)):
            src, dst = arcs_of(g, pick)
            to = rng.integers(0, hi, len(pick)).astype(np.int32)
            apply_host(g, cur, (src, dst, to))
            want = oracle.dinic(g.num_nodes(), index, adj, cur, par, s, t)
            assert sv.apply_updates(src, dst, to) == want
            certify(oracle, g, sv, s, t, want)


@pytest.mark.parametrize("scale,frac", [(9, 0.3), (13, 0.2), (13, 0.002)])
def test_live_list_over_a_stream(dmf, oracle, scale, frac):
    g, s, t = rmat(dmf, scale)
    index, adj, w, par = g.arrays()
    cur = w.copy()
    stream = dmf.gen_batches(g, 12, frac=frac, p_inc=0.3, p_dec=0.3, p_ins=0.1, seed=scale)
    with dmf.Solver(g, s, t) as sv, dmf.Solver(g, s, t) as copy:
        sv.static_maxflow()
        for i, b in enumerate(stream):
            apply_host(g, cur, b)
            want = oracle.dinic(g.num_nodes(), index, adj, cur, par, s, t)
            copy.copy_state_from(sv)
            assert sv.apply_updates(*b) == want
            assert copy.apply_updates_action(i % 4, *b) == want
            certify(oracle, g, sv, s, t, want)
            certify(oracle, g, copy, s, t, want)
            if i % 5 == 4:  # the cut readout revives and rebuilds
                side = sv.cut()
                tail = np.repeat(np.arange(g.num_nodes()), np.diff(index))
                assert int(cur[(side[tail] == 0) & (side[adj] == 1)].sum()) == want


# up to 8 vertices a thread are walked plainly, beyond that in windows of 512 (8192 vertices on 1 block of 512 threads)
@pytest.mark.parametrize("blocks,scale", [(1, 12), (1, 13), (2, 13), (3, 14)])
def test_sweeps_on_few_blocks(dmf, oracle, blocks, scale):
    g, s, t = rmat(dmf, scale)
    index, adj, w, par = g.arrays()
    cur = w.copy()
    with dmf.Solver(g, s, t) as sv:
        o = dmf.Opts()
        dmf._L.dmf_opts_default(ctypes.byref(o))
        o.grid_blocks = blocks
        dmf._check(dmf._L.dmf_solver_set_opts(sv._h, ctypes.byref(o)))
        assert sv.static_maxflow() == oracle.dinic(g.num_nodes(), index, adj, cur, par, s, t)
        for i, b in enumerate(dmf.gen_batches(g, 4, frac=0.1, p_inc=0.3, p_dec=0.3, p_ins=0.1, seed=blocks)):
            apply_host(g, cur, b)
            want = oracle.dinic(g.num_nodes(), index, adj, cur, par, s, t)
            assert sv.apply_updates(*b) == want
            certify(oracle, g, sv, s, t, want)
            side = sv.cut()
            tail = np.repeat(np.arange(g.num_nodes()), np.diff(index))
            assert int(cur[(side[tail] == 0) & (side[adj] == 1)].sum()) == want


# where the staging of a host batch changes: copied by one thread, by several, sent to the device in pieces
@pytest.mark.parametrize("k", [16384, 16385, 262144, 262145])
def test_staging_sizes(dmf, k):
    torch = pytest.importorskip("torch")
    g, s, t = rmat(dmf, 16)
    rng = np.random.default_rng(k)
    pick = rng.permutation(g.num_edges())[:k]
    src, dst = arcs_of(g, pick)
    to = rng.integers(0, 2000, k).astype(np.int32)
    with dmf.Solver(g, s, t) as sv, dmf.Solver(g, s, t) as other:
        sv.static_maxflow()
        d = [torch.from_numpy(x).cuda() for x in (src, dst, to)]
        assert sv.apply_updates(src, dst, to) == other.recompute_device(*(x.data_ptr() for x in d), k)
        assert np.array_equal(sv.state()[0], other.state()[0])


def test_staging_of_a_new_solver_is_bounded(dmf):
    """Staging is not in the footprint that the server admits by: 2^20 updates of five words, whatever the graph."""
    torch = pytest.importorskip("torch")
    g, s, t = dmf.gen_rmat(21, 18 << 21, seed=21, cap_lo=1, cap_hi=1000)
    index, adj, w, _ = g.arrays()
    assert len(adj) // 32 > (1 << 20) + (1 << 19)
    pick = np.random.default_rng(21).permutation(len(adj))[:(1 << 20) + (1 << 19)]
    src, dst = arcs_of(g, pick)
    x = [torch.from_numpy(a).cuda() for a in (src, dst, w[pick])]  # sets what is there already

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    with dmf.Solver(g, s, t) as sv:
        flow = sv.static_maxflow()
        made = free()
        assert sv.apply_updates_device(*(a.data_ptr() for a in x), 1 << 20) == flow
        assert free() == made
        assert sv.apply_updates_device(*(a.data_ptr() for a in x), len(pick)) == flow
        assert 8 << 20 <= made - free() <= 16 << 20  # 30 MiB in the place of 20
