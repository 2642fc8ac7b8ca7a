"""The calls that a program using dyn_maxflow_b200 makes, for timing.

A program holds a graph on the GPU (a Solver, a MultiSolver or a Server) and asks, again and again, for the exact
maximum flow: after a batch of capacity updates (`batch`, `multi`, `serve`), or from scratch (`static`).  Graphs are
the repository's own kinds: R-MAT graphs (a, b, c = 0.57, 0.19, 0.19; capacities U[1,1000]; source and sink = the
vertices of the highest out- and in-degree), 4-neighbour grids, and the small Johnson graph of the test fixture.

A pass of a `batch` or `serve` case takes the next batch of a stream: batches of fresh arcs one after the other, then
one after the other the batches that set these arcs back, and so on round.  Flow values are whole numbers, and so is
the minimum cut: the sink side that is read out is the set of vertices that can still reach the sink, which is the same
for every maximum flow.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import dyn_maxflow_b200 as D

A, B, C = 0.57, 0.19, 0.19  # R-MAT quadrant probabilities
CAP_HI, DELTA_HI = 1000, 500


def listed():
    return [
        # the reference's own fixture graph and a batch of a tenth of its arcs: nothing but latency
        {"name": "johnson_batch", "kind": "batch", "graph": "johnson", "frac": 0.1, "host": True,
         "variant": "data"},
        # a small graph that every test and tool of the repository uses
        {"name": "rmat14_batch", "kind": "batch", "graph": "rmat", "scale": 14, "degree": 16, "frac": 0.01,
         "host": True, "variant": "data"},
        # a few updates on a large graph: one user's change, answered at once
        {"name": "rmat20_few", "kind": "batch", "graph": "rmat", "scale": 20, "degree": 16, "updates": 101,
         "host": True, "variant": "data"},
        # the benchmark's GPU-scale configuration: a 1% batch that is already in device memory
        {"name": "rmat20_batch", "kind": "batch", "graph": "rmat", "scale": 20, "degree": 16, "frac": 0.01,
         "host": False, "variant": "data"},
        # the same on the largest graph of the schedule picker's evaluation (132 M arcs), far beyond the L2
        {"name": "rmat22_batch", "kind": "batch", "graph": "rmat", "scale": 22, "degree": 16, "frac": 0.01,
         "host": False, "variant": "data"},
        # a large batch in host memory (10% of the arcs of a sparser graph), push-pull variant
        {"name": "rmat18_pp_host", "kind": "batch", "graph": "rmat", "scale": 18, "degree": 8, "frac": 0.1,
         "host": True, "variant": "pp"},
        # the topology-driven variant
        {"name": "rmat15_topo", "kind": "batch", "graph": "rmat", "scale": 15, "degree": 16, "frac": 0.01,
         "host": True, "variant": "topo"},
        # from scratch, on the GPU-scale configuration: what a program pays for a new set of capacities
        {"name": "rmat20_static", "kind": "static", "graph": "rmat", "scale": 20, "degree": 16, "cut": False,
         "variant": "data"},
        # the grid configuration: 256 x 256, from scratch with the minimum cut (segmentation), and a 1% batch
        {"name": "grid256_static", "kind": "static", "graph": "grid", "rows": 256, "cols": 256, "cut": True,
         "variant": "data"},
        {"name": "grid256_batch", "kind": "batch", "graph": "grid", "rows": 256, "cols": 256, "frac": 0.01,
         "host": True, "variant": "data"},
        # many independent graphs in one device state, half grids, half R-MAT, all updated in each step
        {"name": "multi24", "kind": "multi", "count": 24, "median": 4000, "frac": 0.02},
        # the serving loop: a request for each of several resident graphs, all in flight together
        {"name": "serve8", "kind": "serve", "count": 8, "scale": 13, "degree": 16, "updates": 1500},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["rmat", "rmat", "rmat", "rmat_static", "grid", "grid", "grid_static", "multi", "serve"])
    variant = rng.choice(["data", "data", "data", "pp", "topo"])
    if kind in ("rmat", "rmat_static"):
        scale = rng.randint(8, 16 if variant == "topo" else 21)
        case = {"kind": "batch", "graph": "rmat", "scale": scale, "degree": rng.randint(5, 24), "variant": variant}
        if kind == "rmat_static":
            return dict(case, kind="static", cut=rng.random() < 0.5)
        return dict(case, frac=round(_log(rng, 0.0002, 0.1), 5), host=rng.random() < 0.5)
    if kind in ("grid", "grid_static"):
        rows = int(_log(rng, 7, 300))
        cols = max(7, min(300, int(_log(rng, 7, 300)), 65536 // rows))
        variant = "data" if variant == "topo" else variant
        case = {"kind": "batch", "graph": "grid", "rows": rows, "cols": cols, "variant": variant}
        if kind == "grid_static":
            return dict(case, kind="static", cut=rng.random() < 0.5)
        return dict(case, frac=round(_log(rng, 0.001, 0.1), 5), host=rng.random() < 0.5)
    if kind == "multi":
        return {"kind": "multi", "count": rng.randint(2, 24), "median": int(_log(rng, 300, 4000)),
                "frac": round(_log(rng, 0.002, 0.05), 5)}
    return {"kind": "serve", "count": rng.randint(2, 8), "scale": rng.randint(8, 14), "degree": rng.randint(5, 16),
            "updates": int(_log(rng, 20, 2000))}


# ---- graphs ------------------------------------------------------------------------------------------------------

_topologies: dict = {}


def _rmat_topology(scale, degree):
    """(index, adj, par on the host, index, adj, forward on the GPU, s, t) of an R-MAT graph: every sampled arc and its
    partner, rows sorted by head; `forward` marks the arcs that were sampled.  The samples depend on the sizes alone
    (one network, whatever its capacities), and the last few networks are kept."""
    key = (scale, degree)
    if key in _topologies:
        return _topologies[key]
    gen = torch.Generator("cuda").manual_seed(1000 * scale + degree)
    n = 1 << scale
    count = degree << scale
    u = torch.zeros(count, dtype=torch.int64, device="cuda")
    v = torch.zeros(count, dtype=torch.int64, device="cuda")
    for _ in range(scale):
        r = torch.rand(count, device="cuda", generator=gen)
        u += u + (r >= A + B)
        v += v + (((r >= A) & (r < A + B)) | (r >= A + B + C))
        del r
    keep = u != v
    fwd = torch.unique((u[keep] << scale) | v[keep])
    del u, v, keep
    back = ((fwd & (n - 1)) << scale) | (fwd >> scale)
    arcs = torch.unique(torch.cat([fwd, back]))
    m = arcs.numel()
    forward = torch.zeros(m, dtype=torch.bool, device="cuda")
    forward[torch.searchsorted(arcs, fwd)] = True
    del back
    out_deg = torch.bincount(fwd >> scale, minlength=n)
    in_deg = torch.bincount(fwd & (n - 1), minlength=n)
    del fwd
    s = int(out_deg.argmax())
    in_deg[s] = -1
    t = int(in_deg.argmax())
    del out_deg, in_deg
    tail, head = arcs >> scale, arcs & (n - 1)
    par = torch.searchsorted(arcs, (head << scale) | tail).to(torch.int32)
    del arcs
    index = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    index[1:] = torch.cumsum(torch.bincount(tail, minlength=n), 0)
    del tail
    index, head = index.to(torch.int32), head.to(torch.int32)
    got = (index.cpu().numpy(), head.cpu().numpy(), par.cpu().numpy(), index, head, forward, s, t)
    torch.cuda.empty_cache()
    while len(_topologies) >= 2:
        _topologies.pop(next(iter(_topologies)))
    _topologies[key] = got
    return got


def _rmat(scale, degree, seed):
    """(graph, s, t, (index, adj, capacities on the GPU))"""
    index, adj, par, d_index, d_adj, forward, s, t = _rmat_topology(scale, degree)
    gen = torch.Generator("cuda").manual_seed(seed)
    w = torch.randint(1, CAP_HI + 1, (len(adj),), dtype=torch.int32, device="cuda", generator=gen) * forward
    return D.Graph.from_csr(index, adj, w.cpu().numpy(), par), s, t, (d_index, d_adj, w)


def _with_arrays(g, s, t):
    return g, s, t, tuple(torch.from_numpy(x).cuda() for x in g.arrays()[:3])


def _grid(rows, cols, seed):
    return _with_arrays(*D.gen_grid(rows, cols, seed=seed, cap_lo=1, cap_hi=100, st_cap=1000))


def _johnson(seed):
    """Johnson graph of the 2-subsets of 8 (disjoint pairs are neighbours): 28 vertices, 210 edges."""
    sub = [(i, j) for i in range(8) for j in range(i + 1, 8)]
    uv = np.array([(a, b) for a in range(28) for b in range(28) if a != b and not set(sub[a]) & set(sub[b])], np.int32)
    w = np.random.default_rng(seed).integers(1, 101, len(uv)).astype(np.int32)
    return _with_arrays(D.Graph.from_edges(uv[:, 0], uv[:, 1], w), 25, 2)


def _graph(case, seed):
    if case["graph"] == "rmat":
        return _rmat(case["scale"], case["degree"], seed)
    if case["graph"] == "grid":
        return _grid(case["rows"], case["cols"], seed)
    return _johnson(seed)


def _updates(case, arrays):
    return case["updates"] if "updates" in case else max(1, int(case["frac"] * int(torch.count_nonzero(arrays[2]))))


def _stream(arrays, k, count, seed):
    """`count` batches of k updates (40% increases, 40% decreases, 10% deletes, 10% inserts into arcs of capacity zero;
    no arc in two of them), then the `count` batches that set the same arcs back: [(src, dst, w)] on the GPU."""
    index, adj, w = arrays
    gen = torch.Generator("cuda").manual_seed(seed)

    def rand(lo, hi, n):
        return torch.randint(lo, hi + 1, (n,), device="cuda", generator=gen, dtype=torch.int32)

    m = adj.numel()
    pool = torch.randint(0, m, (4 * count * k + 64,), device="cuda", generator=gen).unique()
    pool = pool[torch.randperm(pool.numel(), device="cuda", generator=gen)]
    at = w[pool] > 0
    pos, zero = pool[at], pool[~at]
    ins = min(k // 10, zero.numel() // count)
    per = max(1, min(k - ins, pos.numel() // count))
    new, old = [], []
    for b in range(count):
        p, z = pos[b * per:(b + 1) * per], zero[b * ins:(b + 1) * ins]
        step, pick = rand(1, DELTA_HI, p.numel()), torch.rand(p.numel(), device="cuda", generator=gen)
        to = torch.where(pick < 4 / 9, w[p] + step, torch.where(pick < 8 / 9, (w[p] - step).clamp_min(0), 0))
        arcs = torch.cat([p, z])
        src = (torch.searchsorted(index, arcs.to(torch.int32), right=True) - 1).to(torch.int32)
        new.append((src, adj[arcs], torch.cat([to, rand(1, CAP_HI, z.numel())]).to(torch.int32)))
        old.append((src, adj[arcs], w[arcs]))
    return new + old


def _host(batches):
    return [tuple(x.cpu().numpy() for x in b) for b in batches]


# ---- what a program has in hand ----------------------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    if kind in ("batch", "static"):
        g, s, t, arrays = _graph(case, seed)
        sv = D.Solver(g, s, t, variant=case["variant"])
        if kind == "static":
            return {"kind": kind, "sv": sv, "cut": case["cut"]}
        sv.static_maxflow()
        batches = _stream(arrays, _updates(case, arrays), max(2, min(8, int(0.4 / case.get("frac", 0.01)))), seed)
        return {"kind": kind, "sv": sv, "host": case["host"], "batches": _host(batches) if case["host"] else batches,
                "next": 0}
    if kind == "serve":
        made = [_rmat(case["scale"], case["degree"], seed + 7919 * i) for i in range(case["count"])]
        srv = D.Server([x[0] for x in made], [x[1] for x in made], [x[2] for x in made], 8 << 30)
        streams = [_host(_stream(x[3], case["updates"], 4, seed + i)) for i, x in enumerate(made)]
        for i in range(case["count"]):  # a first request each: the graphs are solved
            srv.wait(srv.submit(i, *streams[i][-1]))
        return {"kind": kind, "srv": srv, "batches": list(zip(*streams)), "next": 0}
    # log-normal sizes as in the batched benchmark, spread evenly over the distribution instead of drawn
    made = []
    for i, nv in enumerate(_multi_sizes(case)):
        if i % 2 == 0:
            side = max(4, int(round(math.sqrt(nv))))
            made.append(_grid(side, side + i % 3, seed + 31 * i))
        else:
            g, s, t = D.gen_rmat(max(6, int(round(math.log2(nv)))), None, A, B, C, seed=seed + 31 * i, cap_lo=1,
                                 cap_hi=CAP_HI)
            made.append(_with_arrays(g, s, t))
    sv = D.MultiSolver([x[0] for x in made], [x[1] for x in made], [x[2] for x in made])
    sv.static_maxflow_all()
    streams = [_stream(x[3], _updates(case, x[3]), 2, seed + i) for i, x in enumerate(made)]
    steps, ofs = [], [0]
    for b in zip(*streams):  # every instance's batch of a step, in the union's vertex ids
        steps += [(x[0] + int(sv.vertex_base[i]), x[1] + int(sv.vertex_base[i]), x[2]) for i, x in enumerate(b)]
        ofs.append(ofs[-1] + sum(x[0].numel() for x in b))
    src, dst, w = (torch.cat(x) for x in zip(*steps))
    return {"kind": kind, "sv": sv, "ofs": np.array(ofs, np.int64), "src": src, "dst": dst, "w": w}


# ---- one pass ----------------------------------------------------------------------------------------------------

def run(state):
    kind = state["kind"]
    if kind == "static":
        flow = state["sv"].static_maxflow()
        return [flow, state["sv"].cut()] if state["cut"] else [flow]
    if kind == "multi":
        flows, _ = state["sv"].run_batches(state["ofs"], state["src"].data_ptr(), state["dst"].data_ptr(),
                                           state["w"].data_ptr(), use_graph=True)
        return flows
    b = state["batches"][state["next"]]
    state["next"] = (state["next"] + 1) % len(state["batches"])
    if kind == "serve":
        tickets = [state["srv"].submit(i, *x) for i, x in enumerate(b)]
        return [state["srv"].wait(tk)[0] for tk in tickets]
    if state["host"]:
        return state["sv"].apply_updates(*b)
    return state["sv"].apply_updates_device(b[0].data_ptr(), b[1].data_ptr(), b[2].data_ptr(), b[0].numel())


# ---- what a pass cannot do without -------------------------------------------------------------------------------

def _multi_sizes(case):
    return case["median"] * np.exp(np.linspace(-1.3, 1.3, case["count"]))


def _sizes(case):
    """(vertices, arcs of capacity above zero, CSR arcs), about."""
    if case["graph"] == "rmat":
        n = 1 << case["scale"]
        return n, n * case["degree"], 2 * n * case["degree"]
    if case["graph"] == "grid":
        n = case["rows"] * case["cols"]
        return n, 4 * n, 4 * n
    return 28, 420, 420


def work(case):
    """An update: its three words read, its arc's capacity and residual read and written.  A solve from scratch: heads,
    capacities and row offsets read, residuals written, the cut written where it is asked for."""
    kind = case["kind"]
    if kind == "static":
        n, _, m = _sizes(case)
        return {"bytes": 12 * m + 4 * n + (n if case["cut"] else 0) + 8, "flops": 0}
    if kind == "batch":
        k = case["updates"] if "updates" in case else max(1, int(case["frac"] * _sizes(case)[1]))
        return {"bytes": 28 * k + 8, "flops": 0}
    if kind == "serve":
        return {"bytes": case["count"] * (28 * case["updates"] + 8), "flops": 0}
    arcs = sum((4 if i % 2 == 0 else 16) * nv for i, nv in enumerate(_multi_sizes(case)))
    return {"bytes": 4 * (28 * max(1, int(case["frac"] * arcs)) + 8 * case["count"]), "flops": 0}


def exact(case, seed):
    """Flows and cuts are whole numbers and are compared as they are."""
    return None
