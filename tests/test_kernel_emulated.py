"""The solve kernel's own source on host threads (tests/emu): every warp of it has to stay together by CUDA's rules alone,
with lanes that run as freely as CUDA allows.  Needs g++ and CUDA's headers, no GPU."""
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.fixture(scope="session")
def kernel_main(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("emu") / "kernel_main")
    emu = os.path.join(ROOT, "tests", "emu")
    subprocess.run(["g++", "-std=c++17", "-O0", "-w", "-pthread", f"-I{emu}", f"-I{CUDA}/include",
                    f"-I{ROOT}/dyn_maxflow_b200/csrc", f"-I{ROOT}/include", f"{emu}/kernel_main.cpp", "-o", exe],
                   check=True)
    return exe


def run(*args):
    r = subprocess.run([str(a) for a in args], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, (r.returncode, r.stderr)
    return [[int(x) for x in line.split()] for line in r.stdout.splitlines()]


def ladder(oracle, n, width, seed, hubs=0):
    """Columns of `width` vertices, neighbours both ways, s before the first column and t after the last; `hubs` more
    vertices get flow from s and have an arc to every vertex of the columns (long rows, but no way in)."""
    rng = np.random.default_rng(seed)
    inner, s, t = n - 2 - hubs, n - 2, n - 1
    u = np.arange(inner)
    step, up = u[u + width < inner], u[(u + 1 < inner) & ((u + 1) % width != 0)]
    a = np.concatenate([step, step + width, up, up + 1, np.full(width, s), u[-width:]])
    b = np.concatenate([step + width, step, up + 1, up, u[:width], np.full(width, t)])
    w = rng.integers(1, 50, len(a))
    for h in range(inner, s):
        a = np.concatenate([a, [s], np.full(inner, h)])
        b = np.concatenate([b, [h], u])
        w = np.concatenate([w, [inner], np.ones(inner, np.int64)])
    return oracle.build_csr(a, b, w)


def write(oracle, path, n, width, big=0, hubs=0):
    """A ladder and a batch as kernel_main reads them; the flows before and after the batch."""
    got_n, m, off, adj, cap, par = ladder(oracle, n, width, n, hubs)
    assert got_n == n
    if big:
        cap[0] = big
    rng = np.random.default_rng(n + 1)
    arcs = rng.permutation(m)[:m // 10]
    src, dst = np.searchsorted(off, arcs, side="right") - 1, adj[arcs]
    to = rng.integers(0, 60, len(arcs))
    np.concatenate([[n, m, n - 2, n - 1, len(arcs)], off, adj, cap, par, src, dst, to]).astype(np.int32).tofile(path)
    new = cap.copy()
    new[arcs] = to
    return [oracle.dinic(n, off, adj, c, par, n - 2, n - 1) for c in (cap, new)]


# deep graphs: every warp one window of 32 vertices, some none, some more than others, the most a warp can own
@pytest.mark.parametrize("n,width,blocks,warps", [(64, 1, 1, 2), (64, 2, 2, 2), (30, 1, 1, 2), (96, 1, 1, 2),
                                                  (97, 2, 1, 2), (160, 3, 2, 2), (200, 2, 1, 4), (256, 4, 1, 2)])
def test_deep_solve_stays_together(kernel_main, oracle, tmp_path, n, width, blocks, warps):
    path = str(tmp_path / "graph")
    want = write(oracle, path, n, width)
    got = run(kernel_main, "solve", path, blocks, 32 * warps, 0)
    assert [x[0] for x in got] == want
    assert got[0][1] > 0  # it had barrier-free relabels


# a push phase past its time limit, with one window a warp and with several: a block that other blocks wait for, but
# the first one does not, stops as well, long before the labels of its two vertices have climbed to n
@pytest.mark.parametrize("blocks,n", [(2, 64), (2, 256), (3, 96), (3, 384)])
def test_every_block_keeps_the_time_limit(kernel_main, blocks, n):
    assert run(kernel_main, "push", blocks, n)[0][0] < n


# rows of 9 arcs and more go to a whole warp: below, at and above the arcs it takes at a time, and several times that
@pytest.mark.parametrize("n", [36, 64, 127, 130, 131, 290, 500])
def test_deep_solve_with_long_rows(kernel_main, oracle, tmp_path, n):
    path = str(tmp_path / "graph")
    want = write(oracle, path, n, 1 if n < 64 else 3, hubs=2)
    got = run(kernel_main, "solve", path, 1, 128, 0)
    assert [x[0] for x in got] == want
    assert got[0][1] > 0


# the sink's row by a level of its own before every barrier-free relabel, as for sinks of more than 2,048 arcs
@pytest.mark.parametrize("n,width,hubs", [(64, 1, 0), (97, 2, 0), (130, 3, 2), (256, 40, 1)])
def test_deep_solve_with_a_wide_sink(kernel_main, oracle, tmp_path, n, width, hubs):
    path = str(tmp_path / "graph")
    want = write(oracle, path, n, width, hubs=hubs)
    assert [x[0] for x in run(kernel_main, "solve", path, 1, 128, 4097)] == want
    assert [x[0] for x in run(kernel_main, "solve", path, 2, 128, 4097)] == want


# a batch whose barrier wait runs out leaves capacities and residuals as they were: the claim is in the first phase, or
# (one capacity above 2^30 - 1) in a second one after a barrier
@pytest.mark.parametrize("big,barrier", [(0, 1), (2**30 + 5, 1), (2**30 + 5, 2)])
def test_timed_out_batch_takes_its_claims_back(kernel_main, oracle, tmp_path, big, barrier):
    path = str(tmp_path / "graph")
    write(oracle, path, 200, 20, big)
    err_timeout = 1
    assert run(kernel_main, "timeout", path, 2, 64, barrier) == [[err_timeout, 0]]
