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


def ladder(oracle, n, width, seed):
    """Columns of `width` vertices, neighbours both ways, s before the first column and t after the last."""
    rng = np.random.default_rng(seed)
    u = np.arange(n - 2)
    step, up = u[u + width < n - 2], u[(u + 1 < n - 2) & ((u + 1) % width != 0)]
    a = np.concatenate([step, step + width, up, up + 1, np.full(width, n - 2), u[-width:]])
    b = np.concatenate([step + width, step, up + 1, up, u[:width], np.full(width, n - 1)])
    return oracle.build_csr(a, b, rng.integers(1, 50, len(a)))


def write(oracle, path, n, width, big=0):
    """A ladder and a batch as kernel_main reads them; the flows before and after the batch."""
    got_n, m, off, adj, cap, par = ladder(oracle, n, width, n)
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
    assert got[0][1] > 0  # the greatest distance of a barrier-free relabel: there was one


# a push phase past its time limit, with one window a warp and with several: a block that other blocks wait for, but
# the first one does not, stops as well, long before the labels of its two vertices have climbed to n
@pytest.mark.parametrize("blocks,n", [(2, 64), (2, 256), (3, 96), (3, 384)])
def test_every_block_keeps_the_time_limit(kernel_main, blocks, n):
    assert run(kernel_main, "push", blocks, n)[0][0] < n


# a batch whose barrier wait runs out leaves capacities and residuals as they were: the claim is in the first phase, or
# (one capacity above 2^30 - 1) in a second one after a barrier
@pytest.mark.parametrize("big,barrier", [(0, 1), (2**30 + 5, 1), (2**30 + 5, 2)])
def test_timed_out_batch_takes_its_claims_back(kernel_main, oracle, tmp_path, big, barrier):
    path = str(tmp_path / "graph")
    write(oracle, path, 200, 20, big)
    err_timeout = 1
    assert run(kernel_main, "timeout", path, 2, 64, barrier) == [[err_timeout, 0]]
