"""The device time of the last solve call, Solver.stats()["last_ms"]: fixed when the call ends, whoever asks and when."""
import threading

import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def made(dmf):
    g, s, t = dmf.gen_rmat(14, 16 << 14, seed=5, cap_lo=1, cap_hi=1000)
    return g, s, t, dmf.gen_batches(g, 2, frac=0.01, seed=6)


def test_last_ms_outlives_a_staged_batch(dmf, made):
    g, s, t, batches = made
    with dmf.Solver(g, s, t) as sv:
        sv.static_maxflow()
        sv.features(*batches[0])  # stages the batch, solves nothing
        first = sv.stats()["last_ms"]
        assert first > 0
        for b in batches:
            sv.features(*b)
            assert sv.stats()["last_ms"] == first
        sv.apply_updates(*batches[0])
        second = sv.stats()["last_ms"]
        sv.features(*batches[1])
        assert second > 0 and sv.stats()["last_ms"] == second


def test_threads_read_the_same_time(dmf, made):
    g, s, t, _ = made
    with dmf.Solver(g, s, t) as sv:
        for _ in range(50):
            sv.static_maxflow()
            got, gate = [0.0] * 8, threading.Barrier(8)

            def ask(i):
                gate.wait()
                got[i] = sv.stats()["last_ms"]

            th = [threading.Thread(target=ask, args=(i,)) for i in range(8)]
            for x in th:
                x.start()
            for x in th:
                x.join()
            assert len(set(got)) == 1 and got[0] > 0, got


def test_stats_while_a_stream_is_captured(dmf, made):
    torch = pytest.importorskip("torch")
    g, s, t, _ = made
    x = torch.zeros(8, device="cuda")
    with dmf.Solver(g, s, t) as sv:
        sv.static_maxflow()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            x += 1
            ms = sv.stats()["last_ms"]
        graph.replay()
        torch.cuda.synchronize()
        assert ms > 0 and x.sum().item() == 8
        assert sv.stats()["last_ms"] == ms
