"""Per-phase calls captured into a caller's CUDA graph: the graph holds kernels
only, whatever the size of the table's scratch, and replays of calls in every
window size that has kernels of its own equal the oracle's, beside live calls
of both forms and past the point where the window epochs run out."""
from __future__ import annotations

import numpy as np
import pytest

from lslab_b200 import Map
from lslab_b200 import workload as W
from oracle import OracleMap
from tests.util import dev, first_mismatch, results, results_buf, same_results

pytestmark = pytest.mark.gpu


def _capture(torch, calls):
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        for f in calls:
            f()
    graph.instantiate()
    return graph


def test_captured_calls_are_kernels_only(cuda):
    import torch
    from cuda.bindings import runtime as rt
    m = Map(8)
    k, v = W.key_of_rank(8, np.arange(700)), W.splitmix64(10, 0, 700)
    dk, dv = dev(k), dev(v)
    old = torch.zeros(700, dtype=torch.int64, device="cuda")
    graph = _capture(torch, [lambda: m.put(dk, dv, old), lambda: m.put(dk[:300], dv, old)])
    g = rt.cudaGraph_t(graph.raw_cuda_graph())
    err, _, count = rt.cudaGraphGetNodes(g, 0)
    assert err == rt.cudaError_t.cudaSuccess
    err, nodes, count = rt.cudaGraphGetNodes(g, count)
    kinds = [rt.cudaGraphNodeGetType(n)[1] for n in nodes[:count]]
    assert kinds and all(x == rt.cudaGraphNodeType.cudaGraphNodeTypeKernel for x in kinds), kinds


@pytest.mark.parametrize("n,window", [(300, 0), (512, 0), (513, 0), (20_000, 0), (170_000, 0),
                                      (1_000, 256), (9_000, 4096)])
def test_captured_mixed_calls_replay(cuda, n, window):
    import torch
    rng = np.random.default_rng(71)
    t = rng.choice([0, 1, 2, 3], size=n, p=[0.4, 0.3, 0.1, 0.2]).astype(np.uint8)
    k = W.key_of_rank(8, rng.integers(0, max(20, n // 30), size=n))
    k[rng.random(n) < 0.05] = np.uint64(5)
    v, v2 = W.splitmix64(10, 0, n), W.splitmix64(11, 0, n)
    m, o = Map(8, max_window=window), OracleMap(8)
    dt, dk, dv, dv2 = dev(t), dev(k), dev(v), dev(v2)
    out, live = results_buf(n), results_buf(n)
    graph = _capture(torch, [lambda: m.execute(dt, dk, dv, out)])
    for r in range(135 if n < 1000 else 5):  # 135: the 127 epochs run out
        graph.replay()
        want = o.mixed(t, k, v)
        torch.cuda.synchronize()
        got = results(out)
        assert same_results(got, want), f"replay {r}: " + first_mismatch(got, want)
        (m.execute if r % 2 else m.execute_fused)(dt, dk, dv2, live)
        want = o.mixed(t, k, v2)
        torch.cuda.synchronize()
        got = results(live)
        assert same_results(got, want), f"call {r}: " + first_mismatch(got, want)
    assert m.status() == 0
