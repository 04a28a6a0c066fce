"""GPU parity of mixed batches whose groups sit on both sides of the ordering
paths' limits (one warp, one block, index ranges over several blocks, grid
steps) and spread over narrow and wide parts of the window: every result equals
the oracle's replay, through the per-phase and the persistent form."""
from __future__ import annotations

import numpy as np
import pytest

from lslab_b200 import Map
from lslab_b200 import workload as W
from oracle import OracleMap
from tests.util import dev, first_mismatch, results, results_buf, same_results

pytestmark = pytest.mark.gpu


def _batch(kind):
    rng = np.random.default_rng(41)
    n = 1 << 19
    t = np.zeros(n, np.uint8)
    k = W.key_of_rank(6, rng.integers(0, 5000, size=n))
    # 256 | 257 and 4096 | 4097 change the block's sort, 131072 | 131073 takes
    # the grid steps
    sizes = {"wide": (64, 65, 256, 257, 300, 4096, 4097, 9000, 131_072, 131_073),
             "narrow": (64, 65, 256, 257, 1000, 4096, 4097, 20_000),
             "many": (70,) * 3000 + (4200,) * 3}[kind]
    at = rng.permutation(n) if kind != "narrow" else n - 1 - rng.permutation(60_000)
    for i, c in enumerate(sizes):
        m, at = at[:c], at[c:]
        t[m], k[m] = rng.choice([1, 2, 3], size=c, p=[0.3, 0.2, 0.5]), np.uint64(10 + i)
        # reads of the same key between its mutations
        r = at[:c // 8]
        at = at[c // 8:]
        k[r] = np.uint64(10 + i)
    return t, k, W.splitmix64(8, 0, n)


@pytest.mark.parametrize("fused", [False, True])
@pytest.mark.parametrize("kind", ["wide", "narrow", "many"])
def test_group_sizes_at_path_limits(cuda, kind, fused):
    import torch
    t, k, v = _batch(kind)
    m, o = Map(10), OracleMap(10)
    for _ in range(2):  # the second time the keys that stayed are present
        out = results_buf(len(k))
        (m.execute_fused if fused else m.execute)(dev(t), dev(k), dev(v), out)
        torch.cuda.synchronize()
        got, want = results(out), o.mixed(t, k, v)
        assert same_results(got, want), first_mismatch(got, want)
    assert m.status() == 0


@pytest.mark.parametrize("fused", [False, True])
def test_many_windows_of_one_call(cuda, fused):
    """One call of several hundred windows: the 127 window epochs run out within
    the call, so the group tables are cleared between its windows."""
    import torch
    rng = np.random.default_rng(43)
    n, window = 64 * 300 + 17, 64
    t = rng.choice([0, 1, 2, 3], size=n, p=[0.4, 0.3, 0.1, 0.2]).astype(np.uint8)
    k = W.key_of_rank(7, rng.integers(0, 50, size=n))
    v = W.splitmix64(9, 0, n)
    m, o = Map(6, max_window=window), OracleMap(6)
    for _ in range(2):
        out = results_buf(n)
        (m.execute_fused if fused else m.execute)(dev(t), dev(k), dev(v), out)
        torch.cuda.synchronize()
        got, want = results(out), o.mixed(t, k, v)
        assert same_results(got, want), first_mismatch(got, want)
    assert m.status() == 0


def test_captured_calls_replay_between_live_ones(cuda):
    """put and remove calls captured into a caller's CUDA graph, replayed more
    often than there are window epochs, with live calls on the same keys in
    between: every result equals the oracle's."""
    import torch
    rng = np.random.default_rng(47)
    n = 3000
    k = W.key_of_rank(8, rng.integers(0, 200, size=n))  # groups of ~15: ordered lists
    v, v2 = W.splitmix64(10, 0, n), W.splitmix64(11, 0, n)
    m, o = Map(8), OracleMap(8)
    dk, dv, dv2, part = dev(k), dev(v), dev(v2), dev(k[:500])
    old = torch.zeros(n, dtype=torch.int64, device="cuda")
    out = results_buf(500)
    live = torch.zeros(n, dtype=torch.int64, device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        m.put(dk, dv, old)
        m.remove(part, out)
    for r in range(140):
        graph.replay()
        m.put(dk, dv2, live)
        want_old = o.put(k, v)
        want_out = o.remove(k[:500])
        want_live = o.put(k, v2)
        if r % 10 == 9 or r < 3:
            torch.cuda.synchronize()
            assert np.array_equal(old.cpu().numpy().view(np.uint64), want_old), f"replay {r}"
            got = results(out)
            assert same_results(got, want_out), first_mismatch(got, want_out)
            assert np.array_equal(live.cpu().numpy().view(np.uint64), want_live), f"replay {r}"
    assert m.status() == 0
