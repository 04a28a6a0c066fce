"""GPU parity of hot keys whose mutations lie unevenly in the window (bursts,
key order, clusters at every scale), with updates among them, through the
per-phase and the persistent form: every result equals the oracle's replay."""
from __future__ import annotations

import numpy as np
import pytest

from lslab_b200 import Map
from lslab_b200 import workload as W
from oracle import OracleMap
from tests.util import dev, first_mismatch, results, results_buf, same_results

pytestmark = pytest.mark.gpu

N = 1 << 20


def _hot(kind):
    """[(key, op indices of its mutations)]"""
    rng = np.random.default_rng(61)
    if kind == "burst":  # in a row at the window's end, 4097 and 5000 of them
        return [(1, np.concatenate([[0], np.arange(N - 4_096, N)])),
                (2, np.concatenate([[1], np.arange(N - 20_000, N - 15_000)]))]
    if kind == "runs":  # a batch in key order
        return [(i, np.arange(i * 30_000, i * 30_000 + 5_000 * i)) for i in range(1, 7)] + \
            [(7, np.arange(600_000, 600_000 + 131_072))]
    if kind == "trickle":  # spread over the window, and a burst
        return [(1, np.union1d(np.arange(0, N, 97), np.arange(700_000, 790_000)))]
    at = np.concatenate([2 ** i + np.arange(min(2 ** i, 3_000)) for i in range(20)])
    first = np.unique(np.concatenate([at, N - 1 - 2 ** np.arange(8, 17)]))
    free = np.setdiff1d(np.arange(N), first)
    return [(1, first), (2, free[(rng.random(60_000) ** 6 * len(free)).astype(np.int64)])]


@pytest.mark.parametrize("fused", [False, True])
@pytest.mark.parametrize("kind", ["burst", "runs", "trickle", "clusters"])
def test_uneven_hot_keys(cuda, kind, fused):
    import torch
    rng = np.random.default_rng(67)
    t = np.zeros(N, np.uint8)
    k = W.key_of_rank(6, rng.integers(0, 3000, size=N))
    for key, at in _hot(kind):
        at = np.unique(at)
        t[at], k[at] = rng.choice([1, 2, 3], size=len(at), p=[0.3, 0.2, 0.5]), np.uint64(key)
        reads = rng.integers(0, N, size=500)
        k[reads[t[reads] == 0]] = np.uint64(key)
    v = W.splitmix64(8, 0, N)
    m, o = Map(10), OracleMap(10)
    for _ in range(2):  # the second time the keys that stayed are present
        out = results_buf(N)
        (m.execute_fused if fused else m.execute)(dev(t), dev(k), dev(v), out)
        torch.cuda.synchronize()
        got, want = results(out), o.mixed(t, k, v)
        assert same_results(got, want), first_mismatch(got, want)
    assert m.status() == 0
