"""Groups of more than 2^17 mutations, which the whole grid orders in steps with
barriers between them: two in one window, one whose ops are updates for whole
runs, and two and three of more than 98,304, which takes three to the steps, through the per-phase, the persistent (both probe orders) and the
two-stream form.  Every result and the contents equal the oracle's replay."""
from __future__ import annotations

import numpy as np
import pytest

from lslab_b200 import Map
from lslab_b200 import workload as W
from oracle import OracleMap
from tests.util import dev, first_mismatch, results, results_buf, same_results

pytestmark = pytest.mark.gpu

N = 1 << 19


def _batch(kind):
    rng = np.random.default_rng(79)
    t = rng.choice([0, 1, 2, 3], size=N, p=[0.25, 0.35, 0.2, 0.2]).astype(np.uint8)
    k = W.key_of_rank(6, rng.integers(0, 3000, size=N))
    if kind in ("two_mid", "three_mid"):
        k[:], t[:] = W.key_of_rank(6, np.arange(N) % 3000), 0
        at, last = rng.permutation(N), 98_304 + (kind == "three_mid")
        for i, c in enumerate((98_305, 100_001, last, 60_000)):
            m, at = at[:c], at[c:]
            k[m], t[m] = np.uint64(1 + i), rng.choice([1, 2, 3], size=c, p=[0.4, 0.2, 0.4])
            r, at = at[:2000], at[2000:]
            k[r] = np.uint64(1 + i)
        return t, k, W.splitmix64(8, 0, N)
    if kind == "two":  # one spread over the window, one in a row; a third below the limit
        k[rng.random(N) < 0.75] = np.uint64(1)
        k[300_000:500_000] = np.uint64(2)
        k[rng.random(N) < 0.1] = np.uint64(3)
    else:  # one put, updates only, one remove, updates only
        hot = np.sort(rng.permutation(N)[:300_000])
        k[hot], t[hot] = np.uint64(1), 3
        t[hot[9]], t[hot[170_000]], t[hot[230_001]] = 1, 2, 1
        reads = rng.permutation(N)[:2000]
        k[reads], t[reads] = np.uint64(1), 0
    over = [c for c in np.unique(k[t != 0], return_counts=True)[1] if c > 1 << 17]
    assert len(over) == (2 if kind == "two" else 1)
    return t, k, W.splitmix64(8, 0, N)


@pytest.mark.parametrize("form", ["plain", "fused", "split0", "overlap"])
@pytest.mark.parametrize("kind", ["two", "updates", "two_mid", "three_mid"])
def test_groups_over_the_steps_limit(cuda, kind, form):
    import torch
    t, k, v = _batch(kind)
    m, o = Map(10), OracleMap(10)
    if form in ("split0", "overlap"):
        m.set_tuning(**({"fused_split": 0} if form == "split0" else {"overlap": 1}))
    for _ in range(2):
        out = results_buf(N)
        (m.execute if form == "plain" else m.execute_fused)(dev(t), dev(k), dev(v), out)
        torch.cuda.synchronize()
        got, want = results(out), o.mixed(t, k, v)
        assert same_results(got, want), first_mismatch(got, want)
    kk, vv = m.dump()
    ko, vo = o.dump()
    assert np.array_equal(kk, ko) and np.array_equal(vv, vo)
    assert m.status() == 0
