"""Inserts that meet in a few buckets: thousands of new keys a call in long
chains, then calls that remove some keys and insert others into the slots they
leave, in every lock mode, for the map and the set.  Results, contents and
size equal the oracle's, and no key has two slots."""
from __future__ import annotations

import numpy as np
import pytest

from lslab_b200 import Map, Set
from lslab_b200 import workload as W
from oracle import OracleMap, OracleSet
from tests.util import dev, host, results, results_buf, same_results, first_mismatch

pytestmark = pytest.mark.gpu


def _rounds(keys):
    """Op types and keys of calls: all inserted; a third removed while others
    are written again; removed ones return beside new removals."""
    a, b, c = keys[0::3], keys[1::3], keys[2::3]
    rng = np.random.default_rng(83)
    for put, drop in ((np.concatenate([a, b]), c[:0]), (c, a), (a[::2], b), (b, c[::2]),
                      (np.concatenate([a, c]), b[::3])):
        t = np.concatenate([np.ones(len(put), np.uint8), np.full(len(drop), 2, np.uint8)])
        k = np.concatenate([put, drop])
        order = rng.permutation(len(k))
        yield t[order], k[order]


@pytest.mark.parametrize("lock", ["writer", "rw", "free"])
@pytest.mark.parametrize("log2,n", [(1, 1_500), (3, 6_000), (8, 60_000)])
def test_map_inserts_meet(cuda, lock, log2, n):
    m, o = Map(log2, pool_slabs=n // 8 + 256, lock_mode=lock), OracleMap(log2)
    for r, (t, k) in enumerate(_rounds(W.prefill_keys(9, n))):
        v = W.splitmix64(r, 0, len(k))
        out = results_buf(len(k))
        m.execute(dev(t), dev(k), dev(v), out)
        cuda.cuda.synchronize()
        got, want = results(out), o.mixed(t, k, v)
        assert same_results(got, want), first_mismatch(got, want)
        kk, vv = m.dump()
        ko, vo = o.dump()
        assert np.array_equal(kk, ko) and np.array_equal(vv, vo)
        assert m.size() == len(ko)
    assert m.status() == 0


@pytest.mark.parametrize("lock", ["writer", "rw", "free"])
@pytest.mark.parametrize("log2,n", [(1, 1_500), (8, 60_000)])
def test_set_inserts_meet(cuda, lock, log2, n):
    s, o = Set(log2, pool_slabs=n // 8 + 256, lock_mode=lock), OracleSet(log2)
    for t, k in _rounds(W.set_prefill_keys(9, n)):
        k = k.astype(np.uint32)
        out = cuda.zeros(len(k), dtype=cuda.uint8, device="cuda")
        s.execute(dev(t), dev(k), out)
        cuda.cuda.synchronize()
        assert np.array_equal(host(out, np.uint8), o.mixed(t, k))
        assert np.array_equal(s.dump(), o.dump())
        assert s.size() == len(o.dump())
    assert s.status() == 0
