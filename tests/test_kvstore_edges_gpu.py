"""KV store at the edges of its word copies, prefix sums and compaction: heap
and destination off a word, values of every length around the copy's batches,
destinations that are too small, refused puts, keys of one high byte over many
sort blocks, growing compactions, and entries that a caller wrote into the map
underneath.  Everything equals a Python dict."""
from __future__ import annotations

import numpy as np
import pytest

from lslab_b200 import KVStore, LsbError, _lib
from lslab_b200 import workload as W
from tests.test_kvstore_gpu import _get_all, _pack, _values
from tests.util import dev, host

pytestmark = pytest.mark.gpu


def _put(kv, keys, values):
    buf, off = _pack(values)
    kv.put(dev(keys), dev(buf), dev(off))


def test_lengths_and_alignments(cuda):
    """Every length from 0 to 70 and around 2 KB, from a heap whose size is no
    whole word and is filled to the last byte, to destinations at every offset
    from a word; a destination that ends inside a value leaves that value out."""
    rng = np.random.default_rng(3)
    lens = list(range(71)) + [511, 512, 513, 2047, 2048, 2049, 5001, 0, 3]
    rng.shuffle(lens)
    vals = [rng.integers(0, 256, size=n, dtype=np.uint8).tobytes() for n in lens]
    total = sum(lens)
    kv = KVStore(6, total)
    keys = W.prefill_keys(5, len(vals))
    _put(kv, keys, vals)
    assert kv.usage()["heap_used"] == total
    n = len(keys)
    dk = dev(keys)
    ln = cuda.zeros(n, dtype=cuda.int32, device="cuda")
    off = cuda.zeros(n, dtype=cuda.int64, device="cuda")
    want = b"".join(vals)
    for shift in range(5):
        for cut in (0, 1, 2500):
            buf = cuda.full((total + 16,), 0xAB, dtype=cuda.uint8, device="cuda")
            assert kv.get(dk, ln, off, buf[shift:shift + total], total - cut) == total
            cuda.cuda.synchronize()
            got, o = host(buf, np.uint8), host(off, np.uint64)
            exp = np.full(total + 16, 0xAB, np.uint8)
            for v, at in zip(vals, o):
                if int(at) + len(v) <= total - cut:
                    exp[shift + int(at):shift + int(at) + len(v)] = np.frombuffer(v, np.uint8)
            assert np.array_equal(got, exp), (shift, cut)
    kv.compact()
    assert kv.usage() == {"heap_used": total, "heap_dead": 0, "heap_cap": total}
    assert b"".join(_get_all(kv, keys, cuda)[0]) == want


def test_put_after_a_refused_one(cuda):
    """A value over the limit, offsets that fall and a batch that does not fit
    leave the store as it was, and the next put is taken."""
    kv = KVStore(6, 1 << 25)
    keys = W.prefill_keys(6, 3)
    _put(kv, keys[:2], [b"one", b"two"])
    big = cuda.zeros(1 << 24, dtype=cuda.uint8, device="cuda")
    for off in ([0, 1 << 24], [0, 5, 2], [0, 1 << 26]):
        with pytest.raises(LsbError):
            kv.put(dev(keys[:len(off) - 1]), big, dev(np.array(off, np.uint64)))
        _put(kv, keys[2:], [b"three"])
        assert _get_all(kv, keys, cuda)[0] == [b"one", b"two", b"three"]


def test_compactions_of_many_keys(cuda):
    """Keys 0.. (seven equal high bytes) over many sort blocks, compacted, then
    more and longer values, compacted again with more scratch than was kept."""
    rng = np.random.default_rng(9)
    n = 30_000
    kv = KVStore(10, 1 << 25, pool_slabs=1 << 14)
    ref = {}
    for lo, hi, longest in ((0, n, 20), (n // 2, 2 * n, 300)):
        keys = rng.permutation(np.arange(lo, hi, dtype=np.uint64))
        vals = _values(rng, len(keys), longest)
        _put(kv, keys, vals)
        ref.update(zip(keys.tolist(), vals))
        gone = keys[::7]
        kv.remove(dev(gone))
        for k in gone.tolist():
            del ref[k]
        kv.compact()
        live = sum(len(v) for v in ref.values())
        assert kv.usage() == {"heap_used": live, "heap_dead": 0, "heap_cap": 1 << 25}
        every = np.arange(0, 2 * n, dtype=np.uint64)
        assert _get_all(kv, every, cuda)[0] == [ref.get(k) for k in every.tolist()]


def test_compact_with_entries_of_the_caller(cuda):
    """A second key with a stored value's handle is a value of its own after a
    compaction, as long as the heap takes both; handles past the heap and live
    values past its size are refused without effect."""
    lib = _lib.lib()
    kv = KVStore(6, 1000)
    keys = W.prefill_keys(8, 9)
    _put(kv, keys[:1], [b"x" * 400])
    m = lib.lsb_kvs_map(kv._h)
    st = cuda.cuda.current_stream().cuda_stream
    res = cuda.zeros((1, 2), dtype=cuda.int64, device="cuda")
    dk = dev(keys)
    assert lib.lsb_map_get(m, dk.data_ptr(), res.data_ptr(), 1, st) == 0
    handle = res[:, 1].contiguous()

    def alias(i, h=handle):
        assert lib.lsb_map_put(m, dk[i:].data_ptr(), h.data_ptr(), None, 1, st) == 0

    alias(1)
    kv.compact()
    assert kv.usage()["heap_used"] == 800
    assert _get_all(kv, keys[:3], cuda)[0] == [b"x" * 400, b"x" * 400, None]
    alias(2)  # 1200 bytes
    with pytest.raises(LsbError):
        kv.compact()
    alias(2, cuda.tensor([(997 << 24) | 4], device="cuda"))  # ends at 1001
    with pytest.raises(LsbError):
        kv.compact()
    lib.lsb_map_remove(m, dk[2:].data_ptr(), None, 1, st)
    assert kv.usage()["heap_used"] == 800
    kv.compact()
    assert _get_all(kv, keys[:3], cuda)[0] == [b"x" * 400, b"x" * 400, None]
