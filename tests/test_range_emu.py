"""Hot keys whose mutations are not spread evenly over the window (bursts, key
order, clusters), on the host emulation of the ordering step: lists and
predecessors are in index order, and no block reads a group more often than it
has ranges of it to order."""
from __future__ import annotations

import shutil
import subprocess

import numpy as np
import pytest

from lslab_b200 import workload as W
from tests.test_emu import _build, _write_window

pytestmark = pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")

N, RANGE, BLOCKS = 150_000, 1024, 40


@pytest.fixture(scope="module")
def ranges(tmp_path_factory):
    return _build(tmp_path_factory.mktemp("emu") / "range_emu", "range_emu.cpp", False)


def members(name):
    """Op indices of one key's mutations."""
    rng = np.random.default_rng(53)
    if name == "burst":  # nearly all in a row at the window's end
        return np.concatenate([[0], np.arange(N - 5_000, N)])
    if name == "run":  # a batch in key order
        return np.arange(61_003, 91_004)
    if name == "trickle":  # evenly spread, and a burst
        return np.union1d(np.arange(0, N, 40), np.arange(120_001, 135_000))
    if name == "clusters":  # bursts of every size at growing distances
        at = np.concatenate([[2 ** i + np.arange(min(2 ** i, 700))] for i in range(17)], axis=None)
        return np.unique(np.concatenate([at, np.arange(N - 4_000, N)]))
    return np.sort(rng.permutation(N)[:30_000])  # even


@pytest.mark.parametrize("name", ["burst", "run", "trickle", "clusters", "even"])
def test_hot_key_read_once_per_range(ranges, tmp_path, name):
    m = members(name)
    t = np.zeros(N, np.uint8)
    k = W.key_of_rank(5, np.arange(N))
    t[m], k[m] = np.random.default_rng(59).choice([1, 2, 3], size=len(m)), 7
    path = tmp_path / "w.bin"
    _write_window(path, t, k, N)
    r = subprocess.run([str(ranges), str(path), "256", str(BLOCKS), "3"],
                       capture_output=True, text=True, timeout=900)
    assert r.returncode == 0 and r.stdout.startswith("OK"), r.stdout + r.stderr
    # one range a block (there are more blocks than ranges).  A short group's
    # range may hold all its members: the read that finds so, one of an empty
    # stretch and, per 3072 members, one that takes them and one that is cut
    # again.  A long group's ranges are even: the group once, the sample (256)
    # and one more read where a range holds more than its sort does.
    c = len(m)
    reads = 2 + 2 * -(-c // 3072) if c <= 16_384 else 2
    assert -(-c // RANGE) <= BLOCKS
    assert int(r.stdout.split("MOST")[1]) <= reads * c + 512, r.stdout
