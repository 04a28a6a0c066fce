"""Ordering of a window's groups at the sizes where its path changes (warp,
block, index ranges over several blocks, grid steps), on the host emulation of
the device code: every group's list and predecessors must be the index order.
tests/emu/order_emu.cpp does the checking."""
from __future__ import annotations

import shutil
import subprocess

import numpy as np
import pytest

from lslab_b200 import workload as W
from tests.test_emu import _build, _write_window

pytestmark = pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")


@pytest.fixture(scope="module")
def order(tmp_path_factory):
    return _build(tmp_path_factory.mktemp("emu") / "order_emu", "order_emu.cpp", False)


def _case(name):
    rng = np.random.default_rng(29)
    n, window = 50_000, 1 << 16
    t = np.zeros(n, np.uint8)
    k = W.key_of_rank(5, np.arange(n))

    def group(key, members):  # mutations of one key at these indices
        t[members], k[members] = rng.choice([1, 2, 3], size=len(members)), key

    if name == "edges":  # one group on each side of every limit, spread out
        at = rng.permutation(n)
        for key, c in enumerate((8, 9, 64, 65, 1024, 1025, 4095, 4096, 4097, 8193)):
            group(key, at[:c])
            at = at[c:]
    elif name == "packed":  # a range holds far more than its share of a group
        group(1, np.concatenate([[3], np.arange(20_000, 32_000), [n - 1]]))
        group(2, np.concatenate([np.arange(32_000, 36_096), [0]]))
    elif name == "late":  # every mutation in the last part of the window
        group(1, np.sort(rng.choice(np.arange(45_000, n), 4_500, replace=False)))
        group(2, np.setdiff1d(np.arange(45_000, n), np.nonzero(t)[0]))
    else:  # past the grid steps' limit, beside a group that is not
        n, window = 150_000, 150_001
        t = np.ones(n, np.uint8)
        k = np.full(n, 1, np.uint64)
        group(2, rng.permutation(n)[:n - 131_073])
    return t, k, window


@pytest.mark.parametrize("name", ["edges", "packed", "late", "steps"])
@pytest.mark.parametrize("threads,blocks", [(128, 5), (512, 2)])
def test_ordering_at_path_limits(order, tmp_path, name, threads, blocks):
    t, k, window = _case(name)
    path = tmp_path / "w.bin"
    _write_window(path, t, k, window)
    r = subprocess.run([str(order), str(path), str(threads), str(blocks), "3"],
                       capture_output=True, text=True, timeout=900)
    assert r.returncode == 0 and r.stdout.startswith("OK"), r.stdout + r.stderr
