"""The probe as separate joins and lookups, on the host emulation of the device
code under AddressSanitizer: results equal the oracle's replay."""
from __future__ import annotations

import shutil
import subprocess

import numpy as np
import pytest

from lslab_b200 import workload as W
from oracle import OracleMap
from tests.test_emu import CSRC, EMU, _write_window

pytestmark = pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")


@pytest.mark.parametrize("few", [False, True])
@pytest.mark.parametrize("sort", [False, True])
def test_split_probe_equals_the_oracle(tmp_path, few, sort):
    """Two windows, the second ending within a span; mutations of every type,
    in arrival order and sorted by type (spans without and of only mutations)."""
    exe = tmp_path / "split"
    subprocess.run(["g++", "-fsanitize=address", "-std=c++20", "-O1", "-g", "-pthread",
                    "-DLSB_HOST_EMU", *(["-DSPLIT_FEW"] if few else []), f"-I{EMU}", f"-I{CSRC}",
                    str(EMU / "split_emu.cpp"), "-o", str(exe)], check=True)
    n, window, log2 = 9_000, 6_007, 6
    rng = np.random.default_rng(31)
    t = rng.choice([0, 1, 2, 3], size=n, p=[0.7, 0.15, 0.05, 0.1]).astype(np.uint8)
    if sort:
        t = np.sort(t)
    k = W.key_of_rank(2, rng.integers(0, 300, size=n))
    k[rng.random(n) < 0.3] = np.uint64(77)
    v = W.splitmix64(13, 0, n)
    path, outp = tmp_path / "ops.bin", tmp_path / "out.bin"
    _write_window(path, t, k, window, v)
    want = OracleMap(log2).mixed(t, k, v)
    r = subprocess.run([str(exe), str(path), str(log2), str(4096), "256", str(outp)],
                       capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stdout + r.stderr[-4000:]
    raw = np.fromfile(outp, np.uint8)
    got = raw[: 16 * n].view(np.dtype([("found", "u1"), ("pad", "u1", (7,)), ("value", "<u8")]))
    assert int(raw[16 * n: 16 * n + 4].view(np.uint32)[0]) == 0
    assert np.array_equal(got["found"], want["found"])
    assert np.array_equal(got["value"], want["value"])
