"""The ordering's grid steps (groups too large for index ranges) on the host
emulation of the device code, in a build that takes them for every group of
more than 4096 members: the cases of test_emu, whose hot keys are below the
library's own limit."""
from __future__ import annotations

import shutil
import subprocess

import numpy as np
import pytest

from lslab_b200 import workload as W
from tests import test_emu as emu

pytestmark = pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")


@pytest.fixture(scope="module")
def bins(tmp_path_factory):
    d = tmp_path_factory.mktemp("emu")
    out = {}
    for name, flags in (("order", []), ("window", ["-fsanitize=address"])):
        out[name] = d / f"{name}_emu"
        subprocess.run(["g++", "-std=c++20", "-O1", "-g", "-pthread", "-DLSB_HOST_EMU",
                        "-DLSB_HUGE_STEPS=4096u", *flags, f"-I{emu.EMU}", f"-I{emu.CSRC}",
                        str(emu.EMU / f"{name}_emu.cpp"), "-o", str(out[name])], check=True)
    return out


@pytest.mark.parametrize("case", sorted(emu.ORDER))
def test_steps_match_index_order(bins, tmp_path, case):
    emu.test_ordering_matches_index_order(bins, tmp_path, case, 256, 3)


def test_steps_of_three_groups(bins, tmp_path, monkeypatch):
    """Three groups over the limit and one below it, of different spreads."""
    rng = np.random.default_rng(73)
    n = 40_000
    t = rng.choice([0, 1, 2, 3], size=n, p=[0.1, 0.3, 0.2, 0.4]).astype(np.uint8)
    k = W.key_of_rank(3, np.arange(n))
    k[rng.permutation(n)[:9_000]] = 1
    k[20_000:27_000] = 2
    k[rng.permutation(np.nonzero(k > 2)[0])[:3_000]] = 3
    k[rng.permutation(np.nonzero(k > 3)[0])[:8_000]] = 4
    monkeypatch.setitem(emu.ORDER, "three", (t, k, n))
    emu.test_ordering_matches_index_order(bins, tmp_path, "three", 256, 3)


@pytest.mark.parametrize("mode", ["tiles", "muts_first"])
def test_steps_whole_batch(bins, tmp_path, mode):
    emu.test_whole_batch_in_bounds_and_equal_to_oracle(bins, tmp_path, mode, 16_383)


def test_steps_update_runs(bins, tmp_path):
    emu.test_updates_in_bounds_and_equal_to_oracle(bins, tmp_path, "update_runs", "tiles", 16_384)
