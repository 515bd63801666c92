"""Raises of a pot fraction as the host's best response computes them: the floor of
num * pot / den for every pot that fits the product in 31 bits."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

from conftest import PKG_DIR

SRC = Path(__file__).with_name("raise_target_main.cu")


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    exe = tmp_path_factory.mktemp("raise") / "raise"
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    subprocess.run([nvcc, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", str(SRC),
                    f"-I{PKG_DIR / 'csrc'}", "-o", str(exe)], check=True)
    return exe


def test_targets_are_floors(harness):
    rng = np.random.default_rng(0)
    cases = [(1, 1, 0, 0, 1), (1, 2, 1, 5, 9), (16, 32767, 134_217_727, 100, 300), (16, 1, 134_217_727, 0, 1),
             (16, 32767, 67_137_535, 0, 1),
             (3, 65536, 100, 7, 8)]  # the last denominator does not fit its field: no fraction
    for den in (1, 2, 3, 7, 11, 16384, 16385, 32766, 32767):
        for num in (1, 5, 16):
            top = (2**31 - 1) // num
            pots = [top, top - 1, 6 * 65535, 2**30 // num + 1] + [int(x) for x in rng.integers(0, top, 200)]
            # products just below a multiple of den, where a quotient is first rounded up
            pots += [den * (product // den) // num - 1 for product in (2**30 + 2 * den, 3 * 2**29, 2**31 - 1)]
            for pot in pots:
                if num * pot // den < 2**30:
                    cases.append((num, den, pot, int(rng.integers(0, 65536)), int(rng.integers(1, 65536))))
    text = "\n".join(" ".join(map(str, c)) for c in cases) + "\n"
    out = subprocess.run([str(harness)], input=text, check=True, capture_output=True, text=True).stdout.split()
    assert len(out) == len(cases)
    for (num, den, pot, cb, mrt), got in zip(cases, out):
        frac = num * pot // den if den < 32768 else 0
        assert int(got) == max(mrt, cb + max(1, frac)), (num, den, pot)
