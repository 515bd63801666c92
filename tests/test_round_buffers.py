"""The buffers that a device's rounds share: after any failing call of their set-up
none is left half made, and the next round makes them all."""
from __future__ import annotations

import subprocess
from pathlib import Path

import pytest

from conftest import PKG_DIR
from test_block_pool import OOM, cuda_include

SRC = Path(__file__).with_name("round_buffers_main.cpp")


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    exe = tmp_path_factory.mktemp("round") / "round"
    subprocess.run(["g++", "-O1", "-std=c++17", str(SRC), f"-I{PKG_DIR / 'csrc'}", f"-I{cuda_include()}", "-o",
                    str(exe)], check=True)
    return exe


@pytest.mark.parametrize("fail", range(6))
def test_set_up_is_whole_or_nothing(harness, fail):
    out = subprocess.run([str(harness), str(fail)], check=True, capture_output=True, text=True).stdout.splitlines()
    first, second, end = [tuple(map(int, ln.split())) for ln in out]
    assert first == ((OOM, 0, 0, 0) if fail else (0, 5, 5, 0))
    assert second == (0, 5, 5, 0)
    assert end == (0,)
