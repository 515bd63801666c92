"""The pool of node records on a device short of memory, over an allocator that fails:
fewer blocks are taken, a repeated call keeps what it got, nothing is lost."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

from conftest import PKG_DIR

SRC = Path(__file__).with_name("block_pool_main.cpp")
OOM = 2  # cudaErrorMemoryAllocation


def cuda_include() -> Path:
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    return Path(nvcc).resolve().parent.parent / "include"


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    exe = tmp_path_factory.mktemp("pool") / "pool"
    subprocess.run(["g++", "-O1", "-std=c++17", str(SRC), f"-I{PKG_DIR / 'csrc'}", f"-I{cuda_include()}", "-o",
                    str(exe)], check=True)

    def run(*args):
        out = subprocess.run([str(exe), *map(str, args)], check=True, capture_output=True, text=True).stdout
        lines = [tuple(int(x) for x in ln.split()) for ln in out.splitlines()]
        assert lines[-1] == (0, 0)  # all given back, no error left behind
        return lines[:-1]
    return run


@pytest.mark.parametrize("room,requests,expect", [
    (10_000, [8, 8, 3, 20], [(0, 8, 1), (0, 8, 1), (0, 8, 1), (0, 20, 2)]),
    # 64 -> 32 -> 16 -> 8 blocks; the same and smaller requests keep them
    (1_000, [64, 64, 64, 9], [(0, 8, 4), (0, 8, 4), (0, 8, 4), (0, 8, 4)]),
    (1_000, [64, 65], [(0, 8, 4), (0, 9, 8)]),  # a larger one tries again: 65, 33, 17, 9
    (128, [5, 5], [(0, 1, 4), (0, 1, 4)]),      # 5, 3, 2, 1
    (127, [2, 2], [(OOM, 0, 2), (OOM, 0, 4)]),
    (127, [2, "r5000", 2, 2], [(OOM, 0, 2), (0, 2, 3), (0, 2, 3)]),  # a failed one is tried anew
])
def test_pool_takes_what_there_is_and_keeps_it(harness, room, requests, expect):
    assert harness(room, *requests) == expect
