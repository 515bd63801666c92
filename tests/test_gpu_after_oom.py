"""A call that found no device memory leaves nothing behind: the next one, which needs
less, runs and gives the rows of a trainer that never met the shortage."""
from __future__ import annotations

import pytest
import torch

from conftest import mccfr

L = mccfr.lib
pytestmark = pytest.mark.gpu
OUT_OF_MEMORY = 3  # MCCFR_ERR_OOM
MANY = 1 << 26  # traversals whose deals alone take 4 GB


def _make(hand_table):
    c = L.preset(L.PRESET_HU_20BB)
    c.table_log2 = c.key_bits = 14
    t = mccfr.GPUCFRTrainer(config=c)
    t.set_hand_table(hand_table)
    return t


def _big_table(t):
    c = L.preset(L.PRESET_HU_20BB)
    c.table_log2 = 24  # 4.3 GB
    mccfr.GPUCFRTrainer(config=c)


@pytest.fixture
def two_gigabytes_free():
    held = []
    while (free := torch.cuda.mem_get_info()[0]) > 2 << 30:
        held.append(torch.empty(min(8 << 30, free - (2 << 30) + (2 << 20)), dtype=torch.uint8, device="cuda"))
    yield
    held.clear()
    torch.cuda.empty_cache()


CALLS = {
    "train": lambda t: t.train(1, MANY, verbose=False),
    "step": lambda t: t.step(1, 0, MANY),
    "round": lambda t: mccfr.batch_round([t], [MANY]),
    "batch": lambda t: mccfr.Batch([t], [MANY]),
    "create": _big_table,
}


@pytest.mark.parametrize("call", list(CALLS))
@pytest.mark.parametrize("then", ["train", "round"])
def test_the_call_after_an_allocation_that_failed(hand_table, two_gigabytes_free, call, then):
    t, plain = _make(hand_table), _make(hand_table)
    with pytest.raises(L.MccfrError) as e:
        CALLS[call](t)
    assert e.value.status == OUT_OF_MEMORY
    for x in (t, plain):
        if then == "train":
            x.train(1, 500, verbose=False)
        else:
            mccfr.batch_round([x], [500])
    assert t.digest() == plain.digest()
    t.close()
    plain.close()
