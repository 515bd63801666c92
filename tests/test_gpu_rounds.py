"""Rounds over many tables in the walk form: warps enter and leave tables while
others take the last traversals, and every table equals training it alone."""
from __future__ import annotations

import pytest

from conftest import mccfr

L = mccfr.lib
pytestmark = pytest.mark.gpu


def _game(players, log2, seed):
    c = L.preset(L.PRESET_HU_20BB)
    c.num_players, c.table_log2, c.key_bits, c.seed = players, log2, log2, seed
    return c


def _make(cfgs, table):
    owner = mccfr.GPUCFRTrainer(config=cfgs[0])
    owner.set_hand_table(table)
    ts = [owner]
    for c in cfgs[1:]:
        t = mccfr.GPUCFRTrainer(config=c)
        t.share_hand_table(owner)
        ts.append(t)
    return ts


@pytest.mark.parametrize("tables,most", [(1, 1), (2, 40), (33, 3), (64, 9)])
def test_rounds_whose_tables_run_out_while_warps_enter(hand_table, tables, most):
    """A handful of traversals per table and many more warps than traversals: a
    warp meets tables whose last traversal another warp is taking at that moment."""
    cfgs = [_game(2 + i % 5, 12 + i % 4, 50 + i) for i in range(tables)]
    counts = [1 + (7 * i) % most for i in range(tables)]
    rounds, plain = _make(cfgs, hand_table), _make(cfgs, hand_table)
    for _ in range(12):
        mccfr.batch_round(rounds, counts)
    for t, c, n in zip(plain, cfgs, counts):
        for u in range(12):
            t.step(1 + u // c.num_players, u % c.num_players, n)
    for a, b, c in zip(rounds, plain, cfgs):
        assert a.digest() == b.digest(), c.num_players
        assert a.stats().node_visits == b.stats().node_visits
    for t in plain[::-1] + rounds[::-1]:
        t.close()


def test_a_round_on_a_device_short_of_memory(hand_table):
    """Node records for every resident warp do not fit: the round runs with fewer."""
    import torch

    cfgs = [_game(2, 14, 70), _game(6, 14, 71)]
    counts = [9000, 3000]
    rounds, plain = _make(cfgs, hand_table), _make(cfgs, hand_table)
    mccfr.batch_round(rounds, [3, 3])  # kernels loaded
    mccfr.batch_round(rounds, counts, {"block": 128})  # deals sized, by the form without node records
    for t, c, n in zip(plain, cfgs, counts):
        t.step(1, 0, 3)
        t.step(1, 1, n)
        t.step(1 + 2 // c.num_players, 2 % c.num_players, n)
    torch.cuda.init()
    held, chunk, left = [], 1 << 30, 32 << 20
    while chunk >= 8 << 20:
        if torch.cuda.mem_get_info()[0] < left + chunk:
            chunk //= 2
            continue
        try:
            held.append(torch.empty(chunk, dtype=torch.uint8, device="cuda"))
        except torch.OutOfMemoryError:
            chunk //= 2
    assert torch.cuda.mem_get_info()[0] < 64 << 20  # 87 MB of records do not fit
    try:
        mccfr.batch_round(rounds, counts)
    finally:
        held.clear()
        torch.cuda.empty_cache()
    for a, b in zip(rounds, plain):
        assert a.digest() == b.digest()
    for t in plain[::-1] + rounds[::-1]:
        t.close()
