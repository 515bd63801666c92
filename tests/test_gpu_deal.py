"""The deal kernels at their edges: subgame deals (eight lanes per traversal)
whose draws mostly or always collide, for every player count and both streets,
and full-game deals at block edges, against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

import binding
from conftest import mccfr
from mccfr_b200 import serving

L = mccfr.lib
pytestmark = pytest.mark.gpu


def _subgame(street, players, combos, seed):
    """A request whose players share one range over `combos` hole combos that
    hold only the first `combos`-odd free cards, so that draws collide often
    (with few combos and many players, always)."""
    rng = np.random.default_rng(seed)
    req = serving.make_request(rng, 7)
    board = [int(c) for c in rng.permutation(52)[: street + 2]]
    free = np.flatnonzero(~np.isin(serving.COMBO_CARDS, board).any(axis=1))
    ranges = np.zeros((players, 1326), np.float32)
    ranges[:, free[:combos]] = rng.random((players, combos)).astype(np.float32) + 0.01
    req.street, req.players, req.board, req.ranges, req.pot = street, players, board, ranges, 600 // players * players
    req.table_log2 = 16
    return req


@pytest.mark.parametrize("street", [2, 3])
@pytest.mark.parametrize("players,combos,batch", [(2, 1, 33), (2, 900, 1000), (3, 10, 130), (4, 40, 17), (5, 60, 257),
                                                  (6, 70, 300), (6, 900, 1)])
def test_colliding_subgame_deals_equal_oracle(hand_table, street, players, combos, batch):
    req = _subgame(street, players, combos, 100 * street + players)
    cfg = serving.request_config(req)
    tr = mccfr.GPUCFRTrainer.subgame(cfg, req.street, req.pot, req.board, req.ranges)
    tr.set_hand_table(hand_table)
    orc = binding.Oracle(cfg, hand_table, subgame={"street": req.street, "pot": req.pot, "board": req.board,
                                                   "ranges": req.ranges})
    tr.train(2, batch, verbose=False)
    orc.train(2, batch, threads=1)
    assert tr.digest() == orc.digest()
    # the same deals through the batched kernel
    bt = mccfr.GPUCFRTrainer.subgame(cfg, req.street, req.pot, req.board, req.ranges)
    bt.set_hand_table(hand_table)
    for _ in range(2 * players):
        mccfr.batch_round([bt], [batch])
    assert bt.digest() == tr.digest()
    for t in (tr, bt):
        t.close()
    orc.close()


@pytest.mark.parametrize("players", [2, 3, 4, 5, 6])
@pytest.mark.parametrize("batch", [1, 127, 129])
def test_full_game_deals_equal_oracle(hand_table, players, batch):
    """Every dealt card, bucket, dealer and payoff of one update of the reference game."""
    cfg = L.preset(L.PRESET_REF8)
    cfg.num_players, cfg.table_log2 = players, 16
    tr = mccfr.GPUCFRTrainer(config=cfg)
    tr.set_hand_table(hand_table)
    orc = binding.Oracle(cfg, hand_table)
    g = tr.step(1, 0, batch, trace=True)
    o = orc.step(1, 0, batch, trace=True, trace_dtype=L.TRACE_DTYPE)
    for f in ("hole", "board", "dealer", "hole_bucket", "board_bucket", "n_actions", "actions"):
        assert np.array_equal(g[f], o[f]), f
    assert np.array_equal(g["payoff"].view(np.uint32), o["payoff"].view(np.uint32))
    tr.close()
    orc.close()


def test_deals_beyond_one_grid_equal_oracle(hand_table):
    """More traversals than the deal's grid has threads: each thread deals several."""
    cfg = L.preset(L.PRESET_HU_20BB)
    cfg.table_log2, cfg.key_bits = 18, 17
    tr = mccfr.GPUCFRTrainer(config=cfg)
    tr.set_hand_table(hand_table)
    orc = binding.Oracle(cfg, hand_table)
    batch = 148 * 16 * 128 + 777
    tr.step(1, 0, batch)
    orc.step(1, 0, batch)
    assert tr.digest() == orc.digest()
    tr.close()
    orc.close()
