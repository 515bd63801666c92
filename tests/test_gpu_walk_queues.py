"""The walk's queue of visits off a row's canonical mask: key spaces so small that
most visits share their row with states of other legal actions, bit-exact with the
oracle for full and partly full queues."""
from __future__ import annotations

import pytest

import binding
from conftest import mccfr

L = mccfr.lib
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [1, 4, 8])
@pytest.mark.parametrize("players,batch", [(2, 3000), (6, 1), (6, 33), (6, 2000)])
def test_visits_off_the_canonical_mask_equal_oracle(hand_table, bits, players, batch):
    cfg = L.preset(L.PRESET_6MAX_100BB)
    cfg.num_players, cfg.table_log2, cfg.key_bits = players, 10, bits
    tr, orc = mccfr.GPUCFRTrainer(config=cfg), binding.Oracle(cfg, hand_table)
    tr.set_hand_table(hand_table)
    for it in (1, 2, 3):
        tr.train(1, batch, verbose=False)
        orc.train(1, batch, threads=1)
        assert tr.digest() == orc.digest(), it
    tr.close()
    orc.close()
