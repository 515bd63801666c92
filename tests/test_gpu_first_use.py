"""A handle used the moment it exists: its table's clearing and its copies are done
before the first update on any stream reads them."""
from __future__ import annotations

import pytest

import binding
from conftest import mccfr

L = mccfr.lib
pytestmark = pytest.mark.gpu


def _reference_rule():
    return L.preset(L.PRESET_REF8)  # 2^26 rows, clearing takes milliseconds; no copy follows a share


def _external():
    c = L.preset(L.PRESET_HU_20BB)
    c.table_log2, c.key_bits = 26, 26
    return c


@pytest.mark.parametrize("rounds", [False, True], ids=["train", "round"])
@pytest.mark.parametrize("make", [_reference_rule, _external], ids=["ref8", "hu"])
def test_training_right_after_creation_equals_oracle(hand_table, make, rounds):
    small = make()
    small.table_log2 = 20
    owner = mccfr.GPUCFRTrainer(config=small)
    owner.set_hand_table(hand_table)
    cfg = make()
    if rounds:
        cfg.sampling, cfg.max_depth = L.SAMPLING_EXTERNAL, min(cfg.max_depth, 9)
    orc = binding.Oracle(cfg, hand_table)
    orc.train(1, 300, threads=1)
    for _ in range(2):  # the second table lies where the first one left its rows
        tr = mccfr.GPUCFRTrainer(config=cfg)
        tr.share_hand_table(owner)
        if rounds:
            for _ in range(cfg.num_players):
                mccfr.batch_round([tr], [300])
        else:
            tr.train(1, 300, verbose=False)
        assert tr.digest() == orc.digest()
        tr.close()
    owner.close()
    orc.close()
