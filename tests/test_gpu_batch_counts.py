"""Rows touched and folded wide of a table's last update: the same from a timed train()
of a table in a batch, whose graph is captured again around it, as from single steps."""
from __future__ import annotations

import pytest

from conftest import mccfr

L = mccfr.lib
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("big", [100, 9000])
def test_timed_training_between_batch_iterations_counts_its_rows(hand_table, big):
    def make():
        ts = []
        for n in (2, 3):
            c = L.preset(L.PRESET_HU_20BB)
            c.num_players, c.table_log2, c.key_bits, c.seed = n, 16, 15, n
            t = mccfr.GPUCFRTrainer(config=c)
            t.set_hand_table(hand_table)
            ts.append(t)
        return ts
    batched, plain = make(), make()
    trav = [700, 300]
    b = mccfr.Batch(batched, trav)
    for it in (1, 3):
        b.train(1)
        for t, n in zip(plain, trav):
            for p in range(t.config.num_players):
                t.step(it, p, n)
        for t, s in zip(batched, plain):
            t.train(1, big, verbose=False, timed=True)
            for p in range(t.config.num_players):
                s.step(it + 1, p, big)
            a, o = t.stats(), s.stats()
            assert (a.touched_last, a.wide_rows_last) == (o.touched_last, o.wide_rows_last)
            assert a.touched_last > a.wide_rows_last > 0
            assert t.digest() == s.digest()
    b.close()
    for t in batched + plain:
        t.close()
