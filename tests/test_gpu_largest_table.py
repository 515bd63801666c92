"""Tables above 2^28 rows, whose runs of rows carry marks of their own: every form and
both rules equal the oracle over updates that touch few and many of the runs."""
from __future__ import annotations

import pytest

import binding
from conftest import mccfr

L = mccfr.lib
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def owner(hand_table):
    t = mccfr.GPUCFRTrainer(config=L.preset(L.PRESET_HU_20BB), table_log2=10)
    t.set_hand_table(hand_table)
    yield t
    t.close()


def _trainer(cfg, owner):
    t = mccfr.GPUCFRTrainer(config=cfg)
    t.share_hand_table(owner)
    return t


def _config(bits, sampling):
    c = L.preset(L.PRESET_HU_20BB)
    c.table_log2, c.key_bits, c.sampling = 29, bits, sampling
    if sampling == L.SAMPLING_REFERENCE:
        c.max_depth = 48
    return c


def _oracle(cfg, table):
    small = L.Config.from_buffer_copy(cfg)
    small.table_log2 = 24  # the same rows, found by probing
    return binding.Oracle(small, table)


@pytest.mark.parametrize("bits", [29, 0], ids=["direct", "probed"])
@pytest.mark.parametrize("form", ["reference", "walk", "lanes", "levels"])
def test_marked_runs_equal_oracle(hand_table, owner, form, bits):
    cfg = _config(bits, L.SAMPLING_REFERENCE if form == "reference" else L.SAMPLING_EXTERNAL)
    cfg.traversal_form = {"lanes": L.FORM_LANES, "levels": L.FORM_LEVELS}.get(form, L.FORM_AUTO)
    tr, orc = _trainer(cfg, owner), _oracle(cfg, hand_table)
    it = 0
    for batch in (1, 3000, 1, 40_000):
        it += 1
        tr.train(1, batch, verbose=False)
        orc.train(1, batch, threads=4)
        assert tr.digest() == orc.digest(), (it, batch)
    for p in range(2):
        tr.step(it + 1, p, 500)
        orc.step(it + 1, p, 500, threads=1)
    assert tr.digest() == orc.digest()
    tr.close()
    orc.close()


@pytest.mark.parametrize("tuning", [None, {"block": 128}], ids=["walk", "persistent"])
def test_rounds_with_and_without_marked_runs(hand_table, owner, tuning):
    """One table with marked runs and one without in a round, and in a batch."""
    cfgs, counts = [_config(0, L.SAMPLING_EXTERNAL), L.preset(L.PRESET_HU_20BB)], [700, 900]
    cfgs[1].table_log2 = cfgs[1].key_bits = 18
    ts, orcs = [_trainer(c, owner) for c in cfgs], [_oracle(c, hand_table) for c in cfgs]
    for _ in range(4):
        mccfr.batch_round(ts, counts, tuning)
    b = mccfr.Batch(ts, counts)
    b.set_tuning(form=L.BATCH_PERSISTENT if tuning else L.BATCH_TABLE_GRAPHS)
    b.train(2)
    for t, o, n in zip(ts, orcs, counts):
        o.train(4, n, threads=4)
        assert t.digest() == o.digest()
    b.close()
    for t in ts + orcs:
        t.close()
