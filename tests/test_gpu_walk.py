"""The walk form (an external-sampling update's default): bit-exact with the
oracle where its lists and pools are at their edges, and with the same level
counts as the level-synchronous form."""
from __future__ import annotations

import numpy as np
import pytest

import binding
from conftest import mccfr

L = mccfr.lib
pytestmark = pytest.mark.gpu


def _six(log2=21):
    c = L.preset(L.PRESET_6MAX_100BB)
    c.table_log2, c.key_bits = log2, log2 - 1
    return c


def _hu_probed():
    c = L.preset(L.PRESET_HU_20BB)
    c.table_log2, c.key_bits = 20, 0  # full 64-bit keys, open addressing
    return c


def _hu_cap(cap):
    c = L.preset(L.PRESET_HU_20BB)
    c.table_log2, c.key_bits, c.raise_cap = 20, 20, cap
    return c


def _thirds():
    """Three players, pot fractions with denominators that are no powers of two."""
    c = L.preset(L.PRESET_HU_20BB)
    c.num_players, c.starting_stack, c.table_log2, c.key_bits = 3, 12345, 20, 20
    slots = [(L.ACT_FOLD, 0, 1), (L.ACT_CHECK_CALL, 0, 1), (L.ACT_RAISE_MIN, 0, 1), (L.ACT_RAISE_POT, 1, 3),
             (L.ACT_RAISE_POT, 5, 7), (L.ACT_RAISE_POT, 16, 11), (L.ACT_ALL_IN, 0, 1)]
    c.num_actions = len(slots)
    for a, (k, n, d) in enumerate(slots):
        c.action_kind[a], c.action_num[a], c.action_den[a] = k, n, d
    return c


def _deep():
    """Eight slots and no raise cap: up to eight children per node, as many
    decisions as the depth cut allows."""
    c = L.preset(L.PRESET_REF8)
    c.sampling, c.max_depth = L.SAMPLING_EXTERNAL, 9
    return c


CASES = {
    "six-1": (_six, 1), "six-31": (_six, 31), "six-129": (_six, 129), "six-5000": (_six, 5000),
    "hu-probed-1000": (_hu_probed, 1000), "thirds-700": (_thirds, 700),
    "hu-cap6-28-decisions": (lambda: _hu_cap(6), 200), "hu-cap7-32-decisions": (lambda: _hu_cap(7), 200),
    "eight-slots-no-cap": (_deep, 64),
}


@pytest.mark.parametrize("name", CASES)
def test_walk_form_equals_oracle(hand_table, name):
    make, batch = CASES[name]
    cfg = make()
    tr, lv, orc = mccfr.GPUCFRTrainer(config=cfg), None, binding.Oracle(cfg, hand_table)
    tr.set_hand_table(hand_table)
    cfg.traversal_form = L.FORM_LEVELS
    lv = mccfr.GPUCFRTrainer(config=cfg)
    lv.set_hand_table(hand_table)
    for it in (1, 2, 3):
        for t in (tr, lv):
            t.train(1, batch, verbose=False)
        orc.train(1, batch, threads=1)
        assert tr.digest() == orc.digest(), it
        if lv.level_counts()["deferred"] == 0:
            assert tr.level_counts() == lv.level_counts(), it
    st, oc = tr.stats(), orc.counters()
    assert (st.traversals, st.node_visits, st.traverser_updates, st.terminals) == (
        oc["traversals"], oc["visits"], oc["updates"], oc["terminals"])
    for t in (tr, lv):
        t.close()
    orc.close()


def test_imported_regrets_are_sampled(hand_table):
    """Rows written from outside an update (a checkpoint) are sampled from like
    rows that training wrote: training on from them equals the oracle's."""
    cfg = _six(18)
    a = mccfr.GPUCFRTrainer(config=cfg)
    a.set_hand_table(hand_table)
    a.train(3, 2000, verbose=False)
    orc = binding.Oracle(cfg, hand_table)
    orc.import_rows(a.export_rows(), 3)
    import tempfile
    from pathlib import Path
    with tempfile.TemporaryDirectory() as d:
        f = Path(d) / "c.bin"
        a.save_checkpoint_v2(f)
        b = mccfr.GPUCFRTrainer(config=cfg)
        b.set_hand_table(hand_table)
        b.load_checkpoint_v2(f)
    b.train(1, 2000, verbose=False)
    for p in range(cfg.num_players):
        orc.step(4, p, 2000, threads=1)
    assert b.digest() == orc.digest()
    r = b.export_rows()
    assert np.count_nonzero(r["regrets"]) > 0
    a.close()
    b.close()
    orc.close()


@pytest.mark.parametrize("mixed", [False, True], ids=["path-hash-direct", "any-mix"])
@pytest.mark.parametrize("tuning", [None, {"block": 64, "grab": 2}], ids=["walk", "persistent"])
def test_rounds_of_uneven_tables_equal_plain(hand_table, mixed, tuning):
    """Rounds over tables of different games and sizes (with a probed table and a
    table of FNV slots among them: the general kernel), by the walk and by a tuned
    persistent kernel: every table equals the same updates trained alone."""
    cfgs = [_six(16), _hu_cap(2), _thirds()]
    if mixed:
        ref = L.preset(L.PRESET_REF8)
        ref.sampling, ref.max_depth, ref.table_log2 = L.SAMPLING_EXTERNAL, 9, 22
        cfgs += [_hu_probed(), ref]
    counts = [50, 1, 700, 33, 20][:len(cfgs)]

    def make():
        ts = []
        for c in cfgs:
            t = mccfr.GPUCFRTrainer(config=c)
            t.set_hand_table(hand_table)
            ts.append(t)
        return ts
    rounds, plain = make(), make()
    for _ in range(7):
        mccfr.batch_round(rounds, counts, tuning)
    for t, c, n in zip(plain, cfgs, counts):
        for u in range(7):
            t.step(1 + u // c.num_players, u % c.num_players, n)
    for a, b in zip(rounds, plain):
        assert a.digest() == b.digest()
        sa, sb = a.stats(), b.stats()
        assert (sa.traversals, sa.node_visits, sa.traverser_updates, sa.terminals) == (
            sb.traversals, sb.node_visits, sb.traverser_updates, sb.terminals)
    for t in rounds + plain:
        t.close()
