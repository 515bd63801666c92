"""Reading a table back: rows and strategies come out in ascending key order at
the span edges of the read kernels, from direct-mapped and probed tables, and equal
the oracle's; sizes and capacities as declared."""
from __future__ import annotations

import ctypes
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

import binding
from conftest import mccfr

L = mccfr.lib
pytestmark = pytest.mark.gpu


def _cfg(log2, bits, sampling=1):
    c = L.preset(L.PRESET_6MAX_100BB)
    c.table_log2, c.key_bits, c.sampling = log2, bits, sampling
    if sampling == 0:
        c.max_depth = 64
    return c


@pytest.mark.parametrize("log2,bits,batch", [(10, 1, 3), (10, 5, 40), (10, 10, 300), (12, 11, 500), (16, 13, 2000),
                                             (20, 0, 50)])
@pytest.mark.parametrize("sampling", [0, 1])
def test_rows_and_strategies_equal_oracle(hand_table, log2, bits, batch, sampling):
    cfg = _cfg(log2, bits, sampling)
    tr = mccfr.GPUCFRTrainer(config=cfg)
    tr.set_hand_table(hand_table)
    orc = binding.Oracle(cfg, hand_table)
    assert tr.export_rows()["keys"].size == 0 and tr.strategy_arrays()[0].size == 0
    tr.train(2, batch, verbose=False)
    orc.train(2, batch, threads=1)
    g, o = tr.export_rows(), orc.export_rows()
    for f in ("keys", "visits", "regrets", "strategy_sum"):
        assert np.array_equal(g[f].view(np.uint8), np.asarray(o[f]).view(np.uint8)), f
    assert np.all(np.diff(g["keys"].astype(np.int64)) > 0)
    assert tr.rows_used() == g["keys"].size and tr.digest() == orc.digest()
    assert tr.num_info_sets_active() == int((o["strategy_sum"] > 0).any(axis=1).sum())
    # the strategy: sums divided in slot order, rows without one left out
    s = np.asarray(o["strategy_sum"], np.float32)
    tot = np.zeros(len(s), np.float32)
    for a in range(8):
        tot = tot + s[:, a]
    with np.errstate(all="ignore"):
        p = np.where(tot[:, None] > np.float32(1e-7), s / tot[:, None], np.float32(0))
    t2 = np.zeros(len(s), np.float32)
    for a in range(8):
        t2 = t2 + p[:, a]
    keep = ~(t2 < np.float32(1e-6))
    keys, probs = tr.strategy_arrays()
    assert np.array_equal(keys, o["keys"][keep].astype(np.uint32))
    assert np.array_equal(probs.view(np.uint32), p[keep].view(np.uint32))
    # a capacity below the rows: refused, with their number; null arrays are skipped
    n = ctypes.c_size_t()
    lib = L.load()
    if g["keys"].size > 1:
        one = np.zeros(1, np.uint64)
        assert lib.mccfr_export_rows(tr.handle, L.ptr(one), None, None, None, 1, ctypes.byref(n)) == L.ERR_CAPACITY
        assert n.value == g["keys"].size
    vis = np.zeros(g["keys"].size + 1, np.uint64)
    assert lib.mccfr_export_rows(tr.handle, None, None, None, L.ptr(vis), vis.size, ctypes.byref(n)) == L.OK
    assert np.array_equal(vis[:n.value], g["visits"]) and vis[-1] == 0
    tr.close()
    orc.close()


@pytest.mark.parametrize("n", [1, 15, 16, 17, 1000, 150_001])
def test_eval7_staging_sizes(hand_table, n):
    """Calls of different sizes on one handle share its scratch."""
    cfg = _cfg(10, 10)
    tr = mccfr.GPUCFRTrainer(config=cfg)
    tr.set_hand_table(hand_table)
    rng = np.random.default_rng(n)
    for m in (n, max(1, n // 2), 2 * n):
        cards = rng.random((m, 52)).argpartition(7, axis=1)[:, :7].astype(np.uint8)
        assert np.array_equal(tr.eval7(cards), binding.eval7(hand_table, cards))
    bad = np.zeros((n, 7), np.uint8)
    bad[:] = np.arange(7)
    bad[n - 1, 6] = 52
    with pytest.raises(mccfr.MccfrError, match="52"):
        tr.eval7(bad)
    tr.close()


@pytest.mark.parametrize("threads", [2, 6])
def test_reads_of_one_handle_from_several_threads(hand_table, threads):
    """Rows, strategies and staged hands of one handle, read by several threads at
    once: each gets what it gets alone, though the reads share the handle's scratch."""
    tr = mccfr.GPUCFRTrainer(config=_cfg(16, 13))
    tr.set_hand_table(hand_table)
    tr.train(2, 2000, verbose=False)
    rng = np.random.default_rng(threads)
    hands = [rng.random((m, 52)).argpartition(7, axis=1)[:, :7].astype(np.uint8) for m in (16, 9_001, 150_001)]
    ranks = [binding.eval7(hand_table, c) for c in hands]
    rows, strat, active = tr.export_rows(), tr.strategy_arrays(), tr.num_info_sets_active()

    def read(i):
        for k in range(12):
            w = (i + k) % 4
            if w == 0:
                c = (i + k) // 4 % 3
                assert np.array_equal(tr.eval7(hands[c]), ranks[c])
            elif w == 1:
                got = tr.export_rows()
                assert all(np.array_equal(got[f].view(np.uint8), rows[f].view(np.uint8)) for f in rows)
            elif w == 2:
                assert all(np.array_equal(a.view(np.uint8), b.view(np.uint8)) for a, b in
                           zip(tr.strategy_arrays(), strat))
            else:
                assert tr.num_info_sets_active() == active

    with ThreadPoolExecutor(threads) as pool:
        list(pool.map(read, range(threads)))
    tr.close()
