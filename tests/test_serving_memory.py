"""What the re-solve server counts for a table covers what its handle holds: on the
host by the sizes, on the GPU by the device's free memory."""
from __future__ import annotations

import importlib

import numpy as np
import pytest

from conftest import mccfr

L = mccfr.lib
sv = importlib.import_module("mccfr_b200.serving")


@pytest.mark.parametrize("log2", range(10, 23))
def test_counted_bytes_cover_rows_bitmaps_and_kept_scratch(log2):
    req = sv.make_request(np.random.default_rng(0), 0)
    req.table_log2 = log2
    rows = 1 << log2
    keys = 1 << sv.request_config(req).key_bits
    export = keys * (4 + 32)
    scratch = max(export + export // 4, 1 << 20)
    luts = 22400 + 32487834 // 53 + 52 * 52 + 6 * 1326 * 4
    assert sv.table_bytes(req) >= rows * 256 + rows // 4 + scratch + luts
    srv = sv.ReSolveServer(None)
    srv.pool = {log2: [None, None], 12: [None]}
    req.table_log2 = 12
    assert srv.pooled_bytes() == (2 * sv.capacity_bytes(log2) + sv.table_bytes(req) if log2 != 12
                                  else sv.table_bytes(req))


@pytest.mark.parametrize("log2", [10, 14, 21])
def test_a_table_that_fits_the_budget_is_served_alone(log2):
    """The budget holds the table but not the scratch that it may leave: accepted on
    an idle server (pooled tables freed for it), not beside another one."""
    req = sv.make_request(np.random.default_rng(1), 0)
    req.table_log2 = log2
    own = (1 << log2) * 260 + (1 << 20)
    assert own < sv.table_bytes(req)
    for budget in (own, sv.table_bytes(req) - 1):
        srv = sv.ReSolveServer(None, hbm_budget=budget, free_memory=lambda: own + (1 << 30))
        assert srv.admit_ok(req, 0, 0)
        assert not srv.admit_ok(req, 1, 1)
        assert not sv.ReSolveServer(None, hbm_budget=own - 1, free_memory=lambda: 1 << 40).admit_ok(req, 0, 0)
        assert not sv.ReSolveServer(None, hbm_budget=budget, free_memory=lambda: own + (1 << 30) - 1).admit_ok(req, 0, 0)

        class Pooled:
            closed = False

            def close(self):
                self.closed = True

        other = Pooled()
        srv.pool[9] = [other]
        assert srv.admit_ok(req, 0, 0) and other.closed


@pytest.mark.gpu
@pytest.mark.parametrize("log2", [18, 20])
def test_device_memory_of_solved_tables_is_counted(hand_table, log2):
    """Six solved tables with every key in use, their strategies read."""
    import torch

    owner = mccfr.GPUCFRTrainer(config=L.preset(L.PRESET_HU_20BB), table_log2=10)
    owner.set_hand_table(hand_table)
    rng = np.random.default_rng(log2)

    def solve(i):
        req = sv.make_request(rng, i)
        req.street, req.players, req.table_log2 = 2, 6, log2
        req.board = [int(c) for c in rng.permutation(52)[:4]]
        req.ranges, req.pot = np.ones((6, 1326), np.float32), 1200
        t = mccfr.GPUCFRTrainer.subgame(sv.request_config(req), 2, req.pot, req.board, req.ranges)
        t.share_hand_table(owner)
        for _ in range(6):
            mccfr.batch_round([t], [60_000])
        keys, _ = t.strategy_arrays()
        return t, t.rows_used(), keys.size, sv.table_bytes(req)

    first = solve(0)  # kernels and the rounds' shared buffers
    before = torch.cuda.mem_get_info()[0]
    solved = [solve(i) for i in range(1, 7)]
    held = before - torch.cuda.mem_get_info()[0]
    assert all(rows > 0.95 * (1 << (log2 - 1)) for _, rows, _, _ in solved)
    assert held <= sum(counted for _, _, _, counted in solved)
    for t, *_ in [first] + solved:
        t.close()
    owner.close()
