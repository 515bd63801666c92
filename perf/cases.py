"""Performance cases: what a user of this trainer has it do, through its public
entry points.

  listed()             the cases, plain dicts
  draw(rng)            one more case of the same ranges
  prepare(case, seed)  trainers, tables, requests and buffers on the GPU
  run(state)           one pass; returns what it computed
  work(case)           bytes a pass cannot do without
  exact(case, seed)    None: see there

Kinds of pass:
  train     GPUCFRTrainer.train(iters, batch) on a trainer that has already begun
            its run, then what such a program reads next: the average strategy or
            the rows into its own arrays, or, for a table of many GB, which no
            program copies out between iterations, the 64-bit digest over every
            bit of every row and the counters of its work
  resolve   one subgame re-solve on a kept trainer: reset_subgame, train, strategy
  serve     ReSolveServer.run on a burst of requests, every strategy returned
  batch     Batch.train over uneven tables, every table's rows returned
  eval      GPUCFRTrainer.eval7 on hands in host memory
  showdown  the device showdown kernels: 7-card hands dealt and ranked, and
            six-seat winner masks
"""
from __future__ import annotations

import ctypes
import importlib
import math

import numpy as np
import torch

import __graft_entry__

mccfr = __graft_entry__.load_package()
L = mccfr.lib
serving = importlib.import_module("mccfr_b200.serving")

# Action slots (kind, numerator, denominator of the pot) by number of actions.
ACTIONS = {
    3: [(L.ACT_FOLD, 0, 1), (L.ACT_CHECK_CALL, 0, 1), (L.ACT_ALL_IN, 0, 1)],
    4: [(L.ACT_FOLD, 0, 1), (L.ACT_CHECK_CALL, 0, 1), (L.ACT_RAISE_POT, 1, 1), (L.ACT_ALL_IN, 0, 1)],
    5: [(L.ACT_FOLD, 0, 1), (L.ACT_CHECK_CALL, 0, 1), (L.ACT_RAISE_POT, 1, 2), (L.ACT_RAISE_POT, 1, 1),
        (L.ACT_ALL_IN, 0, 1)],
    6: [(L.ACT_FOLD, 0, 1), (L.ACT_CHECK_CALL, 0, 1), (L.ACT_RAISE_POT, 1, 2), (L.ACT_RAISE_POT, 1, 1),
        (L.ACT_RAISE_POT, 2, 1), (L.ACT_ALL_IN, 0, 1)],
}


def listed() -> list[dict]:
    return [
        # The smallest re-solve a server is asked for: a heads-up river spot with the
        # least budget (2 updates per player); latency and launches count.
        {"name": "resolve-river-2p", "kind": "resolve", "street": 3, "players": 2, "sizes": 3, "budget": 2000,
         "table_log2": 16},
        # A large one: six players on the turn (the river card is dealt), five bet sizes.
        {"name": "resolve-turn-6p", "kind": "resolve", "street": 2, "players": 6, "sizes": 5, "budget": 20000,
         "table_log2": 20},
        # A burst at the re-solve server: 20 requests of the serving workload, solved
        # together by continuous batching, strategies exported by two workers.
        {"name": "serve-burst-20", "kind": "serve", "requests": 20, "traversals": 1024},
        # A small heads-up study: a ragged batch, full 64-bit keys in a probed table.
        {"name": "train-hu-small-64bit-keys", "kind": "train", "game": "hu", "rule": "external", "batch": 1000,
         "iters": 50, "table_log2": 24, "key_bits": 0, "warm": 20, "out": "digest"},
        # The heads-up 20BB preset at the trainer's default batch.
        {"name": "train-hu-20bb", "kind": "train", "game": "hu", "rule": "external", "batch": 65536, "iters": 50,
         "table_log2": 27, "key_bits": 26, "warm": 50, "out": "digest"},
        # 6-max 100BB at the default batch with a reduced key space, all rows read back
        # every 20 iterations.
        {"name": "train-6max-64k", "kind": "train", "game": "six", "rule": "external", "batch": 65536, "iters": 20,
         "table_log2": 20, "key_bits": 20, "warm": 4, "out": "rows"},
        # The headline: 6-max 100BB, 2^20 traversals per player-update, the preset's
        # 2^27-row table, one iteration (six updates) per call.
        {"name": "train-6max-headline", "kind": "train", "game": "six", "rule": "external", "batch": 1 << 20,
         "iters": 1, "table_log2": 27, "key_bits": 26, "warm": 5, "out": "digest"},
        # The drop-in default: the reference's constructor defaults (heads-up, its
        # update rule, FNV slots) at its default batch.
        {"name": "train-ref8-hu", "kind": "train", "game": "ref8", "players": 2, "rule": "reference", "batch": 65536,
         "iters": 100, "table_log2": 26, "key_bits": 0, "warm": 10, "out": "digest"},
        # The reference's update rule on the 6-max preset, the average strategy read
        # every 50 iterations.
        {"name": "train-6max-refrule", "kind": "train", "game": "six", "rule": "reference", "batch": 1 << 18,
         "iters": 50, "table_log2": 19, "key_bits": 18, "warm": 5, "out": "strategy"},
        # Several uneven tables (2-6 players, 10-200BB, 3-6 actions) trained as one batch.
        {"name": "batch-16-uneven", "kind": "batch", "tables": 16, "batch": 4096, "iters": 10, "table_log2": 17},
        # A hundred thousand 7-card hands from a host program.
        {"name": "eval7-host-100k", "kind": "eval", "hands": 100_003},
        # Showdown evaluation on the device: 2^24 dealt 7-card hands and 2^22 six-seat deals.
        {"name": "showdown-16m", "kind": "showdown", "hands": 1 << 24, "deals": 1 << 22},
    ]


def _logint(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    k = rng.choice(["resolve", "resolve", "serve", "train", "train", "train", "train", "batch", "eval", "showdown"])
    if k == "resolve":
        players, budget = rng.randint(2, 6), _logint(rng, 2000, 30000)
        return {"kind": k, "street": rng.choice([2, 3]), "players": players, "sizes": rng.randint(3, 5),
                "budget": budget, "table_log2": int(min(20, max(14, math.ceil(math.log2(budget * players * 16)))))}
    if k == "serve":
        return {"kind": k, "requests": rng.randint(3, 20), "traversals": rng.choice([256, 512, 1000, 1024])}
    if k == "batch":
        return {"kind": k, "tables": rng.randint(2, 16), "batch": _logint(rng, 1000, 8000), "iters": rng.randint(2, 10),
                "table_log2": rng.randint(14, 17)}
    if k == "eval":
        return {"kind": k, "hands": _logint(rng, 1, 2_000_000)}
    if k == "showdown":
        return {"kind": k, "hands": _logint(rng, 1000, 1 << 24), "deals": _logint(rng, 1000, 1 << 22)}
    game = rng.choice(["hu", "hu", "six", "six", "ref8", "mixed"])
    log2 = rng.randint(16, 20)
    c = {"kind": "train", "game": game, "rule": "external", "batch": _logint(rng, 300, 1 << 18), "table_log2": log2,
         "key_bits": log2 - rng.choice([0, 1]), "warm": rng.randint(1, 5), "out": rng.choice(["strategy", "rows"])}
    if game == "ref8":
        c.update(players=rng.choice([2, 3, 6]), rule="reference", table_log2=26, key_bits=0, out="digest")
    elif game == "mixed":
        c.update(players=rng.randint(2, 6), stack_bb=rng.randint(10, 200), actions=rng.choice([3, 4, 5, 6]))
    elif rng.random() < 0.25:
        c["rule"] = "reference"
    # up to as much work per pass as the listed cases of these batches
    c["iters"] = max(1, min(100, (1 << 20) // c["batch"]))
    return c


def _config(case: dict, seed: int) -> "L.Config":
    game = case["game"]
    if game == "ref8":
        c = L.preset(L.PRESET_REF8)
        c.num_players = case["players"]
    elif game == "six":
        c = L.preset(L.PRESET_6MAX_100BB)
    else:
        c = L.preset(L.PRESET_HU_20BB)
        if game == "mixed":
            c.num_players, c.starting_stack = case["players"], case["stack_bb"] * c.big_blind
            _set_actions(c, ACTIONS[case["actions"]])
            c.raise_cap = 3
    if game != "ref8":
        c.key_bits = case["key_bits"]
        c.sampling = L.SAMPLING_REFERENCE if case["rule"] == "reference" else L.SAMPLING_EXTERNAL
        if case["rule"] == "reference":
            c.max_depth = 64
    c.table_log2 = case["table_log2"]
    c.seed = seed
    return c


def _set_actions(c, slots) -> None:
    c.num_actions = len(slots)
    for a, (k, n, d) in enumerate(slots):
        c.action_kind[a], c.action_num[a], c.action_den[a] = k, n, d


def _trainer(cfg):
    t = mccfr.GPUCFRTrainer(config=cfg)
    t.set_hand_table(L.hand_table())
    return t


def _owner():
    """Holds the rank table that re-solve and batch trainers share."""
    return _trainer_small(L.preset(L.PRESET_HU_20BB))


def _trainer_small(cfg):
    cfg.table_log2, cfg.key_bits = 10, 10
    return _trainer(cfg)


def _request(rng: np.random.Generator, rid: int, case: dict):
    """A re-solve request as the serving workload draws them, with the case's
    street, players, number of sizes and budget."""
    r = serving.make_request(rng, rid)
    board = [int(c) for c in rng.permutation(52)[: case["street"] + 2]]
    ranges = rng.dirichlet(np.full(1326, 0.5), size=case["players"])
    ranges[:, np.isin(serving.COMBO_CARDS, board).any(axis=1)] = 0.0
    ranges /= ranges.sum(axis=1, keepdims=True)
    r.street, r.players, r.board = case["street"], case["players"], board
    r.pot = int(round(rng.uniform(2.0, 200.0) * serving.CHIPS_PER_BB / r.players)) * r.players
    r.ranges = ranges.astype(np.float32)
    pick = rng.choice(len(serving.BET_SIZES), size=case["sizes"], replace=False)
    r.sizes = sorted((serving.BET_SIZES[i] for i in pick), key=lambda f: f[0] / f[1])
    r.budget, r.table_log2 = case["budget"], case["table_log2"]
    return r


def prepare(case: dict, seed: int) -> dict:
    rng = np.random.default_rng([seed, 77])
    k, s = case["kind"], {"case": case}
    if k == "train":
        s["trainer"] = _trainer(_config(case, seed))
        s["trainer"].train(case["warm"], case["batch"], verbose=False)
        if case["out"] != "digest":
            s.update(_store(1 << case["key_bits"], case["out"] == "rows"))
    elif k == "resolve":
        s["owner"] = _owner()
        r = s["request"] = _request(rng, seed % 100_000, case)
        s["trainer"] = mccfr.GPUCFRTrainer.subgame(serving.request_config(r), r.street, r.pot, r.board, r.ranges)
        s["trainer"].share_hand_table(s["owner"])
        s.update(_store(1 << (r.table_log2 - 1)))
    elif k == "serve":
        s["owner"] = _owner()
        s["requests"] = [serving.make_request(rng, i) for i in range(case["requests"])]
        # budgets kept to the lower part of the workload's range, so that a burst is
        # served within a second
        for r in s["requests"]:
            r.budget, r.table_log2 = min(r.budget, 12_000), min(r.table_log2, 17)
        s.update(_store(sum(1 << (r.table_log2 - 1) for r in s["requests"])), counts=np.zeros(64, np.int64))
        s["server"] = serving.ReSolveServer(s["owner"], hbm_budget=16 << 30, traversals=case["traversals"],
                                            retire_workers=2)
    elif k == "batch":
        s["owner"] = _owner()
        s["trainers"], counts = [], []
        for i in range(case["tables"]):
            c = L.preset(L.PRESET_HU_20BB)
            c.num_players = int(rng.integers(2, 7))
            c.starting_stack = int(rng.integers(10, 201)) * c.big_blind
            _set_actions(c, ACTIONS[int(rng.integers(3, 7))])
            c.raise_cap, c.table_log2, c.key_bits, c.seed = 3, case["table_log2"], case["table_log2"] - 1, seed + i
            t = mccfr.GPUCFRTrainer(config=c)
            t.share_hand_table(s["owner"])
            s["trainers"].append(t)
            counts.append(max(64, int(case["batch"] * rng.lognormal(-0.5, 1.0))))
        s["stores"] = [_store(1 << (case["table_log2"] - 1), True) for _ in s["trainers"]]
        s["batch"] = mccfr.Batch(s["trainers"], [min(n, 4 * case["batch"]) for n in counts])
    elif k == "eval":
        s["trainer"] = _trainer_small(L.preset(L.PRESET_HU_20BB))
        s["cards"] = rng.random((case["hands"], 52), dtype=np.float32).argpartition(7, axis=1)[:, :7].astype(np.uint8)
    else:
        c = L.preset(L.PRESET_6MAX_100BB)
        c.seed = seed
        s["trainer"] = _trainer_small(c)
        s["ranks"] = torch.empty(case["hands"], dtype=torch.int16, device="cuda")
        s["masks"] = torch.empty(case["deals"], dtype=torch.uint8, device="cuda")
    return s


def _store(rows: int, whole: bool = False) -> dict:
    """Host arrays that a program keeps for what it reads back of a table of up to
    `rows` rows: keys and strategies, or whole rows.  Entries past the rows in
    use stay zero."""
    if whole:
        return {"keys": np.zeros(rows, np.int64), "regrets": np.zeros((rows, 8), np.float32),
                "strategy_sum": np.zeros((rows, 8), np.float32), "visits": np.zeros(rows, np.int64)}
    return {"keys": np.zeros(rows, np.int32), "probs": np.zeros((rows, 8), np.float32)}


def _strategy(t, s: dict) -> tuple:
    n = ctypes.c_size_t()
    L.check(L.load().mccfr_get_strategy(t.handle, L.ptr(s["keys"]), None, L.ptr(s["probs"]), len(s["keys"]),
                                        ctypes.byref(n)), t.handle)
    return s["keys"], s["probs"], int(n.value)


def _rows(t, s: dict) -> tuple:
    n = ctypes.c_size_t()
    L.check(L.load().mccfr_export_rows(t.handle, L.ptr(s["keys"]), L.ptr(s["regrets"]), L.ptr(s["strategy_sum"]),
                                       L.ptr(s["visits"]), len(s["keys"]), ctypes.byref(n)), t.handle)
    return s["keys"], s["regrets"], s["strategy_sum"], s["visits"], int(n.value)


def run(s: dict):
    case = s["case"]
    k = case["kind"]
    if k == "train":
        t = s["trainer"]
        t.train(case["iters"], case["batch"], verbose=False)
        if case["out"] == "strategy":
            return _strategy(t, s)
        if case["out"] == "rows":
            return _rows(t, s)
        (digest, rows), st = t.digest(), t.stats()
        return {"digest": np.array([digest], np.uint64).view(np.int64), "rows": rows,
                "counters": [int(st.traversals), int(st.node_visits), int(st.traverser_updates), int(st.terminals)]}
    if k == "resolve":
        t, r = s["trainer"], s["request"]
        t.reset_subgame(serving.request_config(r), r.street, r.pot, r.board, r.ranges)
        t.train(serving.updates_for(r, 1024), 1024, verbose=False)
        return _strategy(t, s)
    if k == "serve":
        at = 0
        for r in sorted(s["server"].run(s["requests"], realtime=False), key=lambda r: r.rid):
            n = len(r.keys)
            s["keys"][at:at + n], s["probs"][at:at + n], s["counts"][r.rid] = r.keys.view(np.int32), r.probs, n
            at += n
        return s["keys"], s["probs"], s["counts"]
    if k == "batch":
        s["batch"].train(case["iters"])
        return [_rows(t, st)[:3] for t, st in zip(s["trainers"], s["stores"])]
    if k == "eval":
        return s["trainer"].eval7(s["cards"]).view(np.int16)
    lib, h, ms = L.load(), s["trainer"].handle, ctypes.c_float()
    L.check(lib.mccfr_deal_eval7(h, 0, case["hands"], ctypes.c_void_p(s["ranks"].data_ptr()), ctypes.byref(ms)), h)
    L.check(lib.mccfr_showdown_masks(h, 1, 0, case["deals"], ctypes.c_void_p(s["masks"].data_ptr()), ctypes.byref(ms)),
            h)
    return s["ranks"], s["masks"]


# Node visits and updating-player updates of one traversal, about, for `work`
# (they depend on the run: measured a few iterations in).
VISITS = {("hu", "external"): (19.0, 6.5), ("six", "external"): (55.0, 10.0), ("mixed", "external"): (40.0, 10.0),
          ("hu", "reference"): (4.0, 2.0), ("six", "reference"): (8.7, 1.5), ("ref8", "reference"): (3.9, 1.9)}


def work(case: dict) -> dict:
    """Bytes: per node visit its key and regret row (8 + 32 B), per updating-player
    update the regret row written and the strategy row read and written (96 B);
    rank-table gathers (4 B) and the outputs."""
    k = case["kind"]
    if k == "train":
        players = {"hu": 2, "six": 6}.get(case["game"]) or case["players"]
        v, u = VISITS[case["game"], case["rule"]]
        n = case["iters"] * players * case["batch"]
        return {"bytes": n * (40.0 * v + 96.0 * u + 28.0), "flops": 0.0}
    if k == "resolve":
        n = 1024 * serving.updates_for(type("R", (), {"budget": case["budget"]}), 1024) * case["players"]
        return {"bytes": n * (40.0 * 30 + 96.0 * 12 + 28.0), "flops": 0.0}
    if k == "serve":
        return {"bytes": case["requests"] * 6000.0 * 4 * (40.0 * 30 + 96.0 * 12 + 28.0), "flops": 0.0}
    if k == "batch":
        return {"bytes": case["iters"] * case["tables"] * 4.0 * case["batch"] * (40.0 * 40 + 96.0 * 10 + 28.0),
                "flops": 0.0}
    if k == "eval":
        return {"bytes": case["hands"] * (7.0 + 2.0), "flops": 0.0}
    return {"bytes": case["hands"] * 2.0 + case["deals"] * 1.0, "flops": 0.0}


def exact(case: dict, seed: int):
    """None for every case.  Ranks, masks, keys and counts are whole numbers.  A
    trained table's regrets and strategies follow from sampled actions, whose draws
    are decided by the trainer's own rounded strategies from the first iteration
    on, so there is no 64-bit value that they approximate (a run in another
    precision samples other trees); replaying the millions of traversals of a pass
    in plain Python would also take hours."""
    return None
