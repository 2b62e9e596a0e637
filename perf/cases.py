"""Timed cases of the solver's public paths, from a single query to a whole datagen batch.

Each case is a dict of plain values with a "kind"; `prepare` makes what a program
holds before the call (inputs and handles, from the seed alone), `run` is one pass
through the public entry points, `work` the bytes and operations that pass cannot
do without, and `exact` the 64-bit value of outputs that have a closed form.

Kinds, and the use each stands for:
  river_batch    river datagen: a batch of spots with ~Beta(0.5, 0.5) ranges (30% of the
                 combos zeroed), pot U[20, 200], SPR U[0.5, 10] and one of three bet menus,
                 solved to 0.3% of the pot (at most 300 iterations), results and training
                 records taken; now and then with rake
  river_game     one river game through the game API, from its configuration to the root
                 strategy and EVs (a study tool's call)
  turn_game      the same for a turn game with its 48 river deals: the widest single tree
  game_query     exploitability and both root values of a game in hand: the smallest call
  turn_interval  one interval of the turn datagen loop: boundary values in, a few DCFR
                 iterations of a batch of depth-limited turn spots, boundary reach out
  turn_adjoint   forward and backward of the fixed-strategy root values of such a batch:
                 the solver's part of a training step
  net_rows       boundary-network input rows (f32 for training, bf16 for inference)
  first_layer    the boundary network's first layer, factored over the river cards
  river_reduce   reach-weighted 48-river average of the network's outputs (inference)
  river_average  the same average with its backward (training)
  sample         random situations for datagen: river or turn boards, plain or by SPR
"""

from __future__ import annotations

import math

import numpy as np
import torch

import poker_solver_rust_b200 as ps
from poker_solver_rust_b200 import datagen, sampler, trainer

MENUS = ("50%, a", "33%, 75%, a", "25%, 50%, 100%, 150%, a")
COMBOS, ROW, RIVERS = 1326, 2720, 48
_PAIRS = [(a, b) for a in range(52) for b in range(a + 1, 52)]


def listed():
    return [
        # a datagen job's batch, and a small one whose tail does not fill the device
        {"name": "river_batch_4096", "kind": "river_batch", "n": 4096, "raked": False},
        {"name": "river_batch_301", "kind": "river_batch", "n": 301, "raked": False},
        # single games: 1081 hands on a small tree, 1128 hands on 12,285 nodes
        {"name": "river_game", "kind": "river_game", "stack": 200, "menu": "50%, 100%, a", "iterations": 1000},
        {"name": "turn_game", "kind": "turn_game", "stack": 300, "iterations": 60},
        {"name": "game_query", "kind": "game_query", "stack": 200, "menu": "50%, 100%, a"},
        # the turn datagen loop's interval (boundaries re-evaluated every 10 iterations) and a training step's tree
        {"name": "turn_interval_1024", "kind": "turn_interval", "n": 1024, "iterations": 10},
        {"name": "turn_adjoint_1024", "kind": "turn_adjoint", "n": 1024},
        # the steps around the boundary network, one evaluation chunk each
        {"name": "net_rows_733", "kind": "net_rows", "n": 733, "bf16": True},
        {"name": "first_layer_1024", "kind": "first_layer", "n": 1024, "h": 500, "bf16": True},
        {"name": "river_reduce_1024", "kind": "river_reduce", "n": 1024, "bf16": True},
        {"name": "river_average_512", "kind": "river_average", "n": 512},
        {"name": "sample_turn_1500", "kind": "sample", "n": 1500, "cards": 4, "spr": False},
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice([c["kind"] for c in listed()])
    if kind == "river_batch":
        return {"kind": kind, "n": log_int(8, 4096), "raked": rng.random() < 0.25}
    if kind == "river_game":
        return {"kind": kind, "stack": log_int(50, 400), "menu": rng.choice(MENUS[:2] + ("50%, 100%, a",)),
                "iterations": log_int(50, 1000)}
    if kind == "turn_game":
        return {"kind": kind, "stack": log_int(60, 300), "iterations": log_int(10, 60)}
    if kind == "game_query":
        return {"kind": kind, "stack": log_int(50, 400), "menu": rng.choice(MENUS)}
    if kind == "turn_interval":
        return {"kind": kind, "n": log_int(8, 1024), "iterations": log_int(2, 20)}
    if kind == "turn_adjoint":
        return {"kind": kind, "n": log_int(8, 1024)}
    if kind == "net_rows":
        return {"kind": kind, "n": log_int(4, 1024), "bf16": rng.random() < 0.5}
    if kind == "first_layer":
        return {"kind": kind, "n": log_int(4, 1024), "h": log_int(64, 640), "bf16": rng.random() < 0.5}
    if kind == "river_reduce":
        return {"kind": kind, "n": log_int(4, 1024), "bf16": rng.random() < 0.7}
    if kind == "river_average":
        return {"kind": kind, "n": log_int(4, 512)}
    return {"kind": kind, "n": log_int(16, 4096), "cards": rng.choice((4, 5)), "spr": rng.random() < 0.5}


# ---- inputs ----
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda")


def _boards(g, n, k):
    """[n, k] distinct cards."""
    return _rand(g, n, 52).topk(k, dim=1).indices


def _live(boards):
    """[n, 1326]: combos that share no card with the board."""
    pairs = torch.tensor(_PAIRS, device="cuda")
    return (pairs[None, :, :, None] != boards[:, None, None, :]).all(dim=3).all(dim=2)


def _ranges(g, boards):
    """[n, 2, 1326] weights ~Beta(0.5, 0.5) (the arcsine law) with 30% zeroed, board-masked."""
    n = boards.shape[0]
    w = torch.sin(_rand(g, n, 2, COMBOS) * (math.pi / 2)).square()
    return w * (_rand(g, n, 2, COMBOS) >= 0.3) * _live(boards)[:, None, :]


def _card_config(ranges, board):
    b = [int(x) for x in board]
    return ps.CardConfig([ps.Range(ranges[0]), ps.Range(ranges[1])], b[:3], b[3] if len(b) > 3 else ps.NOT_DEALT,
                         b[4] if len(b) > 4 else ps.NOT_DEALT)


def _batch(g, n, river, raked=False):
    """A BatchSolver of n river spots, or of n turn spots with a depth boundary at every non-fold turn
    terminal.  Pots, stacks and menus (so the trees and the number of boundaries) go with n, boards and
    ranges with the seed."""
    boards = _boards(g, n, 5 if river else 4)
    ranges = _ranges(g, boards).cpu().numpy()
    u = np.random.default_rng(n).random((n, 3))
    boards = boards.cpu().numpy()
    cards, trees = [], []
    for i in range(n):
        pot = 20 + int(u[i, 0] * 181)
        stack = max(1, round((0.5 + 9.5 * u[i, 1]) * pot))
        if river:
            s = [ps.BetSizeOptions(MENUS[int(u[i, 2] * 3)], "100%, a")] * 2
            t = ps.TreeConfig(initial_state=ps.BoardState.River, starting_pot=pot, effective_stack=stack,
                              river_bet_sizes=s, rake_rate=0.05 if raked else 0.0, rake_cap=30.0 if raked else 0.0)
        else:
            s = [ps.BetSizeOptions("33%, 75%, a", "60%")] * 2
            t = ps.TreeConfig(initial_state=ps.BoardState.Turn, starting_pot=pot, effective_stack=stack,
                              turn_bet_sizes=s, river_bet_sizes=s, depth_limit=0)
        cards.append(_card_config(ranges[i], boards[i]))
        trees.append(t)
    return ps.BatchSolver(cards, trees)


def _game_config(g, case):
    """One game: ranges U[0, 1] over the live combos, pot 100."""
    turn = case["kind"] == "turn_game"
    board = _boards(g, 1, 4 if turn else 5)
    r = (_rand(g, 1, 2, COMBOS) * _live(board)[:, None, :]).cpu().numpy()[0]
    return _card_config(r, board[0].tolist()), _game_tree(case)


def _game_tree(case):
    if case["kind"] == "turn_game":
        s = [ps.BetSizeOptions("33%, 75%, a", "60%")] * 2
        return ps.TreeConfig(initial_state=ps.BoardState.Turn, starting_pot=100, effective_stack=case["stack"],
                             turn_bet_sizes=s, river_bet_sizes=s)
    s = [ps.BetSizeOptions(case["menu"], "100%")] * 2
    return ps.TreeConfig(initial_state=ps.BoardState.River, starting_pot=100, effective_stack=case["stack"],
                         river_bet_sizes=s)


def _boundary_values(g, batch):
    """[items, 2, 1326] ~N(0, (pot/4)^2), zero on the combos that the board blocks."""
    it = batch.boundary_items()
    boards = torch.as_tensor(it["boards"].astype(np.int64), device="cuda")
    v = torch.randn(len(it["spot"]), 2, COMBOS, generator=g, device="cuda")
    return v * torch.as_tensor(0.25 * it["root_pots"], device="cuda")[:, None, None] * _live(boards)[:, None, :]


def _items(g, n):
    """Boundary items: boards, pots and stacks on the host, reach (range x line probability) on the device."""
    b = _boards(g, n, 4)
    u = _rand(g, n, 2).cpu().numpy()
    pots = np.floor(20 + 400 * u[:, 0]).astype(np.float32)
    stacks = np.floor(5 + 800 * u[:, 1]).astype(np.float32)
    reach = _ranges(g, b) * _rand(g, n, 2, COMBOS)
    return {"boards": b.cpu().numpy().astype(np.uint8), "pots": pots, "stacks": stacks, "reach": reach}


def prepare(case, seed):
    g, kind = _gen(seed), case["kind"]
    if kind == "river_batch":
        b = _batch(g, case["n"], True, case["raked"])
        return {"kind": kind, "batch": b, "target": 0.003 * b.starting_pots}
    if kind in ("river_game", "turn_game"):
        cards, tree = _game_config(g, case)
        return {"kind": kind, "cards": cards, "tree": tree, "iterations": case["iterations"]}
    if kind == "game_query":
        cards, tree = _game_config(g, case)
        game = ps.PostFlopGame.with_config(cards, ps.ActionTree(tree))
        game.allocate_memory()
        for t in range(20):
            ps.solve_step(game, t)
        return {"kind": kind, "game": game}
    if kind == "turn_interval":
        b = _batch(g, case["n"], False)
        return {"kind": kind, "batch": b, "values": _boundary_values(g, b), "iterations": case["iterations"]}
    if kind == "turn_adjoint":
        b = _batch(g, case["n"], False)
        v = _boundary_values(g, b)
        b.set_boundary_cfvs(v)
        b.run_iterations(0, 10)
        cot = torch.randn(case["n"], 2, COMBOS, generator=g, device="cuda")
        return {"kind": kind, "batch": b, "values": v.requires_grad_(), "cot": cot}
    if kind == "sample":
        return {"kind": kind, "n": case["n"], "config": sampler.SamplerConfig(
            board_size=case["cards"], seed=seed,
            spr_intervals=[[0.0, 0.5], [0.5, 1.5], [1.5, 4.0], [4.0, 8.0]] if case["spr"] else None)}
    s = {"kind": kind, "bf16": case.get("bf16", False), **_items(g, case["n"])}
    if kind == "first_layer":
        k = 1 / math.sqrt(ROW)
        dt = torch.bfloat16 if case["bf16"] else torch.float32
        s["weight"] = ((2 * _rand(g, case["h"], ROW) - 1) * k).to(dt)
        s["bias"] = ((2 * _rand(g, case["h"]) - 1) * k).to(dt)
    elif kind in ("river_reduce", "river_average"):
        y = torch.randn(case["n"], 2, RIVERS, COMBOS, generator=g, device="cuda")
        s["net"] = y.to(torch.bfloat16) if s["bf16"] else y
        s["hands"] = torch.arange(COMBOS, dtype=torch.int32, device="cuda")
        if kind == "river_average":
            s["net"].requires_grad_()
            s["cot"] = torch.randn(case["n"], 2, COMBOS, generator=g, device="cuda")
    return s


def run(s):
    kind = s["kind"]
    if kind == "river_batch":
        b = s["batch"]
        b.solve(300, s["target"])
        expl, iters = b.results()
        rec = b.records()
        return {"expl": expl, "iters": iters, "records": rec.view(np.uint8)}
    if kind in ("river_game", "turn_game"):
        game = ps.PostFlopGame.with_config(s["cards"], ps.ActionTree(s["tree"]))
        game.allocate_memory()
        e = ps.solve(game, s["iterations"], 0.0)
        game.cache_normalized_weights()
        return {"expl": e, "strategy": game.strategy(), "ev": [game.expected_values(p) for p in range(2)]}
    if kind == "game_query":
        game = s["game"]
        return {"expl": ps.compute_exploitability(game), "values": [ps.root_cfvalues(game, p) for p in range(2)]}
    if kind == "turn_interval":
        b = s["batch"]
        b.reset()
        b.set_boundary_cfvs(s["values"])
        b.run_iterations(0, s["iterations"], root=True, exploitability=True)
        return {"expl": b.results()[0], "reach": b.boundary_reach(device=True),
                "values": b.root_cfvalues_all(device=True)}
    if kind == "turn_adjoint":
        cfv = trainer.FixedStrategyRootValues.apply(s["batch"], s["values"])
        (grad,) = torch.autograd.grad(cfv, s["values"], s["cot"])
        return {"values": cfv, "grad": grad}
    if kind == "sample":
        r = sampler.sample_situations(s["config"], 0, s["n"])
        return {k: r[k] for k in ("boards", "pots", "stacks", "ranges")}
    if kind == "net_rows":
        return datagen.boundary_encode(s["boards"], s["pots"], s["stacks"], s["reach"], bf16=s["bf16"])
    if kind == "first_layer":
        return datagen.boundary_first_layer(s["boards"], s["pots"], s["stacks"], s["reach"], s["weight"], s["bias"],
                                            bf16=s["bf16"])
    if kind == "river_reduce":
        return datagen.boundary_river_reduce(s["boards"], s["pots"], s["stacks"], s["net"], s["reach"], s["hands"])
    out = trainer.RiverAverage.apply(s["net"], s["boards"], s["pots"] + s["stacks"], s["reach"])
    (grad,) = torch.autograd.grad(out, s["net"], s["cot"])
    return {"values": out, "grad": grad}


# ---- what a pass cannot do without ----
# A DCFR iteration streams 20 bytes per acting hand and action (regrets read as opponent, read and
# written as traverser, strategy sums read and written), an exploitability check 4, with about as many
# operations. The means over the datagen distribution: 53,000 hand-actions and 112 iterations a river
# spot, 10,500 hand-actions and 17 boundaries a turn spot.
_RIVER_S, _RIVER_ITERS, _TURN_S, _TURN_ITEMS = 53_000, 112, 10_500, 17


def work(case):
    kind, n = case["kind"], case.get("n", 1)
    if kind == "river_batch":
        passes = 20 * _RIVER_ITERS + 4 * (_RIVER_ITERS / 5 + 2)
        return {"bytes": n * (_RIVER_S * passes + 2 * 17_300), "flops": n * _RIVER_S * passes}
    if kind in ("river_game", "turn_game", "game_query"):
        cards = 4 if kind == "turn_game" else 5
        r = [ps.Range(np.array([float(min(p) >= cards) for p in _PAIRS], np.float32)) for _ in range(2)]
        hand_actions = ps.PostFlopGame.with_config(_card_config([x.data for x in r], range(cards)),
                                                   ps.ActionTree(_game_tree(case))).program_info()["S"]
        it = case.get("iterations", 0)
        passes = 20 * it + 4 * (it / 5 + 2)
        return {"bytes": hand_actions * passes, "flops": hand_actions * passes}
    if kind == "turn_interval":
        passes = 20 * case["iterations"] + 8
        values = 2 * _TURN_ITEMS * 2 * COMBOS * 4 + 2 * COMBOS * 4
        return {"bytes": n * (_TURN_S * passes + values), "flops": n * _TURN_S * passes}
    if kind == "turn_adjoint":  # an average-strategy pass each way for both players
        return {"bytes": n * (_TURN_S * 8 + 2 * _TURN_ITEMS * 2 * COMBOS * 4 + 4 * COMBOS * 4), "flops": n * _TURN_S * 8}
    if kind == "sample":
        # a 7-card value per combo (and river card on a turn board), 40 operations each, and the two ranges out
        evals = COMBOS * (46 if case["cards"] == 4 else 1)
        return {"bytes": n * (2 * COMBOS * 4 + 13), "flops": n * evals * 40}
    el = 2 if case.get("bf16") else 4
    reach = n * 2 * COMBOS * 4
    if kind == "net_rows":
        return {"bytes": reach + n * 96 * ROW * el, "flops": n * 2 * RIVERS * COMBOS}
    if kind == "first_layer":  # per card the combos that hold it: every combo twice, for both ranges
        h = case["h"]
        return {"bytes": reach + h * ROW * el + n * 96 * h * el, "flops": 2 * n * 2 * COMBOS * 2 * h + n * 96 * h * 4}
    net = n * 2 * RIVERS * COMBOS * el
    if kind == "river_reduce":
        return {"bytes": net + 2 * reach, "flops": n * 2 * RIVERS * COMBOS * 3}
    return {"bytes": 2 * net + 3 * reach, "flops": n * 2 * RIVERS * COMBOS * 6}


# ---- 64-bit values ----
def _rivers(boards):
    """(river cards [n, 48], keep [n, 48, 1326]: combos without the river card)."""
    b = torch.as_tensor(boards.astype(np.int64), device="cuda")
    cards = torch.arange(52, device="cuda")
    free = (cards[None, :, None] != b[:, None, :]).all(dim=2)
    rivers = cards.expand(len(b), 52)[free].view(-1, RIVERS)
    pairs = torch.tensor(_PAIRS, device="cuda")
    return b, rivers, (pairs[None, None] != rivers[:, :, None, None]).all(dim=3)


def _rows64(s, z):
    """Input rows [m, 2, 48, 2720] in 64 bits: both reaches without the river card's combos, the board's
    cards and ranks, pot and stack over their sum, the player."""
    b, rivers, keep = _rivers(s["boards"][z])
    m = len(b)
    x = torch.zeros(m, 2, RIVERS, ROW, dtype=torch.float64, device="cuda")
    x[..., :2 * COMBOS] = (s["reach"][z].double()[:, None] * keep[:, :, None]).reshape(m, 1, RIVERS, 2 * COMBOS)
    board = torch.cat([b[:, None].expand(m, RIVERS, 4), rivers[:, :, None]], dim=2)
    x[..., 2652:2704].scatter_(3, board[:, None].expand(m, 2, RIVERS, 5), 1.0)
    x[..., 2704:2717].scatter_(3, board[:, None].expand(m, 2, RIVERS, 5) // 4, 1.0)
    pot, stack = (torch.as_tensor(s[k][z].astype(np.float64), device="cuda") for k in ("pots", "stacks"))
    x[..., 2717] = (pot / (pot + stack))[:, None, None]
    x[..., 2718] = (stack / (pot + stack))[:, None, None]
    x[:, 1, :, 2719] = 1.0
    return x


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("net_rows", "first_layer", "river_reduce", "river_average"):
        return None  # iterated from the configuration, or drawn: no closed form
    s, parts = prepare(case, seed), []
    for a in range(0, case["n"], 64):
        z = slice(a, min(case["n"], a + 64))
        if kind == "net_rows":
            parts.append(_rows64(s, z))
        elif kind == "first_layer":
            parts.append(_rows64(s, z) @ s["weight"].double().t() + s["bias"].double())
        else:
            _, _, keep = _rivers(s["boards"][z])
            keep = keep.double()
            opp = s["reach"][z].double().flip(1)
            w = torch.einsum("npc,nrc->npr", opp, keep)
            den = torch.einsum("npr,nrc->npc", w, keep)
            y = s["net"].detach()[z].double()
            scale = torch.as_tensor((s["pots"] + s["stacks"])[z].astype(np.float64), device="cuda")[:, None, None]
            ok = den > 0
            inv = torch.where(ok, scale / den.where(ok, torch.ones_like(den)), torch.zeros_like(den))
            out = (w[..., None] * y * keep[:, None]).sum(2) * inv
            if kind == "river_reduce":
                parts.append(out)
            else:
                parts.append((out, w[..., None] * keep[:, None] * (s["cot"][z].double() * inv)[:, :, None]))
    if kind == "river_average":
        return {"values": torch.cat([p[0] for p in parts]), "grad": torch.cat([p[1] for p in parts])}
    return torch.cat(parts)
