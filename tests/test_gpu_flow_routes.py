"""Batches whose default schedule is the dataflow kernel against the
step-synchronous one, bit for bit: sizes around where the default begins and
around one, two and three spots per SM (where CTAs start with unequal numbers
of spots), for solves and for the adjoint."""

import numpy as np
import pytest

import poker_solver_rust_b200 as ps
from tests import spots

pytestmark = pytest.mark.gpu

STEP = 1


def _batch(sp, **kw):
    return ps.BatchSolver([spots.card_config(r, b) for r, b, _ in sp], [t for _, _, t in sp], **kw)


@pytest.fixture(scope="module")
def river():
    rng = np.random.default_rng(31)
    sp = []
    for _ in range(297):
        r, b, t = spots.datagen_spot(rng)
        for w in r:  # a tenth of the hands: quick, and many sizes
            w[rng.random(1326) < 0.9] = 0.0
        sp.append((r, b, t))
    return sp


@pytest.mark.parametrize("n", [15, 16, 148, 149, 297])
def test_solve_routes(river, n):
    got, want = _batch(river[:n]), _batch(river[:n], scheduler=STEP)
    assert got.config()["scheduler"] == ("dataflow" if n >= 16 else "step-synchronous")
    target = 0.01 * got.starting_pots
    for b in (got, want):
        b.solve(40, target)
    for a, b in zip(got.results(), want.results()):
        assert np.array_equal(a, b)
    assert np.array_equal(got.root_cfvalues_all(), want.root_cfvalues_all())


@pytest.mark.parametrize("n", [15, 16, 150])
def test_adjoint_routes(n):
    sp = spots.turn_boundary_spots(n, seed=5)
    cot = np.random.default_rng(6).normal(0, 1, (n, 2, 1326)).astype(np.float32)
    out = []
    for kw in ({}, {"scheduler": STEP}):
        b = _batch(sp, **kw)
        b.set_boundary_cfvs(spots.boundary_values(np.random.default_rng(7), b))
        b.run_iterations(0, 3)
        out.append((*b.adjoint(cot), b.root_cfvalues_all()))
    for x, y in zip(*out):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("bufs", [0, 23])
def test_wide_hands(bufs):
    """The widest spots there are (1176 hands on a flop) at the default shape,
    and a request of scan buffers whose padding does not fit (one less then)."""
    rng = np.random.default_rng(3)
    sp = []
    for k in range(16):
        board = [int(x) for x in rng.choice(52, 3 if bufs == 0 else 5, replace=False)]
        r = spots.uniform_ranges(rng, board)
        if bufs:
            for w in r:  # 800 hands: a stride of 832 floats
                live = np.flatnonzero(w)
                w[rng.choice(live, len(live) - 800, replace=False)] = 0
        s = [ps.BetSizeOptions("50%, a", "a")] * 2
        sp.append((r, board, ps.TreeConfig(initial_state=ps.BoardState.River if bufs else ps.BoardState.Flop,
                                           starting_pot=60, effective_stack=100, flop_bet_sizes=s, turn_bet_sizes=s,
                                           river_bet_sizes=s, depth_limit=None if bufs else 0)))
    out = []
    for kw in ({"scan_buffers": bufs, "scheduler": 2} if bufs else {}, {"scheduler": STEP}):
        b = _batch(sp, **kw)
        b.run_iterations(0, 2, exploitability=True)
        out.append((b.results()[0], b.root_cfvalues_all()))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
