"""The dataflow kernel with every lane of a CTA in use: more spots than lanes on
the device, so lanes are bound again from the queue, and all of a CTA's spots
are at different steps.  Same bits as the step-synchronous kernel.  And the
requests that test_gpu_flow_routes builds do run on the dataflow kernel."""

import numpy as np
import pytest

import poker_solver_rust_b200 as ps
from tests import spots

pytestmark = pytest.mark.gpu

STEP, FLOW = 1, 2


def _batch(sp, **kw):
    return ps.BatchSolver([spots.card_config(r, b) for r, b, _ in sp], [t for _, _, t in sp], **kw)


@pytest.fixture(scope="module")
def crowd():
    rng = np.random.default_rng(53)
    sp = []
    for _ in range(1500):  # more than 148 CTAs x 8 lanes
        r, b, t = spots.datagen_spot(rng)
        for w in r:
            w[rng.random(1326) < 0.92] = 0.0
        sp.append((r, b, t))
    want = _batch(sp, scheduler=STEP)
    want.solve(30, 0.01 * want.starting_pots)
    return sp, want.results(), want.root_cfvalues_all()


@pytest.mark.parametrize("threads,lanes,parts,bufs", [(1024, 4, 2, 0), (1024, 8, 3, 16), (256, 8, 1, 4), (128, 3, 16, 2)])
def test_full_lanes_and_refills(crowd, threads, lanes, parts, bufs):
    sp, (e, it), cfv = crowd
    b = _batch(sp, scheduler=FLOW, flow_threads=threads, flow_spots_per_cta=lanes, node_parts=parts, scan_buffers=bufs,
               ctas_per_sm=1)
    cfg = b.config()
    assert cfg["spots_per_cta"] == lanes and cfg["grid"] * lanes < len(sp)
    b.solve(30, 0.01 * b.starting_pots)
    assert np.array_equal(b.results()[0], e) and np.array_equal(b.results()[1], it)
    assert np.array_equal(b.root_cfvalues_all(), cfv)


def test_full_lanes_adjoint():
    sp = spots.turn_boundary_spots(400, seed=8)
    rng = np.random.default_rng(9)
    for r, _, _ in sp:
        for w in r:
            w[rng.random(1326) < 0.9] = 0.0
    cot = rng.normal(0, 1, (len(sp), 2, 1326)).astype(np.float32)
    out = []
    for kw in ({"flow_threads": 1024, "flow_spots_per_cta": 2, "ctas_per_sm": 1, "scheduler": FLOW}, {"scheduler": STEP}):
        b = _batch(sp, **kw)
        b.set_boundary_cfvs(spots.boundary_values(np.random.default_rng(10), b))
        b.run_iterations(0, 2)
        out.append((*b.adjoint(cot), b.root_cfvalues_all()))
    for x, y in zip(*out):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("bufs", [0, 23])
def test_wide_hands_run_dataflow(bufs):
    """16 flop spots of 1176 hands at the default shape; 820 hands (a stride of 832 floats) with 23
    buffers, one of which gives way to the others' padding: 23 x 10,128 bytes do not fit, 22 do."""
    rng = np.random.default_rng(3)
    s = [ps.BetSizeOptions("50%, a", "a")] * 2
    sp = []
    for _ in range(16):
        board = [int(x) for x in rng.choice(52, 5 if bufs else 3, replace=False)]
        r = spots.uniform_ranges(rng, board)
        for w in r if bufs else ():
            live = np.flatnonzero(w)
            w[rng.choice(live, len(live) - 820, replace=False)] = 0
        state = ps.BoardState.River if bufs else ps.BoardState.Flop
        sp.append((r, board, ps.TreeConfig(initial_state=state, starting_pot=60, effective_stack=100, flop_bet_sizes=s,
                                           turn_bet_sizes=s, river_bet_sizes=s, depth_limit=None if bufs else 0)))
    out = []
    for kw in ({"scan_buffers": bufs, "scheduler": FLOW} if bufs else {}, {"scheduler": STEP}):
        b = _batch(sp, **kw)
        if not out:
            cfg = b.config()
            assert cfg["scheduler"] == "dataflow" and cfg["scan_buffers"] == (22 if bufs else 16)
        b.run_iterations(0, 2, exploitability=True)
        out.append((b.results()[0], b.root_cfvalues_all()))
    for x, y in zip(*out):
        assert np.array_equal(x, y)
