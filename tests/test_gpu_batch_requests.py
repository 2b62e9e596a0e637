"""Launch requests of a batch: what may be asked for, what it costs and what is
shared between batches (tuned shapes, a kernel's shared-memory limit)."""

import subprocess
import sys
import threading

import numpy as np
import pytest

import poker_solver_rust_b200 as ps
from tests import spots

pytestmark = pytest.mark.gpu

STEP, FLOW = 1, 2


def _thin(n, seed, hands=90, stack=200):
    """River spots of one tree with `hands` hands a player."""
    rng = np.random.default_rng(seed)
    sizes = ps.BetSizeOptions("50%, a", "100%, a")
    t = ps.TreeConfig(initial_state=ps.BoardState.River, starting_pot=100, effective_stack=stack,
                      river_bet_sizes=[sizes, sizes])
    sp = []
    for _ in range(n):
        board = [int(x) for x in rng.choice(52, 5, replace=False)]
        r = np.zeros((2, 1326), np.float32)
        for w in r:
            live = rng.permutation(np.flatnonzero(~spots._board_blocked(board)))[:hands]
            w[live] = rng.random(hands).astype(np.float32) * 0.9 + 0.1
        sp.append((r, board, t))
    return sp


def _batch(sp, **kw):
    return ps.BatchSolver([spots.card_config(r, b) for r, b, _ in sp], [t for _, _, t in sp], **kw)


def _solved(b, iterations=20):
    b.solve(iterations, 0.01 * b.starting_pots)
    return (*b.results(), b.root_cfvalues_all())


def _same(a, b):
    for x, y in zip(a, b):
        assert np.array_equal(x, y)


def test_batches_of_different_sizes_launch_from_several_threads():
    """Each launch sets its kernel's shared-memory limit; another thread's batch of another stride must
    not change it before the launch."""
    batches = [_batch(_thin(16, seed=k, hands=40 + 120 * k)) for k in range(4)]
    want = []
    for b in batches:
        assert b.config()["scheduler"] == "dataflow"
        b.run_iterations(0, 2, root=True)
        want.append(b.root_cfvalues_all())
    errors = []

    def launch(b):
        try:
            for _ in range(400):
                if errors:
                    return
                b.run_iterations(2, 2, root=True)
        except Exception as e:
            errors.append(e)

    def build():
        try:
            for k in range(40):
                _batch(_thin(16, seed=k, hands=30 + 64 * (k % 5)))
        except Exception as e:
            errors.append(e)

    threads = [threading.Thread(target=launch, args=(b,)) for b in batches] + [threading.Thread(target=build)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for b, w in zip(batches, want):
        assert np.array_equal(b.root_cfvalues_all(), w)


@pytest.mark.parametrize("request_", [{"flow_spots_per_cta": 9}, {"node_parts": 17}, {"scan_buffers": 32}])
def test_small_batch_ignores_a_dataflow_request_it_cannot_run(request_):
    """Up to a spot per SM the default schedule takes any dataflow request; more spots, or the dataflow
    scheduler asked for, refuse one that is out of range."""
    sp = _thin(16, seed=3, hands=1000)
    b = _batch(sp, **request_)
    assert b.config()["scheduler"] == "step-synchronous"
    _same(_solved(b), _solved(_batch(sp, scheduler=STEP)))
    for kw in ({"scheduler": FLOW}, {}):
        with pytest.raises(Exception):
            _batch(sp if kw else _thin(150, seed=3, hands=1000), **request_, **kw)


def test_dataflow_with_staged_tables_asked_for():
    """13 scan buffers of 1080 hands and a request to stage the board tables: the dataflow kernel reads
    the tables from global memory, so only the buffers count."""
    sp = _thin(150, seed=4, hands=1080)
    b = _batch(sp, stage_tables=1, scan_buffers=13)
    assert b.config()["scheduler"] == "dataflow" and b.config()["scan_buffers"] == 13
    _same(_solved(b, 5), _solved(_batch(sp, scheduler=STEP), 5))


_SCRATCH = """
import torch
from tests.test_gpu_batch_requests import _batch, _thin
free = lambda: torch.cuda.mem_get_info()[0]
sp = _thin(149, seed=5, hands=1080, stack=2000)
at, used, keep = free(), [], []
for lanes in (1, 8):
    keep.append(_batch(sp, scheduler=2, flow_spots_per_cta=lanes, scan_buffers=8))
    used.append(at - free())
    at -= used[-1]
print("BYTES", *used)
"""


def test_scratch_is_for_spots_not_for_idle_lanes():
    """149 spots take 149 scratch areas whether a CTA may hold one spot or eight (in a process of its
    own, where no freed memory waits in the library's pool)."""
    r = subprocess.run([sys.executable, "-c", _SCRATCH], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    one, eight = [int(x) for x in r.stdout.split("BYTES")[1].split()]
    assert eight <= one + (64 << 20), (one, eight)


def test_shapes_are_tuned_per_batch_size():
    """A shape tuned on little more than a spot per SM is not adopted for many spots per SM."""
    sp = _thin(900, seed=71, hands=212)
    _solved(_batch(sp[:200], block_threads=-1), 5)
    large = _batch(sp, block_threads=-1)
    assert large.autotune_trials()
    _solved(large, 5)
    assert not _batch(sp[:820], block_threads=-1).autotune_trials()  # the same class: no trials


def test_tuned_shape_that_does_not_fit_is_replaced():
    """576 and 608 hands are one hand-count class, and 32 scan buffers fit in shared memory for the
    first only: whatever was tuned for the first, the second is built and solved."""
    for hands in (576, 608):
        sp = _thin(200, seed=72, hands=hands)
        b = _batch(sp, block_threads=-1)
        _same(_solved(b, 10), _solved(_batch(sp, scheduler=STEP), 10))


@pytest.mark.parametrize("n", [40, 320])
def test_staged_tables_with_spots_in_lockstep(n):
    """A CTA that solves several spots in lockstep has no room for each one's tables: results are those
    of tables read from global memory."""
    sp = _thin(n, seed=6, hands=120)
    _same(_solved(_batch(sp, scheduler=STEP, instances_per_cta=4, stage_tables=1), 6),
          _solved(_batch(sp, scheduler=STEP), 6))
