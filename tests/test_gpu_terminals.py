"""Terminal evaluation at the hand counts where its list layout changes: the
3V-entry scan is cut into 32 chunks of odd length C, read eight entries at a
time, and hands are looked up 64 at a time.  From the oracle's state, the
exploitability and root values must agree as in test_gpu_parity (f32 prefix
sums against the oracle's f64 ones)."""

import numpy as np
import pytest

import poker_solver_rust_b200 as ps
from tests import spots
from tests.test_gpu_parity import TOL_EVAL_REL, _set_boundaries, _share_state

pytestmark = pytest.mark.gpu


def _sized_ranges(rng, board, sizes):
    """Ranges of exactly the given numbers of hands; the smallest share no card."""
    live = [i for i in range(1326) if not set(ps.index_to_card_pair(i)) & set(board)]
    first = [i for i in rng.permutation(live)]
    second = sorted(first, key=lambda i: len(set(ps.index_to_card_pair(i)) & set(ps.index_to_card_pair(first[0]))))
    out = []
    for order, k in ((first, sizes[0]), (second, sizes[1])):
        w = np.zeros(1326, np.float32)
        w[order[:k]] = rng.random(k).astype(np.float32) * 0.9 + 0.1
        out.append(w)
    return out


# 3V at and around multiples of 32 (C = 1, 3, 9, 11), C = 1, 3, 5, 7 past a multiple of 8, both ends of the range
@pytest.mark.parametrize("hands", [(1, 1), (2, 33), (10, 11), (32, 64), (85, 86), (96, 107), (341, 128), (1081, 1000)])
@pytest.mark.parametrize("kind", ["river", "raked", "boundary"])
def test_terminal_sizes(kind, hands):
    rng = np.random.default_rng(hands[0] * 2000 + hands[1])
    r, board, tc = spots.river_spot(3) if kind != "boundary" else spots.turn_spot(3)
    if kind == "boundary":
        tc.depth_limit = 0
    if kind == "raked":
        tc.rake_rate, tc.rake_cap = 0.05, 3.0
    r = _sized_ranges(rng, board, hands)
    g, o = spots.product_game(r, board, tc), spots.oracle_game(r, board, tc)
    assert (g.num_private_hands(0), g.num_private_hands(1)) == hands
    if kind == "boundary":
        _set_boundaries(g, o)
    for t in range(2):
        o.solve_step(t)
    _share_state(g, o)
    e, eo = ps.compute_exploitability(g), o.compute_exploitability()
    assert abs(e - eo) <= TOL_EVAL_REL * max(abs(eo), 1e-3 * tc.starting_pot), (e, eo)
    for p in range(2):
        v, vo = ps.root_cfvalues(g, p), o.root_cfvalues(p)
        assert np.abs(v - vo).max() <= 10 * TOL_EVAL_REL * max(np.abs(vo).max(), 1e-30)
