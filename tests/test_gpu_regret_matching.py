"""Regret matching against IEEE division: with regrets seeded, the strategy
sums after iteration 0 (its discount clears the old sums) are the strategy
itself, which must be numpy's correctly rounded quotients bit for bit - for
zero, tiny, huge and mixed regrets, around the limits where the kernel's
shared-reciprocal quotients hand over to the divide."""

import numpy as np
import pytest

import poker_solver_rust_b200 as ps
from tests import spots

pytestmark = pytest.mark.gpu


def _regrets(kind, rng, shape):
    x = rng.normal(0, 1, shape).astype(np.float32)
    if kind == "mixed":  # every magnitude, a third negative, some zero
        x = (rng.random(shape) * np.exp2(rng.uniform(-120, 60, shape))).astype(np.float32)
        x[rng.random(shape) < 0.3] *= -1
        x[rng.random(shape) < 0.2] = 0
    elif kind == "limits":  # 2^-100 (numerators, denominators) and 2^20 (denominators), one ulp around
        e = np.exp2(rng.choice([-126.0, -100.0, -99.0, 0.0, 19.0, 20.0], shape)).astype(np.float32)
        x = np.nextafter(e, e * rng.choice([0.5, 1.0, 2.0], shape).astype(np.float32))
    elif kind == "subnormal":
        x = np.float32(1e-45) * rng.integers(0, 1 << 20, shape).astype(np.float32)
    elif kind == "negative":
        x = -np.abs(x)
    elif kind == "near_one":  # quotients close to 1 and to 1/2
        x = (1 + rng.integers(0, 4, shape) * np.float32(2.0**-23)).astype(np.float32)
    return x


@pytest.mark.parametrize("kind", ["normal", "mixed", "limits", "subnormal", "negative", "near_one"])
def test_strategy_is_correctly_rounded(kind):
    r, board, tc = spots.river_spot(4)
    g = spots.product_game(r, board, tc)
    rng = np.random.default_rng(11)
    want = {}
    for i in range(g.num_nodes()):
        info = g.node_info(i)
        if info["player"] & (4 | 8) or info["num_children"] < 2:
            continue
        na, H = info["num_children"], g.num_private_hands(info["player"])
        x = _regrets(kind, rng, (na, H))
        g.seed_node_storage(i, 2, x.reshape(-1))
        m = np.where(x > 0, x, np.float32(0))
        d = m[0].copy()
        for a in range(1, na):
            d = d + m[a]
        with np.errstate(all="ignore"):
            want[i] = np.where(d == 0, np.float32(1) / np.float32(na), m / d)
    # player 0's pass divides in its backward op; player 1's reads what the
    # forward op of player 0's pass cached
    ps.solve_step(g, 0)
    for i, w in want.items():
        assert np.array_equal(g.node_storage(i, 1).reshape(w.shape), w), (kind, i)
