"""Values written into a game are the ones read back and solved from at once:
the write, the copy to the host and the kernels go through one stream."""

import numpy as np
import pytest

import poker_solver_rust_b200 as ps
from tests import spots

pytestmark = pytest.mark.gpu


def test_seeded_storage_reads_back_at_once():
    r, board, tc = spots.river_spot(4)
    g = spots.product_game(r, board, tc)
    nodes = [i for i in range(g.num_nodes()) if not g.node_info(i)["player"] & (4 | 8)]
    rng = np.random.default_rng(0)
    for k in range(300):
        i = nodes[k % len(nodes)]
        info = g.node_info(i)
        x = rng.random(info["num_children"] * g.num_private_hands(info["player"])).astype(np.float32)
        which = 1 + k % 2
        g.seed_node_storage(i, which, x)
        assert np.array_equal(g.node_storage(i, which), x), k
