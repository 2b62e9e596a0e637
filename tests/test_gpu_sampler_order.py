"""The sampler's strength order on many boards: ties, full houses, flushes and
straights decide it, and the ranges follow it bit for bit."""

import numpy as np
import pytest

from oracle import sampler as S
from poker_solver_rust_b200.sampler import SamplerConfig, sample_situations

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", range(4))
def test_sampled_river_ranges(seed):
    cfg = SamplerConfig(board_size=5, seed=100 + seed)
    got = sample_situations(cfg, 0, 40)["ranges"].cpu().numpy()
    for i in range(40):
        want = S.sample_situation(5, cfg.initial_stack, cfg.pot_intervals, cfg.spr_intervals, cfg.seed, i)[3]
        assert np.array_equal(got[i].view(np.uint32), want.view(np.uint32)), i
