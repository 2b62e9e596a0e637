"""Host copies of large device results: records of batches whose bytes are
below, just over and several times a copy piece (4 MB) equal the same records
packed into a device tensor."""

import ctypes as C

import numpy as np
import pytest
import torch

import poker_solver_rust_b200 as ps
from poker_solver_rust_b200 import _native as N
from tests import spots

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 122, 123, 400])
def test_records_on_host_equal_device(n):
    sp = spots.datagen_spots(n, seed=17)
    b = ps.BatchSolver([spots.card_config(r, bd) for r, bd, _ in sp], [t for _, _, t in sp])
    b.solve(2, 0.0)
    host = b.records().view(np.uint8).reshape(-1)
    dev = torch.zeros(host.size, dtype=torch.uint8, device="cuda")
    N.check(N.lib().ps_batch_records(b._h, C.c_void_p(dev.data_ptr()), 1))
    assert np.array_equal(host, dev.cpu().numpy())
