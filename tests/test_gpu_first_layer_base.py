"""ps_boundary_first_layer, the C call that is given the product of the whole
reach (base): against the dense layer over the input rows in f64, at one and at
two columns per thread and around the metadata chunk.  f32 products and sums of
about 2700 terms stay within 2^-18 of the largest output."""

import ctypes as C

import numpy as np
import pytest
import torch

from poker_solver_rust_b200 import _native as N
from poker_solver_rust_b200 import datagen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,h", [(1, 1), (3, 514), (1025, 7), (1025, 64)])
def test_given_base(n, h):
    rng = np.random.default_rng(n + h)
    boards = np.stack([rng.choice(52, 4, replace=False) for _ in range(n)]).astype(np.uint8)
    pots, stacks = (rng.uniform(20, 400, n).astype(np.float32) for _ in range(2))
    reach = torch.tensor(rng.random((n, 2, 1326), dtype=np.float32), device="cuda")
    w = ((torch.rand(h, 2720, device="cuda") - 0.5) / 26)
    bias = torch.randn(h, device="cuda")
    flat, wr = reach.view(n, 2652).double(), w[:, :2652].double()
    pairs = torch.tensor([(a, b) for a in range(52) for b in range(a + 1, 52)], device="cuda").repeat(2, 1)
    base = (flat @ wr.t()).float()
    percard = torch.stack([(flat * (pairs == k).any(1)) @ wr.t() for k in range(52)], 1).float()
    wcols = w[:, 2652:].t().contiguous()
    z = sorted({0, n // 2, n - 1})
    rows = datagen.boundary_encode(boards[z], pots[z], stacks[z], reach[z]).double()
    for b in (bias, None):
        want = rows @ w.double().t() + (0 if b is None else b.double())
        for bf16 in (0, 1):
            out = torch.empty(n, 2, 48, h, device="cuda", dtype=torch.bfloat16 if bf16 else torch.float32)
            N.check(N.lib().ps_boundary_first_layer(
                n, boards.ctypes.data_as(C.POINTER(C.c_uint8)), pots.ctypes.data_as(C.POINTER(C.c_float)),
                stacks.ctypes.data_as(C.POINTER(C.c_float)), C.c_void_p(base.data_ptr()),
                C.c_void_p(percard.data_ptr()), C.c_void_p(wcols.data_ptr()),
                C.c_void_p(0 if b is None else b.data_ptr()), h, C.c_void_p(out.data_ptr()), bf16,
                C.c_void_p(torch.cuda.current_stream().cuda_stream)))
            tol = (2.0**-18 + (2.0**-8 if bf16 else 0)) * want.abs().max()
            assert (out[z].double() - want).abs().max() <= tol
