"""Edges of the datagen kernels: item counts around the metadata chunk, output
hands that are not adjacent pairs, tensors aligned to one value only, and the
average's gradient against the f64 formula.  Tolerances: encode and chunking
are exact; averages and gradients are f64 rounded to f32 (2^-23 relative)."""

import numpy as np
import pytest
import torch

from poker_solver_rust_b200 import datagen, trainer

pytestmark = pytest.mark.gpu


def _items(n, seed=0):
    rng = np.random.default_rng(seed)
    boards = np.stack([rng.choice(52, 4, replace=False) for _ in range(n)]).astype(np.uint8)
    reach = torch.tensor(rng.random((n, 2, 1326), dtype=np.float32), device="cuda")
    return boards, rng.uniform(20, 400, n).astype(np.float32), rng.uniform(0, 400, n).astype(np.float32), reach


def _weights(boards, reach):
    keep = trainer.river_keep_mask(boards, "cuda").double()
    w = torch.einsum("npc,nrc->npr", reach.flip(1).double(), keep)
    return keep, w, torch.einsum("npr,nrc->npc", w, keep)


@pytest.mark.parametrize("n", [1, 1024, 1025])
def test_chunks_equal_single_items(n):
    boards, pots, stacks, reach = _items(n)
    net = torch.randn(n, 2, 48, 1326, device="cuda", dtype=torch.bfloat16)
    hands = torch.arange(1326, dtype=torch.int32, device="cuda")
    rows = datagen.boundary_encode(boards, pots, stacks, reach, bf16=True)
    out = datagen.boundary_river_reduce(boards, pots, stacks, net, reach, hands)
    for i in sorted({0, n // 2, n - 1}):
        z = slice(i, i + 1)
        assert torch.equal(rows[z], datagen.boundary_encode(boards[z], pots[z], stacks[z], reach[z], bf16=True))
        assert torch.equal(out[z], datagen.boundary_river_reduce(boards[z], pots[z], stacks[z], net[z], reach[z], hands))


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("hands", ["odd", "shuffled", "one", "outside"])
def test_reduce_hands_and_alignment(bf16, hands):
    boards, pots, stacks, reach = _items(3, seed=1)
    reach[0, 1] = 0  # no weight: every value 0
    reach[1, 0, 5:] = 0  # a few hands: rivers without weight
    flat = torch.randn(3 * 2 * 48 * 1326 + 1, device="cuda").to(torch.bfloat16 if bf16 else torch.float32)
    net = flat[1:].view(3, 2, 48, 1326)  # aligned to one value
    idx = {"odd": torch.arange(1, 1326), "shuffled": torch.randperm(1326)[:701], "one": torch.tensor([77]),
           "outside": torch.tensor([-1, 0, 1326, 1325])}[hands].to(torch.int32).cuda()
    got = datagen.boundary_river_reduce(boards, pots, stacks, net, reach, idx)
    same = datagen.boundary_river_reduce(boards, pots, stacks, net.clone(), reach, idx)
    assert torch.equal(got, same)
    keep, w, den = _weights(boards, reach)
    want = torch.einsum("npr,npra,nra->npa", w, net.double(), keep) / den.clamp_min(1e-300)
    want = torch.where(den > 1e-9, want, torch.zeros_like(want)) * torch.tensor(pots.astype(np.float64) + stacks,
                                                                                device="cuda")[:, None, None]
    ok = ((idx >= 0) & (idx < 1326)).cuda()
    assert (got[:, :, ~ok] == 0).all()
    a, b = got[:, :, ok].double(), want[:, :, idx[ok].long()]
    assert (a - b).abs().max() <= 2.0**-22 * b.abs().max()


@pytest.mark.parametrize("n", [1, 3])
def test_average_gradient(n):
    boards, pots, stacks, reach = _items(n, seed=2)
    reach[0, 1] = 0
    y = torch.randn(n, 2, 48, 1326, device="cuda", requires_grad=True)
    g = torch.randn(n, 2, 1326, device="cuda")
    out = trainer.RiverAverage.apply(y, boards, pots, reach)
    (kernel,) = torch.autograd.grad(out, y, g, retain_graph=True)
    g2 = g.clone().requires_grad_()  # a differentiated gradient takes the torch formula
    (formula,) = torch.autograd.grad(out, y, g2, create_graph=True)
    assert formula.requires_grad
    assert (kernel - formula.detach()).abs().max() <= 2.0**-22 * formula.detach().abs().max()
    assert (kernel[0, 0] == 0).all()  # player 0 is weighted by the reach that was cleared


@pytest.mark.parametrize("h", [1, 7, 64, 514])
@pytest.mark.parametrize("n", [1, 1025])
def test_first_layer_widths(n, h):
    """Odd and even widths (one column or two per thread), one and several
    rounds of a block, against the dense layer in f64: the f32 products and
    sums of about 2700 terms stay within 2^-18 of the largest output."""
    boards, pots, stacks, reach = _items(n, seed=3)
    w = (torch.rand(h, 2720, device="cuda") - 0.5) / 26
    bias = torch.randn(h, device="cuda")
    z = sorted({0, n - 1})
    rows = datagen.boundary_encode(boards[z], pots[z], stacks[z], reach[z]).double()
    for b in (bias, None):
        got = datagen.boundary_first_layer(boards, pots, stacks, reach.requires_grad_(), w, b)
        want = rows @ w.double().t() + (0 if b is None else b.double())
        assert (got[z].double() - want).abs().max() <= 2.0**-18 * want.abs().max()
        half = datagen.boundary_first_layer(boards, pots, stacks, reach, w, b, bf16=True)
        assert torch.equal(half, got.to(torch.bfloat16))
