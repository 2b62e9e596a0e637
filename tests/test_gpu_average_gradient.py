"""RiverAverage.backward where something looks through the gradient: batched
gradients, derivatives of the gradient with respect to the reach, forward-mode
tangents, negative views and values that are not finite.  Each is compared with
the formula of the backward in f64 (within the f32 rounding of the result,
2^-23 relative, and as much for the tangents and second derivatives that torch
rounds to f32)."""

import numpy as np
import pytest
import torch
from torch.autograd import forward_ad

from poker_solver_rust_b200 import trainer

pytestmark = pytest.mark.gpu


def _case(n, seed=0):
    rng = np.random.default_rng(seed)
    boards = np.stack([rng.choice(52, 4, replace=False) for _ in range(n)]).astype(np.uint8)
    reach = torch.tensor(rng.random((n, 2, 1326), dtype=np.float32), device="cuda")
    scale = rng.uniform(20, 400, n).astype(np.float32)
    y = torch.tensor(rng.normal(0, 1, (n, 2, 48, 1326)).astype(np.float32), device="cuda", requires_grad=True)
    return boards, scale, reach, y


def _formula(boards, scale, reach, g):
    """d/dy of sum(g * average) in f64."""
    keep = trainer.river_keep_mask(boards, "cuda").double()
    w = torch.einsum("npc,nrc->npr", reach.double().flip(1), keep)
    den = torch.einsum("npr,nrc->npc", w, keep)
    k = g.double() * torch.tensor(scale, device="cuda").double()[:, None, None] / den
    return w[..., None] * keep[:, None] * k[:, :, None]


def _close(a, b):
    assert (a.double() - b).abs().max() <= 2.0**-22 * b.abs().max()


def test_batched_gradients():
    boards, scale, reach, y = _case(2)
    out = trainer.RiverAverage.apply(y, boards, scale, reach)
    g = torch.randn(3, *out.shape, device="cuda")
    (got,) = torch.autograd.grad(out, y, g, is_grads_batched=True)
    for k in range(3):
        _close(got[k], _formula(boards, scale, reach, g[k]))


def test_second_derivative_with_respect_to_the_reach():
    boards, scale, reach, y = _case(1, seed=1)
    r = reach.requires_grad_()
    out = trainer.RiverAverage.apply(y, boards, scale, r)
    g = torch.randn_like(out)
    (grad,) = torch.autograd.grad(out, y, g, create_graph=True)
    v = torch.randn_like(grad)
    (got,) = torch.autograd.grad((grad * v).sum(), r)
    r2 = reach.detach().clone().requires_grad_()
    (want,) = torch.autograd.grad((_formula(boards, scale, r2, g) * v).sum(), r2)
    assert (got - want).abs().max() <= 1e-4 * want.abs().max()


def test_forward_mode_tangent():
    boards, scale, reach, y = _case(1, seed=2)
    out = trainer.RiverAverage.apply(y, boards, scale, reach)
    g, t = torch.randn_like(out), torch.randn_like(out)
    with forward_ad.dual_level():
        (grad,) = torch.autograd.grad(out, y, forward_ad.make_dual(g, t))
        value, tangent = forward_ad.unpack_dual(grad)
    _close(value, _formula(boards, scale, reach, g))
    _close(tangent, _formula(boards, scale, reach, t))  # linear in g


def test_negative_view():
    boards, scale, reach, y = _case(1, seed=3)
    out = trainer.RiverAverage.apply(y, boards, scale, reach)
    g = torch.randn_like(out)
    (got,) = torch.autograd.grad(out, y, torch._neg_view(g))
    _close(got, _formula(boards, scale, reach, -g))


def test_non_finite_gradient():
    """A blocked river's weight is zero times the coefficient, as in the formula."""
    boards, scale, reach, y = _case(1, seed=4)
    out = trainer.RiverAverage.apply(y, boards, scale, reach)
    g = torch.randn_like(out)
    g[0, 0, ::7], g[0, 1, ::5], g[0, 1, 3::5] = float("inf"), float("nan"), float("-inf")
    (got,) = torch.autograd.grad(out, y, g)
    want = _formula(boards, scale, reach, g)
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())


def test_reach_on_another_device_is_refused():
    """A saved-tensor hook that hands the reach back on the host: no kernel may take its address."""
    boards, scale, reach, y = _case(1, seed=5)
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t.cpu(), lambda t: t):
        out = trainer.RiverAverage.apply(y, boards, scale, reach)
    with pytest.raises(RuntimeError):
        torch.autograd.grad(out, y, torch.randn_like(out))
