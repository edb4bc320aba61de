"""The cross-entropy's derivatives beyond the first, forward mode and vmap: as the library's loss gives them."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _data(n=37):
    torch.manual_seed(n)
    return torch.randn(n, 6, device="cuda"), torch.randn(6, device="cuda", requires_grad=True), (torch.rand(n, device="cuda") < 0.4).float()


def test_second_derivatives_through_a_head():
    from autodist_b200.ops import functional as Fn
    found = []
    for loss in (Fn.bce_with_logits, F.binary_cross_entropy_with_logits):
        x, w, y = _data()
        g, = torch.autograd.grad(loss(x @ w, y) * 3, w, create_graph=True)
        assert g.requires_grad
        found.append(torch.cat([g.detach(), torch.autograd.grad(g.square().sum(), w)[0]]))
    assert torch.allclose(found[0], found[1], rtol=1e-5, atol=1e-7)


def test_hessian_forward_mode_and_vmap():
    from autodist_b200.ops import functional as Fn
    found = []
    for loss in (Fn.bce_with_logits, F.binary_cross_entropy_with_logits):
        x, w, y = _data()
        w = w.detach()
        hess = torch.func.hessian(lambda v: loss(x @ v, y))(w)
        _, slope = torch.func.jvp(lambda v: loss(x @ v, y), (w,), (torch.ones_like(w),))
        each = torch.func.vmap(lambda v: loss(x @ v, y))(torch.stack([w, 2 * w, -w]))
        with torch.autograd.forward_ad.dual_level():
            dual = torch.autograd.forward_ad.make_dual(w, torch.ones_like(w))
            tangent = torch.autograd.forward_ad.unpack_dual(loss(x @ dual, y)).tangent
        found.append([hess, slope, each, tangent])
    for a, b in zip(*found):
        assert torch.allclose(a, b, rtol=1e-5, atol=1e-7)
