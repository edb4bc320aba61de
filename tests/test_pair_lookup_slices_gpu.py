"""Gradients that reach the pair lookup as slices of larger tensors, starting anywhere."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("off_gmf,off_x", [(0, 1), (1, 0), (3, 2), (2, 5)])
def test_gradients_off_a_vector(off_gmf, off_x):
    from autodist_b200.ops import functional as Fn
    torch.manual_seed(off_x)
    found = []
    for shifted in (False, True):
        torch.manual_seed(9)
        tables = [torch.randn(k, 24, device="cuda").requires_grad_(True) for k in (30, 40)]
        for t in tables:
            t.grad, t._direct_grad = torch.zeros_like(t), True
        users, items = torch.arange(20, device="cuda"), torch.arange(20, device="cuda") + 5      # one addition per element: no order to it
        gmf, x = Fn.pair_lookup(*tables, users, items, 8)
        dgmf, dx = torch.randn(20 * 8 + 8, device="cuda"), torch.randn(20 * 32 + 8, device="cuda").bfloat16()
        slices = dgmf[off_gmf:off_gmf + 160].view(20, 8), dx[off_x:off_x + 640].view(20, 32)
        torch.autograd.backward([gmf, x], list(slices) if shifted else [t.clone() for t in slices])
        found.append([t.grad for t in tables])
    assert all(torch.equal(a, b) for a, b in zip(*found)) and found[0][0].abs().sum() > 0
