"""Pair lookups, binary cross-entropy and many-row column sums against plain PyTorch in fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,mf,h,nu,ni", [(1, 4, 4, 1, 3), (7, 8, 20, 5, 9), (1000, 64, 128, 50, 30), (4097, 12, 8, 3, 2)])
def test_pair_lookup(n, mf, h, nu, ni):
    from autodist_b200.ops import functional as Fn
    torch.manual_seed(n)
    tables = [torch.randn(k, mf + h, device="cuda").requires_grad_(True) for k in (nu, ni)]
    users, items = torch.randint(0, nu, (n,), device="cuda"), torch.randint(0, ni, (n,), device="cuda")
    assert Fn.pair_lookup(*tables, users, items, mf) is None                     # no flat gradient buffers: the library's lookups
    seen = []
    for t in tables:
        t.grad = torch.full_like(t, 0.5)
        t._direct_grad, t._grad_ready_hook = True, seen.append
    gmf, x = Fn.pair_lookup(*tables, users, items, mf)
    u, i = (t.detach().double().requires_grad_(True) for t in tables)
    ru, ri = u[users], i[items]
    want = ru[:, :mf] * ri[:, :mf], torch.cat([ru[:, mf:], ri[:, mf:]], 1)
    assert torch.allclose(gmf.double(), want[0], rtol=2.0 ** -23) and torch.equal(x, want[1].float().bfloat16())
    dboth = torch.randn(n, mf + 4, device="cuda")                                # a slice, as the gradient of a concatenation arrives
    dgmf, dx = dboth[:, :mf], torch.randn_like(x.float()).bfloat16()
    torch.autograd.backward([gmf, x], [dgmf, dx])
    torch.autograd.backward(list(want), [dgmf.double(), dx.double()])
    Fn.check_errors()
    for t, r in zip(tables, (u, i)):                                             # up to n additions per element in fp32, any order
        assert ((t.grad.double() - 0.5 - r.grad).abs() <= 2.0 ** -22 * (n * 4.0) ** 0.5 * 4 + 2.0 ** -16 * r.grad.abs()).all()
    assert len(seen) == 2


@pytest.mark.parametrize("n", [1, 31, 1025, 16384, 16385, 70000])
def test_bce_with_logits(n):
    from autodist_b200.ops import functional as Fn
    torch.manual_seed(n)
    x = (torch.randn(n, device="cuda") * 20).requires_grad_(True)
    y = (torch.rand(n, device="cuda") < 0.3).float()
    (Fn.bce_with_logits(x, y) * 3).backward()
    r = x.detach().double().requires_grad_(True)
    ref = torch.nn.functional.binary_cross_entropy_with_logits(r, y.double())
    (ref * 3).backward()
    assert abs(Fn.bce_with_logits(x, y).item() - ref.item()) <= 2.0 ** -18 * ref.item() + 1e-9
    assert ((x.grad.double() - r.grad).abs() <= 2.0 ** -20 * r.grad.abs() + 2.0 ** -22 / n * 3).all()


def test_hooked_layers_keep_their_own_inputs():
    """A watched layer gets the tables' dtype, as on the plain route; results agree within the roundings of bf16."""
    from autodist_b200.models.ncf import NeuMF, NeuMFConfig
    torch.manual_seed(3)
    m = NeuMF(NeuMFConfig.tiny(dense_gradient=True)).cuda()
    for p in m.parameters():
        p.grad = torch.zeros_like(p)
    for t in (m.user_emb, m.item_emb):
        t._direct_grad = True
    users, items = torch.randint(0, 200, (65,), device="cuda"), torch.randint(0, 120, (65,), device="cuda")
    labels = (torch.arange(65, device="cuda") % 5 == 0).float()
    runs = []
    for hooked in (False, True):
        types = []
        h = m.mlp[1].register_forward_pre_hook(lambda _, a: types.append(a[0].dtype)) if hooked else None
        for p in m.parameters():
            p.grad.zero_()
        loss = m(users, items, labels)
        loss.backward()
        runs.append([loss.detach()] + [p.grad.clone() for p in m.parameters()])
        if h is not None:
            h.remove()
            assert types == [torch.float32]
    for a, b in zip(*runs):
        assert (a - b).norm() <= 2.0 ** -7 * b.norm() + 1e-7


@pytest.mark.parametrize("rows,H", [(255, 8), (4096, 72), (5000, 64), (16384, 256), (20000, 24)])
def test_column_sums_of_many_rows(rows, H):
    from autodist_b200 import ops
    E = ops.ext(required=True)
    x = torch.randn(rows, H, device="cuda").bfloat16()
    out = torch.ones(H, device="cuda")
    part = torch.empty(E.colsum_parts(rows) * H, device="cuda")
    E.keyed_colsum(x, None, part, out, 1, True)
    s = x.double()
    assert ((out.double() - 1 - s.sum(0)).abs() <= 2.0 ** -18 * s.abs().sum(0)).all()
