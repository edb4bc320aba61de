"""The whole-sequence LSTM layer and the dense table lookup against plain PyTorch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _reference(x, w, b, p, fb):
    B, T, _ = x.shape
    h, c = x.new_zeros(B, p.shape[0]), x.new_zeros(B, p.shape[1])
    outs = []
    for t in range(T):
        i, j, f, o = (torch.cat([x[:, t], h], 1) @ w.t() + b).chunk(4, 1)
        c = torch.sigmoid(f + fb) * c + torch.sigmoid(i) * torch.tanh(j)
        h = (torch.sigmoid(o) * torch.tanh(c)) @ p.t()
        outs.append(h)
    return torch.stack(outs, 1)


@pytest.mark.parametrize("direct", [False, True])
@pytest.mark.parametrize("B,T,D,P,S", [(1, 1, 8, 8, 8), (3, 5, 24, 16, 40), (128, 4, 64, 32, 128), (7, 9, 128, 128, 512)])
def test_lstm_layer(B, T, D, P, S, direct):
    from autodist_b200.ops import functional as Fn
    torch.manual_seed(B + T + S)
    # values that bf16 holds exactly, so that the reference starts from the same weights
    x = (torch.randn(B, T, D, device="cuda") * 0.5).bfloat16()
    w, p = ((torch.randn(*s, device="cuda") / s[1] ** 0.5).bfloat16().float().requires_grad_(True) for s in ((4 * S, D + P), (P, S)))
    b = torch.randn(4 * S, device="cuda").mul_(0.1).requires_grad_(True)
    seen = []
    if direct:
        for k, q in enumerate((w, b, p)):
            q.grad = torch.full_like(q, 0.25)
            q._direct_grad, q._grad_ready_hook = True, lambda _, k=k: seen.append(k)
    xg = x.detach().requires_grad_(True)
    out = Fn.lstm_layer(xg, w, b, p, 1.0)
    dy = torch.randn_like(out)
    out.backward(dy)
    Fn.check_errors()
    ref_in = [t.detach().double().requires_grad_(True) for t in (x, w, b, p)]
    ref = _reference(*ref_in, 1.0)
    ref.backward(dy.double())
    # every step rounds gates, state and projection to bf16 (2^-9 each); the recurrence carries them over T steps
    tol = 2.0 ** -8 * (4 + T)
    assert (out.double() - ref).norm() <= tol * ref.norm()
    got = [xg.grad, w.grad, b.grad, p.grad]
    for g, r, off in zip(got, ref_in, (0.0, 0.25, 0.25, 0.25) if direct else (0.0,) * 4):
        assert (g.double() - off - r.grad).norm() <= tol * r.grad.norm() + 1e-6
    assert sorted(seen) == ([0, 1, 2] if direct else [])


@pytest.mark.parametrize("V,H,n", [(1, 1, 3), (50, 192, 1000), (7, 6, 64), (1000, 4, 5)])
def test_dense_lookup_adds_into_the_gradient_buffer(V, H, n, monkeypatch):
    from autodist_b200.ops import functional as Fn
    torch.manual_seed(V)
    table = torch.randn(V, H, device="cuda", requires_grad=True)
    ids = torch.randint(0, V, (n,), device="cuda")
    dy = torch.randn(n, H, device="cuda")
    plain = torch.nn.functional.embedding(ids, table)
    want = torch.zeros(V, H, device="cuda", dtype=torch.float64).index_add_(0, ids, dy.double())
    table.grad, table._direct_grad = torch.ones_like(table), True
    out = Fn.dense_lookup(table, ids)
    assert torch.equal(out, plain)
    out.backward(dy)
    mag = torch.zeros(V, H, device="cuda", dtype=torch.float64).index_add_(0, ids, dy.double().abs()) + 1
    assert ((table.grad.double() - 1 - want).abs() <= n * 2.0 ** -23 * mag).all()         # n fp32 additions in any order
    monkeypatch.setenv("AUTODIST_DETERMINISTIC", "1")
    assert type(Fn.dense_lookup(table, ids).grad_fn).__name__ == "EmbeddingBackward0"
