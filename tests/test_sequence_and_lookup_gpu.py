"""The dense table lookup against plain PyTorch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


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
