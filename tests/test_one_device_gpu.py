"""Tensors on the host are refused before a kernel gets their addresses: as the library refuses them where it is the other route, by an
error of the binding where it is called directly."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _tables():
    tables = [torch.randn(9, 24, device="cuda").requires_grad_(True) for _ in range(2)]
    for t in tables:
        t.grad, t._direct_grad = torch.zeros_like(t), True
    return tables


def test_host_ids_of_a_pair_lookup():
    from autodist_b200 import ops
    from autodist_b200.models.ncf import NeuMF, NeuMFConfig
    from autodist_b200.ops import functional as Fn
    E = ops.ext(required=True)
    tables, dev = _tables(), torch.zeros(5, dtype=torch.int64, device="cuda")
    host = dev.cpu()
    assert Fn.pair_lookup(*tables, dev, dev, 8) is not None
    m = NeuMF(NeuMFConfig.tiny(dense_gradient=True)).cuda()
    for t in (m.user_emb, m.item_emb):
        t.grad, t._direct_grad = torch.zeros_like(t), True
    for users, items in ((host, dev), (dev, host), (host, host)):
        assert Fn.pair_lookup(*tables, users, items, 8) is None
        with pytest.raises(RuntimeError):
            m.logits(users, items)
        out = [torch.empty(5, w, dtype=d, device="cuda") for w, d in ((8, torch.float32), (32, torch.bfloat16), (16, torch.float32))]
        with pytest.raises(RuntimeError, match="one GPU"):
            E.pair_lookup(tables[0].detach(), tables[1].detach(), users, items, 8, *out, torch.zeros(1, dtype=torch.int32, device="cuda"))
        with pytest.raises(RuntimeError, match="one GPU"):
            E.pair_lookup_bwd(out[0], out[1], out[2], users, items, tables[0].grad, tables[1].grad)


def test_host_tensors_of_the_losses():
    from autodist_b200 import ops
    from autodist_b200.ops import functional as Fn
    E = ops.ext(required=True)
    x, y = torch.randn(7, device="cuda", requires_grad=True), torch.zeros(7, device="cuda")
    with pytest.raises(RuntimeError):
        Fn.bce_with_logits(x, y.cpu())
    with pytest.raises(RuntimeError, match="one GPU"):
        E.bce_logits(x.detach(), y.cpu(), torch.empty(1, device="cuda"), 1.0)
    with pytest.raises(RuntimeError, match="one GPU"):
        E.bce_logits_bwd(x.detach(), y, torch.ones(()), torch.empty_like(y), 1.0)
    raw, dot = torch.randn(4, 8, device="cuda").bfloat16(), torch.randn(4, device="cuda").bfloat16()
    bias, neg, own = torch.zeros(9, device="cuda"), torch.zeros(8, dtype=torch.int64, device="cuda"), torch.zeros(4, dtype=torch.int64, device="cuda")
    args = [raw, dot, bias, neg, own]
    assert Fn.sampled_softmax_of(*args, 8) is not None
    scratch = [torch.empty(12, 2, device="cuda"), torch.empty(12, dtype=torch.int32, device="cuda"), torch.empty(4, 9, device="cuda")]
    for k in range(5):
        mixed = [t.cpu() if i == k else t for i, t in enumerate(args)]
        assert Fn.sampled_softmax_of(*mixed, 8) is None
        if k > 0:
            with pytest.raises(RuntimeError, match="one GPU"):
                E.sampled_logits(*mixed, 0.5, 8.0, *scratch, torch.zeros(1, dtype=torch.int32, device="cuda"))
