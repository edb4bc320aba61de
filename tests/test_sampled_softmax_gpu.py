"""The sampled-softmax kernels against the same loss in fp64: rows that do not fill a block, classes that do not fill a chunk, accidental hits.

Products and gradients are bf16 (2^-8 per value); the sums over at most K + P terms are fp32 (below 2^-16 of the sum of magnitudes).
"""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _loss(raw, out, true_w, bias, neg, targets, S):
    def correction(ids):
        f = ids.double()
        return bias[ids] - torch.log(S * torch.log((f + 2) / (f + 1)) / math.log(bias.numel() + 1.0))
    logits = (raw + correction(neg)).masked_fill(neg[None] == targets[:, None], -1e9)
    true = (out * true_w).sum(1) + correction(targets)
    return torch.nn.functional.cross_entropy(torch.cat([true[:, None], logits], 1), torch.zeros_like(targets))


@pytest.mark.parametrize("direct,ordered", [(False, False), (True, False), (True, True)])
@pytest.mark.parametrize("N,K,P,V", [(1, 8, 8, 50), (5, 264, 24, 300), (33, 2048, 64, 60), (131, 8192, 512, 20000), (2560, 512, 128, 1000)])
def test_sampled_softmax(N, K, P, V, direct, ordered, monkeypatch):
    from autodist_b200.ops import functional as Fn
    monkeypatch.setenv("AUTODIST_DETERMINISTIC", "1" if ordered else "0")
    torch.manual_seed(N + K)
    raw = (torch.randn(N, K, device="cuda") * 3).bfloat16().requires_grad_(True)
    out, true_w = ((torch.randn(N, P, device="cuda") * P ** -0.25).bfloat16().requires_grad_(True) for _ in range(2))
    bias = (torch.randn(V, device="cuda") * 0.3).requires_grad_(True)
    # small ids, whose probabilities fp32 resolves; some of them the rows' own classes, some repeated
    neg, targets = torch.randint(0, min(V, 200), (K,), device="cuda"), torch.randint(0, min(V, 200), (N,), device="cuda")
    seen = []
    if direct:
        bias.grad = torch.full_like(bias, 0.5)
        bias._direct_grad, bias._grad_ready_hook = True, lambda p: seen.append(p)
    loss = Fn.sampled_softmax(raw, out, true_w, bias, neg, targets, K)
    (loss * 7.0).backward()
    Fn.check_errors()
    ref_in = [t.detach().double().requires_grad_(True) for t in (raw, out, true_w, bias)]
    ref = _loss(*ref_in, neg, targets, K)
    (ref * 7.0).backward()
    assert abs(loss.item() - ref.item()) <= 2.0 ** -16 * (abs(ref.item()) + 10)
    for got, want in zip((raw, out, true_w), ref_in):
        assert ((got.grad.double() - want.grad).abs() <= 2.0 ** -8 * want.grad.abs() + 2.0 ** -16 * want.grad.abs().max()).all()
    g = bias.grad.double() - (0.5 if direct else 0.0)
    # a class's gradient sums up to N probabilities and, for its own rows, (p - 1): magnitudes bounded by 7 / N per row it occurs in
    assert ((g - ref_in[3].grad).abs() <= 2.0 ** -16 * 7.0 * K).all() and (g - ref_in[3].grad).norm() <= 1e-4 * ref_in[3].grad.norm() + 1e-6
    assert len(seen) == (1 if direct else 0)


def test_refused_forms_take_the_composite_route():
    from autodist_b200.ops import functional as Fn
    raw, out = torch.randn(4, 12, device="cuda").bfloat16(), torch.randn(4, 8, device="cuda").bfloat16()
    ids = torch.zeros(12, dtype=torch.int64, device="cuda")
    b = torch.zeros(5, device="cuda")
    assert Fn.sampled_softmax(raw, out, out, b, ids, ids[:4], 12) is None                    # 12 classes: rows off 16 bytes
    assert Fn.sampled_softmax(raw[:, :8], out.float(), out, b, ids[:8], ids[:4], 8) is None
    assert Fn.sampled_softmax(raw[:, :8], out, out, b, ids[:8], ids[:4], 8) is not None      # a view: copied
