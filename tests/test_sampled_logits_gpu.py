"""The sampled softmax's kernels repeat, bit for bit, what the expression they stand for gives: logits off the edges of blocks, accidental hits,
repeated ids, ids over the whole vocabulary, more places than the ordered bias sums take at once."""
import math

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _expression(raw, dot, bias, neg, targets, S):
    def count(ids):
        f = ids.float()
        return torch.log(S * (torch.log((f + 2.0) / (f + 1.0)) / math.log(bias.numel() + 1.0)))
    own = dot.float() + bias[targets] - count(targets)
    others = raw.float() + bias[neg]
    others = (others - count(neg)).masked_fill(neg[None, :] == targets[:, None], -1e9)
    return F.cross_entropy(torch.cat([own[:, None], others], 1), torch.zeros_like(targets))


@pytest.mark.parametrize("N,K,V,dtype", [(1, 8, 50, torch.bfloat16), (5, 264, 300, torch.float32), (33, 2048, 60, torch.bfloat16),
                                         (131, 8192, 793471, torch.bfloat16), (2560, 8192, 793471, torch.bfloat16), (2563, 1032, 5000, torch.float32),
                                         (32000, 1024, 4000, torch.bfloat16)])
def test_bits_of_the_expression(N, K, V, dtype):
    from autodist_b200.ops import functional as Fn
    torch.manual_seed(N + K)
    def ids(n):
        return (torch.rand(n, device="cuda") * math.log(V + 1.0)).exp().long().clamp_(1, V) - 1
    neg, targets = ids(K), ids(N)
    raw, dot = (torch.randn(N, K, device="cuda") * 3).bfloat16(), (torch.randn(N, device="cuda") * 3).to(dtype)
    bias = torch.randn(V, device="cuda") * 0.3
    runs = []
    for fn in (Fn.sampled_softmax_of, Fn.sampled_softmax_of, _expression):
        args = [t.clone().requires_grad_(True) for t in (raw, dot, bias)]
        loss = fn(*args, neg, targets, K)
        (loss * 20).backward()
        runs.append([loss.detach()] + [t.grad for t in args])
    Fn.check_errors()
    assert all(torch.equal(a, b) for a, b in zip(runs[0], runs[1]))             # repeats itself
    assert all(torch.equal(a, b) for a, b in zip(runs[0][:3], runs[2][:3]))     # loss, gradients of the products and of dot
    a, b = runs[0][3].double(), runs[2][3].double()                             # fp32 sums of up to N terms in another order
    assert (a - b).norm() <= 2.0 ** -20 * math.sqrt(N) * b.norm()


def test_a_gradient_that_is_differentiated_again():
    from autodist_b200.ops import functional as Fn
    torch.manual_seed(1)
    neg, targets = torch.randint(0, 40, (16,), device="cuda"), torch.randint(0, 40, (6,), device="cuda")
    found = []
    for fn in (Fn.sampled_softmax_of, _expression):
        torch.manual_seed(2)
        args = [torch.randn(6, 16, device="cuda").bfloat16(), torch.randn(6, device="cuda"), torch.randn(40, device="cuda")]
        args = [t.requires_grad_(True) for t in args]
        d_bias, = torch.autograd.grad(fn(*args, neg, targets, 16), args[2:], create_graph=True)
        found.append(torch.autograd.grad(d_bias.square().sum(), args[1:]))
    for a, b in zip(*found):
        assert b.abs().max() > 0 and torch.allclose(a, b, rtol=1e-4, atol=1e-7)


@pytest.mark.parametrize("seed", [0, 1])
def test_lm1b_step_repeats_the_composite(seed, monkeypatch):
    """Gradients of the recurrent layer, which twenty steps of rounding stand in front of."""
    from autodist_b200.models import lm1b
    c = lm1b.LM1BConfig(vocab_size=3000, emb_size=64, state_size=256, projected_size=64, num_sampled=512, num_steps=20)
    runs = []
    for composite in (False, False, True):
        torch.manual_seed(seed)
        with torch.device("cuda"):
            m = lm1b.LM1B(c)
        batch = {k: v.cuda() for k, v in lm1b.zipf_tokens(16, 20, 3000, seed=seed).items()}
        if composite:
            for name in ("sampled_softmax_of", "sampled_softmax"):
                monkeypatch.setattr(lm1b, name, lambda *a: None, raising=False)
        torch.manual_seed(seed + 10)
        loss = m(batch["x"], batch["y"])
        loss.backward()
        runs.append([loss.detach(), m.W.grad, m.B.grad, m.W_P.grad])
    assert all(torch.equal(a, b) and torch.equal(a, c) for a, b, c in zip(*runs))
