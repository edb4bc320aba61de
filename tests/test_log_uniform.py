"""Probabilities of the log-uniform sampler over vocabularies that fp32 quotients do not resolve."""
import math

import pytest
import torch


def _exact(ids, vocab):
    i = ids.double()
    return torch.log1p(1.0 / (i + 1.0)) / math.log(vocab + 1.0)


def test_probabilities_of_large_ids():
    from autodist_b200.models.lm1b import log_uniform_prob
    vocab = 50_000_000
    ids = torch.tensor([2 ** 20, 2 ** 20 + 1, 3_000_001, 2 ** 24 - 1, 2 ** 24 + 5, 40_000_003, vocab - 1])
    assert torch.allclose(log_uniform_prob(ids, vocab).double(), _exact(ids, vocab), rtol=2.0 ** -21, atol=0)


def test_smaller_ids_keep_their_values():
    from autodist_b200.models.lm1b import log_uniform_prob
    ids = torch.cat([torch.arange(1000), torch.arange(1000, 2 ** 20, 997)])
    f = ids.float()
    assert torch.equal(log_uniform_prob(ids, 793471), torch.log((f + 2.0) / (f + 1.0)) / math.log(793472.0))


@pytest.mark.gpu
def test_the_kernels_logits_over_a_large_vocabulary():
    from autodist_b200.ops import functional as Fn
    vocab, K, N = 40_000_000, 264, 50
    torch.manual_seed(3)
    neg, own = (torch.randint(2 ** 20, vocab, (n,), device="cuda") for n in (K, N))
    raw, dot = torch.randn(N, K, device="cuda").bfloat16(), torch.randn(N, device="cuda")
    loss = Fn.sampled_softmax_of(raw, dot, torch.zeros(vocab, device="cuda"), neg, own, K)
    Fn.check_errors()
    logits = torch.cat([(dot.double() - torch.log(K * _exact(own, vocab)))[:, None], raw.double() - torch.log(K * _exact(neg, vocab))], 1)
    logits[:, 1:].masked_fill_(neg[None] == own[:, None], -1e9)
    want = torch.nn.functional.cross_entropy(logits, torch.zeros_like(own))
    assert abs(loss.item() - want.item()) <= 2.0 ** -18 * (abs(want.item()) + 20)
