"""Cross-entropy at infinite, huge and undefined logits: the library's values, one logit at a time."""
import math

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("logit", [math.inf, -math.inf, math.nan, 3e38, -3e38, 100.0, -100.0, 0.0])
@pytest.mark.parametrize("label", [0.0, 1.0, 0.25])
def test_extreme_logits(logit, label):
    from autodist_b200.ops import functional as Fn
    found = []
    for loss in (Fn.bce_with_logits, F.binary_cross_entropy_with_logits):
        x = torch.full((1,), logit, device="cuda", requires_grad=True)
        v = loss(x, torch.full((1,), label, device="cuda"))
        v.backward()
        found.append(torch.stack([v.detach(), x.grad[0]]))
    assert torch.allclose(found[0], found[1], rtol=2.0 ** -22, atol=1e-30, equal_nan=True)
