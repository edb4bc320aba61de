"""The auxiliary operand of the GEMM epilogue (addend, GELU derivative) where it travels by TMA - the 256-wide and the two-CTA tiles -
with several tiles per CTA, ragged extents, batches and an output that is its own addend."""
import pytest
import torch

from test_gemm_split_gpu import _close, _operands

pytestmark = pytest.mark.gpu

ADD, MUL_GELU_GRAD = 4, 3


def _aux(M, N, batch, ldc):
    return (torch.randn(batch, M, ldc, device="cuda") * 1.5).bfloat16()[..., :N]


# (M, N, K, batch): fewer tiles than CTAs; two to five tiles per CTA with ragged last rows and columns; a short and a long contraction
@pytest.mark.parametrize("M,N,K,batch", [(256, 512, 256, 1), (5000, 1800, 72, 1), (900, 1288, 136, 5), (3001, 2600, 1032, 1)])
@pytest.mark.parametrize("bn", [256, 512])
def test_auxiliary_operand(M, N, K, batch, bn):
    from autodist_b200 import ops
    E = ops.ext(required=True)
    torch.manual_seed(M + bn)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    a, b, ref, mag = _operands(M, N, K, False, True, batch)
    alpha = 0.5
    for ldc in (N, N + 8):                                                # tight rows and rows that lie further apart
        x = _aux(M, N, batch, ldc)
        x64 = x.double()
        out = torch.full((batch, M, ldc), float("nan"), dtype=torch.bfloat16, device="cuda")
        E.gemm(a, b, out[..., :N], False, True, ADD, None, None, x, alpha, 0.0, err, bn)
        _close(out[..., :N], alpha * ref + x64, alpha * mag + x64.abs(), K, 2.0 ** -8)
        assert torch.isnan(out[..., N:]).all()                             # nothing past the matrix is written
        own = x.clone() if ldc == N else _aux(M, N, batch, ldc).copy_(x)
        E.gemm(a, b, own, False, True, ADD, None, None, own, alpha, 0.0, err, bn)
        assert torch.equal(own, out[..., :N])                              # its own addend
        E.gemm(a, b, out[..., :N], False, True, MUL_GELU_GRAD, None, None, x, alpha, 0.0, err, bn)
        k = 0.7978845608028654
        t = torch.tanh(k * (x64 + 0.044715 * x64 ** 3))
        dt = k * (1 + 3 * 0.044715 * x64 ** 2)
        want = alpha * ref * (0.5 * (1 + t) + 0.5 * x64 * (1 - t * t) * dt)
        # tanh.approx: 2^-11 relative, so the derivative errs by 2^-11 * (0.5 + |x t| dt); one bf16 rounding (doubled); the sums as in _close
        bound = (alpha * ref).abs() * 2.0 ** -10.9 * (0.5 + (x64 * t).abs() * dt) + 1.2 * alpha * K * 2.0 ** -22 * mag + 2.0 ** -8 * want.abs() + 1e-30
        worst = ((out[..., :N].double() - want).abs() / bound).max().item()
        assert worst <= 1.0, f"{worst} times the bound"
    assert err.item() == 0
