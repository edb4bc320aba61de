"""The row-walking batch-norm passes at channel counts and row counts where their layout changes, against fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("relu,with_res", [(True, False), (True, True), (False, True), (False, False)])
@pytest.mark.parametrize("n,c,h", [(1, 8, 3), (2, 24, 1), (3, 96, 17), (2, 1000, 5), (5, 2048, 4), (2, 2056, 3), (1, 4096, 2), (64, 64, 14)])
def test_training_batch_norm(n, c, h, relu, with_res):
    from autodist_b200.ops import functional as Fn
    torch.manual_seed(c + n)
    store = torch.randn(2 * c + 1, device="cuda")                       # parameters that start off a 16-byte boundary
    gamma, beta = store[1:c + 1].clone().requires_grad_(True), store[c + 1:].detach().requires_grad_(True)
    x = torch.randn(n, c, h, h, device="cuda").bfloat16().contiguous(memory_format=torch.channels_last).requires_grad_(True)
    res = torch.randn(n, c, h, h, device="cuda").bfloat16().contiguous(memory_format=torch.channels_last).requires_grad_(True) if with_res else None
    rm, rv = torch.zeros(c, device="cuda"), torch.ones(c, device="cuda")
    y = Fn.batch_norm(x, gamma, beta, rm, rv, True, 0.1, 1e-3, relu, res)
    dy = torch.randn_like(y)
    y.backward(dy)
    xd, gd, bd = (t.detach().double().requires_grad_(True) for t in (x, gamma, beta))
    rd = res.detach().double().requires_grad_(True) if with_res else None
    mean, var = torch.zeros(c, device="cuda", dtype=torch.float64), torch.ones(c, device="cuda", dtype=torch.float64)
    z = torch.nn.functional.batch_norm(xd, mean, var, gd, bd, True, 0.1, 1e-3)
    z = z + rd if with_res else z
    # the mask the kernel used: y as stored; where fp64 and bf16 disagree the value is within rounding of zero
    ref = torch.where(y.detach() > 0, z, torch.zeros_like(z)) if relu else z
    ref.backward(dy.double())
    rows = n * h * h
    tol = 2.0 ** -8                                                     # results are rounded to bf16; sums are fp32 (2^-20 of sum |terms|)
    assert ((y.detach().double() - (z.clamp_min(0) if relu else z)).abs() <= tol * z.abs() + 1e-4).all()
    rstd = (xd.detach().var((0, 2, 3), unbiased=False) + 1e-3).rsqrt().view(1, -1, 1, 1)
    scale = gd.detach().abs().view(1, -1, 1, 1) * rstd
    assert ((x.grad.double() - xd.grad).abs() <= tol * xd.grad.abs() + 2.0 ** -14 * scale * 8).all()
    s = dy.abs().double().sum((0, 2, 3))
    assert ((beta.grad.double() - bd.grad).abs() <= 2.0 ** -18 * s + 1e-6).all()
    assert ((gamma.grad.double() - gd.grad).abs() <= 2.0 ** -15 * s * 5 + 1e-5).all()
    if with_res:
        assert ((res.grad.double() - rd.grad).abs() <= tol * rd.grad.abs()).all()
    if rows > 1:
        assert ((rm.double() - mean).abs() <= 1e-5 + 1e-5 * mean.abs()).all() and ((rv.double() - var).abs() <= 1e-4 * var.abs() + 1e-5).all()
