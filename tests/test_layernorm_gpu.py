"""Layernorm kernels at the edges of their lane layout (one to four vectors of 256 columns per warp, rows that do not fill a block), against fp64.

The inputs are bf16 values, sums are fp32 over at most 1024 terms (relative error below 2^-13), results are rounded to bf16 (2^-8).
"""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _kept(n, seed, p):
    """Decisions of the counter-based dropout function for elements 0 .. n - 1: four per 64-bit hash, 16 bits each."""
    def c(x):
        return x - (1 << 64) if x >= 1 << 63 else x

    def shr(x, k):
        return (x >> k) & ((1 << (64 - k)) - 1)

    i = torch.arange((n + 3) // 4, device="cuda", dtype=torch.int64)
    x = i * c(0x9E3779B97F4A7C15) + seed
    x = (x ^ shr(x, 30)) * c(0xBF58476D1CE4E5B9)
    x = (x ^ shr(x, 27)) * c(0x94D049BB133111EB)
    x = x ^ shr(x, 31)
    bits = torch.stack([shr(x, 16 * j) & 0xFFFF for j in range(4)], 1).reshape(-1)[:n]
    return bits >= int(p * 65536.0)


@pytest.mark.parametrize("p", [0.0, 0.1, 1.0])
@pytest.mark.parametrize("rows,H", [(1, 8), (3, 248), (5, 256), (2, 264), (9, 512), (4, 520), (7, 768), (6, 776), (1201, 1024), (5000, 64)])
def test_layernorm(rows, H, p):
    from autodist_b200 import ops
    E = ops.ext(required=True)
    torch.manual_seed(rows + H)
    def bf():
        return torch.randn(rows, H, device="cuda").bfloat16()
    x, res, dy, dadd = bf(), bf(), bf(), bf()
    gamma, beta = torch.rand(H, device="cuda") + 0.5, torch.randn(H, device="cuda")
    z, y, dz, dx = (torch.empty_like(x) for _ in range(4))
    mean, rstd = torch.empty(rows, device="cuda"), torch.empty(rows, device="cuda")
    step = torch.tensor([3], device="cuda")
    eps = 1e-3
    E.ln_fwd(x, res, gamma, beta, z, y, mean, rstd, eps, p, 7, step)
    scale = torch.zeros(rows, H, device="cuda", dtype=torch.float64)
    if p == 0.0:
        scale.fill_(1.0)
    elif p < 1.0:
        scale[_kept(rows * H, 7 + 3 * 0x100000001B3, p).view(rows, H)] = float(torch.tensor(1.0) / (1.0 - torch.tensor(p)))
    v = x.double() * scale + res.double()
    slack = 2.0 ** -22 * ((x.double() * scale).abs() + res.double().abs())           # the two fp32 terms may cancel
    assert ((z.double() - v).abs() <= 2.0 ** -8 * v.abs() + slack).all()
    mu, var = v.mean(1, keepdim=True), v.var(1, unbiased=False, keepdim=True)
    want = (v - mu) * (var + eps).rsqrt() * gamma.double() + beta.double()
    assert ((y.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -12).all()
    assert (mean.double() - mu[:, 0]).abs().max() < 2.0 ** -13 * 4
    # backward, from the stored statistics
    part = torch.zeros(E.ln_bwd_part_floats(H), device="cuda")
    dg, db, ds = (torch.empty(H, device="cuda") for _ in range(3))
    E.ln_bwd(dy, z, mean, rstd, gamma, dadd, dz, dx if p > 0 else None, part, dg, db, p, 7, step, False, ds)
    xh = (z.double() - mean.double()[:, None]) * rstd.double()[:, None]
    g = dy.double() * gamma.double()
    o = rstd.double()[:, None] * (g - g.mean(1, keepdim=True) - xh * (g * xh).mean(1, keepdim=True))
    slack = 2.0 ** -12 * (rstd.double()[:, None] * (g.abs() + 1 + xh.abs()))       # fp32 terms that cancel
    want = o + dadd.double()
    assert ((dz.double() - want).abs() <= 2.0 ** -8 * want.abs() + slack).all()
    out = dz
    if p > 0:
        want = want * scale
        assert ((dx.double() - want).abs() <= 2.0 ** -8 * want.abs() + slack * 1.2).all()
        out = dx
    for got, terms in ((dg, dy.double() * xh), (db, dy.double()), (ds, out.double())):
        assert ((got.double() - terms.sum(0)).abs() <= 2.0 ** -18 * terms.abs().sum(0) + 1e-6).all()
    assert not part.any()
