"""The updates of flat buffers and of flagged table rows at the edges of their vector forms, against the formulas in fp64.

Every step rounds a handful of fp32 operations on values of order one: 16 units in the last place of the largest value bound the difference.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu
TOL = 16 * 2.0 ** -23


def _close(a, b):
    assert (a.double() - b).abs().max().item() <= TOL * max(1.0, b.abs().max().item())


def _adagrad(p, g, s, lr, eps):
    s = s + g * g
    return p - lr * g / (s.sqrt() + eps), s


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("n", [1, 3, 4, 7, 2050, 1300007])
@pytest.mark.parametrize("rule", ["sgd", "momentum", "nesterov", "adagrad"])
def test_flat_update(rule, n, shift):
    from autodist_b200 import ops
    E = ops.ext(required=True)
    torch.manual_seed(n)
    p, g, s = (torch.randn(n + shift, device="cuda")[shift:] for _ in range(3))       # shift 1: no buffer starts on a 16-byte boundary
    s.abs_()
    p16 = torch.empty(n + shift, dtype=torch.bfloat16, device="cuda")[shift:]
    lr, step = torch.tensor([0.125], device="cuda"), torch.zeros(1, dtype=torch.int64, device="cuda")
    rp, rs = p.double(), s.double()
    for it in range(2):
        E.increment(step)
        G = g.double()
        if rule == "adagrad":
            E.adagrad_update(p, g, s, p16, lr, 1e-10, 0.0, 1.0)
            rp, rs = _adagrad(rp, G, rs, 0.125, 1e-10)
        else:
            mu = 0.0 if rule == "sgd" else 0.5
            E.sgd_update(p, g, s if mu else None, p16, lr, mu, 0.25 if rule == "momentum" else 0.0, 0.0625, rule == "nesterov", step, 0.5)
            G = 0.5 * G + 0.0625 * rp
            if mu:
                rs = G if it == 0 else mu * rs + (0.75 if rule == "momentum" else 1.0) * G
                G = G + mu * rs if rule == "nesterov" else rs
            rp = rp - 0.125 * G
    _close(p, rp)
    _close(s, rs)
    assert torch.equal(p16, p.bfloat16())


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("rows,H", [(1, 4), (3, 512), (4, 7), (127, 20), (129, 132), (50001, 8)])
@pytest.mark.parametrize("kind", [0, 1, 2])
def test_flagged_rows(kind, rows, H, shift):
    from autodist_b200 import ops
    E = ops.ext(required=True)
    torch.manual_seed(rows + H)
    p, g, s1, s2 = (torch.randn(rows * H + shift, device="cuda")[shift:] for _ in range(4))
    s1.abs_(), s2.abs_()
    flags = torch.zeros(rows + shift, dtype=torch.uint8, device="cuda")[shift:]
    flags.copy_(torch.rand(rows, device="cuda") < 0.3)
    flags[0], flags[-1] = 1, 1
    hit = flags.bool()[:, None].expand(rows, H).reshape(-1)
    p16 = p.bfloat16()
    lr, step = torch.tensor([0.125], device="cuda"), torch.tensor([3], device="cuda")
    P, G, A, B = (t.double() for t in (p, g, s1, s2))
    if kind == 0:
        want = P - 0.125 * G
    elif kind == 2:
        want, A1 = _adagrad(P, G, A, 0.125, 1e-10)
    else:
        A1, B1 = 0.5 * A + 0.5 * G, 0.75 * B + 0.25 * G * G
        want = P - 0.125 * (A1 / (1 - 0.5 ** 3)) / ((B1 / (1 - 0.75 ** 3)).sqrt() + 1e-6)
    keep16, eps = p16.clone(), 1e-6 if kind == 1 else 1e-10
    E.flagged_rows_update(p, s1, s2, p16, g, flags, rows, H, kind, lr, 0.5, 0.75, eps, step)
    _close(p, torch.where(hit, want, P))
    if kind:
        _close(s1, torch.where(hit, A1, A))
    if kind == 1:
        _close(s2, torch.where(hit, B1, B))
    assert not flags.any() and torch.equal(g, torch.where(hit, torch.zeros_like(g), G.float()))
    assert torch.equal(p16, torch.where(hit, p.bfloat16(), keep16))
