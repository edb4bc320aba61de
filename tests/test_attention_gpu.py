"""Fused attention kernels against fp64, with the dropout decisions of the stand-alone softmax kernel."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _decisions(count, pd, seed):
    """Which of ``count`` scores dropout keeps: 16 bits of a counter-based 64-bit hash each, four per counter."""
    def wrap(v):
        return v - (1 << 64) if v >= 1 << 63 else v

    def shift(x, n):                                            # logical, on signed words
        return (x >> n) & ((1 << (64 - n)) - 1)
    x = torch.arange((count + 3) // 4, dtype=torch.int64, device="cuda") * wrap(0x9E3779B97F4A7C15) + wrap(seed & ((1 << 64) - 1))
    x = (x ^ shift(x, 30)) * wrap(0xBF58476D1CE4E5B9)
    x = (x ^ shift(x, 27)) * wrap(0x94D049BB133111EB)
    x = x ^ shift(x, 31)
    fields = torch.stack([shift(x, 16 * j) & 0xFFFF if j else x & 0xFFFF for j in range(4)], 1).reshape(-1)[:count]
    return fields >= int(pd * 65536)


def _run(B, S, nh, pd, seed=5, masked=True, mask=None):
    from autodist_b200 import ops
    E = ops.ext(required=True)
    torch.manual_seed(B * S + nh)
    dev, H = "cuda", nh * 64
    err = torch.zeros(1, dtype=torch.int32, device=dev)
    step = torch.tensor([3], dtype=torch.int64, device=dev)
    qkv = (torch.randn(B * S, 3 * H, device=dev) * 1.5).bfloat16()
    if mask is None and masked:
        mask = torch.zeros(B, S, device=dev)
        for b in range(B):
            mask[b, S - (b * 7) % (S // 4 + 1):] = -10000.0
    scale = 1 / math.sqrt(64)
    ctx, dqkv = torch.empty(B * S, H, device=dev, dtype=torch.bfloat16), torch.full_like(qkv, float("nan"))
    lse = torch.empty(B, nh, S, device=dev)
    keep_bits = torch.full((B, nh, S, (S + 127) // 128 * 4), -1, dtype=torch.int32, device=dev) if pd > 0 else None
    E.attn_fwd(qkv, mask, ctx, lse, B, S, nh, scale, pd, seed, step, err, keep_bits)
    dctx = torch.randn(B * S, H, device=dev).bfloat16()
    E.attn_bwd(qkv, mask, ctx, dctx, lse, torch.empty_like(lse), dqkv, B, S, nh, scale, pd, err, keep_bits)
    torch.cuda.synchronize()
    assert err.item() == 0
    keep = torch.ones(B, nh, S, S, device=dev, dtype=torch.float64)
    if pd > 0 and S not in (64, 128, 256, 512, 1024):          # the softmax kernels take no such rows: the same decisions row by row
        keep = _decisions(B * nh * S * S, pd, seed + int(step) * 0x100000001B3).view(B, nh, S, S).double() / (1 - pd)
    elif pd > 0:
        zero, u, d = torch.zeros(B, nh, S, S, device=dev, dtype=torch.bfloat16), *(torch.empty(B, nh, S, S, device=dev, dtype=torch.bfloat16) for _ in range(2))
        E.softmax_fwd(zero, None, u, d, 1.0, pd, seed, step)
        keep = (d != 0).double() / (1 - pd)
        assert 0.5 * pd < (d == 0).float().mean().item() < 2 * pd
    q, k, v = (t.double() for t in qkv.view(B, S, 3, nh, 64).permute(2, 0, 3, 1, 4))
    g = dctx.double().view(B, S, nh, 64).permute(0, 2, 1, 3)
    s = q @ k.transpose(-1, -2) * scale + (0 if mask is None else mask.double()[:, None, None])
    P = torch.softmax(s, -1)
    Pk = P * keep
    o = Pk @ v
    dP = (g @ v.transpose(-1, -2)) * keep
    D = (P * dP).sum(-1, keepdim=True)
    dS = P * (dP - D) * scale
    grads = (dS @ k, dS.transpose(-1, -2) @ q, Pk.transpose(-1, -2) @ g)
    # bounds: P and dS are rounded to bf16 (2^-9) before their products; the row sums come from the rounded context (2^-9 of sum |dO| |O|);
    # fp32 scores and exponentials err by about 2^-18 of P; the results are rounded to bf16 (2^-9); doubled
    ep, u = 2.0 ** -9 + 2.0 ** -17, 2.0 ** -8
    dD = 2.0 ** -9 * (g.abs() * o.abs()).sum(-1, keepdim=True)
    eS = ep * dS.abs() + scale * P * (dD + 2.0 ** -17 * (dP.abs() + D.abs()))
    bounds = (2 * eS @ k.abs(), 2 * eS.transpose(-1, -2) @ q.abs(), 2 * ep * Pk.transpose(-1, -2) @ g.abs())
    got = [t.double() for t in dqkv.view(B, S, 3, nh, 64).permute(2, 0, 3, 1, 4)]
    out = ctx.double().view(B, S, nh, 64).permute(0, 2, 1, 3)
    assert ((out - o).abs() <= 2 * ep * Pk @ v.abs() + u * o.abs() + 1e-6).all()
    assert ((lse.double() - torch.logsumexp(s, -1)).abs() <= 1e-4).all()
    for name, a, r, e in zip("qkv", got, grads, bounds):
        worst = ((a - r).abs() / (e + u * r.abs() + 1e-6)).max().item()
        assert worst <= 1.0, f"d{name}: {worst} times the bound"
    return out, got


@pytest.mark.parametrize("pd", [0.0, 0.1])
@pytest.mark.parametrize("B,S,nh", [(1, 64, 1), (3, 128, 2), (2, 256, 3), (1, 512, 2), (1, 1024, 1), (20, 128, 16), (5, 64, 7), (9, 256, 12)])
def test_attention_matches_fp64(B, S, nh, pd):
    _run(B, S, nh, pd)


@pytest.mark.parametrize("low", [-math.inf, torch.finfo(torch.float32).min])
@pytest.mark.parametrize("B,S,nh", [(2, 64, 2), (3, 256, 2), (2, 512, 1)])
def test_keys_out_of_reach(B, S, nh, low):
    """Masks of minus infinity and of the lowest float, among them whole leading tiles, with at least one key left per row."""
    mask = torch.zeros(B, S, device="cuda")
    mask[0, :S // 2 + 9] = low
    mask[1, 3:] = low
    mask[1, S - 1] = 0.0
    if B > 2:
        mask[2, ::3] = low
    _run(B, S, nh, 0.1, mask=mask)


def test_a_row_without_any_key_is_not_a_number():
    from autodist_b200 import ops
    E = ops.ext(required=True)
    qkv, ctx = torch.randn(256, 192, device="cuda").bfloat16(), torch.zeros(256, 64, device="cuda", dtype=torch.bfloat16)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    E.attn_fwd(qkv, torch.full((1, 256), -math.inf, device="cuda"), ctx, torch.empty(1, 1, 256, device="cuda"), 1, 256, 1, 0.125, 0.0, 0, None, err, None)
    assert torch.isnan(ctx).all() and err.item() == 0


def test_attention_without_mask_and_repeatable():
    a, ga = _run(2, 256, 2, 0.1, masked=False)
    b, gb = _run(2, 256, 2, 0.1, masked=False)
    assert torch.equal(a, b) and all(torch.equal(x, y) for x, y in zip(ga, gb))


@pytest.mark.parametrize("B,S,nh", [(2, 64, 1), (3, 128, 2), (1, 512, 2)])
def test_dropout_of_probability_one_leaves_zeros(B, S, nh):
    """Nothing is kept: a context and gradients of zeros, as the softmax kernels and the library's dropout give."""
    from autodist_b200 import ops
    E = ops.ext(required=True)
    H = nh * 64
    err, step = torch.zeros(1, dtype=torch.int32, device="cuda"), torch.tensor([3], device="cuda")
    qkv, dctx = torch.randn(B * S, 3 * H, device="cuda").bfloat16(), torch.randn(B * S, H, device="cuda").bfloat16()
    ctx, dqkv = torch.full_like(dctx, float("nan")), torch.full_like(qkv, float("nan"))
    lse = torch.empty(B, nh, S, device="cuda")
    keep = torch.full((B, nh, S, (S + 127) // 128 * 4), -1, dtype=torch.int32, device="cuda")
    E.attn_fwd(qkv, None, ctx, lse, B, S, nh, 0.125, 1.0, 5, step, err, keep)
    E.attn_bwd(qkv, None, ctx, dctx, lse, torch.empty_like(lse), dqkv, B, S, nh, 0.125, 1.0, err, keep)
    probs, dropped = (torch.empty(B, nh, S, S, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    E.softmax_fwd(torch.zeros_like(probs), None, probs, dropped, 1.0, 1.0, 5, step)
    assert (dropped == 0).all() and (ctx == 0).all() and (dqkv == 0).all() and err.item() == 0


@pytest.mark.parametrize("pd", [0.0, 0.1])
@pytest.mark.parametrize("B,S,nh", [(3, 4, 2), (2, 100, 3), (2, 192, 2), (40, 200, 4), (1, 1000, 2)])
def test_lengths_that_end_inside_a_tile(B, S, nh, pd):
    _run(B, S, nh, pd)


@pytest.mark.parametrize("B,S,nh", [(2, 1, 1), (1, 131, 2)])
def test_odd_lengths_without_dropout(B, S, nh):
    _run(B, S, nh, 0.0)


def test_dropout_takes_multiples_of_four_tokens():
    """One counter decides four neighbouring scores: rows of another length would share their decisions."""
    from autodist_b200 import ops
    E = ops.ext(required=True)
    B, S, nh = 2, 130, 1
    qkv, ctx = torch.randn(B * S, 192, device="cuda").bfloat16(), torch.empty(B * S, 64, device="cuda", dtype=torch.bfloat16)
    lse, keep = torch.empty(B, nh, S, device="cuda"), torch.empty(B, nh, S, 8, dtype=torch.int32, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    with pytest.raises(RuntimeError, match="multiple of 4"):
        E.attn_fwd(qkv, None, ctx, lse, B, S, nh, 0.125, 0.1, 5, None, err, keep)
    with pytest.raises(RuntimeError, match="multiple of 4"):
        E.attn_bwd(qkv, None, ctx, ctx, lse, torch.empty_like(lse), torch.empty_like(qkv), B, S, nh, 0.125, 0.1, err, keep)
