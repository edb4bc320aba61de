"""The GEMM that splits the contraction over a thread-block cluster, at the edges of its tiles, splits and layouts."""
import os
import subprocess
import sys

import pytest
import torch

pytestmark = pytest.mark.gpu


def _operands(M, N, K, a_mn, b_mn, batch=1):
    """bf16 operands whose leading dimension is padded to a multiple of 8 (the tensor maps' stride rule)."""
    def make(rows, cols):
        t = torch.zeros(batch, rows, (cols + 7) // 8 * 8, dtype=torch.bfloat16, device="cuda")
        t[..., :cols] = torch.randn(batch, rows, cols, device="cuda")
        return t[..., :cols]
    a = make(K, M) if a_mn else make(M, K)
    b = make(K, N) if b_mn else make(N, K)
    A = a.double().transpose(1, 2) if a_mn else a.double()
    B = b.double() if b_mn else b.double().transpose(1, 2)
    return a, b, A @ B, A.abs() @ B.abs()


def _close(out, ref, mag, K, rounding):
    """bf16 products are exact in fp32; K additions that may truncate err by at most K * 2^-23 of the sum of magnitudes (the
    operands of the partial sums included). ``rounding`` is the relative rounding of the stored type."""
    bound = K * 2.0 ** -22 * mag + rounding * ref.abs() + 1e-30
    worst = ((out.double() - ref).abs() / bound).max().item()
    assert worst <= 1.0, f"{worst} times the bound"


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("M,N,K,bn,split", [(128, 64, 128, 64, 2), (129, 72, 136, 64, 3), (1, 8, 512, 64, 8), (200, 130, 1000, 128, 5),
                                            (32, 1000, 4096, 128, 8), (3, 264, 456, 256, 7), (256, 512, 264, 256, 4), (300, 257, 390, 256, 6)])
def test_split_matches_fp64(a_mn, b_mn, M, N, K, bn, split):
    from autodist_b200 import ops
    E = ops.ext(required=True)
    torch.manual_seed(M + N + K)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    a, b, ref, mag = _operands(M, N, K, a_mn, b_mn)
    ldc = (N + 7) // 8 * 8 if split % 2 else N                       # padded and tight (possibly unaligned) output rows
    c32 = torch.ones(1, M, ldc, device="cuda")[..., :N]
    E.gemm_split(a, b, c32, a_mn, b_mn, 0, None, None, None, 0.5, 1.0, err, bn, split)           # adds into the output
    _close(c32 - 1.0, 0.5 * ref, 0.5 * mag + 2, K, 2.0 ** -23)
    bias = torch.randn(N, device="cuda")
    pre, act = (torch.empty(1, M, ldc, dtype=torch.bfloat16, device="cuda")[..., :N] for _ in range(2))
    E.gemm_split(a, b, pre, a_mn, b_mn, 2, bias, act, None, 0.1, 0.0, err, bn, split)            # bias + GELU, two outputs
    _close(pre, 0.1 * ref + bias, 0.1 * mag + bias.abs(), K, 2.0 ** -8)
    want = torch.nn.functional.gelu(0.1 * ref + bias, approximate="tanh")
    # GELU through tanh.approx (2^-11 relative) and one bf16 rounding
    assert ((act.double() - want).abs() <= 2.0 ** -7 * want.abs() + 2.0 ** -9 * (0.1 * ref + bias).abs() + 1e-3).all()
    out = pre.clone()
    E.gemm_split(a, b, out, a_mn, b_mn, 4, None, None, out, 1.0, 0.0, err, bn, split)            # addend aliasing the output
    _close(out, ref + pre.double(), mag + pre.double().abs(), K, 2.0 ** -8)
    again = pre.clone()
    E.gemm_split(a, b, again, a_mn, b_mn, 4, None, None, again, 1.0, 0.0, err, bn, split)
    assert err.item() == 0
    assert torch.equal(out, again)                                                              # the order of the sums is fixed


@pytest.mark.parametrize("M,N,K,batch", [(64, 128, 16384, 1), (32, 1000, 4096, 1), (640, 1024, 4104, 1), (768, 768, 1792, 1), (40, 72, 1024, 3)])
def test_the_chooser_splits_products_with_few_tiles(M, N, K, batch):
    from autodist_b200 import ops
    E = ops.ext(required=True)
    torch.manual_seed(K)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    a, b, ref, mag = _operands(M, N, K, True, True, batch)
    bn, split = E.gemm_choice(M, N, K, batch, 0, True)
    assert bn < 512 and split >= 2
    c = torch.empty(batch, M, N, device="cuda")
    E.gemm(a, b, c, True, True, 0, None, None, None, 1.0, 0.0, err, 0)
    assert err.item() == 0
    _close(c, ref, mag, K, 2.0 ** -23)


@pytest.mark.parametrize("env,chosen", [({"AUTODIST_GEMM_PAIR_MIN_K": "512"}, (True, True, True, False)),
                                        ({"AUTODIST_GEMM_PAIR_MIN_K": "1000000"}, (False, False, True, False)),
                                        ({"AUTODIST_GEMM_PAIR_MIN_K": "0", "AUTODIST_GEMM_PAIR": "0"}, (False, False, False, False))])
def test_a_fixed_rule_for_the_pair_kernel(env, chosen):
    """AUTODIST_GEMM_PAIR_MIN_K: products of at least one pair tile whose tiles fill the SM pairs or whose contraction is that long."""
    code = ("from autodist_b200 import ops; E = ops.ext(required=True); print([E.gemm_choice(*s, 1, 0, False)[0] == 512 for s in "
            "((512, 512, 600), (1024, 4096, 4096), (2560, 2304, 64), (200, 4096, 4096))])")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    out = subprocess.run([sys.executable, "-c", code], cwd=root, env=dict(os.environ, **env), capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    assert out.stdout.strip().splitlines()[-1] == str(list(chosen))


@pytest.mark.parametrize("bn,split", [(64, 1), (128, 1), (256, 1), (512, 1), (64, 2), (256, 3)])
@pytest.mark.parametrize("offset", [1, 4])
def test_outputs_that_start_anywhere_in_their_storage(bn, split, offset):
    """Rows off the 16-byte boundaries of the vector stores: output, second output and auxiliary operand."""
    from autodist_b200 import ops
    E = ops.ext(required=True)
    torch.manual_seed(bn + split)
    M, N, K, ld = 300, 272, 264, 280
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    a, b, ref, mag = _operands(M, N, K, False, False)
    ref, mag = ref[0], mag[0]

    def view(dtype, at):
        return torch.zeros(at + M * ld, dtype=dtype, device="cuda")[at:].view(M, ld)[:, :N]

    def run(c, epilogue, bias, c2, aux, beta):
        args = (a[0], b[0], c, False, False, epilogue, bias, c2, aux, 1.0, beta, err, bn)
        E.gemm(*args) if split == 1 else E.gemm_split(*args, split)

    c32 = view(torch.float32, offset)
    for times in (1, 2):
        run(c32, 0, None, None, None, 1.0)
        _close(c32, times * ref, times * mag, K, 2.0 ** -22)
    bias = torch.randn(offset + N, device="cuda")[offset:]
    pre, act = view(torch.bfloat16, offset), view(torch.bfloat16, offset)
    run(pre, 2, bias, act, None, 0.0)
    _close(pre, ref + bias.double(), mag + bias.double().abs(), K, 2.0 ** -8)
    for where in (0, offset):                                       # the output, then the addend alone off the boundary
        out, add = view(torch.bfloat16, offset - where), view(torch.bfloat16, where)
        add.copy_(pre)
        run(out, 4, None, None, add, 0.0)
        _close(out, ref + pre.double(), mag + pre.double().abs(), K, 2.0 ** -8)
    assert err.item() == 0
