"""Tiles of 192 columns: every operand layout and epilogue at ragged extents, one and several tiles per CTA, tight and padded output rows."""
import pytest
import torch

from test_gemm_split_gpu import _close, _operands

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K,batch", [(128, 192, 64, 1), (264, 200, 72, 1), (1000, 776, 264, 3), (136, 96, 1032, 1), (5000, 1160, 136, 1)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True)])
def test_plain_bias_and_fp32_outputs(M, N, K, batch, a_mn, b_mn):
    from autodist_b200 import ops
    E = ops.ext(required=True)
    torch.manual_seed(M + N)
    M = M if a_mn else M - 7
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    a, b, ref, mag = _operands(M, N, K, a_mn, b_mn, batch)
    bias = torch.randn(N, device="cuda")
    for ldc in (N, N + 8):
        out = torch.full((batch, M, ldc), float("nan"), dtype=torch.bfloat16, device="cuda")
        E.gemm(a, b, out[..., :N], a_mn, b_mn, 1, bias, None, None, 0.5, 0.0, err, 192)
        _close(out[..., :N], 0.5 * ref + bias.double(), 0.5 * mag + bias.double().abs(), K, 2.0 ** -8)
        assert ldc == N or torch.isnan(out[..., N:]).all()
        acc = torch.ones(batch, M, ldc, device="cuda")
        E.gemm(a, b, acc[..., :N], a_mn, b_mn, 0, None, None, None, 1.0, 1.0, err, 192)
        _close(acc[..., :N], ref + 1, mag + 1, K, 2.0 ** -22)
        E.gemm(a, b, acc[..., :N], a_mn, b_mn, 0, None, None, None, 1.0, 0.0, err, 192)
        _close(acc[..., :N], ref, mag, K, 2.0 ** -22)
        assert ldc == N or (acc[..., N:] == 1).all()
    assert err.item() == 0


@pytest.mark.parametrize("M,N,K", [(128, 192, 128), (390, 456, 200), (6000, 1544, 72)])
def test_activations_and_auxiliary_operand(M, N, K):
    from autodist_b200 import ops
    E = ops.ext(required=True)
    torch.manual_seed(M)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    a, b, ref, mag = _operands(M, N, K, False, False)
    a, b, ref, mag = a[0], b[0], ref[0], mag[0]
    bias = torch.randn(N, device="cuda")
    pre, act, th, own = (torch.empty(M, N, dtype=torch.bfloat16, device="cuda") for _ in range(4))
    E.gemm(a, b, pre, False, False, 2, bias, act, None, 1.0, 0.0, err, 192)
    want = ref + bias.double()
    _close(pre, want, mag + bias.double().abs(), K, 2.0 ** -8)
    # tanh.approx errs by 2^-11, a slope of at most 1.13 carries the error of the sums over
    gelu = torch.nn.functional.gelu(want, approximate="tanh")
    assert ((act.double() - gelu).abs() <= 2.0 ** -8 * gelu.abs() + 2.0 ** -11 * want.abs() + 1.2 * K * 2.0 ** -22 * mag + 1e-6).all()
    E.gemm(a, b, th, False, False, 5, bias, None, None, 1.0, 0.0, err, 192)
    assert ((th.double() - torch.tanh(want)).abs() <= 2.0 ** -8 + 1.2 * K * 2.0 ** -22 * mag).all()
    x = torch.randn(M, N, device="cuda").bfloat16()
    own.copy_(x)
    E.gemm(a, b, own, False, False, 4, None, None, own, 1.0, 0.0, err, 192)
    _close(own, ref + x.double(), mag + x.double().abs(), K, 2.0 ** -8)
    wide = torch.empty_like(pre)
    for bn, out in ((192, th), (256, wide)):                              # the same arithmetic in tiles of another width
        E.gemm(a, b, out, False, False, 3, None, None, x, 0.5, 0.0, err, bn)
    assert torch.equal(th, wide) and err.item() == 0


def test_the_chooser_takes_192_columns_where_they_fill_the_gpu():
    from autodist_b200 import ops
    E = ops.ext(required=True)
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the counts below are for 148 SMs")
    assert E.gemm_choice(3072, 1024, 4096, 1, 1, False) == (192, 1)
    assert E.gemm_choice(4096, 768, 3072, 1, 1, False) == (192, 1)
    assert E.gemm_choice(4096, 4096, 1024, 1, 2, False) == (512, 1)
    assert E.gemm_choice(512, 384, 128, 1, 1, False)[0] == 64
