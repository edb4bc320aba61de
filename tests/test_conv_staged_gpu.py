"""The staged epilogue of the convolution where its state travels from tile to tile: several tiles per CTA, several column tiles, every
tile width (64, 128, 256 channels), with batch-norm sums, with an addend, at stride 1 and 2."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _data(n, cin, h, w, cout, k):
    torch.manual_seed(cin + cout + h)
    x = torch.randn(n, h, w, cin, device="cuda").bfloat16()
    wt = (torch.randn(cout, k, k, cin, device="cuda") / (cin * k * k) ** 0.5).bfloat16()
    return x, wt


def _nchw(t):
    return t.double().permute(0, 3, 1, 2)


@pytest.mark.parametrize("n,cin,h,w,cout,k,stride", [(21, 16, 61, 53, 64, 1, 1), (21, 16, 61, 53, 128, 1, 1), (21, 16, 61, 53, 200, 3, 1),
                                                     (21, 24, 61, 53, 520, 1, 1), (83, 16, 55, 57, 264, 3, 2), (1, 8, 3, 5, 8, 3, 1)])
def test_forward_with_sums(n, cin, h, w, cout, k, stride):
    from autodist_b200 import ops
    E = ops.ext(required=True)
    x, wt = _data(n, cin, h, w, cout, k)
    pad = k // 2
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    ref = torch.nn.functional.conv2d(_nchw(x), _nchw(wt), None, stride, pad).permute(0, 2, 3, 1)
    mag = torch.nn.functional.conv2d(_nchw(x).abs(), _nchw(wt).abs(), None, stride, pad).permute(0, 2, 3, 1)
    y = torch.full(ref.shape, float("nan"), dtype=torch.bfloat16, device="cuda")
    stats = torch.zeros(2, cout, device="cuda")
    E.conv_fprop(x, wt, y, None, False, stats, stride, pad, err)
    K = cin * k * k
    bound = K * 2.0 ** -22 * mag + 2.0 ** -8 * ref.abs() + 1e-30           # fp32 sums of K exact products, one bf16 rounding (doubled)
    assert ((y.double() - ref).abs() <= bound).all()
    rows = y.numel() // cout
    y64 = y.double().reshape(rows, cout)
    for got, terms in zip(stats.double(), (y64, y64 * y64)):
        # fp32 sums of the stored values, in pieces of 128 rows that meet in atomics: at most rows / 16 + 128 additions in a chain
        assert ((got - terms.sum(0)).abs() <= (rows / 16 + 128) * 2.0 ** -24 * terms.abs().sum(0) + 1e-30).all()
    again = torch.empty_like(y)
    E.conv_fprop(x, wt, again, None, False, None, stride, pad, err)
    assert torch.equal(y, again) and err.item() == 0                      # the sums change nothing


@pytest.mark.parametrize("n,cin,h,w,cout,k,stride", [(21, 64, 61, 53, 16, 1, 1), (21, 128, 61, 53, 24, 3, 1), (21, 264, 61, 53, 16, 1, 1),
                                                     (21, 512, 61, 53, 16, 3, 1), (25, 64, 107, 111, 16, 3, 2), (25, 264, 107, 111, 16, 3, 2),
                                                     (25, 512, 107, 111, 8, 1, 2), (1, 8, 3, 5, 8, 3, 2)])
def test_input_gradient_with_addend(n, cin, h, w, cout, k, stride):
    from autodist_b200 import ops
    E = ops.ext(required=True)
    _, wt = _data(n, cin, 1, 1, cout, k)
    pad = k // 2
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    oh, ow = (h + 2 * pad - k) // stride + 1, (w + 2 * pad - k) // stride + 1
    dy = torch.randn(n, oh, ow, cout, device="cuda").bfloat16()
    add = torch.randn(n, h, w, cin, device="cuda").bfloat16()
    shape = (n, cin, h, w)
    ref = torch.nn.grad.conv2d_input(shape, _nchw(wt), _nchw(dy), stride, pad).permute(0, 2, 3, 1)
    mag = torch.nn.grad.conv2d_input(shape, _nchw(wt).abs(), _nchw(dy).abs(), stride, pad).permute(0, 2, 3, 1)
    for extra in (add, None):
        dx = torch.full((n, h, w, cin), float("nan"), dtype=torch.bfloat16, device="cuda")
        E.conv_dgrad(dy, wt, dx, stride, pad, err, extra)
        want = ref if extra is None else ref + extra.double()
        size = mag if extra is None else mag + extra.double().abs()
        bound = cout * k * k * 2.0 ** -22 * size + 2.0 ** -8 * want.abs() + 1e-30
        assert ((dx.double() - want).abs() <= bound).all()
    assert err.item() == 0
