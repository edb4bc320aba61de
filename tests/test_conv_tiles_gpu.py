"""Every tile width of the convolutions over several column tiles, and every split of the weight gradient, asked for instead of estimated: batch-norm
sums flushed between column tiles, addends, the evaluation epilogue's coefficients rebuilt, ragged channels, stride 1 and 2."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# images of one size: several tiles per CTA (21 x 61 x 53), and fewer tiles than SMs (3 x 7 x 9)
CASES = [(21, 16, 61, 53, 264, 1, 1), (3, 72, 7, 9, 520, 3, 1), (5, 264, 15, 13, 200, 3, 2), (19, 64, 9, 8, 384, 1, 2)]


def _nchw(t):
    return t.double().permute(0, 3, 1, 2)


def _widths(columns):
    return [bn for bn in (64, 128, 256) if bn == 64 or columns > bn // 2]


def _data(n, cin, h, w, cout, k, stride):
    torch.manual_seed(cin + cout)
    x = torch.randn(n, h, w, cin, device="cuda").bfloat16()
    wt = (torch.randn(cout, k, k, cin, device="cuda") / (cin * k * k) ** 0.5).bfloat16()
    pad = k // 2
    oh, ow = (h + 2 * pad - k) // stride + 1, (w + 2 * pad - k) // stride + 1
    return x, wt, torch.randn(n, oh, ow, cout, device="cuda").bfloat16(), pad, torch.zeros(1, dtype=torch.int32, device="cuda")


@pytest.mark.parametrize("n,cin,h,w,cout,k,stride", CASES)
def test_forward_and_its_sums(n, cin, h, w, cout, k, stride):
    from autodist_b200 import ops
    E = ops.ext(required=True)
    x, wt, like, pad, err = _data(n, cin, h, w, cout, k, stride)
    ref = torch.nn.functional.conv2d(_nchw(x), _nchw(wt), None, stride, pad).permute(0, 2, 3, 1)
    mag = torch.nn.functional.conv2d(_nchw(x).abs(), _nchw(wt).abs(), None, stride, pad).permute(0, 2, 3, 1)
    first = None
    for tile in _widths(cout):
        y, stats = torch.full_like(like, float("nan")), torch.zeros(2, cout, device="cuda")
        E.conv_fprop(x, wt, y, None, False, stats, stride, pad, err, tile)
        # fp32 sums of exact products, one bf16 rounding (doubled)
        assert ((y.double() - ref).abs() <= cin * k * k * 2.0 ** -22 * mag + 2.0 ** -8 * ref.abs() + 1e-30).all()
        first = y if first is None else first
        assert torch.equal(y, first)                                             # a width changes no bit
        rows = y.numel() // cout
        terms = y.double().reshape(rows, cout)
        for got, t in zip(stats.double(), (terms, terms * terms)):
            assert ((got - t.sum(0)).abs() <= (rows / 16 + 128) * 2.0 ** -24 * t.abs().sum(0) + 1e-30).all()
    assert err.item() == 0


@pytest.mark.parametrize("n,cin,h,w,cout,k,stride", CASES)
def test_evaluation_epilogue(n, cin, h, w, cout, k, stride):
    from autodist_b200 import ops
    E = ops.ext(required=True)
    x, wt, res, pad, err = _data(n, cin, h, w, cout, k, stride)
    gamma, beta, mean, bias = torch.randn(4, cout, device="cuda")
    var = torch.rand(cout, device="cuda") + 0.5
    plain = torch.empty_like(res)
    E.conv_fprop(x, wt, plain, bias, False, None, stride, pad, err, 64)
    want = torch.nn.functional.batch_norm(_nchw(plain), mean.double(), var.double(), gamma.double(), beta.double(), False, 0.0, 1e-5).permute(0, 2, 3, 1)
    # the normalised value is rounded, the residual added, the sum rounded: two roundings of at most 2^-9 of what they round
    slack = 2.0 ** -8 * (want.abs() + (want + res.double()).abs()) + 2.0 ** -20 * (gamma.double().abs() * 4 + beta.double().abs() + plain.double().abs() * 4)
    first = None
    for tile in _widths(cout):
        y = torch.full_like(res, float("nan"))
        E.conv_fprop_bn_eval(x, wt, y, bias, True, gamma, beta, mean, var, 1e-5, res, stride, pad, err, tile)
        assert ((y.double() - (want + res.double()).clamp_min(0)).abs() <= slack).all()
        first = y if first is None else first
        assert torch.equal(y, first)
    assert err.item() == 0


@pytest.mark.parametrize("n,cin,h,w,cout,k,stride", CASES)
def test_gradients(n, cin, h, w, cout, k, stride):
    from autodist_b200 import ops
    E = ops.ext(required=True)
    x, wt, dy, pad, err = _data(n, cin, h, w, cout, k, stride)
    add = torch.randn(x.shape, device="cuda").bfloat16()
    shape = (n, cin, h, w)
    ref = torch.nn.grad.conv2d_input(shape, _nchw(wt), _nchw(dy), stride, pad).permute(0, 2, 3, 1)
    mag = torch.nn.grad.conv2d_input(shape, _nchw(wt).abs(), _nchw(dy).abs(), stride, pad).permute(0, 2, 3, 1)
    first = None
    for tile in _widths(cin):
        dx = torch.full_like(x, float("nan"))
        E.conv_dgrad(dy, wt, dx, stride, pad, err, add, tile)
        want, size = ref + add.double(), mag + add.double().abs()
        assert ((dx.double() - want).abs() <= cout * k * k * 2.0 ** -22 * size + 2.0 ** -8 * want.abs() + 1e-30).all()
        first = dx if first is None else first
        assert torch.equal(dx, first)
    ref = torch.nn.grad.conv2d_weight(_nchw(x), (cout, cin, k, k), _nchw(dy), stride, pad).permute(0, 2, 3, 1)
    mag = torch.nn.grad.conv2d_weight(_nchw(x).abs(), (cout, cin, k, k), _nchw(dy).abs(), stride, pad).permute(0, 2, 3, 1)
    for tile in _widths(cin):
        for ksplit in (1, 2, 3):
            for accumulate in (False, True):
                dw = torch.ones(cout, k, k, cin, device="cuda")
                E.conv_wgrad(dy, x, dw, stride, pad, err, accumulate, tile, ksplit)
                want = ref + (1.0 if accumulate else 0.0)
                assert ((dw.double() - want).abs() <= dy.numel() // cout * 2.0 ** -22 * (mag + 1)).all()
    assert err.item() == 0


def test_widths_that_do_not_suit_are_refused():
    from autodist_b200 import ops
    E = ops.ext(required=True)
    x, wt, dy, pad, err = _data(2, 64, 9, 8, 72, 1, 1)
    for tile in (-1, 32, 192, 256):
        with pytest.raises(RuntimeError, match="tile must be"):
            E.conv_fprop(x, wt, torch.empty_like(dy), None, False, None, 1, pad, err, tile)
    with pytest.raises(RuntimeError, match="one CTA per"):
        E.conv_wgrad(dy, x, torch.empty(72, 1, 1, 64, device="cuda"), 1, pad, err, False, 64, 1000)
