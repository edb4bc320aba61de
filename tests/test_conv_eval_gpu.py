"""Evaluation-mode convolution + batch-norm + residual + ReLU as one kernel, and batch-norm alone: against fp64, and bit for bit
against the same layers run one by one."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _bn(c, device="cuda"):
    g = torch.rand(c, device=device) + 0.5
    return g, torch.randn(c, device=device), torch.randn(c, device=device) * 0.1, torch.rand(c, device=device) + 0.2


def _conv64(x, w, bias, stride, pad):
    return torch.nn.functional.conv2d(x.double(), w.double().permute(0, 3, 1, 2), None if bias is None else bias.double(), stride, pad)


def _reference(x, w, bias, stride, pad, g, b, m, v, eps, relu, res):
    y = _conv64(x, w, bias, stride, pad)
    s = (1, -1, 1, 1)
    y = (y - m.double().view(s)) * (v.double() + eps).rsqrt().view(s) * g.double().view(s) + b.double().view(s)
    if res is not None:
        y = y + res.double()
    return y.clamp_min(0) if relu else y


@pytest.mark.parametrize("n,cin,h,cout,k,stride,pad,bias,relu,with_res", [
    (2, 64, 9, 64, 1, 1, 0, False, True, True), (1, 8, 5, 8, 3, 1, 1, True, True, False), (3, 72, 13, 264, 3, 2, 1, False, False, True),
    (13, 128, 7, 512, 1, 1, 0, False, True, True), (2, 3, 21, 64, 7, 2, 3, False, True, False), (1, 256, 1, 2048, 1, 1, 0, True, False, True),
    (2, 3, 12, 16, 3, 1, 1, True, True, True),
    # several tiles per CTA and column tiles that change between them, for each tile width (64, 128, 256)
    (9, 16, 56, 64, 1, 1, 0, False, True, True), (17, 24, 49, 200, 3, 1, 1, False, True, False), (13, 64, 63, 520, 1, 1, 0, False, True, True)])
def test_conv_bn_eval(n, cin, h, cout, k, stride, pad, bias, relu, with_res):
    from autodist_b200.ops import functional as Fn
    torch.manual_seed(cin + cout)
    x = torch.randn(n, cin, h, h, device="cuda").bfloat16().contiguous(memory_format=torch.channels_last)
    w = (torch.randn(cout, k, k, cin, device="cuda") / (cin * k * k) ** 0.5).bfloat16().float()
    b = torch.randn(cout, device="cuda") if bias else None
    g, be, m, v = _bn(cout)
    oh = (h + 2 * pad - k) // stride + 1
    res = torch.randn(n, cout, oh, oh, device="cuda").bfloat16() if with_res else None
    with torch.no_grad():
        y = Fn.conv_bn_eval(x, w, b, stride, pad, g, be, m, v, 1e-3, relu, res)
    assert y is not None and y.dtype == torch.bfloat16
    Fn.check_errors()
    ref = _reference(x, w, b, stride, pad, g, be, m, v, 1e-3, relu, res)
    # bf16 roundings (2^-9 each, doubled) of the convolution's result, scaled by the normalisation, of the normalised value and of the
    # sum, plus fp32 sums of K products (error about K * 2^-24 of terms below 4 standard deviations)
    s = (1, -1, 1, 1)
    scale = g.double().view(s) * (v.double() + 1e-3).rsqrt().view(s)
    conv = _conv64(x, w, b, stride, pad)
    norm = (conv - m.double().view(s)) * scale + be.double().view(s)
    bound = 2.0 ** -8 * (conv.abs() * scale + norm.abs() + ref.abs()) + 1e-4 + 2.0 ** -20 * (cin * k * k) ** 0.5 * 64
    assert ((y.double() - ref).abs() <= bound).all()
    # convolution, batch-norm, addition and ReLU as kernels of their own, one bf16 tensor after another: the same bits
    with torch.no_grad():
        plain = torch.nn.functional.batch_norm(Fn.conv2d(x, w, b, stride, pad), m, v, g, be, False, 0.0, 1e-3)
        plain = plain if res is None else plain + res
    assert torch.equal(y, torch.relu(plain) if relu else plain)


def test_it_steps_aside_where_it_does_not_apply():
    from autodist_b200.ops import functional as Fn
    x = torch.randn(2, 16, 6, 6, device="cuda").bfloat16()
    w = torch.randn(16, 3, 3, 16, device="cuda")
    p = _bn(16)
    assert Fn.conv_bn_eval(x, w, None, 1, 1, *p, 1e-5) is None                           # a gradient could be recorded
    with torch.no_grad():
        assert Fn.conv_bn_eval(x, w, None, 1, 1, *p, 1e-5, residual=torch.randn(2, 16, 6, 6, device="cuda")) is None   # fp32 residual promotes
        assert Fn.conv_bn_eval(x, w, None, 3, 1, *p, 1e-5) is None
        assert Fn.conv_bn_eval(x, w, None, 1, 1, p[0].double(), *p[1:], 1e-5) is None
        assert Fn.batch_norm_eval(x.float(), *p, 1e-5) is None


@pytest.mark.parametrize("shape", [(1, 8, 1, 1), (3, 24, 7, 5), (16, 1024, 7, 7)])
def test_batch_norm_eval_keeps_nan_and_infinity(shape):
    from autodist_b200.ops import functional as Fn
    torch.manual_seed(1)
    x = torch.randn(*shape, device="cuda").bfloat16()
    x[0, 0, 0, 0] = float("nan")
    x[0, 1, 0, 0] = float("inf")
    g, b, m, v = _bn(shape[1])
    with torch.no_grad():
        y = Fn.batch_norm_eval(x, g, b, m, v, 1e-5, True, None)
        res = torch.randn_like(x)
        plain = torch.nn.functional.batch_norm(x.contiguous(memory_format=torch.channels_last), m, v, g, b, False, 0.0, 1e-5)
        fine = ~torch.isnan(plain)
        for r, out in ((None, y), (res, Fn.batch_norm_eval(x, g, b, m, v, 1e-5, True, res))):
            assert torch.equal(out[fine], torch.relu(plain if r is None else plain + r)[fine])              # the separate layers' bits
        ref = torch.nn.functional.batch_norm(x.double(), m.double(), v.double(), g.double(), b.double(), False, 0.0, 1e-5).relu()
    assert torch.isnan(y[0, 0, 0, 0]) and torch.isinf(y[0, 1, 0, 0])
    ok = torch.isfinite(ref)
    assert ((y.double() - ref)[ok].abs() <= 2.0 ** -8 * ref[ok].abs() + 1e-5).all()


@pytest.mark.parametrize("backbone", ["resnet", "densenet121"])
def test_network_evaluation_matches_the_library_route(backbone, monkeypatch):
    from autodist_b200.models import cnn
    torch.manual_seed(0)
    net = (cnn.ResNet((1, 1, 1, 1)) if backbone == "resnet" else cnn.DenseNet121(growth=8, blocks=(2, 2, 2, 2))).cuda().eval()
    with torch.no_grad():
        for name, buf in net.named_buffers():
            if name.endswith("running_var"):
                buf.uniform_(0.05, 0.15)
    x = torch.randn(2, 3, 75, 75, device="cuda").contiguous(memory_format=torch.channels_last)
    with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
        fused = net(x)
        seen = []
        hooks = [m.register_forward_hook(lambda *a: seen.append(1)) for m in net.modules() if isinstance(m, cnn.BatchNormAct)]
        monkeypatch.setattr(cnn, "NORM_POOL_MODE", "library")
        plain = net(x)
        monkeypatch.undo()
        n = len(seen)
        hooked = net(x)
        assert len(seen) == 2 * n                                                        # hooks still see every batch-norm
    for h in hooks:
        h.remove()
    # the fused layers round where the separate ones do
    for out in (fused, hooked):
        assert torch.equal(out, plain)


@pytest.mark.parametrize("own", ["subclass", "instance"])
def test_a_convolution_with_a_forward_of_its_own_is_called(own):
    from autodist_b200.models import cnn

    class Doubled(cnn.Conv2d):
        def forward(self, x, stats=None, fork=None):
            return 2 * super().forward(x, stats, fork)

    torch.manual_seed(0)
    layer = cnn.ConvBN(16, 24, 3, 1, 1).cuda().eval()
    x = torch.randn(2, 16, 7, 7, device="cuda").bfloat16().contiguous(memory_format=torch.channels_last)
    with torch.no_grad():
        y = layer(x)
        if own == "subclass":
            conv = Doubled(16, 24, 3, 1, 1).cuda().eval()
            conv.load_state_dict(layer.conv.state_dict())
            layer.conv = conv
        else:
            plain = layer.conv.forward
            layer.conv.forward = lambda x, stats=None, fork=None: 2 * plain(x, stats, fork)
        twice = layer(x)
    assert y.any() and torch.allclose(twice.float(), 2 * y.float(), rtol=2.0 ** -7, atol=1e-3)
