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


@pytest.mark.parametrize("layout", [torch.channels_last, torch.contiguous_format])
@pytest.mark.parametrize("n,c,extra,h,w", [(2, 24, 8, 5, 3), (1, 64, 32, 1, 1), (3, 96, 4, 2, 7), (1, 8, 8, 1, 9), (4, 16, 16, 1, 1)])
def test_concatenation_gradient_is_added_inside_batch_norm(n, c, extra, h, w, layout):
    """Sliced rows that the kernel can read in place, and (4 extra channels, channels apart) ones it cannot."""
    from autodist_b200.ops import functional as Fn
    torch.manual_seed(c)
    x0 = torch.randn(n, c, h, w, device="cuda").bfloat16().contiguous(memory_format=torch.channels_last)
    new = torch.randn(n, extra, h, w, device="cuda").bfloat16().contiguous(memory_format=torch.channels_last)
    gamma, beta = torch.rand(c, device="cuda") + 0.5, torch.randn(c, device="cuda")
    dcat, dy = (torch.randn(n, k, h, w, device="cuda").bfloat16().contiguous(memory_format=layout) for k in (c + extra, c))
    assert torch.allclose(Fn.channel_sums(x0)[1], x0.double().pow(2).sum((0, 2, 3)).float(), rtol=1e-5)
    grads = []
    for fused in (True, False):
        x = x0.clone().requires_grad_(True)
        g, b = gamma.clone().requires_grad_(True), beta.clone().requires_grad_(True)
        y = Fn.batch_norm(x * 1, g, b, relu=True, sums=Fn.channel_sums(x0), alias=True) if fused else Fn.batch_norm(x, g, b, relu=True, sums=Fn.channel_sums(x0))
        y, xc = y if fused else (y, x)
        out = torch.cat([xc, new], 1)
        torch.autograd.backward([out, y], [dcat, dy])
        grads.append(x.grad)
    # one rounding to bf16 instead of three
    assert ((grads[0].float() - grads[1].float()).abs() <= 2.0 ** -7 * grads[1].float().abs() + 2.0 ** -7 * dcat[:, :c].float().abs() + 1e-3).all()


def test_dense_network_step_matches_the_plain_route(monkeypatch):
    from autodist_b200.models import cnn
    torch.manual_seed(0)
    net = cnn.DenseNet121(growth=8, blocks=(2, 2, 2, 2), num_classes=16).cuda()
    x = torch.randn(4, 3, 64, 64, device="cuda").contiguous(memory_format=torch.channels_last)
    state = {k: v.clone() for k, v in net.state_dict().items()}
    outs = []
    for plain in (False, True):
        net.load_state_dict(state)
        net.zero_grad()
        monkeypatch.setattr(cnn, "FUSE_BN_STATS", not plain)
        with torch.autocast("cuda", dtype=torch.bfloat16):
            y = net(x)
        y.float().pow(2).sum().backward()
        outs.append((y.detach().float(), net.features[0].bn.running_var.clone(), net.fc.weight.grad.clone(),
                     net.features[-1].running_mean.clone()))
    for a, b in zip(*outs):                    # the same values in another order of summation and with fewer roundings
        assert (a - b).norm() <= 0.05 * b.norm()


def test_dense_network_step_records_no_more_functions_than_the_plain_route(monkeypatch):
    """An eager step is bound by the host, where every autograd function written in Python costs as much as a launch."""
    from autodist_b200.models import cnn
    torch.manual_seed(0)
    net = cnn.DenseNet121(growth=8, blocks=(2, 2, 2, 2), num_classes=16).cuda()
    x = torch.randn(4, 3, 64, 64, device="cuda").contiguous(memory_format=torch.channels_last)
    counts = []
    for fused in (True, False):
        monkeypatch.setattr(cnn, "FUSE_BN_STATS", fused)
        with torch.autocast("cuda", dtype=torch.bfloat16):
            stack, seen = [net(x).sum().grad_fn], set()
        while stack:
            node = stack.pop()
            if node is not None and node not in seen:
                seen.add(node)
                stack += [n for n, _ in node.next_functions]
        counts.append(sum("FnBackward" in n.name() for n in seen))
    assert 0 < counts[0] <= counts[1]


def test_a_changed_layer_keeps_to_the_plain_route():
    from autodist_b200.models import cnn
    net = cnn.DenseNet121(growth=8, blocks=(2, 2, 2, 2), num_classes=16).cuda()
    x = torch.randn(2, 3, 64, 64, device="cuda").contiguous(memory_format=torch.channels_last)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        assert net._plan(x) is not None
        net.features[3].f.append(torch.nn.Dropout(0.5))                # five modules where the kernel path expects four
        assert net._plan(x) is None
        net(x).float().sum().backward()
    assert torch.isfinite(net.fc.weight.grad).all()
