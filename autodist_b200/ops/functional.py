"""Autograd-visible wrappers of the hand-written kernels for models that keep using ``torch.autograd``.

``linear`` runs forward, dX and dW on the tcgen05 GEMM (bf16 operands, fp32 accumulation; the weight gradient is
produced in fp32). On CPU tensors the same functions fall back to the plain PyTorch expression, which is also the
numerics reference of the tests.
"""
import math
import os
import warnings

import torch
import torch.nn.functional as F

from autodist_b200 import ops

_err = {}


def _error_flag(device):
    if device not in _err:
        _err[device] = torch.zeros(1, dtype=torch.int32, device=device)
    return _err[device]


#: Per device a word of pinned host memory that kernels write when an id lies outside its table (they read nothing there), and its numpy
#: view: the host looks at it without waiting for the device.
_id_flags = {}
_ID_ERRORS = {71: "a sampled softmax met an id outside its vocabulary", 72: "a lookup of (user, item) pairs met an id outside its table"}


def _id_flag(device):
    if device not in _id_flags:
        flag = torch.zeros(1, dtype=torch.int32).pin_memory()
        _id_flags[device] = flag, flag.numpy()
    return _id_flags[device][0]


def raise_bad_ids():
    """Raises for ids outside their tables that kernels have reported so far, once each. Costs no wait."""
    for dev, (_, seen) in _id_flags.items():
        if seen[0]:
            code = int(seen[0])
            seen[0] = 0
            raise RuntimeError(f"{_ID_ERRORS.get(code, 'an id outside its table')} on {dev}: its row counted as zeros, the results are not valid")


def check_errors():
    for dev in _id_flags:
        torch.cuda.synchronize(dev)
    raise_bad_ids()
    for dev, flag in _err.items():
        code = int(flag.item())
        if code:
            raise RuntimeError(f"a GEMM kernel on {dev} gave up waiting (code {code})")


#: ``bn`` of a product whose sums must not depend on which kernel is the fastest: a recurrence carries an ulp on (see csrc/bindings.cpp)
_FIXED_SHARES = -1


class _LinearFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, weight, bias, activation, bn):
        E = ops.ext(required=True)
        shape = x.shape
        x2 = x.reshape(-1, shape[-1]).to(torch.bfloat16).contiguous()
        w16 = _bf16_weight(weight)
        y = torch.empty(x2.shape[0], weight.shape[0], dtype=torch.bfloat16, device=x.device)
        err = _error_flag(x.device)
        pre = None
        b32 = bias.float().contiguous() if bias is not None else None
        gathered = getattr(weight, "_gathered", None) if activation is None else None
        ctx.gathered = gathered
        if gathered is not None:
            # the weight's row shards stay with their owners: B tiles are fetched over NVLink inside the GEMM
            E.gemm_gathered_b(x2, gathered["ptrs"], gathered["rows"], y, 1 if b32 is not None else 0, b32, err, 0)
        elif activation == "gelu":
            pre = torch.empty_like(y)
            E.gemm(x2, w16, pre, False, False, 2, b32 if b32 is not None else torch.zeros(weight.shape[0], device=x.device),
                   y, None, 1.0, 0.0, err, bn)
        elif b32 is not None:
            E.gemm(x2, w16, y, False, False, 1, b32, None, None, 1.0, 0.0, err, bn)
        else:
            E.gemm(x2, w16, y, False, False, 0, None, None, None, 1.0, 0.0, err, bn)
        ctx.save_for_backward(x2, w16, pre)
        ctx.weight = weight
        _count_use(ctx, weight, 1)
        ctx.has_bias = bias is not None
        ctx.shape, ctx.bn = shape, bn
        ctx.w_dtype = weight.dtype
        return y.view(*shape[:-1], weight.shape[0])

    @staticmethod
    def backward(ctx, dy):
        E = ops.ext(required=True)
        x2, w16, pre = ctx.saved_tensors
        bn = ctx.bn
        err = _error_flag(dy.device)
        dy2 = dy.reshape(-1, dy.shape[-1]).to(torch.bfloat16).contiguous()
        if pre is not None:
            du = torch.empty_like(dy2)
            E.gelu_bwd(dy2, pre, du)
            dy2 = du
        dx = torch.empty_like(x2)
        if ctx.gathered is not None:
            E.gemm_gathered_bt(dy2, ctx.gathered["ptrs"], ctx.gathered["rows"], w16.shape[1], dx, err)   # dX = dY . W, W from its owners
        else:
            E.gemm(dy2, w16, dx, False, True, 0, None, None, None, 1.0, 0.0, err, bn)      # dX = dY . W
        acc = _direct_grad(ctx.weight)
        if acc is not None:
            E.gemm(dy2, x2, acc, True, True, 0, None, None, None, 1.0, 1.0, err, bn)       # dW += dY^T . X, in the gradient buffer
            dw = None
        else:
            dw = torch.empty(w16.shape, dtype=torch.float32, device=dy.device)
            E.gemm(dy2, x2, dw, True, True, 0, None, None, None, 1.0, 0.0, err, bn)        # dW = dY^T . X
        db = None
        if ctx.has_bias:
            n = dy2.shape[1]
            if n % 8 == 0:
                db = torch.empty(n, dtype=torch.float32, device=dy.device)
                part = torch.empty(E.colsum_parts(dy2.shape[0]) * n, dtype=torch.float32, device=dy.device)
                E.keyed_colsum(dy2, None, part, db, 1, False)
            else:
                db = dy2.float().sum(0)
        if dw is None:
            _grad_written(ctx.weight)
        return dx.view(ctx.shape).to(dy.dtype), None if dw is None else dw.to(ctx.w_dtype), db, None, None


def linear(x, weight, bias=None, activation=None, fixed_shares=False):
    """``activation(x @ weight.T + bias)`` with ``activation`` in ``{None, "gelu"}`` (tanh form). ``fixed_shares``: how many CTAs share a
    contraction, and with it the order of its sums, does not follow the kernels' timings."""
    if x.is_cuda and x.shape[-1] % 8 == 0 and (weight.shape[0] % 8 == 0):
        return _LinearFn.apply(x, weight, bias, activation, _FIXED_SHARES if fixed_shares else 0)
    y = F.linear(x, weight.to(x.dtype), None if bias is None else bias.to(x.dtype))
    return F.gelu(y, approximate="tanh") if activation == "gelu" else y


class Linear(torch.nn.Linear):
    """Drop-in ``nn.Linear`` whose CUDA path is the tcgen05 GEMM."""

    def forward(self, x):
        return linear(x, self.weight, self.bias)


class _LSTMCellFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, gates, c_prev, forget_bias):
        E = ops.ext(required=True)
        gates = gates.float().contiguous()
        c_prev = c_prev.float().contiguous()
        c = torch.empty_like(c_prev)
        h = torch.empty(c_prev.shape, dtype=torch.bfloat16, device=c_prev.device)
        E.lstm_cell_fwd(gates, c_prev, c, h, forget_bias)
        ctx.save_for_backward(gates, c_prev, c)
        ctx.fb = forget_bias
        return c, h

    @staticmethod
    def backward(ctx, dc_next, dh):
        E = ops.ext(required=True)
        gates, c_prev, c = ctx.saved_tensors
        dh = torch.zeros_like(c) if dh is None else dh.float().contiguous()
        dgates = torch.empty_like(gates)
        dc_prev = torch.empty_like(c)
        E.lstm_cell_bwd(gates, c_prev, c, dh, None if dc_next is None else dc_next.float().contiguous(), dgates, dc_prev, ctx.fb)
        return dgates, dc_prev, None


def lstm_cell(gates, c_prev, forget_bias=1.0):
    """Pointwise part of an LSTM step: ``gates`` [B, 4S] in the order i, j, f, o -> ``(c_new fp32, h bf16)``."""
    if gates.is_cuda:
        return _LSTMCellFn.apply(gates, c_prev, forget_bias)
    i, j, f, o = gates.float().chunk(4, 1)
    c = torch.sigmoid(f + forget_bias) * c_prev + torch.sigmoid(i) * torch.tanh(j)
    return c, torch.sigmoid(o) * torch.tanh(c)


class _LSTMLayerFn(torch.autograd.Function):
    """A projected LSTM layer over a whole sequence. Per step: one product for the gates, the cell, one product for the
    projection, which lands in the next step's operand; backward likewise, the gradient of the carried state being added in the
    product's epilogue. The weight gradients are one product each over all steps instead of one read-modify-write of the
    gradient buffer per step."""

    @staticmethod
    def forward(ctx, inputs, weight, bias, proj, forget_bias):
        E = ops.ext(required=True)
        dev, err = inputs.device, _error_flag(inputs.device)
        B, T, D = inputs.shape
        P, S = proj.shape
        w16, p16, b32 = _bf16_weight(weight), _bf16_weight(proj), bias.detach().float().contiguous()
        xh = torch.empty(T + 1, B, D + P, dtype=torch.bfloat16, device=dev)           # [x_t, h_{t-1}]; the last slot only holds h
        xh[:T, :, :D].copy_(inputs.transpose(0, 1))
        xh[0, :, D:].zero_()
        gates = torch.empty(T, B, 4 * S, dtype=torch.bfloat16, device=dev)
        c = torch.empty(T + 1, B, S, dtype=torch.float32, device=dev)
        c[0].zero_()
        hid = torch.empty(T, B, S, dtype=torch.bfloat16, device=dev)
        for t in range(T):
            E.gemm(xh[t], w16, gates[t], False, False, 1, b32, None, None, 1.0, 0.0, err, _FIXED_SHARES)
            E.lstm_seq_fwd(gates[t], c[t], c[t + 1], hid[t], forget_bias)
            E.gemm(hid[t], p16, xh[t + 1, :, D:], False, False, 0, None, None, None, 1.0, 0.0, err, _FIXED_SHARES)
        ctx.save_for_backward(xh, gates, c, hid, w16, p16)
        ctx.params, ctx.fb, ctx.dims, ctx.x_dtype = (weight, bias, proj), forget_bias, (B, T, D, P, S), inputs.dtype
        for k, p in ((1, weight), (2, bias), (3, proj)):
            _count_use(ctx, p, k)
        return xh[1:, :, D:].transpose(0, 1).contiguous()                             # [B, T, P]

    @staticmethod
    def backward(ctx, dout):
        E = ops.ext(required=True)
        xh, gates, c, hid, w16, p16 = ctx.saved_tensors
        weight, bias, proj = ctx.params
        B, T, D, P, S = ctx.dims
        dev, err = dout.device, _error_flag(dout.device)
        # slot t: gradient of [x_t, h_{t-1}]; h_{t-1} starts with what the layer's output brings
        dxh = torch.empty(T + 1, B, D + P, dtype=torch.bfloat16, device=dev)
        dxh[:T, :, :D].zero_()
        dxh[0, :, D:].zero_()
        dxh[1:, :, D:].copy_(dout.transpose(0, 1))
        dgates = torch.empty_like(gates)
        dhid = torch.empty(B, S, dtype=torch.bfloat16, device=dev)
        dc = torch.empty(B, S, dtype=torch.float32, device=dev)
        for t in range(T - 1, -1, -1):
            E.gemm(dxh[t + 1, :, D:], p16, dhid, False, True, 0, None, None, None, 1.0, 0.0, err, _FIXED_SHARES)
            E.lstm_seq_bwd(gates[t], c[t], c[t + 1], dhid, dc if t + 1 < T else None, dgates[t], dc, ctx.fb)
            E.gemm(dgates[t], w16, dxh[t], False, True, 4, None, None, dxh[t], 1.0, 0.0, err, _FIXED_SHARES)
        rows = T * B
        dg2, x2, h2 = dgates.view(rows, 4 * S), xh[:T].view(rows, D + P), hid.view(rows, S)
        dh2 = dxh[1:].view(rows, D + P)[:, D:]
        grads = []
        for p, a, b in ((weight, dg2, x2), (proj, dh2, h2)):
            acc = _direct_grad(p)
            g = acc if acc is not None else torch.empty(p.shape, dtype=torch.float32, device=dev)
            E.gemm(a, b, g, True, True, 0, None, None, None, 1.0, 1.0 if acc is not None else 0.0, err, _FIXED_SHARES)
            if acc is not None:
                _grad_written(p)
            grads.append(None if acc is not None else g.to(p.dtype))
        acc = _direct_grad(bias)
        db = acc if acc is not None else torch.empty(4 * S, dtype=torch.float32, device=dev)
        E.keyed_colsum(dg2, None, torch.empty(E.colsum_parts(rows) * 4 * S, dtype=torch.float32, device=dev), db, 1, acc is not None)
        if acc is not None:
            _grad_written(bias)
        dx = dxh[:T, :, :D].transpose(0, 1).to(ctx.x_dtype) if ctx.needs_input_grad[0] else None
        return dx, grads[0], None if acc is not None else db.to(bias.dtype), grads[1], None


def lstm_layer(inputs, weight, bias, proj, forget_bias=1.0):
    """Outputs ``[B, T, P]`` of a projected LSTM over ``inputs`` [B, T, D] from a zero state: ``gates = [x_t, h] @ weight.T + bias``
    (order i, j, f, o), ``h = (o * tanh(c)) @ proj.T``."""
    B, T, D = inputs.shape
    P, S = proj.shape
    fused = inputs.is_cuda and B > 0 and T > 0 and D % 8 == 0 and P % 8 == 0 and S % 8 == 0 and \
        tuple(weight.shape) == (4 * S, D + P) and bias is not None and bias.numel() == 4 * S and \
        getattr(weight, "_gathered", None) is None and getattr(proj, "_gathered", None) is None
    if fused:
        return _LSTMLayerFn.apply(inputs, weight, bias, proj, float(forget_bias))
    h = torch.zeros(B, P, dtype=inputs.dtype, device=inputs.device)
    cell = torch.zeros(B, S, dtype=torch.float32, device=inputs.device)
    outs = []
    for t in range(T):
        cell, hidden = lstm_cell(linear(torch.cat([inputs[:, t], h], 1), weight, bias), cell, forget_bias)
        h = linear(hidden.to(inputs.dtype), proj)
        outs.append(h)
    return torch.stack(outs, 1)


def clip_by_global_norm_(grads, max_norm, weights=None, all_reduce=None):
    """Scale fp32 CUDA gradients in place so that their joint L2 norm is at most ``max_norm``; the norm stays on the
    device. ``weights`` weighs each tensor's squared sum (replicated tensors count once across ranks);
    ``all_reduce`` (optional callable) sums the squared norm over ranks."""
    E = ops.ext(required=True)
    acc = torch.zeros(1, dtype=torch.float32, device=grads[0].device)
    for k, g in enumerate(grads):
        E.sumsq(g, acc, 1.0 if weights is None else weights[k])
    if all_reduce is not None:
        all_reduce(acc)
    for g in grads:
        E.clip_scale(g, acc, max_norm)
    return acc


def _nhwc(x):
    """bf16 ``[N, H, W, C]`` contiguous view / copy of a logical ``[N, C, H, W]`` tensor (free for channels-last bf16)."""
    return x.permute(0, 2, 3, 1).to(torch.bfloat16).contiguous()


def _bf16_weight(weight):
    """bf16 copy of a parameter: the engine's flat compute copy when the parameter lives in flat buffers, else a cast."""
    view = getattr(weight, "_bf16_view", None)
    if view is not None and view.device == weight.device:
        return view
    return weight.detach().to(torch.bfloat16).contiguous()


def _direct_grad(param):
    """The fp32 gradient buffer of ``param`` when its owner (a flat-buffer engine) asked for gradients to be accumulated
    in place by the producing kernel instead of travelling through autograd's accumulation; else ``None``."""
    if not getattr(param, "_direct_grad", False):
        return None                 # (asked first: reading .grad of a non-leaf tensor makes PyTorch warn)
    g = param.grad
    if g is not None and g.dtype == torch.float32 and g.is_contiguous() and g.is_cuda:
        return g
    return None


def _count_use(ctx, param, index):
    """Forward side of the direct accumulation: remember that one more kernel call will add into ``param``'s gradient."""
    if ctx.needs_input_grad[index] and getattr(param, "_direct_grad", False):
        param._pending_uses = getattr(param, "_pending_uses", 0) + 1


def _grad_written(param):
    """Backward side: one pending call has added its part; after the last one tell the owner that the gradient is final."""
    param._pending_uses = getattr(param, "_pending_uses", 1) - 1
    hook = getattr(param, "_grad_ready_hook", None)
    if hook is not None and param._pending_uses <= 0:
        hook(param)


def _colsum(E, dy2):
    n = dy2.shape[1]
    db = torch.empty(n, dtype=torch.float32, device=dy2.device)
    part = torch.empty(E.colsum_parts(dy2.shape[0]) * n, dtype=torch.float32, device=dy2.device)
    E.keyed_colsum(dy2, None, part, db, 1, False)
    return db


def _rowtap_geometry(h, w, kh, kw, stride, padding):
    """Padded-image extents of the first-layer path: the halo is written out and rows are long enough for the last
    64-element read of every output column."""
    oh, ow = (h + 2 * padding - kh) // stride + 1, (w + 2 * padding - kw) // stride + 1
    hp = max(h + 2 * padding, (oh - 1) * stride + kh)
    wp = max(w + 2 * padding, (ow - 1) * stride + 8)
    return oh, ow, hp, wp + (wp & 1)


class GradFork:
    """Meeting point of the two consumers of a forked tensor (the input of a residual block feeds the block's first
    convolution and its skip connection). Whichever consumer's backward runs first leaves its gradient here and returns
    none; the second adds it inside its own kernel (the input-gradient convolution's epilogue) and returns the sum, so
    the fork costs no elementwise pass of its own."""
    __slots__ = ("grad",)

    def __init__(self):
        self.grad = None

    def take(self):
        g, self.grad = self.grad, None
        return g


class _ForkFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, box):
        ctx.box = box
        ctx.set_materialize_grads(False)
        return x.view_as(x), x.view_as(x)

    @staticmethod
    def backward(ctx, ga, gb):
        # a gradient left behind (its partner never ran, or could not fuse the add) still counts
        parts = [g for g in (ga, gb, ctx.box.take()) if g is not None]
        if not parts:
            return None, None
        out = parts[0]
        for g in parts[1:]:
            out = out + g
        return out, None


def fork(x):
    """Two aliases of ``x`` for its two consumers plus the ``GradFork`` both pass to their kernels (``conv2d(fork=...)``,
    ``batch_norm(fork=...)``); ``(x, x, None)`` where no gradient flows."""
    if not (x.is_cuda and x.requires_grad and torch.is_grad_enabled()):
        return x, x, None
    box = GradFork()
    a, b = _ForkFn.apply(x, box)
    return a, b, box


class _ConvFn(torch.autograd.Function):
    """2-D convolution as an implicit GEMM on tcgen05 (``csrc/conv_tcgen05.cu``): forward, input gradient and weight
    gradient read the channels-last bf16 activations in place through TMA boxes, one per filter tap; bias, ReLU and the
    per-channel sums a following batch-norm needs are fused into the forward epilogue. ``weight`` is ``[Cout, KH, KW, Cin]``."""

    @staticmethod
    def forward(ctx, x, weight, bias, stride, padding, relu, stats, fork=None):
        E = ops.ext(required=True)
        ctx.fork = fork
        cout, kh, kw, cin = weight.shape
        err = _error_flag(x.device)
        b32 = bias.detach().float().contiguous() if bias is not None else None
        w16 = _bf16_weight(weight)
        ctx.rowtap = cin % 8 != 0
        if ctx.rowtap:
            n, _, h, w = x.shape
            oh, ow, hp, wp = _rowtap_geometry(h, w, kh, kw, stride, padding)
            xh = torch.empty(n, hp, wp, 8, dtype=torch.bfloat16, device=x.device)
            E.pad_image8(x, xh, padding)
            wr = F.pad(F.pad(w16, (0, 8 - cin)).reshape(cout, kh, kw * 8), (0, 64 - kw * 8)).contiguous()
            y = torch.empty(n, oh, ow, cout, dtype=torch.bfloat16, device=x.device)
            E.conv_rowtap_fprop(xh, wr, y, b32, relu, stats, stride, err)
        else:
            xh = _nhwc(x)
            n, h, w, _ = xh.shape
            oh, ow = (h + 2 * padding - kh) // stride + 1, (w + 2 * padding - kw) // stride + 1
            y = torch.empty(n, oh, ow, cout, dtype=torch.bfloat16, device=x.device)
            E.conv_fprop(xh, w16, y, b32, relu, stats, stride, padding, err)
        ctx.save_for_backward(xh, w16, y if relu else None)
        ctx.weight, ctx.bias = weight, bias
        _count_use(ctx, weight, 1)
        if bias is not None:
            _count_use(ctx, bias, 2)
        ctx.geom = (stride, padding, tuple(weight.shape), tuple(x.shape))
        ctx.has_bias = bias is not None
        ctx.dtypes = (x.dtype, weight.dtype)
        return y.permute(0, 3, 1, 2)

    @staticmethod
    def backward(ctx, dy):
        E = ops.ext(required=True)
        xh, w16, y = ctx.saved_tensors
        stride, padding, (cout, kh, kw, cin), x_shape = ctx.geom
        err = _error_flag(dy.device)
        dyh = _nhwc(dy)
        db = None
        bias = ctx.bias
        acc_b = _direct_grad(bias) if bias is not None else None
        if bias is not None:
            # bias gradient (and the ReLU mask) in one pass over dy
            db = acc_b if acc_b is not None else torch.empty(cout, dtype=torch.float32, device=dy.device)
            masked = torch.empty_like(dyh) if y is not None else None
            E.relu_bwd_colsum(dyh, y, masked, db, acc_b is not None)
            dyh = masked if masked is not None else dyh
        elif y is not None:
            masked = torch.empty_like(dyh)
            E.relu_bwd(dyh, y, masked)
            dyh = masked
        dx = None
        if ctx.rowtap:
            dwr = torch.empty(cout, kh, 64, dtype=torch.float32, device=dy.device)
            E.conv_rowtap_wgrad(dyh, xh, dwr, stride, err)
            dw = dwr[:, :, :kw * 8].reshape(cout, kh, kw, 8)[..., :cin].contiguous()
            if ctx.needs_input_grad[0]:
                w_oihw = w16.float().permute(0, 3, 1, 2)
                dx = torch.nn.grad.conv2d_input(x_shape, w_oihw, dy.float(), stride, padding).to(ctx.dtypes[0])
        else:
            acc = _direct_grad(ctx.weight)
            if acc is not None:
                E.conv_wgrad(dyh, xh, acc, stride, padding, err, True)       # split-K atomics land in the parameter's gradient buffer
                dw = None
            else:
                dw = torch.empty(cout, kh, kw, cin, dtype=torch.float32, device=dy.device)
                E.conv_wgrad(dyh, xh, dw, stride, padding, err, False)
            if ctx.needs_input_grad[0]:
                dxh = torch.empty_like(xh)
                other = ctx.fork.take() if ctx.fork is not None else None
                E.conv_dgrad(dyh, w16, dxh, stride, padding, err, None if other is None else _nhwc(other))
                dx = dxh.permute(0, 3, 1, 2).to(ctx.dtypes[0])
                if ctx.fork is not None and other is None:
                    ctx.fork.grad, dx = dx, None            # first of the two consumers: the other one adds this in its kernel
        if dw is None:
            _grad_written(ctx.weight)
        if acc_b is not None:
            _grad_written(bias)
            db = None
        return dx, None if dw is None else dw.to(ctx.dtypes[1]), db, None, None, None, None, None


def conv2d(x, weight, bias=None, stride=1, padding=0, relu=False, stats=None, fork=None):
    """Convolution of a logical ``[N, C, H, W]`` tensor with a ``[Cout, KH, KW, Cin]`` weight (+ bias, + ReLU).

    On a GPU it runs on the implicit-GEMM kernels when the channel counts allow it: ``Cin`` and ``Cout`` multiples of 8,
    or ``Cin <= 8`` with ``KW <= 8`` (the first layer of an image network, whose input is padded to 8 channels). ``stats``
    (fp32 ``[2, Cout]``, zeroed by the caller) receives the per-channel sum and sum of squares of the output. Other shapes
    and CPU tensors use the library convolution."""
    if _own_conv(x, weight, stride):
        return _ConvFn.apply(x, weight, bias, int(stride), int(padding), bool(relu), stats, fork)
    y = F.conv2d(x, weight.permute(0, 3, 1, 2).to(x.dtype), None if bias is None else bias.to(x.dtype), stride, padding)
    y = F.relu(y) if relu else y
    if stats is not None:
        with torch.no_grad():
            yf = y.float()
            stats[0] += yf.sum((0, 2, 3))
            stats[1] += (yf * yf).sum((0, 2, 3))
    return y


def _own_conv(x, weight, stride):
    """Whether the implicit-GEMM kernels take a convolution of ``x`` with a ``[Cout, KH, KW, Cin]`` weight."""
    cout, kh, kw, cin = weight.shape
    return x.is_cuda and cout % 8 == 0 and stride in (1, 2) and kh * kw <= 49 and (cin % 8 == 0 or (cin <= 8 and kw <= 8))


def _eval_norm_ready(gamma, beta, mean, var, channels):
    """fp32 affine parameters and running statistics of ``channels`` entries each, as the evaluation kernels read them."""
    return all(t is not None and t.is_cuda and t.dtype == torch.float32 and t.is_contiguous() and t.numel() == channels
               for t in (gamma, beta, mean, var))


class _ConvBNEvalFn(torch.autograd.Function):
    """Evaluation-mode ``relu?(batch_norm(conv(x)) + residual)`` as one kernel. Only called where no gradient is recorded; being
    an autograd function keeps transforms that it does not support (forward-mode derivatives, vmap) refused."""

    @staticmethod
    def forward(ctx, x, weight, bias, stride, padding, gamma, beta, mean, var, eps, relu, residual):
        E = ops.ext(required=True)
        cout, kh, kw, cin = weight.shape
        err = _error_flag(x.device)
        b32 = bias.float().contiguous() if bias is not None else None
        w16 = _bf16_weight(weight)
        res = _nhwc(residual) if residual is not None else None
        if cin % 8 != 0:
            n, _, h, w = x.shape
            oh, ow, hp, wp = _rowtap_geometry(h, w, kh, kw, stride, padding)
            xh = torch.empty(n, hp, wp, 8, dtype=torch.bfloat16, device=x.device)
            E.pad_image8(x, xh, padding)
            wr = F.pad(F.pad(w16, (0, 8 - cin)).reshape(cout, kh, kw * 8), (0, 64 - kw * 8)).contiguous()
            y = torch.empty(n, oh, ow, cout, dtype=torch.bfloat16, device=x.device)
            E.conv_rowtap_fprop_bn_eval(xh, wr, y, b32, relu, gamma, beta, mean, var, eps, res, stride, err)
        else:
            xh = _nhwc(x)
            n, h, w, _ = xh.shape
            oh, ow = (h + 2 * padding - kh) // stride + 1, (w + 2 * padding - kw) // stride + 1
            y = torch.empty(n, oh, ow, cout, dtype=torch.bfloat16, device=x.device)
            E.conv_fprop_bn_eval(xh, w16, y, b32, relu, gamma, beta, mean, var, eps, res, stride, padding, err)
        return y.permute(0, 3, 1, 2)

    @staticmethod
    def backward(ctx, dy):
        raise RuntimeError("the fused evaluation path records no gradient")


def conv_bn_eval(x, weight, bias, stride, padding, gamma, beta, running_mean, running_var, eps, relu=False, residual=None):
    """``relu?(batch_norm(conv2d(x, weight, bias)) + residual)`` with the running statistics, in one kernel, or ``None`` where
    that kernel does not apply (a gradient is recorded, CPU tensors, shapes or types it does not take)."""
    if torch.is_grad_enabled() or not x.is_cuda:
        return None
    if weight.shape[3] % 8 == 0 and running_mean is not None and running_var is not None and gamma is not None and beta is not None:
        y = ops.ext(required=True).conv_bn_eval_nchw(x, _bf16_weight(weight), bias, stride, padding, gamma, beta, running_mean, running_var, eps,
                                                     relu, residual, _error_flag(x.device))
        if y is not None:
            return y
    cout, kh, kw, _ = weight.shape
    if x.dim() != 4 or not _own_conv(x, weight, stride) or cout > 2048 or \
            not _eval_norm_ready(gamma, beta, running_mean, running_var, cout):
        return None
    if residual is not None:
        oh, ow = (x.shape[2] + 2 * padding - kh) // stride + 1, (x.shape[3] + 2 * padding - kw) // stride + 1
        if residual.dtype != torch.bfloat16 or tuple(residual.shape) != (x.shape[0], cout, oh, ow) or not residual.is_cuda:
            return None
    return _ConvBNEvalFn.apply(x, weight, bias, int(stride), int(padding), gamma, beta, running_mean, running_var, eps, bool(relu), residual)


class _BNEvalFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, gamma, beta, mean, var, eps, relu, residual):
        xh = _nhwc(x)
        y = torch.empty_like(xh)
        ops.ext(required=True).bn_eval(xh, _nhwc(residual) if residual is not None else None, y, gamma, beta, mean, var, eps, relu)
        return y.permute(0, 3, 1, 2)

    @staticmethod
    def backward(ctx, dy):
        raise RuntimeError("the fused evaluation path records no gradient")


def batch_norm_eval(x, gamma, beta, running_mean, running_var, eps, relu=False, residual=None):
    """``relu?(batch_norm(x) + residual)`` of a bf16 tensor with the running statistics, in one kernel, or ``None`` where that
    kernel does not apply."""
    if torch.is_grad_enabled() or not x.is_cuda or x.dim() != 4 or x.dtype != torch.bfloat16 or x.shape[1] % 8 or x.shape[1] > 4096 or \
            not _eval_norm_ready(gamma, beta, running_mean, running_var, x.shape[1]):
        return None
    if residual is not None and (residual.dtype != torch.bfloat16 or residual.shape != x.shape or not residual.is_cuda):
        return None
    return _BNEvalFn.apply(x, gamma, beta, running_mean, running_var, eps, bool(relu), residual)


def channel_sums(x):
    """Per-channel sum and sum of squares (fp32 ``[2, C]``) of a CUDA tensor, as ``conv2d(stats=...)`` leaves them."""
    with torch.no_grad():
        return ops.ext(required=True).bn_sums(_nhwc(x.detach()))


class _BatchNormFn(torch.autograd.Function):
    """Training-mode batch-norm over channels-last activations on the hand-written kernels, with the tail of a residual
    block fused in: ``y = relu?(bn(x) + residual)``. ``sums`` (fp32 ``[2, C]``: sum and sum of squares per channel, as the
    convolution's epilogue leaves them) skips the statistics pass."""

    @staticmethod
    def forward(ctx, x, gamma, beta, residual, eps, relu, sums, running, fork=None, alias=False):
        E = ops.ext(required=True)
        ctx.fork = fork
        run_mean, run_var, batches, momentum = running if running is not None else (None, None, None, 0.0)
        # keep: which outputs the ReLU let through
        xh, y, keep, mean, rstd, g32 = E.bn_fwd_nchw(x, gamma, beta, residual, eps, relu, sums, run_mean, run_var, batches, momentum)
        ctx.save_for_backward(xh, keep, mean, rstd, g32)
        ctx.params = (gamma, beta)
        ctx.set_materialize_grads(False)                     # mean / rstd carry no gradient: no zero tensors for them
        _count_use(ctx, gamma, 1)
        _count_use(ctx, beta, 2)
        ctx.relu = relu
        ctx.has_res = residual is not None
        ctx.dtypes = (x.dtype, gamma.dtype, residual.dtype if residual is not None else None)
        ctx.mark_non_differentiable(mean, rstd)
        return y, mean, rstd, x.view_as(x) if alias else None

    @staticmethod
    def backward(ctx, dy, _dm, _dr, other):
        E = ops.ext(required=True)
        xh, keep, mean, rstd, g32 = ctx.saved_tensors
        if dy is None:
            return (other,) + (None,) * 9
        dyh = _nhwc(dy)
        dx = torch.empty_like(xh)
        dres = None
        if ctx.has_res and ctx.needs_input_grad[3]:
            dres = torch.empty_like(xh) if ctx.relu else dyh                    # without a ReLU the residual gradient is dy itself
        gamma, beta = ctx.params
        acc_g, acc_b = _direct_grad(gamma), _direct_grad(beta)
        direct = acc_g is not None and acc_b is not None
        add = other if other is not None and other.dtype == torch.bfloat16 else None       # what x's alias received: added in the same pass
        sums = E.bn_bwd(dyh, xh, keep, mean, rstd, g32, dx, dres if ctx.relu else None, ctx.relu, acc_g if direct else None,
                        acc_b if direct else None, add)
        gx = dx.permute(0, 3, 1, 2).to(ctx.dtypes[0])
        if other is not None and add is None:
            gx = gx + other
        dr = dres.permute(0, 3, 1, 2).to(ctx.dtypes[2]) if dres is not None else None
        if ctx.fork is not None and dr is not None:
            other = ctx.fork.take()
            if other is None:
                ctx.fork.grad, dr = dr, None            # the residual's other consumer adds this in its input-gradient kernel
            else:
                dr = dr + other
        if direct:
            _grad_written(gamma)
            _grad_written(beta)
            return gx, None, None, dr, None, None, None, None, None, None
        return gx, sums[1].to(ctx.dtypes[1]), sums[0].to(ctx.dtypes[1]), dr, None, None, None, None, None, None


def batch_norm(x, gamma, beta, running_mean=None, running_var=None, training=True, momentum=0.1, eps=1e-5, relu=False,
               residual=None, sums=None, num_batches_tracked=None, fork=None, alias=False):
    """``relu?(batch_norm(x) + residual)`` of an NCHW / channels-last tensor; updates the running statistics like
    ``F.batch_norm``. ``sums``: per-channel sum / sum of squares of ``x`` when a preceding kernel already produced them;
    ``fork``: the ``GradFork`` of ``residual`` when that tensor has a second consumer. ``alias``: returns ``(y, x)`` with an ``x``
    for its second consumer, whose gradient is added inside the backward pass (a channel slice is read in place)."""
    if not (x.is_cuda and training and x.shape[1] % 8 == 0):
        y = F.batch_norm(x, running_mean, running_var, gamma.to(x.dtype) if x.dtype != gamma.dtype and not x.is_cuda else gamma,
                         beta, training, momentum, eps)
        if residual is not None:
            y = y + residual
        y = F.relu(y) if relu else y
        return (y, x) if alias else y
    running = None
    if running_mean is not None and running_mean.dtype == torch.float32 and running_var.dtype == torch.float32:
        running = (running_mean, running_var, num_batches_tracked, float(momentum))     # folded into the statistics kernel
    y, mean, rstd, x_alias = _BatchNormFn.apply(x, gamma, beta, residual, eps, relu, sums, running, fork, alias)
    if running is None and running_mean is not None:
        with torch.no_grad():
            n = x.numel() // x.shape[1]
            var = (1.0 / (rstd * rstd) - eps).clamp_(min=0) * (n / max(n - 1, 1))
            running_mean.mul_(1 - momentum).add_(mean.to(running_mean.dtype), alpha=momentum)
            running_var.mul_(1 - momentum).add_(var.to(running_var.dtype), alpha=momentum)
        if num_batches_tracked is not None:
            num_batches_tracked.add_(1)
    return (y, x_alias) if alias else y


class _MaxPoolFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, k, stride, pad):
        E = ops.ext(required=True)
        xh = x.permute(0, 2, 3, 1).to(torch.bfloat16).contiguous()
        n, h, w, c = xh.shape
        ho, wo = (h + 2 * pad - k) // stride + 1, (w + 2 * pad - k) // stride + 1
        y = torch.empty(n, ho, wo, c, dtype=torch.bfloat16, device=x.device)
        code = torch.empty(n, ho, wo, c, dtype=torch.uint8, device=x.device)
        E.maxpool_fwd(xh, y, code, k, stride, pad)
        ctx.save_for_backward(code)
        ctx.geom = (k, stride, pad)
        ctx.x_shape = tuple(xh.shape)
        ctx.x_dtype = x.dtype
        return y.permute(0, 3, 1, 2)

    @staticmethod
    def backward(ctx, dy):
        E = ops.ext(required=True)
        (code,) = ctx.saved_tensors
        dx = torch.empty(ctx.x_shape, dtype=torch.bfloat16, device=dy.device)
        E.maxpool_bwd(code, dy.permute(0, 2, 3, 1).to(torch.bfloat16).contiguous(), dx, *ctx.geom)
        return dx.permute(0, 3, 1, 2).to(ctx.x_dtype), None, None, None


def max_pool2d(x, kernel_size, stride=None, padding=0):
    stride = stride or kernel_size
    if x.is_cuda and x.shape[1] % 8 == 0:
        return _MaxPoolFn.apply(x, int(kernel_size), int(stride), int(padding))
    return F.max_pool2d(x, kernel_size, stride, padding)


class _SparseLookupFn(torch.autograd.Function):
    """Rows ``ids`` of an fp32 table as bf16 (gather with the cast fused); the gradient is row-sparse like
    ``F.embedding(sparse=True)`` so only the looked-up rows travel to the table's owner."""

    @staticmethod
    def forward(ctx, table, ids):
        E = ops.ext(required=True)
        flat = ids.reshape(-1).contiguous()
        out = torch.empty(flat.numel(), table.shape[1], dtype=torch.bfloat16, device=table.device)
        E.gather_rows_f32(table.detach(), flat, out)
        ctx.save_for_backward(flat)
        ctx.shape = tuple(table.shape)
        return out.view(*ids.shape, table.shape[1])

    @staticmethod
    def backward(ctx, dy):
        (flat,) = ctx.saved_tensors
        vals = dy.reshape(flat.numel(), -1).float()
        with warnings.catch_warnings():
            warnings.simplefilter("ignore")                                   # the library's notice that invariants are unchecked
            return torch.sparse_coo_tensor(flat[None], vals, ctx.shape, check_invariants=False), None


class _DenseLookupFn(torch.autograd.Function):
    """Rows ``ids`` of an fp32 table whose gradient lives in an engine's flat buffer: the backward pass adds the gradient rows
    straight into it (no sort, no table-sized temporary, no accumulation pass)."""

    @staticmethod
    def forward(ctx, table, ids):
        ctx.save_for_backward(ids)
        ctx.table = table
        _count_use(ctx, table, 0)
        return F.embedding(ids, table)

    @staticmethod
    def backward(ctx, dy):
        (ids,) = ctx.saved_tensors
        acc = _direct_grad(ctx.table)
        rows = dy.reshape(-1, dy.shape[-1]).float().contiguous()
        flat = ids.reshape(-1).contiguous()
        if acc is None:
            acc = torch.zeros(ctx.table.shape, dtype=torch.float32, device=dy.device)
            ops.ext(required=True).scatter_add_rows_f32(acc, flat, rows)
            return acc.to(ctx.table.dtype), None
        ops.ext(required=True).scatter_add_rows_f32(acc, flat, rows)
        _grad_written(ctx.table)
        return None, None


def dense_lookup(table, ids):
    """``F.embedding(ids, table)``. Where an engine keeps the table's gradient in a flat buffer, the gradient rows are added
    into it by atomics (the order of addition varies); deterministic runs and all other tables use the library."""
    direct = table.is_cuda and table.dtype == torch.float32 and table.dim() == 2 and ids.dtype == torch.int64 and _direct_grad(table) is not None
    if direct and torch.is_grad_enabled() and not _ordered():
        return _DenseLookupFn.apply(table, ids)
    return F.embedding(ids, table)


def _one_gpu(*tensors):
    """Whether all of ``tensors`` lie on one GPU: a kernel is handed their addresses."""
    return all(t.is_cuda and t.device == tensors[0].device for t in tensors)


def _reverse_mode_only():
    """Whether nothing but reverse-mode differentiation can be going on: no ``torch.func`` transform, no forward-mode level. The kernels'
    autograd functions know of nothing else."""
    return not torch._C._are_functorch_transforms_active() and torch.autograd.forward_ad._current_level < 0


class _PairLookupFn(torch.autograd.Function):
    """Both lookups of (user, item) pairs with the product of their first columns and the concatenation of the others; the
    gradients go straight into the tables' flat gradient buffers."""

    @staticmethod
    def forward(ctx, users_table, items_table, users, items, mf):
        E = ops.ext(required=True)
        raise_bad_ids()
        n, h, dev = users.numel(), users_table.shape[1] - mf, users_table.device
        gmf, kept = (torch.empty(n, w, dtype=torch.float32, device=dev) for w in (mf, 2 * mf))
        x = torch.empty(n, 2 * h, dtype=torch.bfloat16, device=dev)
        E.pair_lookup(users_table.detach(), items_table.detach(), users, items, mf, gmf, x, kept, _id_flag(dev))
        ctx.save_for_backward(kept, users, items)
        ctx.tables = users_table, items_table
        for k, table in enumerate(ctx.tables):
            _count_use(ctx, table, k)
        return gmf, x

    @staticmethod
    def backward(ctx, dgmf, dx):
        E = ops.ext(required=True)
        kept, users, items = ctx.saved_tensors
        direct = [_direct_grad(t) for t in ctx.tables]
        into = [torch.zeros(t.shape, dtype=torch.float32, device=dx.device) if g is None else g for t, g in zip(ctx.tables, direct)]
        dgmf, dx = dgmf.float(), dx.to(torch.bfloat16).contiguous()
        if dgmf.stride(1) != 1 or dgmf.stride(0) % 4 or dgmf.data_ptr() % 16:
            dgmf = dgmf.clone(memory_format=torch.contiguous_format)
        if dx.data_ptr() % 8:                       # a slice: the kernel reads four values at once
            dx = dx.clone()
        E.pair_lookup_bwd(dgmf, dx, kept, users, items, *into)
        grads = []
        for t, g, d in zip(ctx.tables, into, direct):
            if d is not None:
                _grad_written(t)
            grads.append(g if d is None else None)
        return grads[0], grads[1], None, None, None


def pair_lookup(users_table, items_table, users, items, mf):
    """``(u[:, :mf] * i[:, :mf], [u[:, mf:], i[:, mf:]] as bf16)`` for the rows ``u``, ``i`` of two fp32 tables whose gradients an engine
    keeps in a flat buffer (the gradient rows are added by atomics); ``None`` where ``dense_lookup`` would use the library, or the
    layout does not fit."""
    tables = (users_table, items_table)
    if not all(t.is_cuda and t.dtype == torch.float32 and t.dim() == 2 and t.is_contiguous() and t.shape[1] == users_table.shape[1] and
               t.requires_grad and t.data_ptr() % 16 == 0 and t.shape[1] % 4 == 0 and _direct_grad(t) is not None for t in tables):
        return None
    if not _one_gpu(users_table, items_table, users, items) or not _reverse_mode_only():
        return None
    if users_table is items_table or mf % 4 or not 0 < mf < users_table.shape[1] or any(i.dtype != torch.int64 or i.dim() != 1 for i in (users, items)) or \
            users.numel() != items.numel() or not users.numel() or _ordered() or not torch.is_grad_enabled():
        return None
    if any(g.data_ptr() % 16 for g in (_direct_grad(t) for t in tables)):
        return None
    return _PairLookupFn.apply(users_table, items_table, users.contiguous(), items.contiguous(), int(mf))


class _BCEFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, logits, labels):
        E = ops.ext(required=True)
        n = logits.numel()
        part = torch.empty(E.bce_logits_parts(n), dtype=torch.float32, device=logits.device)
        E.bce_logits(logits, labels, part, 1.0 / n)
        ctx.save_for_backward(logits, labels)
        return part.view(()) if part.numel() == 1 else part.sum()

    @staticmethod
    def backward(ctx, grad):
        logits, labels = ctx.saved_tensors
        if torch.is_grad_enabled():                 # create_graph: a gradient that can itself be differentiated
            return (torch.sigmoid(logits) - labels) * (grad / logits.numel()), None
        dx = torch.empty_like(logits)
        ops.ext(required=True).bce_logits_bwd(logits, labels, grad.float().contiguous(), dx, 1.0 / logits.numel())
        return dx, None


def bce_with_logits(logits, labels):
    """``F.binary_cross_entropy_with_logits(logits, labels)`` (the mean), one kernel each way for fp32 CUDA logits."""
    if _one_gpu(logits, labels) and logits.dtype == labels.dtype == torch.float32 and logits.shape == labels.shape and logits.numel() and \
            not labels.requires_grad and _reverse_mode_only():
        return _BCEFn.apply(logits.contiguous(), labels.contiguous())
    return F.binary_cross_entropy_with_logits(logits, labels)


class _ShardedLookupFn(torch.autograd.Function):
    """Lookup in a table that is kept as one row shard per rank (``parallel.fused_engine.ShardedRows``): rows are gathered
    from their owners inside the kernel; the backward pass adds the gradient rows straight into the owners' shards, so the
    table has no gradient tensor at all. ``anchor`` is a dummy that requires grad, so that autograd runs the backward pass."""

    @staticmethod
    def forward(ctx, anchor, handle, ids):
        ctx.handle = handle
        ctx.save_for_backward(ids)
        return handle.lookup(ids).view(*ids.shape, handle.H)

    @staticmethod
    def backward(ctx, dy):
        (ids,) = ctx.saved_tensors
        ctx.handle.push(ids, dy.reshape(-1, ctx.handle.H))
        return None, None, None


_ANCHORS = {}


def sparse_lookup(table, ids):
    """``F.embedding(ids, table, sparse=True)`` returning bf16 on CUDA (fp32 elsewhere).

    A module that reads a table only through this function may list it in ``sparse_lookup_parameters()``; an engine can
    then keep the table as one row shard per rank and attach the shard handle to the parameter (``_sparse_rows``), in which
    case the lookup and its gradient run on the peer-memory kernels."""
    handle = getattr(table, "_sparse_rows", None)
    if handle is not None and ids.is_cuda:
        anchor = _ANCHORS.get(ids.device)
        if anchor is None:
            anchor = _ANCHORS[ids.device] = torch.zeros((), device=ids.device, requires_grad=True)
        return _ShardedLookupFn.apply(anchor, handle, ids)
    if table.is_cuda and table.dtype == torch.float32 and table.is_contiguous() and table.shape[1] % 8 == 0:
        return _SparseLookupFn.apply(table, ids)
    return F.embedding(ids, table, sparse=True)


def _ordered():
    """Whether gradients have to be added up in a fixed order (no atomics)."""
    return os.environ.get("AUTODIST_DETERMINISTIC") == "1" or torch.are_deterministic_algorithms_enabled()


def log_uniform_steps(ids):
    """``log((i + 2) / (i + 1))`` in fp32. Ids from 2^20 on take ``log1p(1 / (i + 1))``: the quotient's distance from 1 has few digits there and
    none from 2^24 on, where its logarithm would be 0. Smaller ids keep the quotient, and with it the results of vocabularies that size."""
    f = ids.float()
    return torch.where(f < 2.0 ** 20, torch.log((f + 2.0) / (f + 1.0)), torch.log1p(1.0 / (f + 1.0)))


def _sampled_chain(neg_logits, dot, bias, neg, targets, num_sampled):
    """What the sampled-softmax kernels compute, as PyTorch expressions (the log-softmax and the mean are theirs too)."""
    def correction(ids):
        return torch.log(num_sampled * (log_uniform_steps(ids) / math.log(bias.numel() + 1.0)))
    own = dot.float() + bias[targets] - correction(targets)
    others = neg_logits.float() + bias[neg] - correction(neg)
    others = others.masked_fill(neg[None, :] == targets[:, None], -1e9)     # remove accidental hits
    return F.cross_entropy(torch.cat([own[:, None], others], 1), torch.zeros_like(targets))


class _SampledSoftmaxFn(torch.autograd.Function):
    """Mean cross-entropy of the true class against shared sampled classes (csrc/sampled_softmax.cu)."""

    @staticmethod
    def forward(ctx, raw, dot, bias, neg, targets, num_sampled):
        E = ops.ext(required=True)
        raise_bad_ids()
        n, k = raw.shape
        dev = raw.device
        corrections, ids = torch.empty(k + n, 2, dtype=torch.float32, device=dev), torch.empty(k + n, dtype=torch.int32, device=dev)
        logits = torch.empty(n, k + 1, dtype=torch.float32, device=dev)
        E.sampled_logits(raw, dot, bias.detach(), neg, targets, 1.0 / math.log(bias.numel() + 1.0), num_sampled, corrections, ids, logits, _id_flag(dev))
        logp = torch.log_softmax(logits, 1)
        ctx.save_for_backward(raw, dot, logp, ids, neg, targets)
        ctx.bias, ctx.num_sampled = bias, num_sampled
        _count_use(ctx, bias, 2)
        return F.nll_loss(logp, torch.zeros_like(targets))

    @staticmethod
    def backward(ctx, grad):
        E = ops.ext(required=True)
        raw, dot, logp, ids, neg, targets = ctx.saved_tensors
        acc = _direct_grad(ctx.bias) if ctx.needs_input_grad[2] else None
        if torch.is_grad_enabled():                 # create_graph: a gradient that can itself be differentiated
            wanted = [t for t, w in zip((raw, dot, ctx.bias), ctx.needs_input_grad) if w]
            found = iter(torch.autograd.grad(_sampled_chain(raw, dot, ctx.bias, neg, targets, ctx.num_sampled), wanted, grad, create_graph=True))
            draw, ddot, d_bias = (next(found) if w else None for w in ctx.needs_input_grad[:3])
            if acc is not None:
                acc.add_(d_bias.detach())
        else:
            n, k = raw.shape
            part = torch.empty(E.sampled_grad_chunks(n, k), k, dtype=torch.float32, device=raw.device)
            draw, ddot, dadj = torch.empty_like(raw), torch.empty_like(dot), torch.empty(k + n, dtype=torch.float32, device=raw.device)
            E.sampled_grad(logp, ids, grad.float().contiguous(), part, draw, ddot, dadj)
            d_bias = None
            if ctx.needs_input_grad[2]:
                d_bias = torch.zeros(ctx.bias.shape, dtype=torch.float32, device=raw.device) if acc is None else acc
                if k + n <= E.SAMPLED_SCAN_MOST:
                    scratch = torch.empty(2, E.sampled_bias_chunks(k + n), k + n, dtype=torch.float32, device=raw.device)
                    E.sampled_bias_grad(ids, dadj, scratch[0], scratch[1].view(torch.int32), d_bias)
                else:
                    d_bias.index_put_((ids.long().clamp_min_(0),), torch.where(ids >= 0, dadj, 0.0), accumulate=True)
        if acc is not None:
            d_bias = None
            _grad_written(ctx.bias)
        return draw, ddot, d_bias, None, None, None


def sampled_softmax_of(neg_logits, dot, bias, neg, targets, num_sampled):
    """Mean over rows of ``-log softmax`` of the true class among itself and the sampled classes ``neg`` (log-uniform over ``bias.numel()``
    classes). ``neg_logits``: ``out @ W[neg].T``; ``dot``: the rows' products with their own classes, bf16 or fp32; logits are corrected by
    ``bias`` and by the log of the expected counts, negatives that hit the row's own class are masked. ``None`` where the kernels do
    not apply."""
    raw = neg_logits
    if not _one_gpu(raw, dot, bias, neg, targets) or not _reverse_mode_only():
        return None
    if not (raw.dtype == torch.bfloat16 and raw.dim() == 2 and raw.shape[0] and raw.shape[1] and raw.shape[1] % 8 == 0):
        return None
    if dot.shape != raw.shape[:1] or dot.dtype not in (torch.bfloat16, torch.float32) or targets.shape != dot.shape or neg.shape != raw.shape[1:]:
        return None
    if bias.dtype != torch.float32 or bias.dim() != 1 or not bias.is_contiguous() or neg.dtype != torch.int64 or targets.dtype != torch.int64:
        return None
    return _SampledSoftmaxFn.apply(raw.contiguous(), dot.contiguous(), bias, neg.contiguous(), targets.contiguous(), float(num_sampled))


def sampled_softmax(neg_logits, out, true_w, bias, neg, targets, num_sampled):
    """``sampled_softmax_of`` with the products of the rows ``out`` and their own classes' weights ``true_w`` (``W[targets]``) in fp32."""
    mats = (neg_logits, out, true_w)
    if not _one_gpu(*mats) or not all(t.dtype == torch.bfloat16 and t.dim() == 2 and t.shape[0] and t.shape[1] and t.shape[1] % 8 == 0 for t in mats):
        return None
    return sampled_softmax_of(neg_logits, (out.float() * true_w.float()).sum(1), bias, neg, targets, num_sampled)


_SPARSE_KINDS = {"sgd": 0, "lazy_adam": 1, "adagrad": 2}


def sparse_rows_update_(kind, table, grad, lr, state1=None, state2=None, step=None, betas=(0.9, 0.999), eps=1e-8,
                        grad_scale=1.0, table_bf16=None):
    """Apply a row-sparse gradient to ``table`` in place, touching only the rows that carry a gradient.

    ``kind``: ``"sgd"``, ``"lazy_adam"`` (moments of untouched rows do not decay; ``step`` is the int64 device counter
    already incremented for this step) or ``"adagrad"``. ``grad`` is a sparse COO tensor (it is coalesced first: the
    kernel needs unique rows) or a ``(rows, values)`` pair that is already unique. ``lr`` is a float or a device
    tensor. The reference reaches the same updates through TensorFlow's ``ResourceSparseApply*`` family
    (``autodist/kernel/common/op_info.py:24-117``)."""
    E = ops.ext(required=True)
    if isinstance(grad, tuple):
        rows, vals = grad
    else:
        g = grad.coalesce()
        rows, vals = g.indices()[0], g.values()
    if not torch.is_tensor(lr):
        lr = torch.tensor([float(lr)], dtype=torch.float32, device=table.device)
    E.sparse_rows_update(table, state1, state2, table_bf16, rows.contiguous(), vals.float().contiguous(), _SPARSE_KINDS[kind], lr,
                         betas[0], betas[1], eps, step, grad_scale)
    return table
