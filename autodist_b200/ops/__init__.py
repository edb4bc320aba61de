"""Python face of the hand-written sm_100a kernels.

``ext()`` returns the compiled extension module. On a machine with a CUDA device
a missing or stale extension is an error (no silent PyTorch fallback); without a
device ``ext()`` returns ``None`` and only the host-side logic is usable.
"""
import importlib.util
import os
import sys

import torch

from autodist_b200.ops import build as _build

_EXT = None
_TRIED = False
launch_count = 0      # kernels launched through the extension by this process (a graph replay re-launches its capture)


def _dgrad_launches(dy, w, dx, stride, pad, *_):
    """One launch per parity class of the input pixels that a filter tap reaches."""
    kh, kw = w.shape[1:3]
    return sum(1 for ph in range(min(stride, dx.shape[1])) for pw in range(min(stride, dx.shape[2]))
               if any((ph + pad - r) % stride == 0 for r in range(kh)) and any((pw + pad - s) % stride == 0 for s in range(kw)))


def _copy_list_launches(taken, dst, src):
    """One launch per sixteen pairs that have something to copy; none when the list was refused."""
    if not taken:
        return 0
    full = 0
    for d, s in zip(dst, src):
        if d.numel() and d.data_ptr() != s.data_ptr():
            if len(dst) <= 16:
                return 1                        # (a step's time: the first pair settles a short list)
            full += 1
    return (full + 15) // 16


class _Counting:
    """Thin proxy over the extension module that counts kernel-launching calls."""
    _NO_LAUNCH = {"ln_bwd_part_floats", "sampled_grad_chunks", "sampled_bias_chunks", "bce_logits_parts", "colsum_parts", "gemm_choice", "gemm_set_trace", "conv_set_trace", "MAX_COMM_BLOCKS"}
    #: kernels per call where that is not one: a number, or a function of the call's arguments
    _MULTI = {"ln_bwd": 2, "keyed_colsum": 2, "relu_bwd_colsum": 2, "bn_sums": 2, "bn_bwd": 2,
              "bn_fwd": lambda *a: 1 if a[9] is not None else 3, "bn_fwd_nchw": lambda *a: 1 if a[6] is not None else 3,       # sums given or not
              "attn_bwd": lambda *a: 2 if a[8] <= 128 else 3,                                                                # tokens
              "xent": lambda *a: 2 if a[7] else 1,                                                                           # sums the weights
              "sampled_logits": 2, "sampled_grad": 2, "sampled_bias_grad": 2, "conv_dgrad": _dgrad_launches}

    #: kernels per call where that depends on what the call returned
    _AFTER = {"copy_list": _copy_list_launches}

    def __init__(self, mod):
        self._mod = mod
        for name in dir(mod):
            if name.startswith("_"):
                continue
            attr = getattr(mod, name)
            if callable(attr) and name not in self._NO_LAUNCH:
                setattr(self, name, self._wrap_after(attr, self._AFTER[name]) if name in self._AFTER else self._wrap(attr, self._MULTI.get(name, 1)))
            else:
                setattr(self, name, attr)

    @staticmethod
    def _wrap_after(fn, launches):
        def call(*args):
            global launch_count
            result = fn(*args)
            launch_count += launches(result, *args)
            return result
        return call

    @staticmethod
    def _wrap(fn, n):
        if callable(n):
            def call(*args):
                global launch_count
                launch_count += n(*args)
                return fn(*args)
        else:
            def call(*args):
                global launch_count
                launch_count += n
                return fn(*args)
        return call


def ext(required=None):
    global _EXT, _TRIED
    if _EXT is not None:
        return _EXT
    if required is None:
        required = torch.cuda.is_available()
    if not _TRIED or required:
        _TRIED = True
        path = _build.so_path()
        stale = os.path.exists(path) and not _build.is_current()
        if (not os.path.exists(path) or stale) and required:
            path = _build.build()              # rebuilds when the sources changed since the shared object was made
        elif stale:
            raise RuntimeError("the sm_100a extension is older than its sources: run `python -m autodist_b200.ops.build`")
        if os.path.exists(path):
            spec = importlib.util.spec_from_file_location(_build.NAME, path)
            mod = importlib.util.module_from_spec(spec)
            spec.loader.exec_module(mod)
            sys.modules[_build.NAME] = mod
            _EXT = _Counting(mod)
    if _EXT is None and required:
        raise RuntimeError("the sm_100a extension is not built: run `python -m autodist_b200.ops.build`")
    return _EXT
