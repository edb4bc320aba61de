"""The launch counter over calls whose kernels depend on what they returned."""
import types

import torch

from autodist_b200 import ops


def _counted(counting, *args):
    before = ops.launch_count
    counting.copy_list(*args)
    return ops.launch_count - before


def test_copies_count_as_launched():
    taken = ops._Counting(types.SimpleNamespace(copy_list=lambda dst, src: True))
    refused = ops._Counting(types.SimpleNamespace(copy_list=lambda dst, src: False))
    src, empty = [torch.ones(3) for _ in range(17)], [torch.ones(0)] * 20
    dst = [torch.empty(3) for _ in range(17)]
    assert _counted(refused, dst, src) == 0
    assert _counted(taken, dst[:16], src[:16]) == 1
    assert _counted(taken, dst, src) == 2
    assert _counted(taken, empty + dst[:1], empty + src[:1]) == 1
    assert _counted(taken, empty, empty) == _counted(taken, [], []) == _counted(taken, src, src) == 0
