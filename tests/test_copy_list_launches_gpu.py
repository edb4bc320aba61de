"""One launch per sixteen copies that have something to copy, whatever stands between them."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _launches(fn):
    fn()
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        fn()
        torch.cuda.synchronize()
    return sum(e.count for e in prof.key_averages() if "copy_list_kernel" in e.key)


@pytest.mark.parametrize("empty,full,launches", [(0, 16, 1), (24, 16, 1), (5, 17, 2), (40, 1, 1), (3, 0, 0)])
def test_empty_pairs_take_no_place(empty, full, launches):
    from autodist_b200 import ops
    E = ops.ext(required=True)
    src = [torch.randn(0 if i < empty else 9, device="cuda") for i in range(empty + full)]
    dst = [torch.empty_like(t) for t in src]
    assert _launches(lambda: E.copy_list(dst, src)) == launches
    assert all(torch.equal(a, b) for a, b in zip(dst, src))
