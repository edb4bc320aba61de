"""Feeds that start anywhere in their storage (slices of a data set on the device): right at every offset, and no slower than the bytes ask for."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [1, 2, 3, 4, 6, 7, 8, 12, 13])
@pytest.mark.parametrize("size", [1, 4, 5, 7, 8, 9, 255, 16379, 16384, 16389, 50003])
def test_every_offset(offset, size):
    from autodist_b200 import ops
    E = ops.ext(required=True)
    whole = torch.randint(0, 255, (size + 32,), device="cuda", dtype=torch.uint8)
    for into in (0, 4, 8, 3):
        out = torch.full((size + 48,), 7, device="cuda", dtype=torch.uint8)
        assert E.copy_list([out[into:into + size]], [whole[offset:offset + size]])
        assert torch.equal(out[into:into + size], whole[offset:offset + size])
        assert (out[:into] == 7).all() and (out[into + size:] == 7).all()


def _time(fn):
    for _ in range(3):
        fn()
    times = []
    for _ in range(15):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        for _ in range(10):
            fn()
        b.record()
        torch.cuda.synchronize()
        times.append(a.elapsed_time(b))
    return sorted(times)[7]


@pytest.mark.parametrize("offset", [4, 8, 1, 2])
def test_an_offset_costs_no_multiple(offset):
    """64 MB, so that launches do not count. The bytes moved are the same; a word of 4 bytes takes four times the instructions of one of 16."""
    from autodist_b200 import ops
    E = ops.ext(required=True)
    n = 1 << 26
    whole, out = torch.empty(n + 16, device="cuda", dtype=torch.uint8), torch.empty(n, device="cuda", dtype=torch.uint8)
    aligned = _time(lambda: E.copy_list([out], [whole[:n]]))
    assert _time(lambda: E.copy_list([out], [whole[offset:offset + n]])) < 3 * aligned
