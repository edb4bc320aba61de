"""Several copies in one launch: sizes around a block and a vector, bases off 16 bytes, more copies than a launch takes, refused pairs."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [0, 1])
def test_copy_list(shift):
    from autodist_b200 import ops
    E = ops.ext(required=True)
    sizes = [0, 1, 15, 16, 17, 16383, 16384, 16385, 70001, 3] * 3
    src = [torch.randint(0, 255, (n + shift,), device="cuda", dtype=torch.uint8)[shift:] for n in sizes]
    dst = [torch.full((n + 33,), 7, device="cuda", dtype=torch.uint8) for n in sizes]
    assert E.copy_list([d[:n] for d, n in zip(dst, sizes)], src)
    for d, s, n in zip(dst, src, sizes):
        assert torch.equal(d[:n], s) and (d[n:] == 7).all()
    a = [torch.randn(3, 5, device="cuda"), torch.arange(9, device="cuda"), torch.tensor(2.5, device="cuda")]
    b = [torch.empty_like(x) for x in a]
    assert E.copy_list(b, a) and all(torch.equal(x, y) for x, y in zip(a, b))


def test_pairs_that_do_not_qualify_are_left_alone():
    from autodist_b200 import ops
    E = ops.ext(required=True)
    a, b = torch.randn(4, 6, device="cuda"), torch.zeros(4, 6, device="cuda")
    for d, s in ((b, a.double()), (b, a.t().contiguous().t()), (b, a[:2]), (b, a.cpu()), (b.cpu(), a)):
        assert not E.copy_list([b[:, 0].clone(), d], [a[:, 0].contiguous(), s])
    assert not b.any()
