"""The max-pool kernels over the windows that have their own path and the general one: odd sizes, padding, ties, infinities.

Values and routes are exact: the oracle is the library's pooling in float32 on the same bf16 values, whose backward sends each window's
gradient to its first maximum too. A pixel sums at most ceil(k / stride)^2 bf16 gradients in float32 and is rounded to bf16 once."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,stride,pad", [(3, 2, 0), (3, 2, 1), (2, 2, 0), (2, 2, 1), (3, 1, 1), (2, 3, 0)])
@pytest.mark.parametrize("shape", [(1, 8, 3, 3), (2, 24, 13, 14), (3, 64, 17, 9), (1, 264, 6, 31)])
def test_max_pool_values_and_routes(k, stride, pad, shape):
    from autodist_b200.ops import functional as Fn
    torch.manual_seed(5)
    x = torch.relu(torch.randn(shape, device="cuda"))                          # ties at 0
    x[:, ::3, 1] = float("-inf")
    x[:, 1::3, 2, 1] = float("inf")
    x[:, 2::3] *= 1e-38                                                        # many of them below the smallest normal number
    x = x.bfloat16().contiguous(memory_format=torch.channels_last)
    ours, ref = x.clone().requires_grad_(True), x.float().requires_grad_(True)
    y, want = Fn.max_pool2d(ours, k, stride, pad), torch.nn.functional.max_pool2d(ref, k, stride, pad)
    assert torch.equal(y.float(), want)
    dy = torch.randn(want.shape, device="cuda").bfloat16()
    y.backward(dy)
    want.backward(dy.float())
    mag = torch.nn.functional.max_pool2d(ref, k, stride, pad)
    ref_grad, ref.grad = ref.grad, None
    mag.backward(dy.float().abs())                                             # sum of the magnitudes that meet in a pixel
    assert ((ours.grad.float() - ref_grad).abs() <= 2.0 ** -8 * ref_grad.abs() + 2.0 ** -20 * ref.grad).all()
