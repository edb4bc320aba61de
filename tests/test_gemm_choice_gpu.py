"""``gemm_choice`` names the kernel that ``gemm`` launches, for outputs of both types and operands of both layouts."""
import re

import pytest
import torch

pytestmark = pytest.mark.gpu


def _launched(fn):
    fn()
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        fn()
        torch.cuda.synchronize()
    names = [e.key for e in prof.key_averages() if "gemm" in e.key]
    assert len(names) == 1, names
    if "gemm2_kernel" in names[0]:
        return 512, False
    return int(re.search(r"gemm(?:_split)?_kernel<(?:\(int\))?(\d+)", names[0]).group(1)), "gemm_split" in names[0]


@pytest.mark.parametrize("M,N,K", [(3072, 1024, 4096), (1024, 1024, 1024), (256, 256, 8192), (512, 2048, 512)])
@pytest.mark.parametrize("mn", [False, True])
@pytest.mark.parametrize("fp32", [False, True])
def test_the_named_kernel_runs(M, N, K, mn, fp32):
    from autodist_b200 import ops
    E = ops.ext(required=True)
    a = torch.randn((K, M) if mn else (M, K), device="cuda").bfloat16()
    b = torch.randn((K, N) if mn else (N, K), device="cuda").bfloat16()
    c, err = torch.empty(M, N, dtype=torch.float32 if fp32 else torch.bfloat16, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    bn, split = E.gemm_choice(M, N, K, 1, 0, mn, fp32)
    assert _launched(lambda: E.gemm(a, b, c, mn, mn, 0, None, None, None, 1.0, 0.0, err, 0)) == (bn, split > 1)
    if fp32 == mn:
        assert E.gemm_choice(M, N, K, 1, 0, mn) == (bn, split)
