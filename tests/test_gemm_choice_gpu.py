"""``gemm_choice`` names the kernel that ``gemm`` launches, for outputs of both types and operands of both layouts. In a process of its own: the
profiler that names the launches is used once per process."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CODE = """
import itertools, json, re, torch
from torch.profiler import ProfilerActivity, profile
from autodist_b200 import ops
E = ops.ext(required=True)
err = torch.zeros(1, dtype=torch.int32, device="cuda")
calls, named = [], []
for (M, N, K), mn, fp32, fixed in itertools.product([(3072, 1024, 4096), (1024, 1024, 1024), (256, 256, 8192), (128, 512, 2048)], (False, True),
                                                    (False, True), (False, True)):
    a = torch.randn((K, M) if mn else (M, K), device="cuda").bfloat16()
    b = torch.randn((K, N) if mn else (N, K), device="cuda").bfloat16()
    c = torch.empty(M, N, dtype=torch.float32 if fp32 else torch.bfloat16, device="cuda")
    named.append(E.gemm_choice(M, N, K, 1, 0, mn, fp32, fixed))
    if fp32 == mn and not fixed:
        assert E.gemm_choice(M, N, K, 1, 0, mn) == named[-1]
    calls.append(lambda a=a, b=b, c=c, mn=mn, fixed=fixed: E.gemm(a, b, c, mn, mn, 0, None, None, None, 1.0, 0.0, err, -1 if fixed else 0))
for call in calls:
    call()
torch.cuda.synchronize()
with profile(activities=[ProfilerActivity.CUDA]) as prof:
    for call in calls:
        call()
    torch.cuda.synchronize()
ran = []
for e in sorted((e for e in prof.events() if "gemm" in e.name and "kernel" in e.name), key=lambda e: e.time_range.start):
    ran.append((512, False) if "gemm2_kernel" in e.name else
               (int(re.search(r"gemm(?:_split)?_kernel<(?:\\(int\\))?(\\d+)", e.name).group(1)), "gemm_split" in e.name))
print(json.dumps([ran, [(bn, split > 1) for bn, split in named]]))
"""


def test_the_named_kernel_runs():
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    out = subprocess.run([sys.executable, "-c", CODE], cwd=root, capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr[-2000:]
    ran, named = json.loads(out.stdout.strip().splitlines()[-1])
    assert len(ran) == 32 and ran == named
