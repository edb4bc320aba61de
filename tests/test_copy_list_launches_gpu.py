"""One launch per sixteen copies that have something to copy, whatever stands between them. In a process of its own: the profiler that counts
the launches is used once per process."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CODE = """
import json, sys, torch
from torch.profiler import ProfilerActivity, profile
from autodist_b200 import ops
E = ops.ext(required=True)
lists = []
for empty, full in json.loads(sys.argv[1]):
    src = [torch.randn(0 if i < empty else 9, device="cuda") for i in range(empty + full)]
    lists.append(([torch.empty_like(t) for t in src], src))
for dst, src in lists:
    E.copy_list(dst, src)
    assert all(torch.equal(a, b) for a, b in zip(dst, src))
mark = torch.zeros(1, device="cuda")
torch.cuda.synchronize()
with profile(activities=[ProfilerActivity.CUDA]) as prof:
    for dst, src in lists:
        E.copy_list(dst, src)
        mark.add_(1.0)                                  # stands between the launches of two lists
    torch.cuda.synchronize()
found = [0]
for e in sorted((e for e in prof.events() if "copy_list_kernel" in e.name or "elementwise" in e.name), key=lambda e: e.time_range.start):
    if "copy_list_kernel" in e.name:
        found[-1] += 1
    else:
        found.append(0)
print(json.dumps(found[:len(lists)]))
"""


def test_empty_pairs_take_no_place():
    cases = [(0, 16), (24, 16), (5, 17), (40, 1), (3, 0)]
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    out = subprocess.run([sys.executable, "-c", CODE, json.dumps(cases)], cwd=root, capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr[-2000:]
    assert json.loads(out.stdout.strip().splitlines()[-1]) == [1, 1, 2, 1, 0]
