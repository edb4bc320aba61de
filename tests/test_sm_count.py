"""Grids are sized by the device they run on: no source counts on one number of SMs."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "autodist_b200", "csrc")


@pytest.mark.parametrize("path", [p for p in sorted(glob.glob(os.path.join(CSRC, "*.c*"))) if not p.endswith("sm_count.h")], ids=os.path.basename)
def test_no_literal_number_of_sms(path):
    with open(path) as f:
        code = [line.partition("//")[0] for line in f]
    assert not [line for line in code if re.search(r"\b148\b", line)]
