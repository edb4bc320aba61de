"""Bindings that stand in for library calls launch on their tensors' device, whichever device is current: like the library, they switch to it."""
import os
import re

import pytest

BINDINGS = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "autodist_b200", "csrc", "bindings.cpp")


@pytest.mark.parametrize("name", ["copy_list", "pair_lookup", "pair_lookup_bwd", "bce_logits", "bce_logits_bwd", "sampled_logits", "sampled_grad",
                                  "sampled_bias_grad"])
def test_the_device_is_switched_before_the_stream_is_asked_for(name):
    with open(BINDINGS) as f:
        source = f.read()
    body = re.search(r"^(?:void|bool) %s\((?:[^{]|\n)*?\{\n(.*?)^\}" % name, source, re.M | re.S).group(1)
    assert "STREAM" in body
    assert 0 <= body.find("c10::cuda::CUDAGuard guard(") < body.find("STREAM")
