"""Flat updates on both sides of the size from which weights are taken in groups, at bases on and off a vector, remainders included: the same bits either
way, since every weight has the same operations. And few weights cost no more than a launch."""
import pytest
import torch

pytestmark = pytest.mark.gpu
LEAST = 1 << 20


def _update(E, rule, n, shift):
    torch.manual_seed(n)
    lr, step = torch.tensor([0.125], device="cuda"), torch.tensor([3], device="cuda")
    p, g, s = torch.randn(n, device="cuda"), torch.randn(n, device="cuda"), torch.rand(n, device="cuda")
    buf = [torch.full((n + 9,), 7.0, device="cuda") for _ in range(3)] + [torch.full((n + 9,), 7.0, dtype=torch.bfloat16, device="cuda")]
    at = [b[shift:shift + n] for b in buf]
    for a, v in zip(at, (p, g, s)):
        a.copy_(v)
    P, G, S, P16 = at
    if rule == "adagrad":
        E.adagrad_update(P, G, S, P16, lr, 1e-10, 0.01, 0.5)
    else:
        E.sgd_update(P, G, S if rule == "momentum" else None, P16, lr, 0.9 if rule == "momentum" else 0.0, 0.0, 0.01, False, step, 0.5)
    for b in buf:
        assert (b[:shift] == 7).all() and (b[shift + n:] == 7).all()
    return P.clone(), S.clone(), P16.clone()


@pytest.mark.parametrize("rule", ["sgd", "momentum", "adagrad"])
@pytest.mark.parametrize("n", [LEAST - 1, LEAST, LEAST + 1, LEAST + 3, 3 * LEAST + 2])
def test_groups_and_single_weights_agree(rule, n):
    from autodist_b200 import ops
    E = ops.ext(required=True)
    for a, b in zip(_update(E, rule, n, 0), _update(E, rule, n, 1)):
        assert torch.equal(a, b)


def _time(fn):
    for _ in range(3):
        fn()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for _ in range(50):
            fn()
    times = []
    for _ in range(9):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        graph.replay()
        b.record()
        torch.cuda.synchronize()
        times.append(a.elapsed_time(b))
    return sorted(times)[4]


def test_few_weights_cost_a_launch():
    """4096 weights against one: both are a launch and a few latencies long."""
    from autodist_b200 import ops
    E = ops.ext(required=True)
    p, g, s = torch.randn(4096, device="cuda"), torch.randn(4096, device="cuda"), torch.rand(4096, device="cuda")
    p16, lr = torch.empty(4096, dtype=torch.bfloat16, device="cuda"), torch.tensor([0.1], device="cuda")
    one, many = (_time(lambda: E.adagrad_update(p[:n], g[:n], s[:n], p16[:n], lr, 1e-10, 0.0, 1.0)) for n in (1, 4096))
    assert many < 1.5 * one
