"""Hooks on the containers of the DenseNet model: the kernel path, which calls the layers one by one, steps aside for them."""
import pytest
import torch
from torch import nn


def test_every_kind_of_hook_is_seen():
    from autodist_b200.models.cnn import _hooked
    nop = lambda *a: None      # noqa: E731
    g = nn.modules.module
    kinds = [(lambda m: m.register_forward_hook(nop)), (lambda m: m.register_forward_pre_hook(nop)),
             (lambda m: m.register_full_backward_hook(nop)), (lambda m: m.register_full_backward_pre_hook(nop)),
             (lambda m: g.register_module_forward_hook(nop)), (lambda m: g.register_module_forward_pre_hook(nop)),
             (lambda m: g.register_module_full_backward_hook(nop)), (lambda m: g.register_module_full_backward_pre_hook(nop))]
    a, b = nn.ReLU(), nn.ReLU()
    for register in kinds:
        assert not _hooked(a, b)
        handle = register(b)
        assert _hooked(a, b)
        handle.remove()


def _net():
    from autodist_b200.models.cnn import DenseNet121, ImageClassifier
    torch.manual_seed(0)
    return ImageClassifier(DenseNet121(num_classes=16, growth=8, blocks=(2, 2, 2, 2)), num_classes=16).cuda()


@pytest.mark.gpu
@pytest.mark.parametrize("where", ["features", "layer", "f", "global"])
def test_backward_hooks_on_containers_fire_and_change_gradients(where):
    from autodist_b200.models import cnn
    net = _net()
    images, labels = torch.randn(2, 3, 64, 64, device="cuda"), torch.tensor([1, 2], device="cuda")
    features = net.net.features
    target = {"features": features, "layer": features[2], "f": features[2].f, "global": features[2]}[where]
    seen = []

    def hook(module, grad_input, grad_output):
        if module is target:
            seen.append(module)
            return tuple(None if g is None else torch.zeros_like(g) for g in grad_input)

    handle = nn.modules.module.register_module_full_backward_hook(hook) if where == "global" else target.register_full_backward_hook(hook)
    before = []
    pre = target.register_full_backward_pre_hook(lambda m, g: before.append(m))
    net(images, labels).backward()
    handle.remove()
    pre.remove()
    assert seen == [target] and before == [target]
    stem = features[0].conv.weight.grad
    if where in ("layer", "global"):                        # (`f` is one of two branches, `features` starts at the images)
        assert stem is None or not stem.any()              # the gradient that the hook cleared reaches nothing in front of the container
    net.zero_grad()
    net(images, labels).backward()
    assert seen == [target] and features[0].conv.weight.grad.any()
    assert isinstance(features[2], cnn._DenseLayer)
