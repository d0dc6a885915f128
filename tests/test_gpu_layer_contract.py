"""What the layers take and refuse, on CUDA tensors, does not depend on which host path runs them."""

import numpy as np
import pytest
import torch

from gpu_util import DEV, rel_err, to_np, unique_coords

pytestmark = pytest.mark.gpu

SHAPE, N = [20, 20, 20], 1500


def _input(channels, dtype=torch.float32, grad=False):
    import spconv_triton_b200.pytorch as sp

    torch.manual_seed(4)
    idx = torch.from_numpy(unique_coords(3, N, 1, SHAPE)).to(DEV)
    return sp.SparseConvTensor(torch.randn(N, channels, device=DEV).to(dtype).requires_grad_(grad), idx, SHAPE, 1)


def _both_paths(monkeypatch, run):
    """run() through the layers' native host side and through the operator functions."""
    from spconv_triton_b200.pytorch._impl import host

    first = run()
    monkeypatch.setattr(host, "takes", lambda *a: False)
    return first, run()


@pytest.mark.parametrize("what", ["gradient", "autocast", "mixed", "residual"])
def test_pair_list_layers_in_evaluation_mode(what, monkeypatch):
    """Layers of more than 32 offsets are differentiable, follow autocast, keep the type of their features and add
    `add_input` in evaluation mode too."""
    import spconv_triton_b200.pytorch as sp

    torch.manual_seed(5)
    layer = sp.SubMConv3d(16, 16, 5, padding=2).to(DEV).eval()

    def run():
        x = _input(16, torch.float16 if what == "mixed" else torch.float32, grad=what == "gradient")
        layer.zero_grad()
        with torch.set_grad_enabled(what == "gradient"), torch.autocast("cuda", enabled=what == "autocast"):
            y = layer(x, add_input=x) if what == "residual" else layer(x)
        if what != "gradient":
            return [y.features]
        y.features.square().sum().backward()
        return [y.features.detach(), x.features.grad, layer.weight.grad]

    for a, b in zip(*_both_paths(monkeypatch, run)):
        assert a.dtype == b.dtype
        assert rel_err(to_np(a.double()), to_np(b.double())) <= (2e-3 if a.dtype == torch.float16 else 1e-5)


def _misaligned(t):
    """The same values, contiguous, four bytes off a 16-byte boundary."""
    off = 4 // t.element_size()
    return torch.cat([t.new_zeros(off), t.detach().reshape(-1)])[off:].view(t.shape)


@pytest.mark.parametrize("channels", [16, 64])
@pytest.mark.parametrize("which", ["features", "weight", "gradient"])
def test_operands_that_start_anywhere(channels, which):
    """Views into a larger buffer (flat parameters, slices) need not start at a multiple of 16 bytes."""
    import spconv_triton_b200.pytorch as sp

    torch.manual_seed(6)
    layer = sp.SubMConv3d(channels, channels, 3, padding=1).to(DEV)
    x, g = _input(channels).features, torch.randn(N, channels, device=DEV)
    results = []
    for moved in (False, True):
        if moved and which == "weight":
            layer.weight.data = _misaligned(layer.weight.data)
        feats = (_misaligned(x) if moved and which == "features" else x.clone()).requires_grad_()
        layer.zero_grad()
        y = layer(_input(channels).replace_feature(feats)).features
        y.backward(_misaligned(g) if moved and which == "gradient" else g)
        results.append([y.detach(), feats.grad, layer.weight.grad, layer.bias.grad])
        with torch.no_grad():
            results[-1].append(layer.eval()(_input(channels).replace_feature(feats.detach())).features)
        layer.train()
    for a, b in zip(*results):
        assert torch.equal(a, b)


@pytest.mark.parametrize("kind", ["subm", "down", "max", "avg"])
def test_forward_mode_derivatives_are_refused(kind):
    """... not dropped: the layers have no forward-mode derivative."""
    import spconv_triton_b200.pytorch as sp

    layer = {"subm": lambda: sp.SubMConv3d(16, 16, 3, padding=1), "down": lambda: sp.SparseConv3d(16, 16, 3, 2, 1),
             "max": lambda: sp.SparseMaxPool3d(2, 2), "avg": lambda: sp.SparseAvgPool3d(2, 2)}[kind]().to(DEV).train()
    x = _input(16)
    with torch.autograd.forward_ad.dual_level():
        dual = torch.autograd.forward_ad.make_dual(x.features, torch.ones_like(x.features))
        with pytest.raises((NotImplementedError, RuntimeError), match="forward"):
            layer(x.replace_feature(dual))


@pytest.mark.parametrize("kind", ["subm", "max"])
@pytest.mark.parametrize("transform", ["grad", "vmap"])
def test_function_transforms_are_refused(kind, transform):
    import spconv_triton_b200.pytorch as sp

    layer = (sp.SubMConv3d(16, 16, 3, padding=1) if kind == "subm" else sp.SparseMaxPool3d(2, 2)).to(DEV).train()
    x = _input(16)

    def run(feats):
        y = layer(x.replace_feature(feats)).features
        return y.sum() if transform == "grad" else y

    with pytest.raises(RuntimeError):
        torch.func.grad(run)(x.features) if transform == "grad" else torch.func.vmap(run)(x.features[None])


@pytest.mark.parametrize("train", [False, True])
def test_a_bias_that_does_not_fit_is_no_operand_of_a_kernel(train):
    """A bias of one value is broadcast in training; other shapes, and a bias elsewhere, are errors."""
    import spconv_triton_b200.pytorch as sp

    layer, x = sp.SubMConv3d(16, 16, 3, padding=1, bias=True).to(DEV).train(train), _input(16)
    with torch.set_grad_enabled(train):
        layer.bias = torch.nn.Parameter(torch.zeros(16, device=DEV))
        plain = layer(x).features
        layer.bias = torch.nn.Parameter(torch.full((1,), 0.5, device=DEV))
        if train:
            y = layer(x).features
            assert torch.equal(y, plain + 0.5)
            y.sum().backward()
            assert layer.bias.grad.shape == (1,) and float(layer.bias.grad) == 16 * N
        else:
            with pytest.raises(ValueError):
                layer(x)
        for bias in (torch.zeros(15, device=DEV), torch.zeros(16)):
            layer.bias = torch.nn.Parameter(bias)
            with pytest.raises((ValueError, RuntimeError)):
                layer(x)


def test_weights_on_another_device_are_refused():
    import spconv_triton_b200.pytorch as sp

    with pytest.raises((ValueError, RuntimeError, AssertionError)):
        sp.SubMConv3d(16, 16, 3, padding=1)(_input(16))


def test_a_bias_that_does_not_fit_stays_out_of_the_native_pass():
    import spconv_triton_b200.pytorch as sp

    net = sp.SparseSequential(sp.SubMConv3d(16, 16, 3, padding=1, bias=True)).to(DEV).half().eval()
    x = _input(16, torch.float16)
    with torch.no_grad():
        net(x)
        net[0].bias = torch.nn.Parameter(torch.zeros(1, device=DEV).half())
        with pytest.raises(ValueError):
            net(x)


def test_a_bias_in_double_precision():
    import spconv_triton_b200.pytorch as sp

    layer, x = sp.SubMConv3d(16, 16, 3, padding=1, bias=True).to(DEV), _input(16)
    layer.bias = torch.nn.Parameter(layer.bias.detach().double())
    y = layer(x).features
    y.sum().backward()
    assert y.dtype == torch.float32 and layer.bias.grad.dtype == torch.float64
    assert torch.equal(layer.bias.grad, torch.full_like(layer.bias.grad, N))
