"""Prepared copies of fp32 weights: they belong to a call, so a weight that changes, by whatever route, is never
met by an old copy, and nothing stays on the device when it is gone."""

import gc

import pytest
import torch

from gpu_util import DEV, unique_coords

pytestmark = pytest.mark.gpu

SHAPE = [32, 32, 32]


@pytest.fixture(params=[False, True], ids=["ieee", "tf32"])
def tf32(request):
    from spconv_triton_b200 import constants

    old = constants.SPCONV_ALLOW_TF32
    constants.SPCONV_ALLOW_TF32 = request.param
    yield request.param
    constants.SPCONV_ALLOW_TF32 = old


def _input(channels, grad=False):
    import spconv_triton_b200.pytorch as sp

    idx = torch.from_numpy(unique_coords(3, 3000, 1, SHAPE)).to(DEV)
    feats = torch.randn(3000, channels, device=DEV).requires_grad_(grad)
    return sp.SparseConvTensor(feats, idx, SHAPE, 1)


def test_nothing_stays_when_layers_go(tf32):
    import spconv_triton_b200.pytorch as sp

    def use():
        layer = sp.SubMConv3d(16, 32, 3, padding=1).to(DEV)
        # (a weight that is no contiguous tensor is copied first)
        layer.weight.data = layer.weight.data.transpose(1, 3).contiguous().transpose(1, 3)
        for train in (True, False):
            layer.train(train)(_input(16, grad=train)).features.sum()
        layer.train()(_input(16, grad=True)).features.sum().backward()

    use()
    gc.collect()
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    for _ in range(20):
        use()
    gc.collect()
    torch.cuda.synchronize()
    assert torch.cuda.memory_allocated() <= before


@pytest.mark.parametrize("path", ["layer", "operators"])
def test_weights_written_past_their_version_counter(tf32, path, monkeypatch):
    """Doubling is exact in every step, so the output doubles bit for bit."""
    import spconv_triton_b200.pytorch as sp
    from spconv_triton_b200.pytorch._impl import host

    if path == "operators":
        monkeypatch.setattr(host, "takes", lambda *a: False)
    layer, x = sp.SubMConv3d(16, 32, 3, padding=1, bias=False).to(DEV).eval(), _input(16)
    with torch.no_grad():
        first = layer(x).features
        layer.weight.data.mul_(2.0)  # (a moving average of weights writes like this)
        assert torch.equal(layer(x).features, 2 * first)


def test_captured_layers_follow_their_weight(tf32):
    """A captured layer multiplies the weight of the time of its replay, and what a capture recorded but nobody
    has run yet is no input of other calls."""
    import spconv_triton_b200.pytorch as sp

    layer, x = sp.SubMConv3d(16, 32, 3, padding=1, bias=False, indice_key="k").to(DEV).eval(), _input(16)
    with torch.no_grad():
        x = layer(x).replace_feature(x.features)  # the neighbour map exists before the capture
        layer.weight.mul_(2.0)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            captured = layer(x).features
        eager = layer(x).features
        graph.replay()
        assert torch.equal(captured, eager)
        layer.weight.mul_(2.0)
        graph.replay()
        assert torch.equal(captured, 2 * eager)
