"""Evaluation-mode normalisations folded into the store of the layer before them: made anew by each pass."""

import pytest
import torch
from torch import nn

import spconv_triton_b200.pytorch as sp
from gpu_util import DEV, unique_coords
from spconv_triton_b200 import constants
from spconv_triton_b200.pytorch.modules import _folded_bn, _folded_norms

pytestmark = pytest.mark.gpu

SHAPE, N = (24, 24, 24), 3000


def _bn(channels, dtype=torch.float32, affine=True, eps=1e-3):
    bn = nn.BatchNorm1d(channels, eps=eps, affine=affine)
    g = torch.Generator().manual_seed(channels)
    with torch.no_grad():
        bn.running_mean.copy_(torch.randn(channels, generator=g))
        bn.running_var.copy_(0.1 + torch.rand(channels, generator=g))
        if affine:
            bn.weight.copy_(torch.randn(channels, generator=g))
            bn.bias.copy_(torch.randn(channels, generator=g))
    return bn.to(DEV).to(dtype).eval()


def test_the_kernel_rounds_as_the_functions_do():
    """Every type, without parameters, odd channel counts, more of them than a launch takes."""
    norms = [_bn(c, dtype, affine) for c in (1, 3, 16, 257, 1024) for dtype in (torch.float16, torch.bfloat16, torch.float32)
             for affine in (True, False)] * 2
    norms[4].weight.data = norms[4].weight.data.bfloat16()  # (a type of its own)
    block, places, _ = _folded_norms(norms, torch.zeros(1, device=DEV))
    assert len(norms) > 48
    for bn, (at, to) in zip(norms, places):
        for got, want in zip((block[at:at + bn.num_features], block[to:to + bn.num_features]), _folded_bn(bn)):
            assert torch.equal(got, want)


def test_what_the_kernel_does_not_take():
    like = torch.zeros(1, device=DEV)
    wide = _bn(8).double()
    block, ((at, to),), _ = _folded_norms([wide], like)
    assert torch.equal(block[at:at + 8], _folded_bn(wide)[0]) and torch.equal(block[to:to + 8], _folded_bn(wide)[1])
    strided = _bn(8)
    strided.running_mean = torch.randn(16, device=DEV)[::2]
    block, ((at, to),), _ = _folded_norms([strided], like)
    assert torch.equal(block[to:to + 8], _folded_bn(strided)[1])
    assert _folded_norms([_bn(8).cpu()], like) is None
    short = _bn(8)
    short.num_features = 16
    assert _folded_norms([short], like) is None


def _net():
    torch.manual_seed(0)
    net = sp.SparseSequential(sp.SubMConv3d(16, 32, 3, bias=False, indice_key="a"), _bn(32), nn.ReLU(),
                              sp.SparseConv3d(32, 32, 3, 2, padding=1, bias=False), _bn(32), nn.ReLU())
    return net.to(DEV).half().eval()


def _input():
    idx = torch.from_numpy(unique_coords(3, N, 1, SHAPE)).to(DEV)
    return sp.SparseConvTensor(torch.randn(N, 16, generator=torch.Generator(DEV).manual_seed(1), device=DEV).half(), idx, list(SHAPE), 1)


def _apart(net, x):
    """The modules one by one, none of them folded."""
    constants.SPCONV_FOLD_BN_RELU, was = False, constants.SPCONV_FOLD_BN_RELU
    try:
        return net(x).features
    finally:
        constants.SPCONV_FOLD_BN_RELU = was


@pytest.mark.parametrize("native", [True, False])
def test_statistics_written_past_their_version_counters(native, monkeypatch):
    monkeypatch.setattr(constants, "SPCONV_NATIVE_SEQUENCE", native)
    net, x = _net(), _input()
    with torch.no_grad():
        for scale in (1.0, 3.0, 0.5):
            for i in (1, 4):
                net[i].running_mean.data.mul_(scale).add_(scale)
                net[i].running_var.data.mul_(scale)
                net[i].weight.data.mul_(scale)
            got, want = net(x).features, _apart(net, x)
            assert (got.float() - want.float()).norm() <= 2e-3 * want.float().norm()


@pytest.mark.parametrize("native", [True, False])
def test_passes_on_two_streams(native, monkeypatch):
    """The second stream's pass does not wait for 50 ms of other work on the stream of the first."""
    monkeypatch.setattr(constants, "SPCONV_NATIVE_SEQUENCE", native)
    net, x = _net(), _input()
    with torch.no_grad():
        want = net(x).features.clone()
        torch.cuda.synchronize()
        first, second = torch.cuda.Stream(), torch.cuda.Stream()
        block_first = torch.cuda.Event()
        with torch.cuda.stream(first):
            torch.cuda._sleep(100_000_000)
            _folded_norms([net[1], net[4]], x.features)
            block_first.record()
        with torch.cuda.stream(second):
            got = net(x).features
            second.synchronize()
            assert not block_first.query()
        assert torch.equal(got, want)
    torch.cuda.synchronize()


def test_a_graph_follows_the_statistics(monkeypatch):
    monkeypatch.setattr(constants, "SPCONV_NATIVE_SEQUENCE", False)
    monkeypatch.setattr(constants, "SPCONV_RULEBOOK_RUNAHEAD", False)
    net, x = sp.SparseSequential(*list(_net()._modules.values())[:3]), _input()
    with torch.no_grad():
        x.indice_dict.update(net(x).indice_dict)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = net(x).features
        for scale in (1.0, 3.0):
            net[1].running_mean.mul_(scale)
            net[1].weight.mul_(scale)
            graph.replay()
            want = _apart(net, x)
            assert (out.float() - want.float()).norm() <= 2e-3 * want.float().norm()
