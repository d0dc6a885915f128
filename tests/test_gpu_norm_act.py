"""BatchNorm1d and the activation after it in training, as one operator (csrc/norm.cu), against the torch modules in
fp64 and against the modules run one by one."""

import copy

import pytest
import torch
from torch import nn

import spconv_triton_b200.pytorch as sp
from spconv_triton_b200.pytorch import modules

pytestmark = pytest.mark.gpu

ACTS = {"none": None, "relu": nn.ReLU, "silu": nn.SiLU}
EPS = {torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8, torch.float32: 2.0 ** -24}


def _tensor(features):
    n = features.shape[0]
    idx = torch.stack([torch.zeros(n, dtype=torch.int32), *([torch.arange(n, dtype=torch.int32)] * 3)], 1).cuda()
    return sp.SparseConvTensor(features, idx, [n] * 3, 1)


def _net(channels, act, affine=True):
    net = sp.SparseSequential(nn.BatchNorm1d(channels, eps=1e-3, momentum=0.1, affine=affine), *([ACTS[act]()] if ACTS[act] else []))
    if affine:
        g = torch.Generator().manual_seed(channels)
        net[0].weight.data = 1 + 0.3 * torch.randn(channels, generator=g)
        net[0].bias.data = 0.3 * torch.randn(channels, generator=g)
    return net.cuda().train()


def _apart(net, x):
    """The same modules, none of them in the operator's sight."""
    y = x.features
    for m in net._modules.values():
        y = m(y)
    return y


@pytest.mark.parametrize("act", list(ACTS))
@pytest.mark.parametrize("dtype,rows,channels,shift", [
    (torch.float16, 2, 8, 0.0), (torch.float16, 31, 16, 3.0), (torch.float16, 4099, 32, 0.5), (torch.bfloat16, 1000, 48, 1.0),
    (torch.float32, 777, 4, 50.0), (torch.float32, 70001, 64, 5.0), (torch.float16, 257, 2056, 0.0), (torch.float32, 5, 4096, 0.0)])
def test_against_fp64(act, dtype, rows, channels, shift):
    g = torch.Generator("cuda").manual_seed(rows)
    x = (shift + torch.randn(rows, channels, generator=g, device="cuda") * (0.5 + torch.rand(channels, generator=g, device="cuda"))).to(dtype)
    dy = torch.randn(rows, channels, generator=g, device="cuda").to(dtype)
    net = _net(channels, act)
    wide = copy.deepcopy(net).double()
    f = x.clone().requires_grad_()
    y = net(_tensor(f)).features
    assert y.grad_fn.name() == "SparseBatchNormActBackward" and y.dtype == dtype
    y.backward(dy)
    d = x.double().requires_grad_()
    z = _apart(wide, _tensor(d))
    z.backward(dy.double())
    # one rounding of the result; fp32 arithmetic of about ten operations, the mean's error seen through 1 / std (2.5 at most)
    unit, small = EPS[dtype], 2.0 ** -24 * (16 + 4 * shift)
    scale = z.abs().max().item() + 1
    assert (y.double() - z).abs().max().item() <= (unit + small) * scale
    if rows > 2:  # (two rows: the gradient cancels to nothing, eps times the incoming one)
        assert (f.grad.double() - d.grad).norm() <= (2 * unit + 8 * small) * d.grad.norm() + 1e-12
    for a, b in zip(net.parameters(), wide.parameters()):
        assert (a.grad.double() - b.grad).abs().max().item() <= 8 * small * rows ** 0.5 * (1 + b.grad.abs().max().item())
    bn, ref = net[0], wide[0]
    assert torch.allclose(bn.running_mean.double(), ref.running_mean, rtol=1e-6, atol=1e-6)
    assert torch.allclose(bn.running_var.double(), ref.running_var, rtol=2e-6, atol=1e-6)
    assert int(bn.num_batches_tracked) == 1 and bn.num_batches_tracked._version == 1


def test_no_worse_than_the_modules():
    """Error against fp64 where the mean is large against the spread."""
    x = (100 + torch.randn(50000, 32, generator=torch.Generator("cuda").manual_seed(1), device="cuda"))
    net = _net(32, "none")
    exact = _apart(copy.deepcopy(net).double(), _tensor(x.double()))
    own = net(_tensor(x)).features.double() - exact
    apart = _apart(copy.deepcopy(net), _tensor(x)).double() - exact
    assert own.norm() <= 1.05 * apart.norm()


@pytest.mark.parametrize("act", list(ACTS))
@pytest.mark.parametrize("dtype,rows,channels", [(torch.float16, 4099, 32), (torch.float16, 60000, 64), (torch.bfloat16, 4099, 32),
                                                 (torch.bfloat16, 60000, 64), (torch.float32, 4099, 32), (torch.float32, 60000, 64)])
def test_no_output_is_further_from_fp64_than_the_modules(act, dtype, rows, channels):
    """Result, input gradient and both parameters' gradients, in every type and with every activation."""
    g = torch.Generator("cuda").manual_seed(rows + channels)
    x = (0.5 + torch.randn(rows, channels, generator=g, device="cuda") * (0.5 + torch.rand(channels, generator=g, device="cuda"))).to(dtype)
    dy = torch.randn(rows, channels, generator=g, device="cuda").to(dtype)
    net = _net(channels, act)

    def outputs(run, net, x, dy):
        f = x.clone().requires_grad_()
        y = run(net, f)
        y.backward(dy)
        return [t.double() for t in (y.detach(), f.grad, net[0].weight.grad, net[0].bias.grad)]

    exact = outputs(lambda n, f: _apart(n, _tensor(f)), copy.deepcopy(net).double(), x.double(), dy.double())
    own = outputs(lambda n, f: n(_tensor(f)).features, copy.deepcopy(net), x, dy)
    apart = outputs(lambda n, f: _apart(n, _tensor(f)), copy.deepcopy(net), x, dy)
    for what, a, b, e in zip(("y", "dx", "dweight", "dbias"), own, apart, exact):
        # (both sides round y and dx once to the features' type at least: equal but for the values' luck.  The parameters'
        # gradients are fp32 sums; without an activation those of dy alone, of which both sides see all but the last bits)
        slack = 2.0 ** -24 * 4 * e.norm() if what.startswith("d") else 0.0
        assert (a - e).norm() <= 1.05 * (b - e).norm() + slack, what


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
def test_silu_far_from_zero(dtype):
    """Each value, and the parameters' gradients of rows whose activation is all but flat, where exp(-z) is large."""
    lim = 15.0 if dtype == torch.float16 else 88.0  # below, results of that type are none
    n = 4096
    x = torch.linspace(-1, 1, n, device="cuda", dtype=torch.float64)[torch.randperm(n, generator=torch.Generator().manual_seed(1)).cuda()]
    x = x[:, None].expand(n, 8).contiguous().to(dtype)
    net = _net(8, "silu")
    net[0].weight.data.fill_(lim / 3 ** 0.5)  # (a uniform variable's largest value is 3 ** 0.5 deviations)
    net[0].bias.data.zero_()
    f = x.clone().requires_grad_()
    y = net(_tensor(f)).features
    d = x.double().requires_grad_()
    wide = copy.deepcopy(net).double()
    z = wide[0](d)
    e = nn.functional.silu(z)
    low = (z < -0.8 * lim).float()
    y.backward(low.to(dtype))
    e.backward(low.double())
    # one rounding of the result, a few of exp and the division; z is off by a few roundings of itself and by the mean's error
    # (2^-24 of values up to 1, twice) times the gain, and the activation's slope takes that on
    s, dz = torch.sigmoid(z), 2.0 ** -24 * (8 * z.abs() + 2 * lim)
    bound = (EPS[dtype] + 2.0 ** -24 * 8) * e.abs() + dz * (s * (1 + z * (1 - s))).abs() + dz ** 2 * s
    tiny = 2.0 ** -24 if dtype == torch.float16 else torch.finfo(dtype).tiny
    assert ((y.double() - e).abs() <= bound + tiny).all()
    for a, b in zip(net.parameters(), wide.parameters()):
        assert (a.grad.double() - b.grad).abs().max() <= 2.0 ** -24 * 16 * (1 + lim) * b.grad.abs().max()  # (s is off by dz of itself)


def test_without_affine_and_non_finite():
    net = _net(16, "relu", affine=False)
    x = torch.randn(100, 16, device="cuda")
    x[3, 5] = float("nan")
    x[4, 6] = float("inf")
    a, b = net(_tensor(x)).features, _apart(copy.deepcopy(net), _tensor(x))
    assert torch.equal(torch.isnan(a), torch.isnan(b)) and torch.allclose(a.nan_to_num(), b.nan_to_num(), atol=1e-6)


def test_gradients_of_gradients():
    def penalty(run, net, f):
        y = run(net, f)
        g, gw = torch.autograd.grad(y.square().sum(), [f, net[0].weight], create_graph=True)
        (g.square().sum() + gw.square().sum()).backward()
        return f.grad, net[0].weight.grad, net[0].bias.grad

    x = torch.randn(64, 8, device="cuda")
    own, ref = _net(8, "silu"), _net(8, "silu")
    a = penalty(lambda n, f: n(_tensor(f)).features, own, x.clone().requires_grad_())
    b = penalty(lambda n, f: _apart(n, _tensor(f)), ref, x.clone().requires_grad_())
    for p, q in zip(a, b):
        assert torch.allclose(p, q, rtol=1e-4, atol=1e-4 * q.abs().max().item())


def test_what_stays_with_the_modules():
    x = torch.randn(50, 16, device="cuda")

    def name(net, f=x):
        y = net(_tensor(f.detach().requires_grad_())).features
        return y.grad_fn.name() if y.grad_fn is not None else ""

    own = "SparseBatchNormActBackward"
    assert name(_net(16, "silu")) == own
    seen = []
    hooked = _net(16, "silu")
    hooked[0].register_forward_hook(lambda m, i, o: seen.append(o))
    assert name(hooked) != own and len(seen) == 1
    hooked = _net(16, "silu")
    hooked[1].register_forward_hook(lambda m, i, o: seen.append(o))
    assert name(hooked) != own and len(seen) == 2
    cumulative = _net(16, "relu")
    cumulative[0].momentum = None
    assert name(cumulative) != own
    assert name(_net(16, "relu").eval()) != own
    assert name(_net(18, "relu"), torch.randn(50, 18, device="cuda")) != own          # 72 bytes a row
    assert name(_net(16, "relu"), torch.randn(16, 50, device="cuda").t()) != own      # not contiguous
    assert name(_net(16, "relu"), torch.randn(50 * 16 + 1, device="cuda")[1:].view(50, 16)) != own  # not aligned
    assert name(_net(16, "relu").double(), x.double()) != own
    with pytest.raises(ValueError):
        _net(16, "relu")(_tensor(x[:1]))
    net = _net(16, "silu")
    with torch.autograd.forward_ad.dual_level():
        dual = torch.autograd.forward_ad.make_dual(x, torch.ones_like(x))
        y = net(_tensor(dual)).features
        assert torch.autograd.forward_ad.unpack_dual(y).tangent is not None


def test_saved_tensor_hooks_and_changes_in_place():
    net, x = _net(16, "silu"), torch.randn(50, 16, device="cuda", requires_grad=True)
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(t) or t.cpu(), lambda t: t.cuda()):
        y = net(_tensor(x)).features
    assert packed
    y.sum().backward()
    f = x.detach().clone().requires_grad_() * 1.0
    y = net(_tensor(f)).features
    f.mul_(2)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        y.sum().backward()
    y = net(_tensor(x)).features
    y.sum().backward()
    with pytest.raises(RuntimeError):
        y.sum().backward()


@pytest.mark.parametrize("start", [0, 1])
def test_saved_tensors_come_back_with_other_strides(start):
    """... or from another address; nets of a convolution, a normalisation and each pooling."""

    def other(t):  # the same values, columns first, or starting off a 16-byte boundary
        if not t.is_floating_point():
            return t.clone()
        if start:
            room = torch.empty(t.numel() + start, dtype=t.dtype, device=t.device)
            room[start:].copy_(t.reshape(-1))
            return room[start:].view(t.shape)
        return t.reshape(len(t), -1).t().contiguous().t().reshape(t.shape) if t.dim() == 2 else torch.stack([t, t], -1)[..., 0]

    gen = torch.Generator().manual_seed(2)
    cells = torch.randperm(16 ** 3, generator=gen)[:900]
    idx = torch.stack([torch.zeros_like(cells), cells // 256, cells // 16 % 16, cells % 16], 1).int().cuda()
    f = torch.randn(900, 16, generator=gen).cuda().requires_grad_()
    torch.manual_seed(0)
    for pool in (sp.SparseMaxPool3d, sp.SparseAvgPool3d):
        net = sp.SparseSequential(sp.SubMConv3d(16, 32, 3), nn.BatchNorm1d(32), nn.SiLU(), pool(2, 2)).cuda()

        def grads():
            y = net(sp.SparseConvTensor(f, idx, [16] * 3, 1)).features
            return torch.autograd.grad(y, [f, *net.parameters()], torch.ones_like(y))

        want = grads()
        with torch.autograd.graph.saved_tensors_hooks(other, lambda t: t):
            got = grads()
        assert all(torch.equal(a, b) for a, b in zip(got, want))
