"""The kernels at the sizes where they can go wrong: edges of tiles and splits, remainders, channel widths
whose rows are no power of two, the smallest and the largest of a range.  Each against the CPU oracle or a
plain PyTorch statement of the same operation in fp32 or fp64."""

import numpy as np
import pytest
import torch

from gpu_util import DEV, rel_err, to_np, unique_coords
from oracle import rulebook as orb

pytestmark = pytest.mark.gpu

TOL = {torch.float32: 1e-5, torch.float16: 2e-3, torch.bfloat16: 8e-3}


def _table(n_in, n_out, kv, density, seed):
    g = torch.Generator().manual_seed(seed)
    t = torch.randint(0, n_in, (kv, n_out), generator=g, dtype=torch.int32)
    t[torch.rand((kv, n_out), generator=g) >= density] = -1
    return t.to(DEV)


def _dense_statement(x, g, w, table):
    """out, and dW, of the gathered products in fp64."""
    x, g, w = x.double(), g.double(), w.double()
    out, dw = torch.zeros((table.shape[1], w.shape[0]), dtype=torch.float64, device=DEV), torch.zeros_like(w)
    for k in range(table.shape[0]):
        m = (table[k] >= 0).nonzero()[:, 0]
        rows = x[table[k][m].long()]
        out[m] += rows @ w[:, k].t()
        dw[:, k] = g[m].t() @ rows
    return out, dw


# rows at tile (128) and split (2048 / 4096) edges; channels with 32-, 64- and 128-byte pieces; one and two blocks
# of 128 outputs; narrow (four copy warps) and wide (eight); fp32 with full, ragged and single output groups
SHAPES = [
    (torch.float16, 1, 16, 16, 27), (torch.float16, 129, 48, 96, 27), (torch.float16, 4097, 96, 48, 8),
    (torch.bfloat16, 4096, 96, 192, 3), (torch.float16, 2049, 32, 64, 1), (torch.float16, 300, 128, 256, 27),
    (torch.bfloat16, 130, 256, 512, 2), (torch.float16, 127, 112, 80, 125),
    (torch.float32, 1, 3, 5, 27), (torch.float32, 129, 16, 16, 27), (torch.float32, 1000, 64, 64, 27),
    (torch.float32, 513, 33, 17, 8), (torch.float32, 255, 100, 130, 3),
]


@pytest.mark.parametrize("dtype,n,c_in,c_out,kv", SHAPES)
def test_gather_gemm_and_weight_gradient(dtype, n, c_in, c_out, kv):
    from spconv_triton_b200.pytorch._impl import gemm as G

    n_in = n + 7
    table = _table(n_in, n, kv, 0.4, seed=n + kv)
    gen = torch.Generator().manual_seed(1)
    mk = lambda *s: torch.randn(s, generator=gen).to(DEV).to(dtype)  # noqa: E731
    x, g, w = mk(n_in, c_in), mk(n, c_out), mk(c_out, kv, c_in)
    out, dw = _dense_statement(x, g, w, table)
    assert rel_err(to_np(G.conv_forward(x, w, table, n).double()), to_np(out)) <= TOL[dtype]
    assert rel_err(to_np(G.conv_backward_weight(x, g, table, tuple(w.shape)).double()), to_np(dw)) <= TOL[dtype]
    din = G.conv_backward_input(g, w, _invert(table, n_in), n_in)
    exp = torch.zeros((n_in, c_in), dtype=torch.float64, device=DEV)
    inv = _invert(table, n_in)
    for k in range(kv):
        m = (inv[k] >= 0).nonzero()[:, 0]
        exp[m] += g.double()[inv[k][m].long()] @ w.double()[:, k]
    assert rel_err(to_np(din.double()), to_np(exp)) <= TOL[dtype]
    G.check_device_status()


def _invert(table, n_in):
    """A table over the inputs: one of the outputs that read each input with offset k, or -1."""
    kv, n = table.shape
    inv = torch.full((kv, n_in), -1, dtype=torch.int32)
    t = table.cpu()
    for k in range(kv):
        m = (t[k] >= 0).nonzero()[:, 0]
        inv[k][t[k][m].long()] = m.int()
    return inv.to(DEV)


# (shape, rows, batch, kernel, stride, subm, transposed): cells and rows at the edges of 256-thread blocks, of the
# 8192-row pieces of the tile order, of the windows of a bitmap line, of the slabs of a 125-offset and a
# four-dimensional kernel; a grid too large for a bitmap
BOOKS = [
    ((64, 64, 64), 1, 1, 3, 1, True, False), ((64, 64, 64), 8191, 2, 3, 1, True, False),
    ((40, 33, 65), 8193, 1, 3, 1, True, False), ((128, 128, 32), 16385, 2, 5, 1, True, False),
    ((9, 9, 9, 10), 2000, 1, 3, 1, True, False), ((512, 512), 5000, 3, 3, 1, True, False),
    ((64, 64, 64), 257, 1, 3, 2, False, False), ((41, 50, 63), 8193, 2, 3, 2, False, False),
    ((40, 40, 40), 6000, 1, 2, 2, False, False), ((30, 30, 30), 1500, 2, 3, 1, False, False),
    ((20, 20, 21), 700, 1, 3, 2, False, True), ((1500, 1500, 1500), 3000, 1, 3, 2, False, False),
    ((1500, 1500, 1500), 3000, 1, 3, 1, True, False),
]


@pytest.mark.parametrize("shape,n,batch,k,stride,subm,transposed", BOOKS)
@pytest.mark.parametrize("ordered", [False, True])
def test_layer_rulebook_tables(shape, n, batch, k, stride, subm, transposed, ordered):
    """Tables and coordinates of both sides equal the oracle's, bit for bit."""
    from spconv_triton_b200.pytorch._impl import host

    nd = len(shape)
    idx = unique_coords(n, n, batch, shape)
    if ordered:
        idx = idx[np.lexsort(idx.T[::-1])]
    one, pad = (1,) * nd, ((k // 2,) * nd if k % 2 else (0,) * nd)
    geo, _ = host.geometry(batch, shape, (k,) * nd, (stride,) * nd, pad, one, (0,) * nd, subm, transposed)
    rb = host.ext().build_rulebook(geo, torch.from_numpy(idx).to(DEV), True, True, True)
    exp = orb.igemm_pairs(idx, batch, list(shape), [k] * nd, [stride] * nd, list(pad), [1] * nd, [0] * nd, subm, transposed,
                          True, False)
    np.testing.assert_array_equal(to_np(rb.out_indices), exp[0])
    np.testing.assert_array_equal(to_np(rb.colmajor(False)), exp[2])
    np.testing.assert_array_equal(to_np(rb.rowmajor(False))[:, :geo.kv].T, exp[2])
    if not subm:  # the input side of a submanifold layer is its forward table, offsets reversed
        np.testing.assert_array_equal(to_np(rb.colmajor(True)), exp[3])
        np.testing.assert_array_equal(to_np(rb.rowmajor(True))[:, :geo.kv].T, exp[3])


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("kind,n,k", [("subm", 8193, 3), ("subm", 500, 5), ("down", 4097, 3), ("up", 129, 3)])
def test_trained_layer(kind, n, k, dtype):
    """Output, input, weight and bias gradient of a layer through its autograd node, against fp64 sums over the
    oracle's tables: a row that the tile order lost or doubled would be wrong in one of them."""
    import spconv_triton_b200.pytorch as sp

    shape, ci, co = (48, 48, 48), 32, 48
    idx = unique_coords(n, n, 1, shape)
    cls = {"subm": sp.SubMConv3d, "down": sp.SparseConv3d, "up": sp.SparseConvTranspose3d}[kind]
    stride = 1 if kind == "subm" else 2
    torch.manual_seed(2)
    layer = cls(ci, co, k, stride=stride, padding=k // 2, bias=True).to(DEV).to(dtype)
    x = torch.randn(n, ci).to(DEV).to(dtype).requires_grad_()
    y = layer(sp.SparseConvTensor(x, torch.from_numpy(idx).to(DEV), list(shape), 1)).features
    g = torch.randn(y.shape).to(DEV).to(dtype)
    y.backward(g)
    table = torch.from_numpy(orb.igemm_pairs(idx, 1, list(shape), [k] * 3, [stride] * 3, [k // 2] * 3, [1] * 3, [0] * 3,
                                             kind == "subm", kind == "up", True, False)[2]).to(DEV)
    w = layer.weight.detach().reshape(co, -1, ci)
    out, dw = _dense_statement(x.detach(), g, w, table)
    din = torch.zeros((n, ci), dtype=torch.float64, device=DEV)
    for q in range(table.shape[0]):
        m = (table[q] >= 0).nonzero()[:, 0]
        din.index_add_(0, table[q][m].long(), g[m].double() @ w[:, q].double())
    for got, want in ((y.detach(), out + layer.bias.detach().double()), (x.grad, din), (layer.weight.grad.reshape(w.shape), dw),
                      (layer.bias.grad, g.double().sum(0))):
        assert rel_err(to_np(got.double()), to_np(want)) <= TOL[dtype]


@pytest.mark.parametrize("rows,cols", [(1, 8), (255, 16), (4097, 48), (70000, 128)])
def test_bias_gradient_sums(rows, cols):
    import spconv_triton_b200.pytorch as sp

    idx = unique_coords(rows, rows, 1, (80, 80, 80))
    layer = sp.SubMConv3d(16, cols, 1, bias=True).to(DEV).half()
    y = layer(sp.SparseConvTensor(torch.ones(rows, 16, device=DEV).half(), torch.from_numpy(idx).to(DEV), [80] * 3, 1)).features
    g = torch.randn(rows, cols, device=DEV).half()
    y.backward(g)
    assert rel_err(to_np(layer.bias.grad.double()), to_np(g.double().sum(0))) <= TOL[torch.float16]


@pytest.mark.parametrize("heavy", [255, 256, 257, 3000])
def test_voxels_with_many_points(heavy):
    """Voxels around the number of points up to which a point ranks itself by comparisons."""
    from oracle.voxelize import point_to_voxel
    from spconv_triton_b200.pytorch.utils import PointToVoxel

    g = torch.Generator().manual_seed(heavy)
    pts = torch.rand((5000 + heavy, 4), generator=g) * 50
    at = torch.randperm(len(pts), generator=g)[:heavy]
    pts[at, :3] = torch.rand((heavy, 3), generator=g) * 0.4 + 20.05
    ctor = dict(vsize_xyz=[0.5] * 3, coors_range_xyz=[0.0, 0.0, 0.0, 50.0, 50.0, 50.0], num_point_features=4,
                max_num_voxels=100_000, max_num_points_per_voxel=300)
    out = PointToVoxel(device=torch.device(DEV), **ctor).generate_voxel_with_id(pts.to(DEV))
    for got, want in zip(out, point_to_voxel(pts.numpy(), **ctor)):
        np.testing.assert_array_equal(to_np(got), want)


@pytest.mark.parametrize("n,targets,channels", [(1, 1, 8), (255, 9000, 64), (1025, 8192, 256), (5000, 100_000, 40)])
@pytest.mark.parametrize("average", [False, True])
def test_pool_gradient_in_any_row_order(n, targets, channels, average):
    """The order is a permutation by the first row read, and the average's gradient has the same bits with it and
    without; the maximum's (no order) beside it."""
    from spconv_triton_b200 import _lib

    lib, kv, pitch = _lib.load(), 27, 28
    gen = torch.Generator().manual_seed(n)
    table = torch.randint(0, targets, (n, pitch), generator=gen, dtype=torch.int32)
    table[torch.rand((n, pitch), generator=gen) < 0.6] = -1
    table[:, kv:] = -1
    first = torch.where(table >= 0, table, 0).gather(1, (table >= 0).int().argmax(1, keepdim=True))[:, 0]
    table = table.to(DEV)
    order = torch.empty(n, dtype=torch.int32, device=DEV)
    scratch = torch.empty(lib.spc_pool_row_order_workspace_bytes(n), dtype=torch.uint8, device=DEV)
    st = _lib.current_stream(table.device)
    _lib.check(lib.spc_pool_row_order(_lib.ptr(table), pitch, kv, n, targets, _lib.ptr(order), _lib.ptr(scratch),
                                      scratch.numel(), st))
    assert torch.equal(order.sort().values.cpu(), torch.arange(n, dtype=torch.int32))
    bucket = -(-targets // 8192)
    assert bool((first[order.cpu().long()].diff() > -2 * bucket).all())
    mk = lambda r: torch.randn((r, channels), generator=gen).to(DEV).half()  # noqa: E731
    grad, own, ref = mk(targets), mk(n), mk(targets)
    ref[::2] = own[torch.arange(0, targets, 2) % n]
    count = torch.randint(1, 28, (targets,), generator=gen, dtype=torch.int32).to(DEV)
    got = []
    for rows in (None, order) if average else (None,):
        dst = torch.full((n, channels), 7.0, device=DEV).half()
        _lib.check(lib.spc_pool(2 if average else 3, _lib.ptr(grad), _lib.ptr(own), _lib.ptr(ref), _lib.ptr(table), pitch,
                                _lib.ptr(rows), _lib.ptr(count), _lib.ptr(dst), None, n, channels, kv,
                                _lib.dtype_code(torch.float16), st))
        got.append(dst)
    assert torch.equal(got[0], got[-1])
    t = table[:, :kv].long()
    there, t = (t >= 0)[:, :, None], t.clamp(min=0)
    g = grad.double()[t] * (count.double()[t][:, :, None] if average else (ref[t] == own[:, None]).double())
    assert rel_err(to_np(got[0].double()), to_np((g * there).sum(1))) <= TOL[torch.float16]


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("channels", [32, 128, 40])
def test_average_of_16_bit_rows_is_the_rounded_fp32_average(dtype, channels):
    """Sums and quotients of 16-bit rows have the bits of fp32 sums divided by the count, infinities, NaNs, zeros of
    either sign and the smallest values among them."""
    import spconv_triton_b200.pytorch as sp

    idx = torch.from_numpy(unique_coords(5, 3000, 1, (24, 24, 24))).to(DEV)
    x = torch.randn(3000, channels, device=DEV).to(dtype)
    for at, value in enumerate((float("inf"), -float("inf"), float("nan"), -0.0, 6e-8, 65504.0)):
        x[at::97, at % channels] = value
    pool = sp.SparseAvgPool3d(3, 1, padding=1)
    got = pool(sp.SparseConvTensor(x, idx, [24] * 3, 1)).features
    exp = pool(sp.SparseConvTensor(x.float(), idx, [24] * 3, 1)).features.to(dtype)
    assert torch.equal(got.isnan(), exp.isnan())
    assert torch.equal(got.nan_to_num(7.0), exp.nan_to_num(7.0))
    assert torch.equal(torch.signbit(got)[~got.isnan()], torch.signbit(exp)[~exp.isnan()])


_FIRST_CALLS = """
import ctypes, sys, threading
ctypes.CDLL(sys.argv[2]).cudaFree(None)  # the context, so that the threads meet in the call itself
lib, gate, got = ctypes.CDLL(sys.argv[1]), threading.Barrier(16), []
def first():
    gate.wait()
    got.append(lib.spc_conv_forward_needs_colmajor(64, 64, 27, 0, 0, 0, 0))
threads = [threading.Thread(target=first) for _ in range(16)]
for t in threads: t.start()
for t in threads: t.join()
sys.exit(any(got))
"""


def test_first_calls_of_many_threads():
    """All of them find the tensor cores, also the ones that come while another looks the driver's function up (new processes:
    it happens once in each, and not in each)."""
    import subprocess
    import sys

    from spconv_triton_b200.csrc.build import LIB

    with open("/proc/self/maps") as f:
        runtime = next(line.split()[-1] for line in f if "libcudart.so" in line)
    for _ in range(6):
        subprocess.run([sys.executable, "-c", _FIRST_CALLS, str(LIB), runtime], check=True, timeout=60)


@pytest.mark.parametrize("kv,c_in,c_out,n_out", [(66000, 12, 4, 3), (27, 132, 68, 2100)])
def test_fp32_weight_gradient_of_many_offsets_and_blocks(kv, c_in, c_out, n_out):
    """More offsets than a launch takes, several channel blocks with ragged edges, two splits."""
    import ctypes

    from spconv_triton_b200 import _lib

    lib = _lib.load()
    gen = torch.Generator(DEV).manual_seed(kv)
    n_in = 50
    x, g = torch.randn(n_in, c_in, generator=gen, device=DEV), torch.randn(n_out, c_out, generator=gen, device=DEV)
    table = torch.randint(-1, n_in, (kv, n_out), generator=gen, device=DEV).int()
    dw = torch.full((c_out, kv, c_in), float("nan"), device=DEV)
    ws = torch.empty(lib.spc_conv_backward_weight_workspace_bytes(n_out, c_in, c_out, kv), dtype=torch.uint8, device=DEV)
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    assert lib.spc_conv_backward_weight(p(x), p(g), p(table), p(dw), p(ws), ws.numel(), n_in, n_out, c_in, c_out, kv, _lib.SPC_F32,
                                        _lib.SPC_PREC_IEEE, 0, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    wide = torch.cat([x.double(), x.new_zeros(1, c_in).double()])
    for k in range(0, kv, 1000):  # (index -1: the row of zeros)
        f = wide[table[k:k + 1000].long()]
        want, size = torch.einsum("mn,kmc->nkc", g.double(), f), torch.einsum("mn,kmc->nkc", g.double().abs(), f.abs())
        assert ((dw[:, k:k + 1000].double() - want).abs() <= 2.0 ** -24 * (n_out + 4) * (size + 1e-30)).all()
