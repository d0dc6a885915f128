"""The fp32 gather-GEMM for few rows (csrc/gemm_f32.cu) against fp64, and the layers that run on it."""

import ctypes

import pytest
import torch

import spconv_triton_b200.pytorch as sp
from spconv_triton_b200 import _lib, constants

pytestmark = pytest.mark.gpu


def _p(t):
    return ctypes.c_void_p(0 if t is None else t.data_ptr())


@pytest.mark.parametrize("rows,n,r,kv", [(1, 16, 12, 27), (7, 64, 64, 1), (8, 48, 16, 8), (9, 32, 20, 32), (2000, 16, 16, 27),
                                         (512, 64, 64, 27), (8191, 16, 16, 3)])
def test_against_fp64(rows, n, r, kv):
    lib = _lib.load()
    assert lib.spc_conv_small(rows, n, r, kv) == 1
    gen = torch.Generator("cuda").manual_seed(rows)
    n_in = rows + 5
    x, w = torch.randn(n_in, r, generator=gen, device="cuda"), torch.randn(n, kv, r, generator=gen, device="cuda")
    bias, residual = torch.randn(n, generator=gen, device="cuda"), torch.randn(rows, n, generator=gen, device="cuda")
    table = torch.randint(0, n_in, (rows, kv), generator=gen, device="cuda").int()
    table[torch.rand(rows, kv, generator=gen, device="cuda") < 0.7] = -1
    rm = torch.full((rows, (kv + 3) // 4 * 4), -1, dtype=torch.int32, device="cuda")
    rm[:, :kv] = table
    f = torch.cat([x.double(), x.new_zeros(1, r).double()])[table.long()]  # [rows, kv, r], absent rows zero (index -1)
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    # one fp32 rounding a product and sum, kv * r of them at most
    bound = 2.0 ** -24 * (kv * r + 4)

    def near(got, want, size):
        assert ((got.double() - want).abs() <= bound * (size + 1)).all()

    out = torch.full((rows, n), float("nan"), device="cuda")
    assert lib.spc_conv_forward_residual(_p(x), _p(w), _p(bias), None, _p(rm), None, _p(out), n_in, rows, r, n, kv, _lib.SPC_F32, _lib.SPC_F32,
                                         _lib.SPC_PREC_IEEE, 0, None, None, 1, 0.0, _p(residual), stream) == 0
    want = torch.einsum("akr,nkr->an", f, w.double())
    near(out, torch.relu(want + bias) + residual, torch.einsum("akr,nkr->an", f.abs(), w.double().abs()) + bias.abs() + residual.abs())
    back = w.permute(2, 1, 0).contiguous()  # [r, kv, n] of a layer n -> r
    for reverse in (0, 1):
        din = torch.full((rows, n), float("nan"), device="cuda")
        assert lib.spc_conv_backward_input_tables(_p(x), _p(back), None, _p(rm), None, _p(din), rows, n_in, n, r, kv, reverse, _lib.SPC_F32,
                                                  _lib.SPC_PREC_IEEE, 0, stream) == 0
        m = back.flip(1) if reverse else back
        near(din, torch.einsum("akr,rkn->an", f, m.double()), torch.einsum("akr,rkn->an", f.abs(), m.double().abs()))


@pytest.mark.parametrize("tf32", [False, True])
def test_layers_that_share_the_rulebook(tf32, monkeypatch):
    """A small layer builds it without a row order; a wide one and a 16-bit one use it after."""
    monkeypatch.setattr(constants, "SPCONV_ALLOW_TF32", tf32)
    gen = torch.Generator().manual_seed(3)
    cells = torch.randperm(24 ** 3, generator=gen)[:1500]
    idx = torch.stack([torch.zeros_like(cells), cells // 576, cells // 24 % 24, cells % 24], 1).int().cuda()
    x = torch.randn(1500, 16, generator=gen).cuda()
    small, wide = sp.SubMConv3d(16, 16, 3, indice_key="a").cuda(), sp.SubMConv3d(16, 128, 3, indice_key="a").cuda()
    t = small(sp.SparseConvTensor(x, idx, [24] * 3, 1))
    dense = torch.zeros(1, 16, 24, 24, 24, dtype=torch.float64, device="cuda")
    at = idx.long()
    for layer, bound in ((small, 2e-3 if tf32 else 1e-5), (wide, 2e-3 if tf32 else 1e-5)):
        y = layer(t.replace_feature(x)).features.double()
        dense[0, :, at[:, 1], at[:, 2], at[:, 3]] = x.double().t()
        z = torch.nn.functional.conv3d(dense, layer.weight.double().permute(0, 4, 1, 2, 3), layer.bias.double(), padding=1)
        z = z[0, :, at[:, 1], at[:, 2], at[:, 3]].t()
        assert (y - z).norm() <= bound * z.norm()
    with torch.autocast("cuda", dtype=torch.float16):
        half = small(t.replace_feature(x)).features
    assert half.dtype == torch.float16


@pytest.mark.parametrize("rows", [257, 1024, 1025, 4096])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_a_wide_layer_gets_its_row_order(rows, dtype):
    """... also on the rulebook of a small one, and the same: its results have the bits of a rulebook of its own."""
    gen = torch.Generator().manual_seed(rows)
    cells = torch.randperm(32 ** 3, generator=gen)[:rows]
    idx = torch.stack([torch.zeros_like(cells), cells // 1024, cells // 32 % 32, cells % 32], 1).int().cuda()
    x = sp.SparseConvTensor(torch.randn(rows, 16, generator=gen).cuda(), idx, [32] * 3, 1)
    small, wide = sp.SubMConv3d(16, 16, 3, indice_key="a").cuda(), sp.SubMConv3d(128, 128, 3, indice_key="a").cuda().to(dtype)
    f = torch.randn(rows, 128, generator=gen).cuda().to(dtype)
    lib, launches = _lib.load(), []
    own = wide(x.replace_feature(f)).features
    shared = small(x)
    for _ in range(2):
        before = lib.spc_launch_count()
        assert torch.equal(wide(shared.replace_feature(f)).features, own)
        launches.append(lib.spc_launch_count() - before)
    assert launches[0] == launches[1] + 2  # (keys and sort, once)


def test_row_order_of_a_table():
    """Made later it is the order that the tables come with; more rows than one CTA sorts are refused."""
    from spconv_triton_b200.pytorch._impl import host

    geo = host.geometry(1, (24,) * 3, (3,) * 3, (1,) * 3, (1,) * 3, (1,) * 3, (0,) * 3, True, False)[0]
    cells = torch.randperm(24 ** 3, generator=torch.Generator().manual_seed(0))[:8193]
    idx = torch.stack([torch.zeros_like(cells), cells // 576, cells // 24 % 24, cells % 24], 1).int().cuda()
    lib, stream = _lib.load(), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    g = _lib.make_geometry(1, [24] * 3, [24] * 3, [3] * 3, [1] * 3, [1] * 3, [1] * 3, True, False)
    for n in (1, 31, 2048, 8192, 8193):
        at = idx[:n].contiguous()
        rm = host.ext().build_rulebook(geo, at, False, False, False).rowmajor(False)
        order, keys = torch.full((n,), -1, dtype=torch.int32, device="cuda"), torch.empty(n, dtype=torch.int32, device="cuda")
        rc = lib.spc_rowmajor_order(ctypes.byref(g), _p(rm), n, _p(order), _p(keys), stream)
        if n > 8192:
            assert rc == _lib.SPC_ERR_UNSUPPORTED
            continue
        assert rc == 0
        ws = torch.empty(lib.spc_rulebook_workspace_bytes(ctypes.byref(g), n), dtype=torch.uint8, device="cuda")
        n_out, want, table = ctypes.c_int64(), torch.empty_like(order), torch.empty_like(rm)
        assert lib.spc_rulebook_prepare(ctypes.byref(g), _p(at), n, _p(ws), ws.numel(), ctypes.byref(n_out), stream) == 0
        assert lib.spc_rulebook_tables(ctypes.byref(g), _p(at), n, n, _p(ws), ws.numel(), None, None, _p(table), _p(want), None, None, None,
                                       stream) == 0
        assert torch.equal(order, want) and torch.equal(table, rm)


def test_a_row_order_asked_for_under_capture():
    """It belongs to the graph; a layer outside makes the rulebook's own."""
    gen = torch.Generator().manual_seed(5)
    cells = torch.randperm(32 ** 3, generator=gen)[:2000]
    idx = torch.stack([torch.zeros_like(cells), cells // 1024, cells // 32 % 32, cells % 32], 1).int().cuda()
    x = sp.SparseConvTensor(torch.randn(2000, 16, generator=gen).cuda(), idx, [32] * 3, 1)
    small, wide = sp.SubMConv3d(16, 16, 3, indice_key="a").cuda(), sp.SubMConv3d(128, 128, 3, indice_key="a").cuda().half()
    f = torch.randn(2000, 128, generator=gen).cuda().half()
    with torch.no_grad():
        own, shared = wide(x.replace_feature(f)).features, small(x).replace_feature(f)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            inside = wide(shared).features
        inside.zero_()
        graph.replay()
        assert torch.equal(inside, own) and torch.equal(wide(shared).features, own)
        inside.zero_()
        graph.replay()
        assert torch.equal(inside, own)
