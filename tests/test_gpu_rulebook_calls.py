"""The C ABI of the rulebooks called as its header allows."""

import ctypes

import numpy as np
import pytest
import torch

from gpu_util import DEV, to_np, unique_coords
from oracle import rulebook as orb

pytestmark = pytest.mark.gpu


def _prepared(shape, n, batch, stride, subm):
    from spconv_triton_b200 import _lib

    lib, nd = _lib.load(), len(shape)
    out = list(shape) if subm else [(s + 2 - 3) // stride + 1 for s in shape]
    geo = _lib.make_geometry(batch, list(shape), out, [3] * nd, [stride] * nd, [1] * nd, [1] * nd, subm, False)
    coords = unique_coords(n, n, batch, shape)
    idx = torch.from_numpy(coords).to(DEV)
    ws = torch.empty(int(lib.spc_rulebook_workspace_bytes(ctypes.byref(geo), n)), dtype=torch.uint8, device=DEV)
    n_out = ctypes.c_int64(0)
    st = _lib.current_stream(idx.device)
    _lib.check(lib.spc_rulebook_prepare(ctypes.byref(geo), _lib.ptr(idx), n, _lib.ptr(ws), ws.numel(), ctypes.byref(n_out), st))

    def tables(**want):
        names = ("out_indices", "pair_fwd", "pair_fwd_rowmajor", "order_fwd", "pair_bwd", "pair_bwd_rowmajor", "order_bwd")
        _lib.check(lib.spc_rulebook_tables(ctypes.byref(geo), _lib.ptr(idx), n, n_out.value, _lib.ptr(ws), ws.numel(),
                                           *[_lib.ptr(want.get(k)) for k in names], _lib.current_stream(idx.device)))

    exp = orb.igemm_pairs(coords, batch, list(shape), [3] * nd, [stride] * nd, [1] * nd, [1] * nd, [0] * nd, subm, False, True, False)
    return tables, n, int(n_out.value), exp


@pytest.mark.parametrize("n,subm", [(8191, True), (8193, True), (30000, True), (9000, False), (40000, False)])
def test_a_row_order_asked_for_again(n, subm):
    """... is an order of the rows again, of either side, whether or not the rows fit one piece."""
    tables, n_in, n_out, _ = _prepared((64, 64, 48), n, 2, 2, subm)
    for _ in range(3):
        order = torch.full((n_out,), -1, dtype=torch.int32, device=DEV)
        tables(order_fwd=order, **({} if subm else {"out_indices": torch.empty((n_out, 4), dtype=torch.int32, device=DEV)}))
        assert torch.equal(order.sort().values.cpu(), torch.arange(n_out, dtype=torch.int32))
        if not subm:
            order = torch.full((n_in,), -1, dtype=torch.int32, device=DEV)
            tables(order_bwd=order)
            assert torch.equal(order.sort().values.cpu(), torch.arange(n_in, dtype=torch.int32))


def _node_types(graph):
    """The kinds of nodes of a captured graph."""
    cuda, count = ctypes.CDLL("libcuda.so.1"), ctypes.c_size_t(0)
    handle = ctypes.c_void_p(graph.raw_cuda_graph())
    assert cuda.cuGraphGetNodes(handle, None, ctypes.byref(count)) == 0
    nodes = (ctypes.c_void_p * count.value)()
    assert cuda.cuGraphGetNodes(handle, nodes, ctypes.byref(count)) == 0
    kinds, kind = set(), ctypes.c_int(0)
    for node in nodes:
        assert cuda.cuGraphNodeGetType(ctypes.c_void_p(node), ctypes.byref(kind)) == 0
        kinds.add({0: "kernel", 1: "memcpy", 2: "memset"}.get(kind.value, kind.value))
    return kinds


@pytest.mark.parametrize("start", [0, 1, 2, 3])
@pytest.mark.parametrize("n", [777, 778, 779, 780])
def test_a_table_that_starts_and_ends_anywhere(n, start):
    """The column-major table of a strided layer is a caller's: cleared to its last entry, and nothing beside it,
    by a kernel (no driver memset, which may wait behind the application's transfers)."""
    tables, _, n_out, exp = _prepared((20, 24, 22), n, 1, 2, False)
    room = torch.full((27 * n_out + 8,), 7, dtype=torch.int32, device=DEV)
    table = room[start:start + 27 * n_out]
    out_indices = torch.empty((n_out, 4), dtype=torch.int32, device=DEV)
    tables(pair_fwd=table, out_indices=out_indices)
    np.testing.assert_array_equal(to_np(table).reshape(27, n_out), exp[2])
    assert bool((room[:start] == 7).all()) and bool((room[start + 27 * n_out:] == 7).all())
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        tables(pair_fwd=table, out_indices=out_indices)
    assert _node_types(graph) == {"kernel"}


def test_outputs_numbered_by_hash_after_outputs_numbered_by_bitmap():
    """In a pass of one call, the outputs of a transposed layer on a grid beyond the bitmap's limit are enumerated
    from the coordinates that the strided layer before it writes, not before it has written them."""
    import spconv_triton_b200.pytorch as sp
    from spconv_triton_b200 import constants

    shape, n, batch = [100, 1000, 1000], 20000, 3  # 37 M cells behind the first layer, 296 M behind the second
    net = sp.SparseSequential(sp.SparseConv3d(16, 16, 3, stride=2, padding=1, bias=False),
                              sp.SparseConvTranspose3d(16, 16, 3, stride=2, padding=1, bias=False)).to(DEV).half().eval()
    idx = torch.from_numpy(unique_coords(5, n, batch, shape)).to(DEV)
    x = torch.randn(n, 16, device=DEV).half()
    outs = []
    with torch.no_grad():
        for native in (False, True, True, True):
            old, constants.SPCONV_NATIVE_SEQUENCE = constants.SPCONV_NATIVE_SEQUENCE, native
            try:
                y = net(sp.SparseConvTensor(x, idx, shape, batch))
            finally:
                constants.SPCONV_NATIVE_SEQUENCE = old
            outs.append((y.indices, y.features))
    for indices, features in outs[1:]:
        assert torch.equal(indices, outs[0][0])
        assert torch.equal(features, outs[0][1])
