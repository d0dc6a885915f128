"""Tables that are made when somebody asks for them: on any stream and thread, and under capture."""

import threading

import numpy as np
import pytest
import torch

from gpu_util import DEV, to_np, unique_coords
from oracle import rulebook as orb

pytestmark = pytest.mark.gpu

SHAPE, N = (40, 40, 40), 9000


def _book(colmajor=False):
    """A strided rulebook without its input side, and the oracle's tables of both sides."""
    from spconv_triton_b200.pytorch._impl import host

    idx = unique_coords(11, N, 2, SHAPE)
    geo, _ = host.geometry(2, SHAPE, (3,) * 3, (2,) * 3, (1,) * 3, (1,) * 3, (0,) * 3, False, False)
    rb = host.ext().build_rulebook(geo, torch.from_numpy(idx).to(DEV), False, colmajor, True)
    exp = orb.igemm_pairs(idx, 2, list(SHAPE), [3] * 3, [2] * 3, [1] * 3, [1] * 3, [0] * 3, False, False, True, False)
    return rb, exp[2], exp[3]


def test_a_table_made_on_one_stream_is_read_on_another():
    """Behind 50 ms of other work on the stream that makes it, the table is not there yet when the second stream asks."""
    rb, fwd, bwd = _book()
    torch.cuda.synchronize()
    first, second = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(first):
        torch.cuda._sleep(100_000_000)
        rb.colmajor(False)
        rb.rowmajor(True)
    with torch.cuda.stream(second):
        got = [rb.colmajor(False).clone(), rb.rowmajor(True).clone(), rb.colmajor(True).clone()]
    second.synchronize()
    np.testing.assert_array_equal(to_np(got[0]), fwd)
    np.testing.assert_array_equal(to_np(got[1])[:, :27].T, bwd)
    np.testing.assert_array_equal(to_np(got[2]), bwd)


def test_threads_ask_for_the_same_tables():
    bad = []
    for _ in range(8):
        rb, fwd, bwd = _book()
        torch.cuda.synchronize()
        gate = threading.Barrier(4)

        def work(colmajor_first):
            with torch.cuda.stream(torch.cuda.Stream()):
                gate.wait()
                for input_side, want in ((True, bwd), (False, fwd)):
                    cm = rb.colmajor(input_side) if colmajor_first else None
                    rm = rb.rowmajor(input_side).clone()
                    cm = (rb.colmajor(input_side) if cm is None else cm).clone()
                    torch.cuda.current_stream().synchronize()
                    if not (np.array_equal(to_np(cm), want) and np.array_equal(to_np(rm)[:, :27].T, want)):
                        bad.append(input_side)

        threads = [threading.Thread(target=work, args=(i % 2 == 0,)) for i in range(4)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    assert not bad


def test_tables_asked_for_under_capture():
    """A capture records the making of a table but does not run it: later calls make their own."""
    rb, fwd, bwd = _book()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        inside = [rb.colmajor(False), rb.colmajor(True)]
    np.testing.assert_array_equal(to_np(rb.colmajor(True)), bwd)
    np.testing.assert_array_equal(to_np(rb.colmajor(False)), fwd)
    graph.replay()
    torch.cuda.synchronize()
    np.testing.assert_array_equal(to_np(inside[0]), fwd)
    np.testing.assert_array_equal(to_np(inside[1]), bwd)


def test_a_graph_keeps_what_it_makes_tables_from():
    """... also when a later call has made them for good and other tensors have come and gone."""
    rb, _, bwd = _book()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        inside = rb.colmajor(True)
    assert rb.captured
    np.testing.assert_array_equal(to_np(rb.colmajor(True)), bwd)
    others = [torch.full((size,), 0x55, dtype=torch.uint8, device=DEV) for size in (1 << 16, 1 << 18, 1 << 20, 1 << 22) for _ in range(16)]
    torch.cuda.synchronize()
    for _ in range(2):
        inside.fill_(-7)
        graph.replay()
        np.testing.assert_array_equal(to_np(inside), bwd)
    assert all(bool((t == 0x55).all()) for t in others)


def test_a_graph_keeps_what_a_pending_side_is_made_from():
    """The same for the input side that an inference pass of the operator functions leaves pending."""
    import spconv_triton_b200.pytorch as sp
    from spconv_triton_b200.pytorch import ops
    from spconv_triton_b200.pytorch._impl import pairs

    idx = torch.from_numpy(unique_coords(11, N, 2, SHAPE)).to(DEV)
    layer = sp.SparseConv3d(16, 16, 3, stride=2, padding=1, indice_key="d").to(DEV).half().eval()
    with torch.no_grad(), pairs.deferred_backward("late"):
        res = ops.get_indice_pairs_implicit_gemm(idx, 2, list(SHAPE), layer.algo, layer.kernel_size, layer.stride, layer.padding,
                                                 layer.dilation, [0] * 3)
    late = res[2]._spc_late
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        inside = late.get()[0]
    want = late.get()[0].clone()
    assert late.p is not None
    others = [torch.full((size,), 0x55, dtype=torch.uint8, device=DEV) for size in (1 << 16, 1 << 18, 1 << 20, 1 << 22) for _ in range(16)]
    torch.cuda.synchronize()
    inside.fill_(-7)
    graph.replay()
    assert torch.equal(inside, want)
    assert all(bool((t == 0x55).all()) for t in others)


def test_scratch_goes_with_its_use():
    """The scratch of a rulebook goes once both sides are there."""
    rb, _, _ = _book()
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    rb.rowmajor(True)
    made = rb.n_in * 28 * 4 + rb.n_in * 4
    torch.cuda.synchronize()
    assert torch.cuda.memory_allocated() <= before + made - 100_000  # (the scratch is larger than that)


def test_an_entry_read_on_two_streams():
    import spconv_triton_b200.pytorch as sp

    idx = unique_coords(11, N, 2, SHAPE)
    layer = sp.SparseConv3d(16, 16, 3, stride=2, padding=1, indice_key="d").to(DEV).half().eval()
    with torch.no_grad():
        y = layer(sp.SparseConvTensor(torch.randn(N, 16, device=DEV).half(), torch.from_numpy(idx).to(DEV), list(SHAPE), 2))
    entry = y.indice_dict["d"]
    torch.cuda.synchronize()
    first, second = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(first):
        torch.cuda._sleep(100_000_000)
        entry.pair_fwd, entry.pair_bwd, entry.mask_argsort_fwd_splits
    with torch.cuda.stream(second):
        got = [entry.pair_fwd.clone(), entry.pair_bwd.clone(), entry.mask_argsort_fwd_splits[0].clone()]
    second.synchronize()
    exp = orb.igemm_pairs(idx, 2, list(SHAPE), [3] * 3, [2] * 3, [1] * 3, [1] * 3, [0] * 3, False, False, True, False)
    for g, e in zip(got, (exp[2], exp[3], exp[6][0])):
        np.testing.assert_array_equal(to_np(g), e)


def test_tables_of_the_operator_functions_under_capture():
    """What the operator functions remember on a pair list or a table is not what a capture has recorded."""
    import spconv_triton_b200.pytorch as sp
    from spconv_triton_b200.core import ConvAlgo
    from spconv_triton_b200.pytorch import ops
    from spconv_triton_b200.pytorch._impl import pairs

    idx = torch.from_numpy(unique_coords(11, N, 2, SHAPE)).to(DEV)
    _, lists, num = ops.get_indice_pairs(idx, 2, list(SHAPE), ConvAlgo.Native, [3] * 3, [1] * 3, [1] * 3, [1] * 3, [0] * 3, True)
    layer = sp.SparseConv3d(16, 16, 3, stride=2, padding=1, indice_key="d").to(DEV).half().eval()
    with torch.no_grad(), pairs.deferred_backward("late"):
        res = ops.get_indice_pairs_implicit_gemm(idx, 2, list(SHAPE), layer.algo, layer.kernel_size, layer.stride, layer.padding,
                                                 layer.dilation, [0] * 3)
    late = res[2]._spc_late
    plain = res[2].clone()
    torch.cuda.synchronize()
    with torch.cuda.graph(torch.cuda.CUDAGraph()):
        pairs.native_pair_to_tables(lists, num, N, N, False)
        pairs.rowmajor_of(plain)
        late.get()
    exp = orb.igemm_pairs(to_np(idx), 2, list(SHAPE), [3] * 3, [2] * 3, [1] * 3, [1] * 3, [0] * 3, False, False, True, False)
    fwd, bwd = pairs.native_pair_to_tables(lists, num, N, N, False)
    want = orb.native_pair_to_tables(to_np(lists), N, N, False, True)
    np.testing.assert_array_equal(to_np(fwd), want[0])
    np.testing.assert_array_equal(to_np(bwd), want[1])
    np.testing.assert_array_equal(to_np(pairs.rowmajor_of(plain))[:, :27].T, exp[2])
    np.testing.assert_array_equal(to_np(late.get()[0]), exp[3])


def test_tables_go_when_backward_has_run():
    """... and not with the last tensor that keeps the graph's nodes."""
    import spconv_triton_b200.pytorch as sp

    layer = sp.SparseConv3d(16, 16, 3, stride=2, padding=1).to(DEV)
    idx = torch.from_numpy(unique_coords(11, N, 2, SHAPE)).to(DEV)
    x = torch.randn(N, 16, device=DEV, requires_grad=True)
    loss = layer(sp.SparseConvTensor(x, idx, list(SHAPE), 2)).features.sum()
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    loss.backward()  # (`loss` keeps the graph's nodes)
    grads = sum(t.grad.numel() * 4 for t in (x, *layer.parameters()))
    torch.cuda.synchronize()
    assert torch.cuda.memory_allocated() <= before + grads - N * 28 * 4
    with pytest.raises(RuntimeError, match="second time"):
        loss.backward()
    pool = sp.SparseMaxPool3d(2, 2)
    x = torch.randn(N, 16, device=DEV, requires_grad=True)
    loss = pool(sp.SparseConvTensor(x, idx, list(SHAPE), 2)).features.sum()
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    loss.backward()
    torch.cuda.synchronize()
    assert torch.cuda.memory_allocated() <= before + x.grad.numel() * 4 - N * 8 * 4
