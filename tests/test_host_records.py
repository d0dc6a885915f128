"""Host-side records: entries read by several threads or written by the user, containers that are copied after a
pass, folded statistics.  No GPU needed."""

import copy
import pickle
import threading
import time
import weakref
from types import SimpleNamespace

import numpy as np
import torch

import spconv_triton_b200.pytorch as sp
from spconv_triton_b200.core import ConvAlgo
from spconv_triton_b200.pytorch.core import ImplicitGemmIndiceData


def _entry():
    return ImplicitGemmIndiceData(torch.zeros(3, 4), torch.zeros(3, 4), None, torch.Tensor(), None, [], None, [],
                                  [np.array([0xFFFFFFFF], dtype=np.uint32)], [4] * 3, [2] * 3, False,
                                  ConvAlgo.MaskImplicitGemm, [3] * 3, [2] * 3, [1] * 3, [1] * 3)


class _Late:
    def __init__(self):
        self.calls = 0

    def get(self):
        self.calls += 1
        time.sleep(0.05)
        return torch.ones(2), [torch.ones(3)], [torch.ones(4)]


def test_threads_read_an_entry_whose_tables_are_made_on_demand():
    entry = _entry()
    late, made = _Late(), []

    def slow(result):
        made.append(result)
        time.sleep(0.05)
        return result

    entry._late = late
    entry._pair_fwd_thunk = lambda: slow(torch.zeros(5))
    entry._masks_fwd_thunk = lambda: slow(([torch.zeros(6)], [torch.zeros(7)]))
    seen, gate = [], threading.Barrier(4)

    def read():
        gate.wait()
        seen.append((entry.pair_fwd, entry.pair_mask_fwd_splits, entry.mask_argsort_fwd_splits, entry.pair_bwd,
                     entry.pair_mask_bwd_splits, entry.mask_argsort_bwd_splits))

    threads = [threading.Thread(target=read) for _ in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(seen) == 4 and late.calls == 1 and len(made) == 2
    for values in seen:
        assert [v.numel() if isinstance(v, torch.Tensor) else v[0].numel() for v in values] == [5, 6, 7, 2, 3, 4]


def test_a_table_that_the_user_assigns_stays():
    entry = _entry()
    entry._late = _Late()
    entry._masks_fwd_thunk = lambda: ([torch.zeros(6)], [torch.zeros(7)])
    mine = torch.full((9,), 3.0)
    entry.pair_bwd = mine
    entry.mask_argsort_fwd_splits = [mine]
    assert entry.pair_bwd is mine and entry.mask_argsort_fwd_splits[0] is mine
    assert entry.pair_mask_bwd_splits[0].numel() == 3 and entry.pair_mask_fwd_splits[0].numel() == 6
    assert entry.pair_bwd is mine and entry.mask_argsort_fwd_splits[0] is mine


def test_copies_of_an_entry_hold_its_tables():
    entry = _entry()
    entry._late = _Late()
    entry._pair_fwd_thunk = lambda: torch.zeros(5)
    entry._rb = threading.Lock()  # (like a native rulebook: cannot be copied)
    for clone in (copy.deepcopy, lambda e: pickle.loads(pickle.dumps(e))):
        got = clone(entry)
        assert got.pair_fwd.numel() == 5 and got.pair_bwd.numel() == 2 and got.__dict__.get("_rb") is None
        assert got.ksize == [3] * 3 and got.algo == ConvAlgo.MaskImplicitGemm
    assert entry._rb is not None


def _net():
    return sp.SparseSequential(sp.SubMConv3d(16, 16, 3, padding=1, bias=False, indice_key="s"), torch.nn.BatchNorm1d(16),
                               torch.nn.ReLU()).eval()


def test_a_container_that_has_run_can_be_copied():
    """Plans of the native pass belong to the object that made them, not to its copies."""
    from spconv_triton_b200.pytorch import sequence

    net = _net()
    x = sp.SparseConvTensor(torch.zeros(3, 16), torch.zeros(3, 4, dtype=torch.int32), [4] * 3, 1)
    net.__dict__["_spc_plans"] = {threading.get_ident(): sequence._compile(net, x)}
    net.__dict__["_spc_arena_floor"] = [1 << 30, 6144.0]
    for clone in (copy.deepcopy, lambda n: pickle.loads(pickle.dumps(n))):
        got = clone(net)
        assert "_spc_plans" not in got.__dict__ and "_spc_arena_floor" not in got.__dict__
        assert torch.equal(got[0].weight, net[0].weight)
    assert net.__dict__["_spc_plans"]


class _OnDevice(torch.Tensor):
    is_cuda = True


def test_what_a_graph_makes_tables_from_stays(monkeypatch):
    """... also when a later call outside the capture has made them for good, and when the user has put others there."""
    capturing = True
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: capturing)
    stream = SimpleNamespace(record_event=lambda: None, device="cuda")
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device: stream)

    class Late(_Late):
        def get(self):
            return torch.ones(2).as_subclass(_OnDevice), [], []

    entry = _entry()
    entry._late = Late()
    late = weakref.ref(entry._late)
    entry.pair_bwd, entry.pair_bwd  # (recorded twice, kept once)
    capturing = False
    entry.pair_bwd
    assert entry._late is None and late() is not None and len(entry._captured) == 1
    rb = SimpleNamespace(captured=True)
    entry._rb = rb
    entry.pair_mask_bwd_splits = []
    assert entry._rb is None and entry._captured[-1] is rb
    entry._rb = SimpleNamespace(captured=False)
    entry.mask_argsort_bwd_splits = []
    assert len(entry._captured) == 2
    assert copy.copy(entry)._captured == ()
    entry = None
    assert late() is None


def test_folded_statistics_follow_a_forward_in_training_mode():
    """Training moves the running statistics without telling their version counters."""
    from spconv_triton_b200.pytorch.modules import _folded_bn

    bn = torch.nn.BatchNorm1d(4)
    bn.eval()
    before = [t.clone() for t in _folded_bn(bn)]
    bn.train()(torch.randn(64, 4) * 3 + 1)
    bn.eval()
    x = torch.randn(8, 4)
    scale, shift = _folded_bn(bn)
    assert not torch.equal(shift, before[1])
    torch.testing.assert_close(x * scale + shift, bn(x))


def test_folded_statistics_follow_other_tensors_at_the_same_address():
    from spconv_triton_b200.pytorch.modules import _folded_bn

    bn, store = torch.nn.BatchNorm1d(4).eval(), torch.zeros(4)
    for value in (0.0, 1.0):
        store.fill_(value)
        bn.running_mean = store.data  # (a new tensor on the same memory, its version counter at its start)
        scale, shift = _folded_bn(bn)
        x = torch.randn(8, 4)
        torch.testing.assert_close(x * scale + shift, bn(x))
