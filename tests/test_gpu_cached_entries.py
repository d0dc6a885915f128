"""Cache entries of layers are records of tensors: they can be copied, stored and loaded."""

import copy
import io
import pickle

import numpy as np
import pytest
import torch

from gpu_util import DEV, to_np, unique_coords
from oracle import rulebook as orb

pytestmark = pytest.mark.gpu


def _torch_save(obj):
    buf = io.BytesIO()
    torch.save(obj, buf)
    buf.seek(0)
    return torch.load(buf, weights_only=False)


@pytest.mark.parametrize("clone", [copy.deepcopy, lambda o: pickle.loads(pickle.dumps(o)), _torch_save],
                         ids=["deepcopy", "pickle", "torch.save"])
@pytest.mark.parametrize("train,how", [(False, "layers"), (True, "layers"), (False, "one call")])
def test_copies_of_an_indice_dict(clone, train, how):
    import spconv_triton_b200.pytorch as sp

    shape = [24, 22, 20]
    idx = unique_coords(7, 2500, 2, shape)
    net = sp.SparseSequential(sp.SubMConv3d(16, 16, 3, padding=1, indice_key="s"),
                              sp.SparseConv3d(16, 32, 3, stride=2, padding=1, indice_key="d")).to(DEV).half().train(train)
    wide = sp.SubMConv3d(16, 16, 5, padding=2, indice_key="n").to(DEV).half().train(train)  # 125 offsets: pair lists
    x = sp.SparseConvTensor(torch.randn(2500, 16, device=DEV).half(), torch.from_numpy(idx).to(DEV), shape, 2)
    with torch.set_grad_enabled(train):
        y = net(x) if how == "one call" else net[1](net[0](x))
        entries = dict(y.indice_dict, **wide(x).indice_dict)
        got = clone(entries)
        for key, ksize, stride, subm in (("s", 3, 1, True), ("d", 3, 2, False)):
            exp = orb.igemm_pairs(idx, 2, shape, [ksize] * 3, [stride] * 3, [1] * 3, [1] * 3, [0] * 3, subm, False, True, False)
            for e in (got[key], entries[key]):
                np.testing.assert_array_equal(to_np(e.out_indices), exp[0])
                np.testing.assert_array_equal(to_np(e.pair_fwd), exp[2])
                np.testing.assert_array_equal(to_np(e.pair_mask_fwd_splits[0]), exp[4][0])
                np.testing.assert_array_equal(to_np(e.mask_argsort_fwd_splits[0]), exp[6][0])
                if not subm:
                    np.testing.assert_array_equal(to_np(e.pair_bwd), exp[3])
                    np.testing.assert_array_equal(to_np(e.mask_argsort_bwd_splits[0]), exp[7][0])
        for e in (got["n"], entries["n"]):
            exp = orb.native_pairs(idx, 2, shape, [5] * 3, [1] * 3, [2] * 3, [1] * 3, [0] * 3, True, False)
            np.testing.assert_array_equal(to_np(e.indice_pairs), exp[1])
        # the copy serves a layer, and so does the original
        up = sp.SparseInverseConv3d(32, 16, 3, indice_key="d").to(DEV).half().train(train)
        outs = []
        for d in (got, entries):
            z = y.shadow_copy()
            z.indice_dict = d
            outs.append(up(z).features.detach().float())
        # (the layer's rows come in another tile order: fp16 outputs, sums in another order)
        assert float((outs[0] - outs[1]).abs().max()) <= 4e-3 * float(outs[1].abs().max())
