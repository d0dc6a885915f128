"""The layers' host side in C++ (``csrc/host.cpp``): when a layer takes it, and how its rulebooks look to
the rest of the package.

A layer on CUDA tensors with the default algorithms builds a ``Rulebook`` (its tables in the form the kernels
read) and runs on it.  The reference's interface shows more: sorted masks, column-major tables, pair lists.
Those are made from the rulebook when somebody reads them from the ``indice_dict`` entry.
"""

from __future__ import annotations

import functools
import importlib.machinery
import importlib.util

import numpy as np
import torch

from spconv_triton_b200 import _lib, constants

from . import gemm as _gemm
from . import pairs as _pairs

_ext = None
FLOATS = (torch.float16, torch.bfloat16, torch.float32)
POOL_FLOATS = (torch.float16, torch.bfloat16, torch.float32, torch.float64)


def ext():
    """The extension module; raises if it has not been built."""
    global _ext
    if _ext is None:
        _lib.load()
        path = _lib.LIB_PATH.parent / "_host.so"
        if not path.exists():
            raise RuntimeError(f"{path} is missing: run `python -m spconv_triton_b200.csrc.build`")
        loader = importlib.machinery.ExtensionFileLoader("_host", str(path))
        module = importlib.util.module_from_spec(importlib.util.spec_from_loader("_host", loader))
        loader.exec_module(module)
        module.set_error_type(_lib.SpconvB200Error)
        _ext = module
    return _ext


def takes(features, indices) -> bool:
    """Whether tensors like these go through the extension (everything else: the operator functions)."""
    return (features.is_cuda and indices.is_cuda and features.dtype in FLOATS and indices.dtype == torch.int32
            and _gemm.GEMM_PATH == _lib.SPC_GEMM_AUTO and _gemm.FP32_ON_TENSOR_CORES and constants.SPCONV_DO_SORT)


@functools.lru_cache(maxsize=1024)
def geometry(batch, in_shape, ksize, stride, padding, dilation, out_padding, subm, transposed):
    """(Geometry, output shape) or None where the operator functions raise their own errors."""
    if (any(k <= 0 for k in ksize) or (subm and any(k % 2 == 0 for k in ksize)) or len(in_shape) > _lib.SPC_MAX_NDIM):
        return None
    if subm:
        out_shape = list(in_shape)
    elif transposed:
        out_shape = _pairs.get_deconv_output_size(in_shape, ksize, stride, padding, dilation, out_padding)
    else:
        out_shape = _pairs.get_conv_output_size(in_shape, ksize, stride, padding, dilation)
    if any(v <= 0 for v in out_shape):
        return None
    return (ext().Geometry(batch, list(in_shape), list(out_shape), list(ksize), list(stride), list(padding), list(dilation),
                           subm, transposed), out_shape)


def geometry_of(layer, batch, spatial_shape):
    """``geometry`` of a convolution or pooling layer."""
    return geometry(batch, tuple(spatial_shape), tuple(layer.kernel_size), tuple(layer.stride), tuple(layer.padding),
                    tuple(layer.dilation), tuple(getattr(layer, "output_padding", ())) or (0,) * layer.ndim, bool(layer.subm),
                    bool(getattr(layer, "transposed", False)))


def build(layer, geo, indices, spatial_shape, input_side, colmajor, order=True):
    """The rulebook of ``layer``; raises as the reference does where no point is left."""
    rb = ext().build_rulebook(geo, indices, input_side, colmajor, order)
    if rb.n_out == 0:
        raise ValueError(_pairs._POINT_VANISH_MSG.format(list(spatial_shape), list(layer.kernel_size), list(layer.stride),
                                                         list(layer.padding), list(layer.dilation)))
    return rb


def exact_masks(rowmajor, kv):
    """The mask words of the rows of a table (kv <= 32) sorted ascending, stable, and their argsort: what
    ``igemm_pairs`` gives for one split."""
    weights = torch.ones(kv, dtype=torch.int64, device=rowmajor.device) << torch.arange(kv, device=rowmajor.device)
    words = ((rowmajor[:, :kv] >= 0).to(torch.int64) * weights).sum(1)
    vals, args = torch.sort(words, stable=True)
    vals = torch.where(vals >= 2 ** 31, vals - 2 ** 32, vals)  # the words are unsigned, the tensor is int32
    return [vals.to(torch.int32).reshape(-1, 1)], [args.to(torch.int32)]


class Tables:
    """What an ``indice_dict`` entry shows of a rulebook, made when read."""

    __slots__ = ("rb", "want_bwd")

    def __init__(self, rb, want_bwd):
        self.rb, self.want_bwd = rb, want_bwd

    def forward(self):
        table = self.rb.colmajor(False)
        table._spc_rowmajor = self.rb.rowmajor(False)
        return table

    def masks(self):
        return exact_masks(self.rb.rowmajor(False), self.rb.geometry.kv)

    def get(self):
        """(pair_bwd, its masks, their argsorts)"""
        rb = self.rb
        if not self.want_bwd:
            return torch.Tensor(), [], []
        if rb.geometry.subm:
            return rb.colmajor(False).flip(0), [], []
        table = rb.colmajor(True)
        table._spc_rowmajor = rb.rowmajor(True)
        return (table, *exact_masks(table._spc_rowmajor, rb.geometry.kv))
