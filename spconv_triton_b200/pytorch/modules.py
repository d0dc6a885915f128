"""Containers and thin wrappers (reference: spconv_triton/pytorch/modules.py)."""

from __future__ import annotations

import threading
import time
from collections import OrderedDict

import torch
from torch import nn

from spconv_triton_b200 import _lib

from ._impl import host as _host
from .core import SparseConvTensor

_depth = threading.local()  # nesting depth of SparseSequential.forward on this thread


class SparseModule(nn.Module):
    """Marks a module as taking and returning SparseConvTensor."""

    def __init__(self, name=None):
        super().__init__()
        self.name = name
        self._sparse_unique_name = ""


def is_spconv_module(module):
    return isinstance(module, (SparseModule, SparseBatchNorm, SparseReLU))


def is_sparse_conv(module):
    from .conv import SparseConvolution

    return isinstance(module, SparseConvolution)


class SparseSequential(SparseModule):
    """Sequential container: sparse-aware children receive the SparseConvTensor,
    every other module is applied to its features."""

    def __init__(self, *args, **kwargs):
        super().__init__()
        if len(args) == 1 and isinstance(args[0], OrderedDict):
            for key, module in args[0].items():
                self.add_module(key, module)
        else:
            for idx, module in enumerate(args):
                self.add_module(str(idx), module)
        for name, module in kwargs.items():
            if name in self._modules:
                raise ValueError("name exists.")
            self.add_module(name, module)

    # What the native pass keeps on a container (plans of this process's threads, arena size) is not part of a copy.
    def __getstate__(self):
        return {k: v for k, v in self.__dict__.items() if k not in ("_spc_plans", "_spc_arena_floor")}

    def __len__(self):
        return len(self._modules)

    def __getitem__(self, idx):
        n = len(self)
        if not (-n <= idx < n):
            raise IndexError(f"index {idx} is out of range")
        return list(self._modules.values())[idx % n]

    def add(self, module, name=None):
        if name is None:
            name = str(len(self._modules))
            if name in self._modules:
                raise KeyError("name exists")
        self.add_module(name, module)

    def forward(self, x):
        from . import runahead

        # the outermost container of a CUDA pass looks at the status its device posted during an
        # earlier pass (raises without waiting) and posts the status of this pass when it is done
        device = None
        if isinstance(x, SparseConvTensor) and x.features.is_cuda and not getattr(_depth, "n", 0):
            device = x.features.device
            _lib.raise_posted_status(device)
        if isinstance(x, SparseConvTensor) and getattr(x, "_planner", None) is None:
            from . import sequence

            done = sequence.forward(self, x)  # the whole pass as one library call, where it applies
            if done is not None:
                if device is not None:
                    _lib.post_device_status(device)
                return done
        _depth.n = getattr(_depth, "n", 0) + 1
        entered, owned = x, runahead.begin(self, x)
        try:
            x = self._run(x)
        finally:
            _depth.n -= 1
            if owned is not None:
                owned.join_late()
                entered._planner = None
        if owned is not None and isinstance(x, SparseConvTensor):
            x._planner = None
        if device is not None and not torch.cuda.is_current_stream_capturing():
            _lib.post_device_status(device)
        return x

    def _run(self, x):
        mods = list(self._modules.values())
        i = 0
        while i < len(mods):
            module = mods[i]
            fused = _try_fold_bn_relu(mods, i, x) or _try_train_bn_act(mods, i, x)
            if fused is not None:
                x, i = fused
            else:
                if is_spconv_module(module):
                    x = module(x)
                elif isinstance(x, SparseConvTensor):
                    if x.indices.shape[0] != 0:
                        x = x.replace_feature(module(x.features))
                else:
                    x = module(x)
                i += 1
            # the GEMM of this layer is queued: build the next rulebook beside it
            if is_sparse_conv(module) and isinstance(x, SparseConvTensor) and x._planner is not None:
                x._planner.advance()
        return x


def _folded_bn(bn: nn.BatchNorm1d):
    """fp32 (scale, shift) with bn(x) == x * scale + shift in evaluation mode."""
    with torch.no_grad():
        scale = torch.rsqrt(bn.running_var.float() + bn.eps)
        if bn.weight is not None:
            scale = scale * bn.weight.float()
        shift = -bn.running_mean.float() * scale
        if bn.bias is not None:
            shift = shift + bn.bias.float()
        return scale.contiguous(), shift.contiguous()


def _bn_operands(bn):
    params, buffers = bn._parameters, bn._buffers  # (attributes of a module are a slow look-up)
    if "weight" in params and "bias" in params and "running_mean" in buffers and "running_var" in buffers:
        return buffers["running_mean"], buffers["running_var"], params["weight"], params["bias"], bn.eps, bn.num_features
    return bn.running_mean, bn.running_var, bn.weight, bn.bias, bn.eps, bn.num_features


def _folded_norms(norms, like, launch=True):
    """``_folded_bn`` of each of ``norms`` for features like ``like``: a block of fp32 values, where in it each (scale, shift)
    lies, and the argument of ``spc_fold_norms``, which fills the block (queued here unless ``launch`` is False; empty where
    torch's functions have filled it).  None where a tensor is on another device or of another length.  Made anew by each
    pass: a pair kept from one for the next would have to notice every way in which statistics can change (training writes
    them past their version counters, as ``.data`` does) and wait for the stream that made it."""
    done = _host.ext().norm_folds([_bn_operands(bn) for bn in norms], like)
    if done is None:
        parts = [t for bn in norms for t in _folded_bn(bn)]
        if any(t.device != like.device for t in parts) or [t.shape for t in parts[::2]] != [(bn.num_features,) for bn in norms]:
            return None
        starts = [0]
        for t in parts:
            starts.append(starts[-1] + t.numel())
        return torch.cat(parts), list(zip(starts[0::2], starts[1::2])), b""
    if launch:
        with torch.cuda.device(like.device):
            _lib.check(_lib.load().spc_fold_norms(done[2], len(norms), _lib.current_stream(like.device)))
    return done


def _try_fold_bn_relu(mods, i, x):
    """In evaluation mode a sparse convolution followed by BatchNorm1d (and
    optionally ReLU) runs as ONE kernel: the normalisation becomes a per-channel
    scale and shift applied, with the ReLU, while the GEMM stores its rows.  This
    removes two passes over the activations; the result differs from the
    separate modules only by fp16 rounding order.  Switch:
    ``spconv_triton_b200.constants.SPCONV_FOLD_BN_RELU``.  Returns
    ``(new_x, next_index)`` or None when the pattern does not apply."""
    from spconv_triton_b200 import constants

    from .conv import SparseConvolution

    if not constants.SPCONV_FOLD_BN_RELU or i + 1 >= len(mods) or not isinstance(x, SparseConvTensor):
        return None
    conv, bn = mods[i], mods[i + 1]
    if not (isinstance(conv, SparseConvolution) and conv.can_fold_epilogue()):
        return None
    if not (type(bn) in (nn.BatchNorm1d, SparseBatchNorm) and not bn.training and bn.track_running_stats
            and bn.running_mean is not None and bn.num_features == conv.out_channels):
        return None
    if not x.features.is_cuda or x.features.dtype not in (torch.float16, torch.bfloat16, torch.float32):
        return None
    if x.benchmark or x.indices.shape[0] == 0:
        return None
    relu = i + 2 < len(mods) and type(mods[i + 2]) in (nn.ReLU, SparseReLU)
    folded = _host.ext().fold_norm(*_bn_operands(bn), x.features)
    if folded is None:
        folded = _folded_bn(bn)
        if any(t.device != x.features.device or t.shape != (bn.num_features,) for t in folded):
            return None
    return conv(x, _fold=(*folded, relu)), i + 2 + int(relu)


_HOOKS = ("_forward_hooks", "_forward_pre_hooks", "_backward_hooks", "_backward_pre_hooks")
_GLOBAL_HOOKS = ("_global_forward_hooks", "_global_forward_pre_hooks", "_global_backward_hooks", "_global_backward_pre_hooks")


def _plain(module) -> bool:
    """Nobody looks at what goes in and out of this module."""
    own = module.__dict__
    return "forward" not in own and not any(own.get(h) for h in _HOOKS)


def _watched() -> bool:
    """Something sees or changes the torch functions that the modules would call."""
    return (any(getattr(torch.nn.modules.module, h, None) for h in _GLOBAL_HOOKS) or torch._C._len_torch_function_stack() > 0
            or torch._C._len_torch_dispatch_stack() > 0 or torch._C._functorch.peek_interpreter_stack() is not None
            or torch.compiler.is_compiling() or torch.jit.is_tracing())


def _try_train_bn_act(mods, i, x):
    """In training a BatchNorm1d and the ReLU or SiLU after it run as one operator (``spc_norm_act_*``) that passes over
    the features twice in each direction; the activation sees the normalised features before they are rounded.  Returns
    ``(new_x, next_index)``, or None where the modules run one by one: whatever the operator does not take, and wherever
    something could see the tensor between the two."""
    bn = mods[i]
    if type(bn) not in (nn.BatchNorm1d, SparseBatchNorm) or not bn.training or not isinstance(x, SparseConvTensor):
        return None
    features = x.features
    if (type(features) is not torch.Tensor or not features.is_cuda or features.dim() != 2 or x.indices.shape[0] == 0
            or features.shape[1] != bn.num_features or bn.momentum is None or not bn.track_running_stats
            or bn.running_mean is None or bn.running_var is None or bn.num_batches_tracked is None
            or not _plain(bn) or _watched()):
        return None
    if any(type(t) not in (torch.Tensor, nn.Parameter) for t in (bn.weight, bn.bias) if t is not None):
        return None
    act, after = 0, i + 1
    if after < len(mods) and _plain(mods[after]):
        kind = type(mods[after])
        act = 1 if kind in (nn.ReLU, SparseReLU) else 2 if kind is nn.SiLU else 0
        after += 1 if act else 0
    out = _host.ext().norm_act_train(features, bn.weight, bn.bias, bn.running_mean, bn.running_var, bn.num_batches_tracked,
                                     bn.momentum, bn.eps, act)
    return None if out is None else (x.replace_feature(out), after)


def assign_name_for_sparse_modules(module: nn.Module):
    for k, n in module.named_modules():
        if isinstance(n, SparseModule):
            n._sparse_unique_name = k


def _on_features(base):
    """Subclass of a dense torch module that also accepts a SparseConvTensor."""

    class _Wrapped(base):
        def forward(self, x):
            if isinstance(x, SparseConvTensor):
                return x.replace_feature(super().forward(x.features))
            return super().forward(x)

    return _Wrapped


def _named(cls, name):
    cls.__name__ = cls.__qualname__ = name
    cls.__module__ = __name__
    return cls


SparseBatchNorm = _named(_on_features(nn.BatchNorm1d), "SparseBatchNorm")
SparseSyncBatchNorm = _named(_on_features(nn.SyncBatchNorm), "SparseSyncBatchNorm")
SparseReLU = _named(_on_features(nn.ReLU), "SparseReLU")
SparseIdentity = _named(_on_features(nn.Identity), "SparseIdentity")


class PrintTensorMeta(nn.Module):
    def forward(self, x):
        ft = x.features if isinstance(x, SparseConvTensor) else x
        if isinstance(ft, torch.Tensor):
            print(ft.min(), ft.max(), ft.mean())
        return x


class PrintCurrentTime(nn.Module):
    def __init__(self) -> None:
        super().__init__()
        self.first_time = time.time()

    def forward(self, x, msg="", reset: bool = False):
        if reset:
            self.first_time = time.time()
        torch.cuda.synchronize()
        print(msg, time.time() - self.first_time)
        return x
