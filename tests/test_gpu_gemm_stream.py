"""The gather-GEMM of many tiles a CTA (csrc/gemm_stream.cu) against fp32 matmuls of the same rows: at the fewest rows it
takes, with ragged last tiles, tiles without any pair, every span of a row, each option of the store, and stores whose
pass through shared memory the host narrows to win a third stage."""

import ctypes

import pytest
import torch

from spconv_triton_b200 import _lib

pytestmark = pytest.mark.gpu

CODES = {torch.float16: _lib.SPC_F16, torch.bfloat16: _lib.SPC_BF16, torch.float32: _lib.SPC_F32}
EPS = {torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8, torch.float32: 2.0 ** -22}


def _rows(n_dim, r_dim):
    """The first count that the kernel takes, and a bit."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return (11 if n_dim > 64 and r_dim == 64 else 20) * sms * 128 - 127


def _p(t):
    return ctypes.c_void_p(0 if t is None else t.data_ptr())


def _table(n_out, n_in, kv, gen):
    """Few pairs a row, whole tiles of rows without any, and runs of rows that share one offset."""
    pairs = torch.full((n_out, kv), -1, dtype=torch.int32, device="cuda")
    rows = torch.arange(n_out, device="cuda")
    for _ in range(2):
        k = torch.randint(0, kv, (n_out // 64 + 1,), generator=gen, device="cuda")[rows // 64]
        pairs[rows, k] = torch.randint(0, n_in, (n_out,), generator=gen, device="cuda").int()
    pairs[(rows // 128) % 7 == 3] = -1
    pairs[::5, 0] = torch.randint(0, n_in, (len(pairs[::5]),), generator=gen, device="cuda").int()
    pairs[(rows // 128) % 7 == 5] = -1
    rm = torch.full((n_out, (kv + 3) // 4 * 4), -1, dtype=torch.int32, device="cuda")
    rm[:, :kv] = pairs
    return pairs.t().contiguous(), rm


def _reference(x, w, cm, reverse=False, transposed=False):
    out = 0.0
    for k in range(cm.shape[0]):
        at = (cm[k] >= 0).nonzero()[:, 0]
        m = w[:, cm.shape[0] - 1 - k if reverse else k].float()
        if isinstance(out, float):
            out = torch.zeros(cm.shape[1], m.shape[1] if transposed else m.shape[0], device="cuda")
        out[at] += x[cm[k, at].long()].float() @ (m if transposed else m.t())
    return out


def _close(got, want, magnitude, out_type):
    # products and sums in fp32 (at most 3 pairs of 64 products a row), one rounding of the result
    assert (got.float() - want).abs().max().item() <= EPS[out_type] * want.abs().max().item() * 1.01 + 2.0 ** -20 * magnitude


# (stages of the kernel and bytes of a row that a store passes through shared memory, beside the cases below)
@pytest.mark.parametrize("c_in,c_out,kv,dtype,out_type,ordered,colmajor", [
    (64, 128, 27, torch.float16, torch.float16, True, False), (64, 96, 27, torch.bfloat16, torch.bfloat16, False, False),
    (32, 64, 27, torch.float16, torch.float32, True, False), (32, 112, 33, torch.float16, torch.float16, True, False),
    (16, 16, 27, torch.float16, torch.float16, True, True), (16, 128, 3, torch.bfloat16, torch.float32, False, True),
    (64, 16, 40, torch.float16, torch.float16, True, False),
    (64, 128, 8, torch.float16, torch.float32, True, False),  # 2, 128
    (64, 128, 9, torch.bfloat16, torch.float32, False, False),  # 2, 128
    (64, 112, 27, torch.float16, torch.float32, True, False),  # 2, 128
    (64, 128, 1, torch.float16, torch.float32, True, False),  # 3, 64
    (64, 96, 27, torch.float16, torch.float32, False, False),  # 3, 64
    (64, 64, 27, torch.bfloat16, torch.float32, True, False),  # 3, 128
    (64, 128, 8, torch.float16, torch.float16, True, False),  # 3, 32
    (64, 128, 9, torch.bfloat16, torch.bfloat16, False, False),  # 3, 32
    (64, 112, 27, torch.float16, torch.float16, True, False)])  # 3, 32
def test_forward_and_input_gradient(c_in, c_out, kv, dtype, out_type, ordered, colmajor):
    gen = torch.Generator("cuda").manual_seed(c_in + c_out)
    n_out, n_in = _rows(c_out, c_in), 30001
    cm, rm = _table(n_out, n_in, kv, gen)
    x = torch.randn(n_in, c_in, generator=gen, device="cuda").to(dtype)
    w = (torch.randn(c_out, kv, c_in, generator=gen, device="cuda") / c_in ** 0.5).to(dtype)
    bias = torch.randn(c_out, generator=gen, device="cuda").to(dtype)
    scale, shift = (torch.randn(c_out, generator=gen, device="cuda") for _ in range(2))
    residual = torch.randn(n_out, c_out, generator=gen, device="cuda").to(out_type)
    order = torch.randperm(n_out, generator=gen, device="cuda").int() if ordered else None
    plain = _reference(x, w, cm)
    lib = _lib.load()
    acts = {1: torch.relu, 2: torch.sigmoid, 3: lambda z: torch.nn.functional.leaky_relu(z, 0.1)}
    for act in (0, *acts):
        full = act != 0
        out = torch.full((n_out, c_out), float("nan"), dtype=out_type, device="cuda")
        extra = (_p(scale), _p(shift), act, 0.1, _p(residual)) if full else (None, None, 0, 0.0, None)
        rc = lib.spc_conv_forward_residual(_p(x), _p(w), _p(bias if full else None), _p(cm), _p(None if colmajor else rm), _p(order), _p(out),
                                           n_in, n_out, c_in, c_out, kv, CODES[dtype], CODES[out_type], 0, 0, *extra,
                                           ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert rc == 0
        want = plain
        if full:
            want = acts[act]((plain + bias.float()) * scale + shift) + residual.float()
        _close(out, want, 4 * (1 + scale.abs().max().item()), out_type)
    # the input gradient of a layer with the channels the other way round, of a strided and of a submanifold layer
    weight = w.permute(2, 1, 0).contiguous()  # [c_in, kv, c_out]: its output channels are reduced over
    for reverse in (0, 1):
        din = torch.full((n_out, c_out), float("nan"), dtype=dtype, device="cuda")
        rc = lib.spc_conv_backward_input_tables(_p(x), _p(weight), _p(cm), _p(None if colmajor else rm), _p(order), _p(din), n_out, n_in, c_out,
                                                c_in, kv, reverse, CODES[dtype], 0, 0, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert rc == 0
        _close(din, _reference(x, weight, cm, bool(reverse), True), 4.0, dtype)
