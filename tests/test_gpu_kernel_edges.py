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
