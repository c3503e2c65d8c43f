"""The persistent tcgen05 product on pairs of SMs (csrc/tc_gemm.cu) at the edges of its tiles: one row or one piece of eight columns
more or less than whole tiles, a K below one stage, of whole stages and of more than the ring holds, both widths of tiles."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("gated,m,cols,k,columns", [
    (True, 905, 4864, 896, 192), (True, 1024, 4864, 64, 192), (True, 1025, 4872, 8, 256), (True, 513, 3848, 456, 192),
    (True, 2049, 2440, 520, 256), (False, 2047, 4864, 448, 192), (False, 1793, 2568, 392, 192), (False, 4100, 2568, 904, 256)])
def test_edges_of_pair_tiles(gated, m, cols, k, columns):
    from qwenforge_b200 import ops
    from qwenforge_b200.csrc import library
    g = torch.Generator(device=DEV).manual_seed(m)
    x = torch.randn(m, k, generator=g, device=DEV).bfloat16()
    w = (torch.randn(2 * cols if gated else cols, k, generator=g, device=DEV) * k ** -0.5).bfloat16()
    epilogue = ops.TC_SWIGLU if gated else ops.TC_PLAIN
    assert ops.tc_gemm_is_persistent(epilogue, m, w.shape[0])
    assert library("tc_gemm").qf_tc_gemm_pair_columns(ctypes.c_int(epilogue), ctypes.c_int(m), ctypes.c_int(w.shape[0])) == columns
    rows = torch.full((m + 2, cols + 16), 7.0, dtype=torch.bfloat16, device=DEV)   # what lies around the result stays as it is
    err = torch.zeros(1, dtype=torch.int32, device=DEV)
    ops.tc_gemm(epilogue, x, w, rows[1:m + 1, 8:cols + 8], err)
    sums, most = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    want, slack = sums, most * k * 2.0 ** -24
    if gated:   # |d silu| <= 1.1, so a sum's error counts 1.1 times the other half's size
        gate, up = sums[:, :cols], sums[:, cols:]
        want = gate * torch.sigmoid(gate) * up
        slack = 1.1 * (slack[:, :cols] * (up.abs() + 1) + slack[:, cols:] * (gate.abs() + 1)) + want.abs() * 2.0 ** -20
    got = rows[1:m + 1, 8:cols + 8].double()
    assert int(err) == 0
    assert bool(((got - want).abs() <= want.abs() * 2.0 ** -8 + slack + 1e-30).all())   # float32 sums, rounded once to eight bits
    assert bool((rows[0] == 7).all() and (rows[-1] == 7).all() and (rows[:, :8] == 7).all() and (rows[:, -8:] == 7).all())
