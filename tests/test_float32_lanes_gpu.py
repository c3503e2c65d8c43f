"""Float32 products in tiles of 96 x 96, a lane's rows and columns in runs of two: the bits of the kernel of few rows."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


# whole tiles, ragged ones both ways, a K of no whole piece of 16 and one below it
@pytest.mark.parametrize("m,n,k", [(960, 1344, 32), (1031, 1152, 35), (1030, 1100, 9), (1100, 1060, 48)])
def test_tiles_of_96_by_96(m, n, k):
    from qwenforge_b200 import ops
    from qwenforge_b200.csrc import library
    assert library("gemm_f32").qf_gemm_f32_tile(ctypes.c_int(m), ctypes.c_int(n)) == 96096
    g = torch.Generator(device=DEV).manual_seed(m + n + k)
    x, w, b = torch.randn(m, k, generator=g, device=DEV), torch.randn(n, k, generator=g, device=DEV), torch.randn(n, generator=g, device=DEV)
    out, rows = torch.full((m + 1, n), 7.0, device=DEV), torch.empty(m, n, device=DEV)
    ops.gemm_f32(x, w, b, out[:m])
    for at in range(0, m, 16):
        ops.gemm_f32(x[at:at + 16], w, b, rows[at:at + 16])
    assert torch.equal(out[:m], rows) and bool((out[m] == 7).all())
    wide = torch.zeros(m, k + 3, device=DEV)      # rows that no 16-byte load can address
    wide[:, 1:k + 1] = x
    ops.gemm_f32(wide[:, 1:k + 1], w, b, out[:m])
    assert torch.equal(out[:m], rows)
