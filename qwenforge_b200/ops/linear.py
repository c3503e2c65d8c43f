"""Dense projections: y = x W^T (+ b).

float32 runs this library's own FFMA kernel (true 32-bit, a fixed order of additions for
every output element). bfloat16 calls the cuBLAS matrix product through torch, the same
library call the reference makes for its projections (student_engine.py:563, :664, :666,
:727, :736), until the tensor-core kernel of this library covers the shape.
"""
from __future__ import annotations

from typing import Optional

import torch

from . import kernels

# Plain products of 128 or more token rows can run on this library's own tcgen05 kernel (`csrc/tc_gemm.cu`) instead of
# the cuBLAS call. Off by default: measured on a B200 at 7358 x 2560 x 2048 its persistent form reaches 1,424 TFLOP/s where
# cuBLAS reaches 1,507 (at 11788 x 3584 x 18944: 1,542 against 1,462; at 2048 x 896 x 4864: 475 against 1,023). The gate/up product with the gate in its epilogue
# does not wait for this switch: it is the faster way wherever the persistent kernel runs (`parts/swiglu.py`).
_own_tensor_core_products = False
OWN_PRODUCT_MIN_ROWS = 128


def use_own_tensor_core_products(on: bool) -> None:
    global _own_tensor_core_products
    _own_tensor_core_products = bool(on)


def own_tensor_core_products(x: torch.Tensor, weight: torch.Tensor) -> bool:
    """Whether x @ weight.T is to run on the library's own tcgen05 kernel."""
    return (_own_tensor_core_products and x.dtype == torch.bfloat16 and x.shape[0] >= OWN_PRODUCT_MIN_ROWS
            and weight.shape[0] % 8 == 0 and kernels.tc_gemm_takes(x, weight))


def linear(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor] = None,
           out: Optional[torch.Tensor] = None, out_dtype: Optional[torch.dtype] = None) -> torch.Tensor:
    """x [M, K], weight [N, K] -> [M, N]. `out_dtype=torch.float32` asks a bfloat16 product for
    float32 results (accumulated in float32 and not rounded to bfloat16), as the logits need."""
    if not x.is_cuda:
        raise kernels.KernelError(f"linear: input on {x.device}; this library computes on CUDA devices only")
    m, n = x.shape[0], weight.shape[0]
    if x.dtype == torch.float32:
        if out is None:
            out = torch.empty((m, n), device=x.device, dtype=torch.float32)
        kernels.gemm_f32(x, weight, bias, out)
        return out
    if x.dtype != torch.bfloat16 or weight.dtype != torch.bfloat16:
        raise kernels.KernelError(f"linear: dtypes {x.dtype} x {weight.dtype} are not supported")
    if out_dtype != torch.float32 and bias is None and own_tensor_core_products(x, weight):
        if out is None:
            out = torch.empty((m, n), device=x.device, dtype=torch.bfloat16)
        kernels.tc_gemm(kernels.TC_PLAIN, x, weight, out)
        return out
    if out_dtype == torch.float32:
        result = torch.mm(x, weight.t(), out_dtype=torch.float32)
        if bias is not None:
            result += bias.float()
        if out is not None:
            out.copy_(result)
            return out
        return result
    if out is not None:
        if bias is None:
            torch.mm(x, weight.t(), out=out)
        else:
            torch.addmm(bias, x, weight.t(), out=out)
        return out
    return torch.nn.functional.linear(x, weight, bias)


def linear_rows(x: torch.Tensor, weight: torch.Tensor, out_dtype: Optional[torch.dtype] = None) -> torch.Tensor:
    """`linear` without a bias for parts whose steps may have few rows: up to 16 bfloat16 rows run on this library's
    weight streamer where it takes the shape and is the faster way (`skinny_gemm_takes`, `skinny_gemm_pays`). Unlike
    the library product it is launched as a programmatic dependent, so a chain of such products and the small kernels
    between them runs without gaps: the kernel after it starts its weight copies under this one's tail. Everything else
    goes to `linear`. The result is bfloat16, or float32 with `out_dtype=torch.float32`."""
    m = x.shape[0]
    if (x.dtype == torch.bfloat16 and weight.dtype == torch.bfloat16 and m <= kernels.SKINNY_MAX_ROWS and x.stride(1) == 1
            and kernels.skinny_gemm_takes(m, weight, kernels.EPI_PLAIN, False, ldx=x.stride(0)) and kernels.skinny_gemm_pays(m, weight)):
        out = torch.empty((m, weight.shape[0]), device=x.device, dtype=torch.float32 if out_dtype == torch.float32 else torch.bfloat16)
        kernels.skinny_gemm(kernels.EPI_PLAIN, weight, x=x, out=out)
        return out
    return linear(x, weight, None, out_dtype=out_dtype)


def tail_rides(x: torch.Tensor, joint: torch.Tensor, n: int) -> bool:
    """Whether x @ joint.T runs as one launch whose first n columns are bfloat16 and whose others stay float32 (`kernels.tc_gemm_tail`), and
    is the faster way: more than 64 rows, a K of up to 2,048 and columns enough, twice K, or more than 1,024 rows. Measured for 8 to 64
    float32 columns with the norm ahead, microseconds, two library products / one launch: n 2,688, K 896 14.9 / 9.9 for 100 rows, 21.7 / 15.4 for
    2,048; 6,144, 2,048 15.0 / 14.6 for 65, 47.5 / 42.7 for 2,048; 8,448, 2,048 22.8 / 20.2 for 512, 109.8 / 108.4 for 4,096 (17 rows alone: 14.3 /
    16.9). Beyond, the library cuts K among blocks or has the better rate: 12,288, 4,096 37.2 / 46.6 for 300, 93.5 / 101.3 for 1,200 (301.8 /
    286.2 for 4,096); 768, 2,048 11.6 / 13.0 for 65, 12.7 / 13.9 for 512, 18.8 / 17.4 for 2,048; 1,536, 1,536 12.0 / 12.6 for 512, 15.8 / 14.3 for 1,200."""
    m, k = x.shape
    return (x.is_cuda and x.dtype == torch.bfloat16 and joint.dtype == torch.bfloat16 and m > kernels.WIDE_MAX_ROWS and n % 8 == 0
            and k <= 2048 and (n >= 2 * k or m > 1024)
            and kernels.tc_gemm_takes(x, joint))


def gated_rows(x: torch.Tensor, weight: torch.Tensor, out: torch.Tensor, clamp=None) -> bool:
    """The fused [gate | up] product of a step of few rows with its gate in the product's epilogue, where this library's weight
    streamer takes the shape and is the faster way: out = silu(g) * u, or with clamp = (limit, alpha) the clamped gate of
    `clamped_glu`, on the float32 sums. Returns False, having done nothing, where the caller is to run the product and the gate
    as two kernels."""
    m = x.shape[0]
    if not (x.is_cuda and x.dtype == torch.bfloat16 and weight.dtype == torch.bfloat16 and m <= kernels.SKINNY_MAX_ROWS
            and x.stride(1) == 1 and (clamp is None or float(clamp[0]) > 0)
            and kernels.skinny_gemm_takes(m, weight, kernels.EPI_SWIGLU, False, ldx=x.stride(0)) and kernels.skinny_gemm_pays(m, weight)):
        return False
    kernels.skinny_gemm(kernels.EPI_SWIGLU, weight, x=x, out=out, clamp=clamp)
    return True
