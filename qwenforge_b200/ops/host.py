"""Stretches of a prompt step whose launches native code issues (csrc/host.cpp), kernel by kernel those of `ops.kernels`.

Every function answers None, having launched nothing, for what it does not take; the caller then launches the kernels one by one, where the
same condition is reported or another kernel chosen. So do they while one of these kernels' names in `ops` is not the function of
`ops.kernels`: whoever puts something in its place (`ops.timing.KernelTimer`) sees every call; and where the native module cannot be built.
"""
from __future__ import annotations

import ctypes
import sys
from typing import Optional

import torch

from ..csrc import KernelLibraryError, host_module, library
from . import kernels
from .linear import linear, linear_rows, own_tensor_core_products, tail_rides

_ENTRIES = {"norm": ("qf_add_rms_norm",),
            "tc_gemm": ("qf_tc_gemm_qkv_pairs_pays", "qf_tc_gemm_qkv_pairs", "qf_tc_gemm_is_persistent", "qf_tc_gemm", "qf_tc_gemm_tail"),
            "attention_prefill_tc": ("qf_attention_prefill_tc_ex",), "rope_cache": ("qf_rope_cache_write",), "activation": ("qf_swiglu",), "recurrent": ("qf_stabilized_gates", "qf_gated_group_norm", "qf_causal_conv"),
            "state_chunks": ("qf_state_chunks",), "row_chunks": ("qf_row_chunks",)}
_known: set = set()   # libraries whose entries the module has been told
_module = None
_OWN = {"linear_rows": linear_rows, "tail_rides": tail_rides}   # (of `ops.linear`'s file)


def _host(*libraries: str):
    """The native module, told the entries of these kernel libraries; None where it cannot be had (`host_module` has said why)."""
    global _module
    if _module is None:
        try:
            _module = host_module()
        except KernelLibraryError:
            return None
    for name in libraries:
        if name not in _known:
            loaded = library(name)
            _module.setup(kernels.KernelError, {entry: ctypes.cast(getattr(loaded, entry), ctypes.c_void_p).value for entry in _ENTRIES[name]})
            _known.add(name)
    return _module


def _untouched(*names: str) -> bool:
    """Whether these names in `ops` are the functions of this package."""
    ops = sys.modules[__package__]
    return ops.linear is linear and all(getattr(ops, name) is (_OWN.get(name) or getattr(kernels, name)) for name in names)


def _launch(name: str, launches: int, libraries: tuple, *args) -> Optional[torch.Tensor]:
    """The native module's function `name`; the kernels of this package that it launched are counted."""
    module = _host(*libraries)
    out = None if module is None else getattr(module, name)(*args)
    if out is not None:
        kernels.launches += launches
    return out


def rms_norm(hidden: torch.Tensor, delta: Optional[torch.Tensor], weight: torch.Tensor, eps: float) -> Optional[torch.Tensor]:
    """`add_rms_norm` into a new tensor."""
    if not (hidden.is_cuda and _untouched("add_rms_norm")):
        return None
    return _launch("rms_norm", 1, ("norm",), hidden, delta, weight, eps)


def prompt_attention(x: torch.Tensor, qkv_weight: torch.Tensor, bias: Optional[torch.Tensor], inv_freq: Optional[torch.Tensor], o_weight: torch.Tensor,
                     ctx, site, n_heads: int, kv_heads: int, head_dim: int, scale: float, window: int, write_cache: bool) -> Optional[torch.Tensor]:
    """Queries, keys and values (`qkv_product` where it is the faster way, else the product and `rope_cache_write`), `attention_prefill_tc`, which the
    caller has found to be the kernel, and the output projection without a bias."""
    if not (x.is_cuda and _untouched("qkv_product", "qkv_product_takes", "qkv_product_pays", "rope_cache_write", "attention_prefill_tc")) \
            or own_tensor_core_products(x, o_weight) or own_tensor_core_products(x, qkv_weight):
        return None
    return _launch(
        "prompt_attention", 2, ("tc_gemm", "rope_cache", "attention_prefill_tc"),
        x, qkv_weight, bias, inv_freq, o_weight, ctx.tok_seq, ctx.tok_pos, ctx.slots, ctx.cu_q, site.storage, site.table, ctx.err, n_heads, kv_heads,
        head_dim, ctx.n_seqs, ctx.max_q_len, ctx.max_kv_len, scale, window, int(bool(write_cache)))


def gated_feed_forward(x: torch.Tensor, gate_up: torch.Tensor, down: torch.Tensor, err: torch.Tensor) -> Optional[torch.Tensor]:
    """Gate and up with the gate (`tc_gemm` where it has tiles for every SM, else the product and `swiglu`) and the down projection."""
    if not (x.is_cuda and _untouched("tc_gemm", "tc_gemm_takes", "tc_gemm_is_persistent", "swiglu")) or own_tensor_core_products(x, down) \
            or own_tensor_core_products(x, gate_up):
        return None
    return _launch("gated_feed_forward", 1, ("tc_gemm", "activation"), x, gate_up, down, err)


def matrix_memory(x: torch.Tensor, joint: torch.Tensor, gate_bias: torch.Tensor, norm: torch.Tensor, o_weight: torch.Tensor, ctx, state: torch.Tensor,
                  n_heads: int, dim: int, vdim: int, offsets: tuple, cap: float, eps: float, floor: float) -> Optional[torch.Tensor]:
    """`tc_gemm_tail`, `stabilized_gates`, `state_chunks`, `gated_group_norm` and the output projection, where the float32 columns ride on the
    projections' product and the step runs in chunks."""
    n = x.shape[0]
    if not (x.is_cuda and kernels.state_chunks_pay(n, dim, vdim, n_heads, ctx.max_q_len, ctx.n_seqs)
            and _untouched("tc_gemm_tail", "tail_rides", "stabilized_gates", "state_chunks", "state_chunks_take", "gated_group_norm", "linear_rows")) \
            or own_tensor_core_products(x, o_weight):
        return None
    if not tail_rides(x, joint, 2 * n_heads * (dim + vdim)):
        return None
    records, each = kernels.state_chunk_records(n, ctx.n_seqs, n_heads, dim, vdim)
    return _launch(
        "matrix_memory", 4, ("tc_gemm", "recurrent", "state_chunks"),
        x, joint, gate_bias, norm, o_weight, state, ctx.cu_q, ctx.slots, ctx.err, n_heads, dim, vdim, ctx.max_q_len, records, each, *offsets,
        cap, eps, floor)


def state_space(x: torch.Tensor, joint: torch.Tensor, conv_weight: torch.Tensor, conv_bias: torch.Tensor, dt_bias: torch.Tensor, rate_log: torch.Tensor,
                skip: torch.Tensor, norm: torch.Tensor, o_weight: torch.Tensor, ctx, state: torch.Tensor, n_heads: int, vdim: int, n_state: int, groups: int,
                norm_parts: int, offsets: tuple, eps: float) -> Optional[torch.Tensor]:
    """`tc_gemm_tail`, `causal_conv_silu`, `state_chunks` with the gates formed inside, `gated_group_norm` and the output projection, where the
    float32 columns ride on the projections' product and the step runs in chunks."""
    n = x.shape[0]
    if not (x.is_cuda and kernels.state_chunks_pay(n, n_state, vdim, n_heads, ctx.max_q_len, ctx.n_seqs)
            and _untouched("tc_gemm_tail", "tail_rides", "causal_conv_silu", "state_chunks", "state_chunks_take", "gated_group_norm", "linear_rows")) \
            or own_tensor_core_products(x, o_weight):
        return None
    if not tail_rides(x, joint, joint.shape[0] - n_heads):
        return None
    records, each = kernels.state_chunk_records(n, ctx.n_seqs, n_heads, n_state, vdim)
    return _launch(
        "state_space", 4, ("tc_gemm", "recurrent", "state_chunks"),
        x, joint, conv_weight, conv_bias, dt_bias, rate_log, skip, norm, o_weight, state, ctx.cu_q, ctx.tok_seq, ctx.slots, ctx.err, n_heads, vdim, n_state,
        groups, norm_parts, ctx.max_q_len, records, each, *offsets, eps)


def gated_linear_attention(x: torch.Tensor, joint: torch.Tensor, a2: torch.Tensor, a2_bias: torch.Tensor, norm: torch.Tensor, o_weight: torch.Tensor, ctx,
                           state: torch.Tensor, n_heads: int, dim: int, vdim: int, tau: float, eps: float) -> Optional[torch.Tensor]:
    """The product of [q | k | v | gate | middle] and the middle's in float32, `row_chunks`, `gated_group_norm` and the output projection, where the
    step runs in chunks."""
    n = x.shape[0]
    if not (x.is_cuda and kernels.row_chunks_pay(n, dim, vdim, n_heads, ctx.max_q_len, ctx.n_seqs)
            and _untouched("row_chunks", "row_chunks_take", "gated_group_norm", "linear_rows")) \
            or own_tensor_core_products(x, o_weight) or own_tensor_core_products(x, joint):
        return None
    records, each = kernels.row_chunk_records(n, ctx.n_seqs, n_heads, dim, vdim)
    return _launch(
        "gated_linear_attention", 2, ("recurrent", "row_chunks"),
        x, joint, a2, a2_bias, norm, o_weight, state, ctx.cu_q, ctx.slots, n_heads, dim, vdim, ctx.max_q_len, records, each, 1.0 / tau, eps)
