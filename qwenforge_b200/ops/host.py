"""Stretches of a prompt step whose launches native code issues (csrc/host.cpp), kernel by kernel those of `ops.kernels`.

Every function answers None, having launched nothing, for what it does not take; the caller then launches the kernels one by one, where the
same condition is reported or another kernel chosen. So do they while one of these kernels' names in `ops` is not the function of
`ops.kernels`: whoever puts something in its place (`ops.timing.KernelTimer`) sees every call.
"""
from __future__ import annotations

import ctypes
import sys
from typing import Optional

import torch

from ..csrc import host_module, library
from . import kernels
from .linear import linear, linear_rows, own_tensor_core_products, tail_rides

_ENTRIES = {"norm": ("qf_add_rms_norm",),
            "tc_gemm": ("qf_tc_gemm_qkv_pairs_pays", "qf_tc_gemm_qkv_pairs", "qf_tc_gemm_is_persistent", "qf_tc_gemm", "qf_tc_gemm_tail"),
            "attention_prefill_tc": ("qf_attention_prefill_tc_ex",), "recurrent": ("qf_stabilized_gates", "qf_gated_group_norm"),
            "state_chunks": ("qf_state_chunks",)}
_known: set = set()   # libraries whose entries the module has been told
_module = None
_OWN = {"linear_rows": linear_rows, "tail_rides": tail_rides}   # (of `ops.linear`'s file)


def _host(*libraries: str):
    """The native module, told the entries of these kernel libraries."""
    global _module
    if _module is None:
        _module = host_module()
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


def _counted(out: Optional[torch.Tensor], launches: int) -> Optional[torch.Tensor]:
    if out is not None:
        kernels.launches += launches
    return out


def rms_norm(hidden: torch.Tensor, delta: Optional[torch.Tensor], weight: torch.Tensor, eps: float) -> Optional[torch.Tensor]:
    """`add_rms_norm` into a new tensor."""
    if not (hidden.is_cuda and _untouched("add_rms_norm")):
        return None
    return _counted(_host("norm").rms_norm(hidden, delta, weight, eps), 1)


def prompt_attention(x: torch.Tensor, qkv_weight: torch.Tensor, bias: Optional[torch.Tensor], inv_freq: Optional[torch.Tensor], o_weight: torch.Tensor,
                     ctx, site, n_heads: int, kv_heads: int, head_dim: int, scale: float, window: int, write_cache: bool) -> Optional[torch.Tensor]:
    """`qkv_product`, `attention_prefill_tc` and the output projection without a bias, where the first is the faster way; that the second is,
    the caller has found."""
    if not (x.is_cuda and _untouched("qkv_product", "qkv_product_takes", "qkv_product_pays", "attention_prefill_tc")) or own_tensor_core_products(x, o_weight):
        return None
    return _counted(_host("tc_gemm", "attention_prefill_tc").prompt_attention(
        x, qkv_weight, bias, inv_freq, o_weight, ctx.tok_seq, ctx.tok_pos, ctx.slots, ctx.cu_q, site.storage, site.table, ctx.err, n_heads, kv_heads,
        head_dim, ctx.n_seqs, ctx.max_q_len, ctx.max_kv_len, scale, window, int(bool(write_cache))), 2)


def gated_feed_forward(x: torch.Tensor, gate_up: torch.Tensor, down: torch.Tensor, err: torch.Tensor) -> Optional[torch.Tensor]:
    """`tc_gemm` with the gate in its epilogue, where it has tiles for every SM, and the down projection."""
    if not (x.is_cuda and _untouched("tc_gemm", "tc_gemm_takes", "tc_gemm_is_persistent")) or own_tensor_core_products(x, down):
        return None
    return _counted(_host("tc_gemm").gated_feed_forward(x, gate_up, down, err), 1)


def matrix_memory(x: torch.Tensor, joint: torch.Tensor, gate_bias: torch.Tensor, norm: torch.Tensor, o_weight: torch.Tensor, ctx, state: torch.Tensor,
                  n_heads: int, dim: int, vdim: int, offsets: tuple, cap: float, eps: float, floor: float) -> Optional[torch.Tensor]:
    """`tc_gemm_tail`, `stabilized_gates`, `state_chunks`, `gated_group_norm` and the output projection, where the float32 columns ride on the
    projections' product and the step runs in chunks."""
    n = x.shape[0]
    if not (x.is_cuda and _untouched("tc_gemm_tail", "tail_rides", "stabilized_gates", "state_chunks", "state_chunks_take", "gated_group_norm", "linear_rows")
            and kernels.state_chunks_pay(n, dim, vdim, n_heads, ctx.max_q_len, ctx.n_seqs)) or own_tensor_core_products(x, o_weight):
        return None
    if not tail_rides(x, joint, 2 * n_heads * (dim + vdim)):
        return None
    records, each = kernels.state_chunk_records(n, ctx.n_seqs, n_heads, dim, vdim)
    return _counted(_host("tc_gemm", "recurrent", "state_chunks").matrix_memory(
        x, joint, gate_bias, norm, o_weight, state, ctx.cu_q, ctx.slots, ctx.err, n_heads, dim, vdim, ctx.max_q_len, records, each, *offsets,
        cap, eps, floor), 4)
