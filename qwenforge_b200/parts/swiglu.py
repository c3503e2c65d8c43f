"""SwiGLU feed-forward: (silu(x Wg^T) * (x Wu^T)) Wd^T, no biases (student_engine.py:523-527, :663-666).
Gate and up weights are concatenated by rows so that one product yields both halves."""
from __future__ import annotations

import torch

from .. import ops
from .base import FeedForward, PendingSums, TensorSpec
from .registry import register_part


class SwiGlu(FeedForward):
    """params: hidden_size, intermediate_size. tensors: gate_weight [I, W], up_weight [I, W], down_weight [W, I]."""

    def __init__(self, spec):
        super().__init__(spec)
        self.hidden = int(self.params["hidden_size"])
        self.inter = int(self.params["intermediate_size"])
        self.gate_up_weight = self.down_weight = None

    def tensor_specs(self):
        return [
            TensorSpec(self.file_name("gate_weight"), (self.inter, self.hidden)),
            TensorSpec(self.file_name("up_weight"), (self.inter, self.hidden)),
            TensorSpec(self.file_name("down_weight"), (self.hidden, self.inter)),
        ]

    def kernel_libraries(self, dtype):
        return {"activation"} | ({"gemm_f32"} if dtype == torch.float32 else {"skinny_gemm", "tc_gemm", "wide_gemm", "feed_forward"})

    def bind(self, tensors, dtype, device):
        self.gate_up_weight = torch.cat((tensors[self.file_name("gate_weight")], tensors[self.file_name("up_weight")]),
                                        dim=0).contiguous()
        self.down_weight = tensors[self.file_name("down_weight")]

    def step_weights(self):
        return [self.gate_up_weight, self.down_weight]

    def forward(self, x, ctx):
        if ctx is not None and x.dtype == torch.bfloat16:   # what follows, issued from native code
            out = ops.host.gated_feed_forward(x, self.gate_up_weight, self.down_weight, ctx.err)
            if out is not None:
                return out
        act = torch.empty((x.shape[0], self.inter), dtype=x.dtype, device=x.device)
        # Steps with tiles for every SM run gate/up with the gate in the product's epilogue on this library's
        # persistent tcgen05 kernel: measured at 2048 x 9728 x 896 it takes 27 microseconds where the library product
        # (30) and the gate kernel after it take 45, since the product's 40 MB of output are never written and read.
        own = x.dtype == torch.bfloat16 and self.inter % 8 == 0 and ops.tc_gemm_takes(x, self.gate_up_weight) and (
            ops.own_tensor_core_products(x, self.gate_up_weight)
            or ops.tc_gemm_is_persistent(ops.TC_SWIGLU, x.shape[0], 2 * self.inter))
        if own:
            ops.tc_gemm(ops.TC_SWIGLU, x, self.gate_up_weight, act, ctx.err if ctx is not None else None)
            return ops.linear(act, self.down_weight)
        gate_up = ops.linear(x, self.gate_up_weight)
        ops.swiglu(gate_up, act)
        return ops.linear(act, self.down_weight)

    # ---- the form for steps of up to 64 tokens that works on the residual stream in place: norm + gate/up + SwiGLU in
    # one kernel, down + residual in another. Each of the two products chooses its way for itself: gate/up by `ops.gate_product_way`,
    # down by `ops.residual_product_way`.
    def _ways(self, ctx):
        rows = ctx.n_tokens
        return ops.gate_product_way(rows, self.gate_up_weight), ops.residual_product_way(rows, self.down_weight)

    def fused_takes(self, ctx) -> bool:
        return (ctx.dtype == torch.bfloat16 and ctx.attention == "auto" and self.inter % 8 == 0
                and ctx.n_tokens <= ops.WIDE_MAX_ROWS and self._ways(ctx) != ("unfused", "unfused"))

    def leaves_sums(self, hidden, ctx) -> bool:
        """Whether `fused_forward` with nothing pending runs as one kernel and returns a `PendingSums`: where the model runs the layers."""
        return bool(ctx.step_memo) and "model.resolves_sums" in ctx.step_memo and ops.feed_forward_takes(hidden.shape[0], self.gate_up_weight, self.down_weight)

    def fused_forward(self, hidden, rms, ctx, delta=None):
        """Adds to the stream, or (`leaves_sums`) returns what is still to reach it."""
        if delta is None and self.leaves_sums(hidden, ctx):
            # the whole layer out of the SMs' shared memory, in one kernel; its output stands in rows of its own that all layers share
            key = ("swiglu.sums", tuple(hidden.shape))
            sums = ctx.step_memo.get(key)
            if sums is None:
                sums = ctx.step_memo[key] = torch.zeros_like(hidden)
            ops.feed_forward(hidden, rms[0], rms[1], self.gate_up_weight, self.down_weight, sums, ctx.err)
            return PendingSums(sums)
        gate_up, down = self._ways(ctx)
        act = torch.empty((hidden.shape[0], self.inter), dtype=torch.bfloat16, device=hidden.device)
        if gate_up == "skinny":
            if delta is not None:
                ops.residual_add(hidden, delta)
            ops.skinny_gemm(ops.EPI_SWIGLU, self.gate_up_weight, hidden=hidden, norm_weight=rms[0], eps=rms[1], out=act,
                            constants=True)
        else:
            x = torch.empty(hidden.shape, dtype=torch.bfloat16, device=hidden.device)
            ops.add_rms_norm(hidden, delta, rms[0], rms[1], x, constant_weight=True)   # the norm kernel adds the pending delta on its way
            if gate_up == "wide":
                ops.wide_gemm(ops.EPI_SWIGLU, self.gate_up_weight, x=x, out=act, err=ctx.err)
            else:
                ops.swiglu(ops.linear(x, self.gate_up_weight), act)
        if down == "skinny":
            ops.skinny_gemm(ops.EPI_RESIDUAL, self.down_weight, x=act, residual=hidden)
        elif down == "wide":
            ops.wide_gemm(ops.EPI_RESIDUAL, self.down_weight, x=act, residual=hidden, err=ctx.err)
        else:
            ops.residual_add(hidden, ops.linear(act, self.down_weight))
        return None


register_part("feed_forward", "swiglu", SwiGlu)
