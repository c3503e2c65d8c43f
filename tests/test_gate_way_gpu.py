"""Which kernels make the gate and up product of a step of up to 64 token rows, at both sides of every line of the rule."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


# 0.5B's (17 MB) and 3B's (90 MB) weights, one on either side of 100 MB, 7B's (272 MB), and columns that no streamer takes
@pytest.mark.parametrize("rows,k,ways", [
    (9728, 896, {1: "skinny", 8: "skinny", 9: "wide", 16: "wide", 17: "unfused", 48: "unfused", 64: "unfused"}),
    (22016, 2048, {1: "skinny", 3: "skinny", 4: "wide", 8: "wide", 9: "unfused", 16: "unfused", 48: "unfused", 64: "unfused"}),
    (24400, 2048, {1: "skinny", 8: "wide", 9: "unfused", 64: "unfused"}), (24432, 2048, {1: "wide", 16: "wide", 64: "wide"}),
    (37888, 3584, {1: "wide", 8: "wide", 9: "wide", 64: "wide"}), (37888, 1404, {1: "unfused", 64: "unfused"})])
def test_the_rule(rows, k, ways):
    """Below 100 MB the tcgen05 streamer takes the place of the mma.sync one and of nothing else."""
    from qwenforge_b200 import ops
    weight = torch.empty(rows, k, dtype=torch.bfloat16, device=DEV)
    assert {m: ops.gate_product_way(m, weight) for m in ways} == ways


@pytest.mark.parametrize("rows", [1, 9, 16])
def test_gates_of_the_ways_are_float32s_own(rows):
    """Sums that are exact in any order, from gates far below zero (to -88.5: below -88.7 a float32 e^-z overflows) to far above: both
    streamers leave the same bits, those of the formula."""
    from qwenforge_b200 import ops
    inter, k = 4096, 64
    g = torch.Generator(device=DEV).manual_seed(rows)
    x, w = torch.zeros(rows, k, dtype=torch.bfloat16, device=DEV), torch.zeros(2 * inter, k, dtype=torch.bfloat16, device=DEV)
    x[:, 0], x[:, 1] = torch.linspace(1, 0.25, rows, device=DEV).bfloat16(), 1.0
    w[:inter, 0] = torch.cat((torch.linspace(-88.5, 40, inter // 2, device=DEV), 4 * torch.randn(inter // 2, generator=g, device=DEV))).bfloat16()
    w[inter:, 1] = torch.randn(inter, generator=g, device=DEV).bfloat16()
    outs = [torch.empty(rows, inter, dtype=torch.bfloat16, device=DEV) for _ in range(2)]
    ops.skinny_gemm(ops.EPI_SWIGLU, w, x=x, out=outs[0])
    ops.wide_gemm(ops.EPI_SWIGLU, w, x=x, out=outs[1])
    assert torch.equal(*outs)
    gate = x[:, :1].double() * w[:inter, 0].double()
    want = gate / (1 + torch.exp(-gate)) * w[inter:, 1].double()
    # one rounding to eight bits of a float32 number of a few roundings; no step smaller than bfloat16's 2^-133
    assert bool(((outs[1].double() - want).abs() <= want.abs() * (2.0 ** -8 + 2.0 ** -20) + 2.0 ** -133).all())
