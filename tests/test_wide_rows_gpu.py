"""The tcgen05 weight streamer (csrc/wide_gemm.cu) on tiles of fewer than 128 weight rows, which heavy weights take: sizes whose last tile is
ragged, whose rows per tile are odd, whose K is no whole slab, split along K and not."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("m", [1, 16, 17, 64])
@pytest.mark.parametrize("n,k", [(2048, 4104), (3601, 2408), (7000, 1224), (1030, 8200), (40000, 216)])
def test_into_the_stream(m, n, k):
    from qwenforge_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(m + n)
    assert n * k * 2 >= 16 << 20
    x = torch.randn(m, k, generator=g, device=DEV).bfloat16()
    w = (torch.randn(n, k, generator=g, device=DEV) * k ** -0.5).bfloat16()
    before, err = torch.randn(m, n, generator=g, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    got = before.clone()
    ops.wide_gemm(ops.EPI_RESIDUAL, w, x=x, residual=got, err=err)
    want = before.double() + x.double() @ w.double().T
    slack = (x.double().abs() @ w.double().abs().T) * k * 2.0 ** -24 + want.abs() * 2.0 ** -23   # float32 sums of k products, one addition
    assert int(err) == 0 and bool(((got.double() - want).abs() <= slack + 1e-30).all())
    alone = before[m - 1:].clone()
    ops.wide_gemm(ops.EPI_RESIDUAL, w, x=x[m - 1:].clone(), residual=alone, err=err)
    again = before.clone()
    ops.wide_gemm(ops.EPI_RESIDUAL, w, x=x, residual=again, err=err)
    assert torch.equal(again, got)                             # the same sums in the same order, run after run
    if m <= 16:
        assert torch.equal(alone[0], got[m - 1])               # and, with as many token columns, beside any other rows


@pytest.mark.parametrize("m", [1, 16, 33, 64])
@pytest.mark.parametrize("inter,k", [(4864, 896), (11008, 2048), (2601, 1640), (19001, 232)])
def test_gate_and_up(m, inter, k):
    from qwenforge_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(m + inter)
    x = torch.randn(m, k, generator=g, device=DEV).bfloat16()
    w = (torch.randn(2 * inter, k, generator=g, device=DEV) * k ** -0.5).bfloat16()
    out, err = torch.full((m + 1, inter), 7.0, dtype=torch.bfloat16, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    ops.wide_gemm(ops.EPI_SWIGLU, w, x=x, out=out[:m], err=err)
    sums, slack = x.double() @ w.double().T, (x.double().abs() @ w.double().abs().T) * k * 2.0 ** -24
    gate, up = sums[:, :inter], sums[:, inter:]
    want = gate * torch.sigmoid(gate) * up
    # |d silu| <= 1.1; the gate's exponential and division are the hardware's (2^-20); one rounding to eight bits
    slack = 1.1 * (slack[:, :inter] * (up.abs() + 1) + slack[:, inter:] * (gate.abs() + 1)) + want.abs() * 2.0 ** -20
    assert int(err) == 0 and bool(((out[:m].double() - want).abs() <= want.abs() * 2.0 ** -8 + slack + 1e-30).all())
    assert bool((out[m] == 7).all())


@pytest.mark.parametrize("n,k", [(6656, 1536), (2048, 11008), (3584, 18944), (1030, 8200), (7000, 1224)])
def test_a_row_has_the_same_bits_beside_any_number_of_others(n, k):
    """The split of K, which decides the order of a sum, follows from the weight's shape and not from the step's rows."""
    from qwenforge_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(n)
    x, w = torch.randn(64, k, generator=g, device=DEV).bfloat16(), (torch.randn(n, k, generator=g, device=DEV) * k ** -0.5).bfloat16()
    stream, err = torch.randn(64, n, generator=g, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    results = []
    for m in (1, 16, 17, 33, 64):
        got = stream[:m].clone()
        ops.wide_gemm(ops.EPI_RESIDUAL, w, x=x[:m], residual=got, err=err)
        results.append(got)
    assert int(err) == 0
    for got in results[:-1]:
        assert torch.equal(got, results[-1][:got.shape[0]])
