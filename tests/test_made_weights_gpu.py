"""Norm weights and biases that the kernel directly ahead on the stream makes: the calls that take them read them behind that kernel,
although their own launch starts under its tail, unless the caller promises that they are constants."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def made_row(width, g):
    """(launch, row): a gate kernel over many rows, whose last row is what the next call is given."""
    from qwenforge_b200 import ops
    gu = torch.randn(6000, 2 * width, generator=g, device=DEV).bfloat16()
    out = torch.zeros(6000, width, dtype=torch.bfloat16, device=DEV)
    want = torch.nn.functional.silu(gu[-1, :width].double()) * gu[-1, width:].double()

    def launch():
        ops.swiglu(gu, out)
    return launch, out, want


@pytest.mark.parametrize("width", [896, 2048, 4096, 4100])
def test_norm(width):
    from qwenforge_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(width)
    launch, made, weight = made_row(width, g)
    hidden, out = torch.randn(8, width, generator=g, device=DEV), torch.empty(8, width, dtype=torch.bfloat16, device=DEV)
    want = hidden.double() * torch.rsqrt(hidden.double().square().mean(-1, keepdim=True) + 1e-6) * weight
    for _ in range(5):
        made.zero_()
        torch.cuda.synchronize()
        launch()
        ops.add_rms_norm(hidden, None, made[-1], 1e-6, out)
        # the weight and the result are each rounded to eight bits, float32 between
        assert bool(((out.double() - want).abs() <= want.abs() * (2.0 ** -7 + 2.0 ** -14) + 1e-30).all())
    settled = torch.empty_like(out)
    torch.cuda.synchronize()
    ops.add_rms_norm(hidden, None, made[-1], 1e-6, settled, constant_weight=True)
    assert torch.equal(settled, out)


@pytest.mark.parametrize("rows,n", [(1, 1024), (8, 1024), (16, 1024), (8, 40000)])   # one wave of blocks, and the ring
def test_few_rows_product(rows, n):
    from qwenforge_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(rows + n)
    k = 2048
    launch, made, weight = made_row(k, g)
    launch_bias, made_bias, bias = made_row(n if n < 4096 else 8, g)
    w = (torch.randn(n, k, generator=g, device=DEV) * k ** -0.5).bfloat16()
    hidden = torch.randn(rows, k, generator=g, device=DEV)
    out, settled = (torch.empty(rows, n, device=DEV) for _ in range(2))
    common = dict(hidden=hidden, norm_weight=made[-1], eps=1e-6)
    for _ in range(5):
        made.zero_()
        torch.cuda.synchronize()
        launch()
        ops.skinny_gemm(ops.EPI_PLAIN, w, out=out, **common)
        torch.cuda.synchronize()
        ops.skinny_gemm(ops.EPI_PLAIN, w, out=settled, constants=True, **common)
        assert torch.equal(out, settled)
    want = (hidden.double() * torch.rsqrt(hidden.double().square().mean(-1, keepdim=True) + 1e-6) * weight) @ w.double().T
    assert float((out.double() - want).norm() / want.norm()) < 2 ** -7      # (rows and weights rounded to eight bits)
    if n < 4096:
        x = hidden.bfloat16()
        for _ in range(5):
            made_bias.zero_()
            torch.cuda.synchronize()
            launch_bias()
            ops.skinny_gemm(ops.EPI_PLAIN, w, x=x, bias=made_bias[-1], out=out)
            torch.cuda.synchronize()
            ops.skinny_gemm(ops.EPI_PLAIN, w, x=x, bias=made_bias[-1], out=settled, constants=True)
            assert torch.equal(out, settled)
        want = x.double() @ w.double().T + bias
        assert float((out.double() - want).abs().max()) <= 2 ** -8 * float(bias.abs().max()) + 1e-4
