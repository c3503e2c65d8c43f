"""The float32 path's tile kernels at the edges of their tiles: the product against its own single rows, the attention against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("m", [17, 63, 64, 65, 127, 129, 300])
@pytest.mark.parametrize("n,k", [(64, 16), (65, 20), (130, 33), (6200, 48), (19100, 17)])
def test_products_keep_the_order_of_a_single_chain(m, n, k):
    """Every element is one chain of fused multiply-adds over k, whatever the tile: the bits of the kernel of few rows."""
    from qwenforge_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(m + n + k)
    x, w, b = torch.randn(m, k, generator=g, device=DEV), torch.randn(n, k, generator=g, device=DEV), torch.randn(n, generator=g, device=DEV)
    out, rows = torch.empty(m, n, device=DEV), torch.empty(m, n, device=DEV)
    ops.gemm_f32(x, w, b, out)
    for at in range(0, m, 16):
        ops.gemm_f32(x[at:at + 16], w, b, rows[at:at + 16])
    assert torch.equal(out, rows)
    wide = torch.zeros(m, k + 3, device=DEV)      # rows that no 16-byte load can address
    wide[:, 1:k + 1] = x
    ops.gemm_f32(wide[:, 1:k + 1], w, b, out)
    assert torch.equal(out, rows)


# every size of tile, with ragged last tiles both ways, a K of no whole piece of 16 and one below it
@pytest.mark.parametrize("m,n,k,tile", [(1031, 4865, 33, 96128), (1031, 9728, 20, 96128), (1057, 22016, 17, 96128), (300, 6200, 48, 128128), (700, 1025, 16, 96064),
                                        (65, 19100, 35, 96064), (257, 5000, 9, 64064), (70, 130, 40, 32064)])
def test_every_tile_keeps_the_order_of_a_single_chain(m, n, k, tile):
    import ctypes
    from qwenforge_b200 import ops
    from qwenforge_b200.csrc import library
    assert library("gemm_f32").qf_gemm_f32_tile(ctypes.c_int(m), ctypes.c_int(n)) == tile
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


@pytest.mark.parametrize("dim,heads,kv_heads,window", [(64, 14, 2, 0), (128, 4, 4, 0), (64, 4, 1, 70), (128, 2, 1, 1)])
def test_attention_tiles(dim, heads, kv_heads, window):
    from qwenforge_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(dim + heads + window)
    spans = [(0, 1), (0, 64), (0, 65), (63, 130), (200, 2), (0, 40)]     # (tokens before, tokens of the step)
    slots = [5, 3, 0, 1, 4, -1]
    pages_each, n_slots = 5, 6
    order = torch.randperm(n_slots * pages_each, generator=torch.Generator().manual_seed(1)).to(torch.int32).view(n_slots, pages_each).to(DEV)
    storage = torch.randn(n_slots * pages_each, 2, kv_heads, 64, dim, generator=g, device=DEV)
    cu, pos, total = [0], [], 0
    for start, n in spans:
        cu.append(cu[-1] + n)
        pos += range(start, start + n)
    for (start, n), slot in zip(spans, slots):   # what a sequence has not written yet is no number
        if slot >= 0:
            for p in range(start + n, pages_each * 64):
                storage[order[slot, p // 64], :, :, p % 64] = float("nan")
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    q, out, err = torch.randn(cu[-1], heads * dim, generator=g, device=DEV), torch.empty(cu[-1], heads * dim, device=DEV), ints([0])
    site = ops.KvSiteArgs(storage, order, kv_heads, dim)
    ops.attention_generic(q, out, ints(cu), ints(pos), ints(slots), site, heads, len(spans), max(n for _, n in spans), dim ** -0.5, window, err)
    assert int(err) == 0
    for (start, n), slot, first in zip(spans, slots, cu):
        got = out[first:first + n].view(n, heads, dim).double()
        if slot < 0:
            assert not bool(got.any())
            continue
        kv = storage[order[slot].long()].double().permute(1, 2, 0, 3, 4).reshape(2, kv_heads, -1, dim)[:, :, :start + n].repeat_interleave(heads // kv_heads, 1)
        scores = torch.einsum("nhd,hkd->hnk", q[first:first + n].view(n, heads, dim).double(), kv[0]) * dim ** -0.5
        i, j = torch.arange(start, start + n, device=DEV)[:, None], torch.arange(start + n, device=DEV)[None]
        scores = scores.masked_fill((j > i) | ((j <= i - window) if window else torch.zeros_like(j > i)), float("-inf"))
        want = torch.einsum("hnk,hkd->nhd", torch.softmax(scores, -1), kv[1])
        # scores of size up to about 5 carry a rounding of 128 x 2^-24 of that at worst, the weights and sums as much again
        assert float((got - want).abs().max()) < 2e-5 * float(want.abs().max())
    # a row does not see what else is in the step
    alone = torch.empty(130, heads * dim, device=DEV)
    ops.attention_generic(q[cu[3]:cu[4]].contiguous(), alone, ints([0, 130]), ints(pos[cu[3]:cu[4]]), ints([slots[3]]), site, heads, 1, 130, dim ** -0.5, window, err)
    assert torch.equal(alone, out[cu[3]:cu[4]])


def test_a_value_that_is_not_finite_reaches_no_earlier_row():
    from qwenforge_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(3)
    dim, heads, n, bad = 64, 2, 100, 70
    storage = torch.randn(2, 2, 1, 64, dim, generator=g, device=DEV)
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    site = ops.KvSiteArgs(storage, ints([[0, 1]]), 1, dim)
    q, err, outs = torch.randn(n, heads * dim, generator=g, device=DEV), ints([0]), []
    for value in (1.0, float("inf"), float("nan")):
        storage[1, 1, 0, bad - 64, 5] = value
        out = torch.empty_like(q)
        ops.attention_generic(q, out, ints([0, n]), ints(list(range(n))), ints([0]), site, heads, 1, n, dim ** -0.5, 0, err)
        outs.append(out.view(n, heads, dim))
    for out in outs[1:]:
        assert torch.equal(out[:bad], outs[0][:bad]) and not bool(torch.isfinite(out[bad:, :, 5]).any())


@pytest.mark.parametrize("heads,kv_heads,dim", [(14, 2, 64), (3, 3, 128), (8, 2, 128), (40, 2, 64)])
def test_short_sequences_alone_and_beside_long_ones(heads, kv_heads, dim):
    """Rows in tiles of 16 and of 64 (a step of few tokens, the same beside a longer sequence): the same bits."""
    from qwenforge_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(heads)
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    storage = torch.randn(20, 2, kv_heads, 64, dim, generator=g, device=DEV)
    site, err = ops.KvSiteArgs(storage, ints([list(range(4 * i, 4 * i + 4)) for i in range(5)]), kv_heads, dim), ints([0])
    spans = [(130, 2), (50, 150), (0, 5), (200, 1), (0, 1)]
    cu, pos = [0], []
    for start, n in spans:
        cu.append(cu[-1] + n)
        pos += range(start, start + n)
    q = torch.randn(cu[-1], heads * dim, generator=g, device=DEV)
    out = torch.empty_like(q)
    ops.attention_generic(q, out, ints(cu), ints(pos), ints([0, 1, 2, 3, 4]), site, heads, 5, 150, dim ** -0.5, 0, err)
    for s, (start, n) in enumerate(spans):
        rows = slice(cu[s], cu[s + 1])
        alone = torch.empty(n, heads * dim, device=DEV)
        ops.attention_generic(q[rows].contiguous(), alone, ints([0, n]), ints(pos[rows]), ints([s]), site, heads, 1, n, dim ** -0.5, 0, err)
        assert torch.equal(alone, out[rows])
    assert int(err) == 0


@pytest.mark.parametrize("heads,kv_heads,dim,tokens", [(14, 2, 64, 70), (14, 2, 64, 676), (14, 2, 64, 677), (14, 2, 64, 1360), (14, 2, 64, 2030), (8, 2, 128, 1184),
                                                       (8, 2, 128, 1185), (3, 3, 128, 33)])
def test_a_sequence_alone_in_smaller_tiles_and_alternating_waves(heads, kv_heads, dim, tokens):
    """Alone a sequence takes tiles of 32 rows where 64 leave SMs idle, and waves of alternating order; beside another neither: the same bits."""
    from qwenforge_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(tokens)
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    pages = (tokens + 63) // 64 + 1
    storage = torch.randn(pages + 1, 2, kv_heads, 64, dim, generator=g, device=DEV)
    table = torch.full((2, pages), -1, dtype=torch.int32)
    table[0], table[1, 0] = torch.arange(pages), pages
    site, err = ops.KvSiteArgs(storage, table.to(DEV), kv_heads, dim), ints([0])
    pos = list(range(11, 11 + tokens))
    q = torch.randn(tokens + 1, heads * dim, generator=g, device=DEV)
    both, alone = torch.empty_like(q), torch.full((tokens, heads * dim), float("nan"), device=DEV)
    ops.attention_generic(q, both, ints([0, tokens, tokens + 1]), ints(pos + [0]), ints([0, 1]), site, heads, 2, tokens, dim ** -0.5, 0, err)
    ops.attention_generic(q[:tokens].contiguous(), alone, ints([0, tokens]), ints(pos), ints([0]), site, heads, 1, tokens, dim ** -0.5, 0, err)
    assert int(err) == 0 and torch.equal(alone, both[:tokens])


@pytest.mark.parametrize("rows,inter", [(1, 4), (3, 20), (700, 1028), (1031, 4864)])
def test_the_gate_four_numbers_at_a_time(rows, inter):
    """Rows on 16-byte boundaries and the same rows off them (the kernel of single numbers): the same bits, also of what is not finite."""
    from qwenforge_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(rows)
    gu = 4 * torch.randn(rows, 2 * inter, generator=g, device=DEV)
    gu[0, :4] = torch.tensor([float("inf"), float("-inf"), float("nan"), -200.0], device=DEV)
    out, off = torch.empty(rows, inter, device=DEV), torch.empty(1 + rows * inter, device=DEV)[1:].view(rows, inter)
    ops.swiglu(gu, out)
    ops.swiglu(gu, off)
    assert torch.equal(out.view(torch.int32), off.view(torch.int32).contiguous())
    want = torch.nn.functional.silu(gu[:, :inter].double()) * gu[:, inter:].double()
    fine = torch.isfinite(want) & (want.abs() > 1e-30)
    # expf within 2 units, a sum, a quotient and a product: below eight roundings of 2^-24
    assert bool(((out.double() - want).abs() <= 8 * 2.0 ** -24 * want.abs())[fine].all())
