"""Decode attention of long runs: more pages of a warp than it holds numbers of."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


# whole sequences in one run: 32 pages of 64 positions a warp (8 warps at heads of up to 64, 4 beyond), one position and one page more, 40 pages
@pytest.mark.parametrize("heads,kv,dim,lengths", [(7, 1, 64, [16384, 16385, 16449, 20500, 40]), (4, 2, 128, [8192, 8193, 8257, 10300, 64]),
                                                  (4, 1, 32, [16384, 16449, 20500]), (4, 1, 96, [8192, 8257, 10300])])
def test_against_float64(heads, kv, dim, lengths):
    from qwenforge_b200 import ops
    from qwenforge_b200.measure import Pages
    g = torch.Generator(device=DEV).manual_seed(dim)
    n, ints = len(lengths), lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    pages, q = Pages(n, max(lengths), kv, dim, DEV), torch.randn(n, heads * dim, generator=g, device=DEV).bfloat16()
    pages.storage.normal_(generator=g)
    out, err, scratch = torch.empty_like(q), ints([0]), ops.DecodeScratch(torch.device(DEV))
    cu, pos, slots = ints(list(range(n + 1))), ints([x - 1 for x in lengths]), ints(list(range(n)))
    plan = ops.attention_decode_plan(cu, pos, slots, kv, dim, heads, n, 0, 1, scratch)
    ops.attention_decode(q, out, cu, pos, slots, pages.args(), heads, n, 2 * dim ** -0.5, 0, 1, scratch, err, plan)
    assert int(err) == 0
    for i, length in enumerate(lengths):
        held = pages.storage[pages.table[i].long()].double().permute(1, 2, 0, 3, 4).reshape(2, kv, -1, dim)[:, :, :length]
        keys, values = held.repeat_interleave(heads // kv, dim=1)
        weights = torch.softmax(torch.einsum("hd,hkd->hk", q[i].view(heads, dim).double(), keys) * 2 * dim ** -0.5, dim=-1)
        want = torch.einsum("hk,hkd->hd", weights, values).reshape(-1)
        # weights and output are rounded to eight bits: 2^-9 each at worst
        assert float((out[i].double() - want).norm()) < 2.0 ** -8 * float(want.norm())
