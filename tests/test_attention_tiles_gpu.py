"""The tcgen05 prompt attention at sizes for which it takes one or two tiles a block and shares them among 1, 2, 4 or 8 blocks."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
CASES = [([200] * 6, 0, 14, 2, 64, 0), ([1024], 0, 14, 2, 64, 0), ([256], 8000, 14, 2, 64, 0), ([64], 3000, 14, 2, 64, 0),
         ([200], 2000, 14, 2, 64, 0), ([183, 275, 1, 246], 0, 14, 2, 64, 0), ([300, 17], 3000, 16, 2, 128, 0), ([512], 0, 16, 2, 128, 0),
         ([129, 5], 1215, 3, 1, 128, 0), ([300, 128], 700, 14, 2, 64, 150), ([2], 129, 6, 2, 128, 1000), ([130], 4000, 5, 5, 64, 3000),
         # prompts that small blocks take (three on an SM, two a tile), and their neighbours that they do not
         ([1153], 0, 16, 2, 64, 0), ([1500, 300, 1], 0, 14, 2, 64, 0), ([1409], 0, 14, 14, 64, 1100), ([3500], 0, 14, 2, 64, 0),
         ([1000], 0, 14, 2, 64, 0), ([1153], 64, 16, 2, 64, 0)]


@pytest.mark.parametrize("lens,before,heads,kv_heads,dim,window", CASES)
@pytest.mark.parametrize("with_sinks", [False, True])
def test_against_float64(lens, before, heads, kv_heads, dim, window, with_sinks):
    from qwenforge_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(sum(lens) + before)
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    totals = [n + before for n in lens] + [70]          # a padding entry of 70 rows stands last
    pages = [-(-t // 64) for t in totals[:-1]]
    storage = torch.randn(sum(pages), 2, kv_heads, 64, dim, generator=g, device=DEV).bfloat16()
    order, table, at = torch.randperm(sum(pages), generator=torch.Generator().manual_seed(1)).tolist(), [], 0
    for count in pages:
        table.append(order[at:at + count] + [-1] * (max(pages) - count))
        at += count
    rows = [*lens, 70]
    cu, pos = [0], []
    for n in rows:
        cu.append(cu[-1] + n)
        pos += range(before, before + n)
    q = (1.5 * torch.randn(cu[-1], heads * dim, generator=g, device=DEV)).bfloat16()
    out, err = torch.full_like(q, 7.0), ints([0])
    sinks = torch.randn(heads, generator=g, device=DEV) if with_sinks else None
    site, table_t = ops.KvSiteArgs(storage, ints(table), kv_heads, dim), ints(table)
    ops.attention_prefill_tc(q, out, ints(cu), ints(pos), ints([*range(len(lens)), -1]), site, heads, len(rows), max(rows), dim ** -0.5, window, err,
                             max_kv_len=max(totals), sinks=sinks)
    assert int(err) == 0 and not bool(out[cu[-2]:].any())
    for s, n in enumerate(lens):
        kv = storage[table_t[s, :pages[s]].long()].double().permute(1, 2, 0, 3, 4).reshape(2, kv_heads, -1, dim)[:, :, :totals[s]]
        i, j = torch.arange(before, totals[s], device=DEV)[:, None], torch.arange(totals[s], device=DEV)[None]
        hidden = (j > i) | (j <= i - window if window else torch.zeros_like(j > i))
        for h in sorted({0, heads // 2, heads - 1}):
            kvh = h // (heads // kv_heads)
            scores = (q[cu[s]:cu[s + 1]].view(n, heads, dim)[:, h].double() @ kv[0, kvh].T * dim ** -0.5).masked_fill(hidden, float("-inf"))
            if with_sinks:
                scores = torch.cat((scores, sinks[h].double().expand(n, 1)), dim=1)
            want = torch.softmax(scores, -1)[:, :totals[s]] @ kv[1, kvh]
            got = out[cu[s]:cu[s + 1]].view(n, heads, dim)[:, h].double()
            # weights and outputs are rounded to bfloat16 (2^-9 of each at most, independent: about 2^-9 of the norm)
            assert float((got - want).norm() / want.norm()) < 2 ** -8


@pytest.mark.parametrize("lens,before,heads,kv_heads,window", [([300] * 8, 0, 14, 2, 0), ([257, 130, 1] * 8, 0, 14, 14, 0), ([4100], 0, 14, 2, 256),
                                                              ([200] * 20, 70, 16, 4, 0), ([129, 300] * 9, 700, 12, 2, 0)])
def test_small_blocks_alone_and_in_pairs(lens, before, heads, kv_heads, window):
    """Steps of many tiles at head size 64, which small blocks take: a tile each below 16 pages or beyond two rounds of them, else in pairs."""
    test_against_float64(lens, before, heads, kv_heads, 64, window, True)


@pytest.mark.parametrize("n,before,heads,kv_heads,dim,window", [(300, 0, 5, 5, 64, 0), (300, 0, 3, 1, 128, 0), (700, 130, 6, 2, 64, 0), (64, 3000, 2, 2, 128, 0),
                                                               (400, 700, 4, 4, 64, 150), (400, 690, 4, 4, 128, 200), (130, 4000, 5, 5, 64, 3000), (1153, 0, 16, 2, 64, 0)])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_values_of_pages_that_a_tile_does_not_see(n, before, heads, kv_heads, dim, window, bad):
    """A value that is not finite reaches no tile of 128 rows none of whose rows sees its page."""
    from qwenforge_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(n + before)
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    pages = -(-(n + before) // 64)
    storage = torch.randn(pages, 2, kv_heads, 64, dim, generator=g, device=DEV).bfloat16()
    q, err = torch.randn(n, heads * dim, generator=g, device=DEV).bfloat16(), ints([0])
    site = ops.KvSiteArgs(storage, ints([list(range(pages))]), kv_heads, dim)

    def run():
        out = torch.empty_like(q)
        ops.attention_prefill_tc(q, out, ints([0, n]), ints(list(range(before, before + n))), ints([0]), site, heads, 1, n, dim ** -0.5, window, err,
                                 max_kv_len=n + before)
        return out
    want = run()
    seen = []
    for t0 in range(0, n, 128):
        first, last = before + t0, before + min(t0 + 128, n) - 1
        seen.append(((max(0, first - window + 1) if window else 0) // 64, last // 64))
    for page in range(max(0, pages - 12), pages):
        held = storage[page, 1].clone()
        storage[page, 1] = bad
        got = run()
        storage[page, 1] = held
        for i, (lo, hi) in enumerate(seen):
            if not lo <= page <= hi:
                assert torch.equal(got[128 * i:128 * i + 128], want[128 * i:128 * i + 128]), (page, i)
    assert int(err) == 0


@pytest.mark.parametrize("n,heads,kv_heads,dim", [(300, 4, 2, 128), (130, 3, 3, 64), (1153, 16, 2, 64)])
@pytest.mark.parametrize("scale", [0.0, -0.05, 0.05])
def test_any_scale(n, heads, kv_heads, dim, scale):
    """A scale of zero weighs all keys alike, one below zero prefers the unlike ones."""
    from qwenforge_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(n)
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    pages = -(-n // 64)
    storage = torch.randn(pages, 2, kv_heads, 64, dim, generator=g, device=DEV).bfloat16()
    q, err = torch.randn(n, heads * dim, generator=g, device=DEV).bfloat16(), ints([0])
    out, site = torch.empty_like(q), ops.KvSiteArgs(storage, ints([list(range(pages))]), kv_heads, dim)
    ops.attention_prefill_tc(q, out, ints([0, n]), ints(list(range(n))), ints([0]), site, heads, 1, n, scale, 0, err, max_kv_len=n)
    kv = storage.double().permute(1, 2, 0, 3, 4).reshape(2, kv_heads, -1, dim)[:, :, :n].repeat_interleave(heads // kv_heads, 1)
    scores = torch.einsum("ihd,hjd->hij", q.view(n, heads, dim).double(), kv[0]) * scale
    want = torch.softmax(scores.masked_fill(torch.ones(n, n, dtype=torch.bool, device=DEV).triu(1), float("-inf")), -1) @ kv[1]
    got = out.view(n, heads, dim).transpose(0, 1).double()
    assert int(err) == 0 and float((got - want).norm() / want.norm()) < 2 ** -8   # (weights and outputs rounded to bfloat16)


def test_which_kernel_a_step_takes():
    from qwenforge_b200 import ops
    from qwenforge_b200.parts.attention import prefill_attention
    assert prefill_attention(64, 2, 128) is ops.attention_prefill_tc and prefill_attention(128, 500, 4000, 200) is ops.attention_prefill_tc
    assert prefill_attention(64, 100, 100) is ops.attention_prefill and prefill_attention(32, 500, 500) is ops.attention_prefill
    assert prefill_attention(64, 500, 4000, 100) is ops.attention_prefill


def test_many_short_sequences_keep_the_smaller_tiles():
    """Where both kernels were measured, the rule names the faster one."""
    from qwenforge_b200 import ops
    from qwenforge_b200.parts.attention import prefill_attention
    pick = lambda dim, heads, kv, seqs, tokens, before: prefill_attention(dim, seqs * tokens, before + tokens, max_q_len=tokens, n_seqs=seqs,
                                                                         n_heads=heads, kv_heads=kv) is ops.attention_prefill_tc
    assert not pick(64, 14, 2, 64, 2, 127) and not pick(64, 14, 2, 64, 2, 1000) and not pick(64, 14, 14, 64, 16, 1000)
    assert not pick(128, 28, 4, 64, 8, 127) and not pick(64, 14, 2, 16, 2, 127) and not pick(128, 4, 4, 64, 16, 127)
    assert pick(128, 28, 4, 64, 8, 1000) and pick(64, 14, 2, 16, 2, 1000) and pick(64, 14, 2, 64, 100, 500) and pick(64, 14, 2, 4, 32, 500)
