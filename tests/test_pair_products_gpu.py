"""The persistent tcgen05 product on pairs of SMs (csrc/tc_gemm.cu) at the edges of its tiles: one row or one piece of eight columns
more or less than whole tiles, a K below one stage, of whole stages and of more than the ring holds, both widths of tiles."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("gated,m,cols,k,columns", [
    (True, 905, 4864, 896, 192), (True, 1024, 4864, 64, 192), (True, 1025, 4872, 8, 256), (True, 513, 3848, 456, 192),
    (True, 2049, 2440, 520, 256), (False, 2047, 4864, 448, 192), (False, 1793, 2568, 392, 192), (False, 4100, 2568, 904, 256)])
def test_edges_of_pair_tiles(gated, m, cols, k, columns):
    from qwenforge_b200 import ops
    from qwenforge_b200.csrc import library
    g = torch.Generator(device=DEV).manual_seed(m)
    x = torch.randn(m, k, generator=g, device=DEV).bfloat16()
    w = (torch.randn(2 * cols if gated else cols, k, generator=g, device=DEV) * k ** -0.5).bfloat16()
    epilogue = ops.TC_SWIGLU if gated else ops.TC_PLAIN
    assert ops.tc_gemm_is_persistent(epilogue, m, w.shape[0])
    assert library("tc_gemm").qf_tc_gemm_pair_columns(ctypes.c_int(epilogue), ctypes.c_int(m), ctypes.c_int(w.shape[0])) == columns
    rows = torch.full((m + 2, cols + 16), 7.0, dtype=torch.bfloat16, device=DEV)   # what lies around the result stays as it is
    err = torch.zeros(1, dtype=torch.int32, device=DEV)
    ops.tc_gemm(epilogue, x, w, rows[1:m + 1, 8:cols + 8], err)
    sums, most = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    want, slack = sums, most * k * 2.0 ** -24
    if gated:   # |d silu| <= 1.1, so a sum's error counts 1.1 times the other half's size
        gate, up = sums[:, :cols], sums[:, cols:]
        want = gate * torch.sigmoid(gate) * up
        slack = 1.1 * (slack[:, :cols] * (up.abs() + 1) + slack[:, cols:] * (gate.abs() + 1)) + want.abs() * 2.0 ** -20
    got = rows[1:m + 1, 8:cols + 8].double()
    assert int(err) == 0
    assert bool(((got - want).abs() <= want.abs() * 2.0 ** -8 + slack + 1e-30).all())   # float32 sums, rounded once to eight bits
    assert bool((rows[0] == 7).all() and (rows[-1] == 7).all() and (rows[:, :8] == 7).all() and (rows[:, -8:] == 7).all())


# every width of tiles (64, 128, 192 and 256 columns of heads of 64; 128 and 256 of heads of 128): ragged rows, columns and K, rows without
# a slot, a cache that is not written, no rotation, no bias
@pytest.mark.parametrize("m,heads,kv_heads,dim,k,rotated,biased", [
    (301, 14, 2, 64, 896, True, True), (2047, 14, 2, 64, 72, True, True), (3001, 14, 2, 64, 136, True, False), (4601, 12, 2, 64, 64, True, True),
    (257, 5, 1, 64, 8, False, True), (300, 16, 2, 128, 200, True, True), (1537, 16, 2, 128, 1032, True, True), (130, 3, 1, 128, 64, False, False)])
def test_queries_keys_and_values_of_pairs(m, heads, kv_heads, dim, k, rotated, biased):
    from qwenforge_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(m)
    n, first = (heads + 2 * kv_heads) * dim, [700, 0, 63]
    lengths = [m - m // 3 - 40, 40, m // 3]                    # three sequences, the second one without a slot
    x = torch.randn(m, k, generator=g, device=DEV).bfloat16()
    w = (torch.randn(n, k, generator=g, device=DEV) * k ** -0.5).bfloat16()
    bias = torch.randn(n, generator=g, device=DEV).bfloat16() if biased else None
    inv = 1e6 ** (-torch.arange(0, dim, 2, device=DEV).float() / dim) if rotated else None
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    seq = ints(sum(([i] * c for i, c in enumerate(lengths)), []))
    pos = ints(sum((list(range(f, f + c)) for f, c in zip(first, lengths)), []))
    pages = 2 * (-(-(700 + m) // 64))
    table = torch.randperm(pages, generator=g, device=DEV).int().view(2, -1).contiguous()
    storage = torch.full((pages, 2, kv_heads, 64, dim), 7.0, dtype=torch.bfloat16, device=DEV)
    site, slots, err = ops.KvSiteArgs(storage, table, kv_heads, dim), ints([1, -1, 0]), ints([0])
    q = torch.full((m, heads * dim), 7.0, dtype=torch.bfloat16, device=DEV)
    assert ops.qkv_product_takes(x, w, dim if rotated else 0, site)
    ops.qkv_product(x, w, bias, inv, seq, pos, slots, heads, q, site, True, err)
    want = x.double() @ w.double().T
    slack = (x.double().abs() @ w.double().abs().T + 1) * k * 2.0 ** -24 + want.abs() * 2.0 ** -8   # (sums rounded to eight bits before the bias)
    want = want + (bias.double() if biased else 0)
    want, slack = want.view(m, -1, dim).clone(), slack.view(m, -1, dim)
    if rotated:
        angle = (pos.float()[:, None] * inv).double()[:, None]
        cos, sin, turned = angle.cos(), angle.sin(), want[:, :heads + kv_heads]
        a, b = turned[..., :dim // 2].clone(), turned[..., dim // 2:].clone()
        turned[..., :dim // 2], turned[..., dim // 2:] = a * cos - b * sin, b * cos + a * sin
        slack = slack + slack.roll(dim // 2, -1) + 2.0 ** -21 * (want.abs() + want.roll(dim // 2, -1).abs())   # (angles rounded to float32)
    close = lambda got, want, slack: bool(((got.double() - want).abs() <= want.abs() * 2.0 ** -8 + slack + 1e-30).all())
    assert int(err) == 0
    assert close(q.view(m, heads, dim), want[:, :heads], slack[:, :heads])
    written = torch.zeros(pages, 64, dtype=torch.bool, device=DEV)
    at = table[slots[seq].clamp(min=0).long(), (pos // 64).long()].long()
    held = (seq != 1).nonzero()[:, 0]
    written[at[held], (pos % 64).long()[held]] = True
    got = storage[at, :, :, (pos % 64).long()].reshape(m, 2 * kv_heads, dim)
    assert close(got[held], want[held, heads:], slack[held, heads:])
    assert bool((storage.permute(0, 3, 1, 2, 4)[~written] == 7).all())
    before, again = storage.clone(), torch.empty_like(q)
    ops.qkv_product(x, w, bias, inv, seq, pos, slots, heads, again, site, False, err)   # the queries alone
    assert torch.equal(before, storage) and torch.equal(again, q) and int(err) == 0
    table[0, 0] = -1                                           # the third sequence's first page is not held
    ops.qkv_product(x, w, bias, inv, seq, pos, slots, heads, again, site, True, err)
    assert torch.equal(before, storage) and torch.equal(again, q) and int(err) == ops.ERR_NO_PAGE


@pytest.mark.parametrize("m,heads,kv_heads,dim,rotated,biased", [(301, 14, 2, 64, True, True), (2047, 14, 2, 64, True, False), (600, 16, 2, 128, True, True),
                                                                 (130, 3, 1, 128, False, True)])
def test_the_bits_of_product_and_rotation(m, heads, kv_heads, dim, rotated, biased):
    """Whole numbers, whose sums are exact in any order: queries, keys and values are those of the stored product with the rotation
    kernel behind it, bit for bit, at positions far out as well."""
    from qwenforge_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(m)
    n, k = (heads + 2 * kv_heads) * dim, 264
    x, w = (torch.randint(-9, 10, shape, generator=g, device=DEV).bfloat16() for shape in ((m, k), (n, k)))
    bias = torch.randn(n, generator=g, device=DEV).bfloat16() if biased else None
    inv = 1e6 ** (-torch.arange(0, dim, 2, device=DEV).float() / dim) if rotated else None
    first = 40000
    pages = -(-(first + m) // 64)
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    seq, pos, slots, err = ints([0] * m), ints(list(range(first, first + m))), ints([0]), ints([0])
    table = torch.full((1, pages), -1, dtype=torch.int32)
    table[0, first // 64:] = torch.arange(pages - first // 64)
    results = []
    for own in (True, False):
        storage = torch.zeros(pages - first // 64, 2, kv_heads, 64, dim, dtype=torch.bfloat16, device=DEV)
        site, q = ops.KvSiteArgs(storage, table.to(DEV), kv_heads, dim), torch.empty(m, heads * dim, dtype=torch.bfloat16, device=DEV)
        if own:
            ops.qkv_product(x, w, bias, inv, seq, pos, slots, heads, q, site, True, err)
        else:
            ops.rope_cache_write(ops.linear(x, w), seq, pos, slots, inv, dim if rotated else 0, heads, q, site, True, err, bias=bias)
        results.append((q, storage))
    assert int(err) == 0 and all(torch.equal(a, b) for a, b in zip(*results))

@pytest.mark.parametrize("m,n,extra,k", [(65, 2688, 14, 896), (257, 264, 1, 72), (300, 248, 32, 8), (2049, 2560, 2, 136), (700, 1536, 40, 640)])
def test_columns_that_stay_float32(m, n, extra, k):
    """The tail of a product's columns: inside the last tile, across its border, alone in a tile of its own."""
    from qwenforge_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(m)
    x = torch.randn(m, k, generator=g, device=DEV).bfloat16()
    w = (torch.randn(n + extra, k, generator=g, device=DEV) * k ** -0.5).bfloat16()
    out, tail = torch.full((m + 1, n + 8), 7.0, dtype=torch.bfloat16, device=DEV), torch.full((m + 1, extra), 7.0, device=DEV)
    err = torch.zeros(1, dtype=torch.int32, device=DEV)
    ops.tc_gemm_tail(x, w, out[:m, :n], tail[:m], err)
    want, slack = x.double() @ w.double().T, (x.double().abs() @ w.double().abs().T) * k * 2.0 ** -24
    got = torch.cat((out[:m, :n].double(), tail[:m].double()), dim=1)
    round_off = torch.full((n + extra,), 2.0 ** -8, dtype=torch.float64, device=DEV)
    round_off[n:] = 0
    assert int(err) == 0 and bool(((got - want).abs() <= want.abs() * round_off + slack + 1e-30).all())
    assert bool((out[m] == 7).all() and (out[:, n:] == 7).all() and (tail[m] == 7).all())


@pytest.mark.parametrize("m,cols,columns", [(2047, 4861, 192), (1793, 2561, 192), (4100, 2564, 256), (4100, 2567, 256), (100, 77, 0)])
def test_columns_that_are_no_whole_pieces(m, cols, columns):
    """A last piece of one to seven columns: they are the product's, what stands behind them in the rows' padding stays as it is."""
    from qwenforge_b200 import ops
    from qwenforge_b200.csrc import library
    g = torch.Generator(device=DEV).manual_seed(cols)
    x, w = torch.randn(m, 72, generator=g, device=DEV).bfloat16(), (torch.randn(cols, 72, generator=g, device=DEV) / 8).bfloat16()
    assert ops.tc_gemm_is_persistent(ops.TC_PLAIN, m, cols) == (columns > 0)
    assert columns == 0 or library("tc_gemm").qf_tc_gemm_pair_columns(ctypes.c_int(ops.TC_PLAIN), ctypes.c_int(m), ctypes.c_int(cols)) == columns
    rows = torch.full((m, cols // 8 * 8 + 16), 7.0, dtype=torch.bfloat16, device=DEV)
    err = torch.zeros(1, dtype=torch.int32, device=DEV)
    ops.tc_gemm(ops.TC_PLAIN, x, w, rows[:, :cols], err)
    want = x.double() @ w.double().T
    slack = (x.double().abs() @ w.double().abs().T) * 72 * 2.0 ** -24
    assert int(err) == 0 and bool(((rows[:, :cols].double() - want).abs() <= want.abs() * 2.0 ** -8 + slack + 1e-30).all())
    assert bool((rows[:, cols:] == 7).all())


def test_where_the_qkv_product_on_pairs_pays():
    """Both sides of the rule's lines: rows, pairs at work, and a K that is long for the tiles' columns."""
    from qwenforge_b200 import ops
    pays = lambda m, n, k, dim: ops.qkv_product_pays(m, torch.empty(n, k, dtype=torch.bfloat16, device=DEV), dim)
    assert all(pays(m, 1152, 896, 64) for m in (1, 64, 900, 8192)) and pays(64, 1536, 1280, 64) and pays(5, 320, 192, 64)
    assert not any(pays(m, 512, 4096, 64) for m in (1, 64, 900, 2048)) and not pays(64, 512, 1024, 64) and not pays(300, 1024, 2048, 64)
    assert not pays(900, 1024, 2048, 64) and pays(900, 1152, 1536, 64) and not pays(2048, 512, 3072, 64) and pays(4096, 512, 3072, 64)
    assert pays(7358, 2560, 2048, 128) and not pays(2048, 2560, 2048, 128) and not pays(512, 2560, 2048, 128) and pays(513, 2560, 2048, 128)
    assert not pays(1300, 1280, 4096, 128) and pays(3000, 1280, 4096, 128) and not pays(64, 2304, 2048, 64) and pays(900, 2304, 2048, 64)


def test_where_the_float32_columns_ride():
    """Both sides of the rule's lines: rows, a long K, columns that are few beside K."""
    from qwenforge_b200 import ops
    rides = lambda m, n, extra, k: ops.tail_rides(torch.empty(m, k, dtype=torch.bfloat16, device=DEV), torch.empty(n + extra, k, dtype=torch.bfloat16, device=DEV), n)
    assert rides(65, 2688, 14, 896) and rides(2048, 2688, 14, 896) and rides(65, 6144, 32, 2048) and rides(4206, 8448, 32, 2048)
    assert not rides(64, 2688, 14, 896) and not rides(300, 12288, 64, 4096) and not rides(65, 768, 8, 2048) and not rides(512, 1536, 8, 1536)
    assert not rides(1024, 768, 8, 2048) and rides(1025, 768, 8, 2048) and not rides(300, 2692, 14, 896)
