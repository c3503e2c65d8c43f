"""The recurrence with a decay per row of the state, in chunks, against its token-by-token form in float64."""
import pytest
import torch

from tests import kernel_refs as refs

pytestmark = pytest.mark.gpu
DEV = "cuda"
# A float32 sum of up to 64 scores plus 64 state rows, each a sum of 64 products: a dozen roundings of 2^-23 a level, independent
LIMIT = 4e-6


def rel(got, want):
    return float((got.double() - want.double()).norm() / want.double().norm())


def ints(values):
    return torch.tensor(values, dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("heads,vdim", [(3, 64), (2, 128), (40, 192)])
@pytest.mark.parametrize("lengths", [(1,), (15, 16, 17), (63, 64, 65), (300, 1, 129)])
@pytest.mark.parametrize("form", ["after", "bonus", "double_exp", "sigmoid_root"])
def test_chunks_against_the_recurrence(heads, vdim, lengths, form):
    from qwenforge_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(vdim + len(lengths))
    dim, slots, cu = 64, [3, -1, 1][:len(lengths)], [0]
    for n in lengths:
        cu.append(cu[-1] + n)
    n, s_off = cu[-1], 4
    start = torch.randn(5, s_off + heads * dim * vdim + 3, generator=g, device=DEV)
    wide = torch.randn(n, 2 * heads * dim + heads * vdim + 8, generator=g, device=DEV).bfloat16()
    q, k, v = wide[:, :heads * dim], wide[:, heads * dim:2 * heads * dim], wide[:, 2 * heads * dim:-8]
    bonus = torch.randn(heads, dim, generator=g, device=DEV) if form in ("bonus", "double_exp") else None
    if form in ("after", "bonus"):   # decays from forgetting at once (0 among them) to hardly at all
        decay, decay_from = torch.exp(-torch.exp(3 * torch.randn(n, heads * dim, generator=g, device=DEV) - 3)), None
        decay[n // 2, ::3] = 0.0
    else:
        decay, decay_from = torch.randn(n, heads * dim, generator=g, device=DEV), (form, torch.randn(heads * dim, generator=g, device=DEV), 8.0)
    results = []
    for chunks in (True, False):
        state, y = start.clone(), torch.full((n, heads * vdim), 7.0, device=DEV)
        rest = (state, s_off, heads, dim, vdim, 0.3, y)
        if chunks:
            ops.row_chunks(q, k, v, decay, ints(cu), ints(slots), max(lengths), *rest, bonus=bonus, decay_from=decay_from)
        else:
            refs.outer_state_scan_rows(q, k, v, decay, ints(cu), ints(slots), *rest, bonus=bonus, decay_from=decay_from)
        results.append((state, y))
    (state, y), (want_state, want_y) = results
    assert rel(y, want_y) < LIMIT and rel(state, want_state) < LIMIT
    held = torch.zeros(5, dtype=torch.bool)
    held[[s for s in slots if s >= 0]] = True
    assert torch.equal(state[~held], start[~held])
    assert torch.equal(state[:, :s_off], start[:, :s_off]) and torch.equal(state[:, s_off + heads * dim * vdim:], start[:, s_off + heads * dim * vdim:])


def test_a_value_that_is_not_finite_reaches_no_earlier_token():
    from qwenforge_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(1)
    n, heads, dim, bad = 200, 2, 64, 150
    q, k, v = (torch.randn(n, heads * dim, generator=g, device=DEV).bfloat16() for _ in range(3))
    decay, outs = torch.rand(n, heads * dim, generator=g, device=DEV), []
    for value in (1.0, float("inf"), float("nan")):
        v[bad, 3] = value
        state, y = torch.zeros(1, heads * dim * dim, device=DEV), torch.empty(n, heads * dim, device=DEV)
        ops.row_chunks(q, k, v, decay, ints([0, n]), ints([0]), n, state, 0, heads, dim, dim, 1.0, y)
        outs.append(y)
    for y in outs[1:]:
        assert rel(y[:bad], outs[0][:bad]) < LIMIT and not bool(torch.isfinite(y[bad:, 3]).any())


def test_what_the_chunked_form_takes():
    from qwenforge_b200 import ops
    q, w = torch.zeros(600, 3 * 64, dtype=torch.bfloat16, device=DEV), torch.zeros(600, 64, device=DEV)
    takes = lambda t, dim=64, vdim=64, longest=600: ops.row_chunks_take(t, t, t, w, dim, vdim, longest)
    assert takes(q[:, :64])
    assert not takes(q[:, :64].float()) and not takes(q[:, 1:65]) and not takes(q[:, :64], dim=128) and not takes(q[:, :64], vdim=96)
    assert not takes(q[:, :64], longest=16) and not takes(q[:, :64], vdim=576)


# Where the blocks fill the SMs a block of outputs takes two tiles of 64 columns of v; a call on 64 columns takes one.
@pytest.mark.parametrize("heads,vdim,lengths,form,odd", [
    (40, 128, (300, 1, 129), "after", None), (40, 128, (300, 1, 129), "bonus", None), (40, 128, (300, 1, 129), "sigmoid_root", None),
    (20, 256, (300, 1, 129), "double_exp", None), (74, 128, (63, 64, 65), "after", float("inf")), (74, 128, (63, 64, 65), "bonus", float("nan"))])
def test_two_tiles_of_v_a_block(heads, vdim, lengths, form, odd, monkeypatch):
    from qwenforge_b200 import ops
    from qwenforge_b200.ops import kernels
    g = torch.Generator(device=DEV).manual_seed(heads + vdim)
    dim, slots, cu, s_off = 64, [3, -1, 1], [0], 4
    for n in lengths:
        cu.append(cu[-1] + n)
    n, records = cu[-1], cu[-1] // 64 + len(lengths)
    assert records * heads * (vdim // 128) >= 2 * ops.sm_count(torch.device(DEV))
    q, k, v = (torch.randn(n, heads * c, generator=g, device=DEV).bfloat16() for c in (dim, dim, vdim))
    bad = lengths[0] - 10                                      # a token of the first sequence, and a column of the second tile of head 1
    if odd is not None:
        v[bad, vdim + 70] = odd
    start = torch.randn(5, s_off + heads * dim * vdim, generator=g, device=DEV)
    bonus = torch.randn(heads, dim, generator=g, device=DEV) if form in ("bonus", "double_exp") else None
    if form in ("after", "bonus"):
        decay, decay_from = torch.exp(-torch.exp(3 * torch.randn(n, heads * dim, generator=g, device=DEV) - 3)), None
    else:
        decay, decay_from = torch.randn(n, heads * dim, generator=g, device=DEV), (form, torch.randn(heads * dim, generator=g, device=DEV), 8.0)
    more = dict(bonus=bonus, decay_from=decay_from)

    def whole():
        state, y = start.clone(), torch.full((n, heads * vdim), 7.0, device=DEV)
        ops.row_chunks(q, k, v, decay, ints(cu), ints(slots), max(lengths), state, s_off, heads, dim, vdim, 0.3, y, **more)
        return state, y
    state, y = whole()
    tiles = start[:, s_off:].view(5, heads, dim, vdim // 64, 64)
    bits = lambda t: t.contiguous().view(torch.int32)
    for at in range(vdim // 64):
        part, out = tiles[:, :, :, at].reshape(5, -1).contiguous(), torch.empty(n, heads * 64, device=DEV)
        ops.row_chunks(q, k, v.view(n, heads, -1, 64)[:, :, at].reshape(n, -1).contiguous(), decay, ints(cu), ints(slots), max(lengths), part, 0, heads,
                       dim, 64, 0.3, out, **more)
        assert torch.equal(bits(out), bits(y.view(n, heads, -1, 64)[:, :, at].reshape(n, -1)))
        assert torch.equal(bits(part), bits(state[:, s_off:].view(5, heads, dim, -1, 64)[:, :, :, at].reshape(5, -1)))
    if odd is not None:
        hit = ~torch.isfinite(y.view(n, heads, vdim))
        assert bool(hit[bad:lengths[0], 1, 70].any()) and not bool(hit[:bad].any()) and not bool(hit[lengths[0]:].any())
        hit[:, 1, 70] = False
        assert not bool(hit.any())
    # in portions of two chunks of every sequence a block takes one tile again: the same bits
    assert min(2, -(-max(lengths) // 64)) * len(lengths) * heads * (vdim // 128) < 2 * ops.sm_count(torch.device(DEV)) or heads == 74
    monkeypatch.setattr(kernels, "_chunk_portions", lambda n, n_seqs, chunk, floats: (2 * n_seqs, 2))
    cut_state, cut_y = whole()
    assert torch.equal(bits(cut_y), bits(y)) and torch.equal(bits(cut_state), bits(state))
