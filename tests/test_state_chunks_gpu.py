"""The recurrence of a matrix state in chunks against its token-by-token form in float64."""
import pytest
import torch

from tests import kernel_refs as refs

pytestmark = pytest.mark.gpu
DEV = "cuda"
# A float32 sum of up to 128 scores plus 128 state rows, rounded (or cut) at 2^-23 of its size per addition: sqrt(256) 2^-23 = 2e-6
# of the result's norm if the roundings are independent; the weights add a dozen roundings of 2^-24.
LIMIT = 4e-6


def rel(got, want):
    return float((got.double() - want.double()).norm() / want.double().norm())


def ints(values):
    return torch.tensor(values, dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("heads,groups,dim,vdim,with_n", [(3, 3, 64, 64, True), (4, 1, 128, 128, False), (2, 2, 64, 128, True),
                                                         (3, 1, 128, 64, False), (40, 2, 64, 256, True)])
@pytest.mark.parametrize("lengths", [(1,), (16, 15, 17), (127, 128, 129), (300, 1, 513), (96, 640)])
def test_chunks_against_the_recurrence(heads, groups, dim, vdim, with_n, lengths):
    from qwenforge_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(dim + vdim + len(lengths))
    slots = [3, -1, 1][:len(lengths)]
    cu = [0]
    for n in lengths:
        cu.append(cu[-1] + n)
    n, s_off = cu[-1], 4
    n_off = s_off + heads * dim * vdim + 1
    start = torch.randn(5, n_off + heads * dim + 3, generator=g, device=DEV)
    wide = torch.randn(n, 2 * groups * dim + heads * vdim + 8, generator=g, device=DEV).bfloat16()
    q, k, v = wide[:, :groups * dim], wide[:, groups * dim:2 * groups * dim], wide[:, 2 * groups * dim:-8]
    # decays from forgetting at once (0 among them) to hardly at all
    decay = torch.exp(-torch.exp(3 * torch.randn(n, heads, generator=g, device=DEV) - 3))
    decay[n // 2] = 0.0
    take = 2 * torch.rand(n, heads, generator=g, device=DEV)
    results = []
    for chunks in (True, False):
        state = start.clone()
        y, nq = torch.full((n, heads * vdim), 7.0, device=DEV), torch.full((n, heads), 7.0, device=DEV) if with_n else None
        args = (state, s_off, n_off if with_n else -1, heads, groups, dim, vdim, 0.3, y, nq)
        if chunks:
            ops.state_chunks(q, k, v, decay, take, ints(cu), ints(slots), max(lengths), *args)
        else:
            refs.outer_state_scan(q, k, v, decay, take, ints(cu), ints(slots), *args)
        results.append((state, y, nq))
    (state, y, nq), (want_state, want_y, want_nq) = results
    assert rel(y, want_y) < LIMIT and rel(state, want_state) < LIMIT
    if with_n:
        assert rel(nq, want_nq) < LIMIT
    held = torch.zeros(5, dtype=torch.bool)
    held[[s for s in slots if s >= 0]] = True
    assert torch.equal(state[~held], start[~held])                              # slots that the step does not name
    assert torch.equal(state[:, :s_off], start[:, :s_off]) and torch.equal(state[:, n_off + heads * dim:], start[:, n_off + heads * dim:])
    if not with_n:
        assert torch.equal(state[:, n_off:], start[:, n_off:])


@pytest.mark.parametrize("lengths", [(1,), (130, 7)])
def test_gates_from_their_pre_activations(lengths):
    """The gates formed inside are those of `decay_gates` to a unit or two of their last place, whatever the rows' stride."""
    from qwenforge_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(5)
    n, heads, dim, vdim = sum(lengths), 3, 128, 64
    cu = [0, lengths[0], n][:len(lengths) + 1]
    q, k, v = (torch.randn(n, heads * w, generator=g, device=DEV).bfloat16() for w in (dim, dim, vdim))
    pre = 4 * torch.randn(n, heads + 2, generator=g, device=DEV)[:, :heads]
    dt_bias, rate_log = torch.randn(heads, generator=g, device=DEV), torch.randn(heads, generator=g, device=DEV)
    decay, take = torch.empty(n, heads, device=DEV), torch.empty(n, heads, device=DEV)
    ops.decay_gates(pre, dt_bias, rate_log, decay, take)
    results = []
    for gates in ((decay, take, None), (None, None, (pre, dt_bias, rate_log))):
        state, y = torch.ones(2, heads * dim * vdim, device=DEV), torch.empty(n, heads * vdim, device=DEV)
        ops.state_chunks(q, k, v, *gates[:2], ints(cu), ints([1, 0][:len(lengths)]), max(lengths), state, 0, -1, heads, heads, dim, vdim, 1.0, y,
                         None, decay_gates=gates[2])
        results.append((y, state))
    for got, want in zip(results[1], results[0]):
        assert rel(got, want) < LIMIT


@pytest.mark.parametrize("rows,dim,vdim", [(False, 64, 128), (False, 128, 64), (False, 128, 128), (True, 64, 64), (True, 64, 128)])
@pytest.mark.parametrize("slow", [False, True])
def test_no_less_exact_than_token_by_token(rows, dim, vdim, slow):
    """Against 64 bits the chunked form is as close as the scan, outputs and states: its float32 operands are whole, and its sums over
    tokens and state rows are rounded, not cut off. (Both errors are means over 10^5 numbers and more: 10% covers their spread.)"""
    from qwenforge_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(dim + vdim)
    heads, n, width = 4, 1031, (dim if rows else 1)
    q, k, v = (torch.randn(n, heads * w, generator=g, device=DEV).bfloat16() for w in (dim, dim, vdim))
    logit = torch.randn(n, heads * width, generator=g, device=DEV)
    decay = torch.sigmoid(logit + 4) if slow else torch.exp(-torch.exp(logit - 3))
    take, start = torch.rand(n, heads, generator=g, device=DEV), torch.randn(1, heads * dim * vdim, generator=g, device=DEV)
    results = []
    for form in ("exact", "scan", "chunks"):
        state, y = start.clone(), torch.empty(n, heads * vdim, device=DEV)
        step = (q, k, v, decay) if rows else (q, k, v, decay, take)
        kept = (state, 0, heads, dim, vdim, 0.125, y) if rows else (state, 0, -1, heads, heads, dim, vdim, 0.125, y, None)
        if form == "chunks":
            (ops.row_chunks if rows else ops.state_chunks)(*step, ints([0, n]), ints([0]), n, *kept)
        else:
            source = refs if form == "exact" else ops
            (source.outer_state_scan_rows if rows else source.outer_state_scan)(*step, ints([0, n]), ints([0]), *kept)
        results.append((y, state))
    for want, scan, chunks in zip(*results):
        assert rel(chunks, want) <= 1.1 * rel(scan, want)


@pytest.mark.parametrize("lengths,floor", [((700,), 0), ((300, 1, 2113), 0), ((300, 1, 1300), 13)])
@pytest.mark.parametrize("rows", [False, True])
def test_portions_leave_the_same_bits(lengths, floor, rows, monkeypatch):
    """A step whose records would need more than their bound goes through its chunks in portions: the same operations, also for a
    sequence without a slot, whose state passes from portion to portion in the scratch."""
    from qwenforge_b200 import ops
    from qwenforge_b200.ops import kernels
    g = torch.Generator(device=DEV).manual_seed(len(lengths) + floor)
    heads, dim, vdim, slots, cu = 2, 64, 128, [3, 0, -1][:len(lengths)], [0]
    for n in lengths:
        cu.append(cu[-1] + n)
    n = cu[-1]
    size, sizes = heads * dim * vdim, [heads * dim, heads * dim, heads * vdim]
    q, k, v = (torch.randn(n, w, generator=g, device=DEV).bfloat16() for w in sizes)
    decay = torch.rand(n, heads * dim if rows else heads, generator=g, device=DEV)
    take, start = torch.rand(n, heads, generator=g, device=DEV), torch.randn(4, size + heads * dim, generator=g, device=DEV)
    record = 4 * heads * (dim * vdim + dim + 1)
    results = []
    for bound in (1 << 30, record * floor):
        monkeypatch.setattr(kernels, "CHUNK_SCRATCH_BYTES", bound)
        state, y, nq = start.clone(), torch.empty(n, heads * vdim, device=DEV), torch.empty(n, heads, device=DEV)
        if rows:
            ops.row_chunks(q, k, v, decay, ints(cu), ints(slots), max(lengths), state, 0, heads, dim, vdim, 0.3, y,
                           decay_from=("sigmoid_root", torch.ones(heads * dim, device=DEV), 8.0))
        else:
            ops.state_chunks(q, k, v, decay, take, ints(cu), ints(slots), max(lengths), state, 0, size, heads, heads, dim, vdim, 0.3, y, nq)
        results.append((state, y) if rows else (state, y, nq))
    for whole, portions in zip(*results):
        assert torch.equal(whole, portions)


def test_a_value_that_is_not_finite_reaches_no_earlier_token():
    from qwenforge_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(1)
    n, heads, dim, vdim, bad = 200, 2, 64, 64, 150
    q, k, v = (torch.randn(n, heads * dim, generator=g, device=DEV).bfloat16() for _ in range(3))
    decay, take = torch.rand(n, heads, generator=g, device=DEV), torch.rand(n, heads, generator=g, device=DEV)
    outs = []
    for value in (1.0, float("inf"), float("nan")):
        v[bad, 3] = value
        state, y = torch.zeros(1, heads * dim * vdim, device=DEV), torch.empty(n, heads * vdim, device=DEV)
        ops.state_chunks(q, k, v, decay, take, ints([0, n]), ints([0]), n, state, 0, -1, heads, heads, dim, vdim, 1.0, y, None)
        outs.append(y)
    for y in outs[1:]:
        assert rel(y[:bad], outs[0][:bad]) < LIMIT and not bool(torch.isfinite(y[bad:, 3]).any())


def test_what_the_chunked_form_takes():
    from qwenforge_b200 import ops
    q = torch.zeros(200, 3 * 64, dtype=torch.bfloat16, device=DEV)
    takes = lambda t, dim=64, vdim=64, longest=200: ops.state_chunks_take(t, t, t, dim, vdim, longest)
    assert takes(q[:, :64])
    assert not takes(q[:, :64].float()) and not takes(q[:, 1:65]) and not takes(q[:, :64], dim=32) and not takes(q[:, :64], vdim=96)
    assert not takes(torch.zeros(200, 65, dtype=torch.bfloat16, device=DEV)[:, :64]) and not takes(q[:, :64], longest=16)
