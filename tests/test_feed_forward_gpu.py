"""The feed-forward of a step of few rows as one kernel, and the two kernels that take its sums along."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _layer(width, inter, rows, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    rnd = lambda *shape: torch.randn(*shape, generator=g, device=DEV)
    return (rnd(rows, width), (1 + 0.1 * rnd(width)).bfloat16(), (rnd(2 * inter, width) * width ** -0.5).bfloat16(),
            (rnd(width, inter) * inter ** -0.5).bfloat16(), rnd(rows, width))


# every number of warps a row and of warps a tile (8 to 128 columns a block), a half step of K in the down product, a ragged last block
@pytest.mark.parametrize("width,inter", [(896, 4864), (896, 4872), (1024, 3000), (512, 1184), (128, 2368), (64, 18944), (288, 4720), (1536, 1184)])
@pytest.mark.parametrize("rows", [1, 2, 3, 4, 5, 8])
def test_against_float64(width, inter, rows):
    from qwenforge_b200 import ops
    from qwenforge_b200.csrc import library
    hidden, norm, gate_up, down, before = _layer(width, inter, rows, width + inter + rows)
    blocks = library("feed_forward").qf_feed_forward_blocks(ctypes.c_int(rows), ctypes.c_int(width), ctypes.c_int(inter))
    assert blocks > 0 and ops.feed_forward_takes(rows, gate_up, down) == (blocks * rows * width // 4 <= 250_000 and (width, inter) != (64, 18944))
    sums, kept, err = before.clone(), hidden.clone(), torch.zeros(1, dtype=torch.int32, device=DEV)
    ops.feed_forward(hidden, norm, 1e-6, gate_up, down, sums, err)
    h = hidden.double()
    y = h * torch.rsqrt(h.square().mean(-1, keepdim=True) + 1e-6) * norm.double() @ gate_up.double().T
    want = (torch.nn.functional.silu(y[:, :inter]) * y[:, inter:]) @ down.double().T
    assert int(err) == 0 and torch.equal(hidden, kept)
    # the rows and the activations are rounded to eight bits (2^-9 each at worst); what is added to lies in float32
    assert float(((sums - before).double() - want).norm()) < 2.0 ** -8 * float(want.norm())


def test_what_is_not_taken():
    from qwenforge_b200 import ops
    hidden, norm, gate_up, down, sums = _layer(896, 4864, 9, 1)
    assert not ops.feed_forward_takes(9, gate_up, down)                   # rows
    with pytest.raises(ops.KernelError if hasattr(ops, "KernelError") else Exception):
        ops.feed_forward(hidden, norm, 1e-6, gate_up, down, sums)
    _, _, wide, narrow, _ = _layer(2048, 11008, 1, 1)                     # weights beyond the shared memory
    assert not ops.feed_forward_takes(1, wide, narrow)
    _, _, odd, odd_down, _ = _layer(900, 4864, 1, 1)                      # a width of no whole blocks of 32
    assert not ops.feed_forward_takes(1, odd, odd_down)


@pytest.mark.parametrize("seqs", [1, 2, 3, 8])
def test_decode_steps_with_and_without(seqs, monkeypatch):
    """Three layers of the smallest preset's sizes, prompts and then single tokens: the logits of the layers as two kernels, within the
    rounding of activations to eight bits; launch by launch, each step from the same cache."""
    from qwenforge_b200 import ops
    from qwenforge_b200.config import preset_config
    from qwenforge_b200.engine import Model
    config = preset_config("qwen2.5-0.5b", num_hidden_layers=3, vocab_size=512)
    model = Model.from_random(config, 3)
    logits, ran = {}, []
    real = ops.feed_forward
    monkeypatch.setattr(ops, "feed_forward", lambda *a, **k: (ran.append(1), real(*a, **k))[1])
    for on in (True, False):
        if not on:
            monkeypatch.setattr(ops, "feed_forward_takes", lambda *a: False)
        cache = model.new_cache(64 * 4 * seqs, seqs)
        slots = [cache.open() for _ in range(seqs)]
        model.step(cache, [(s, list(range(1, 20 + 7 * i))) for i, s in enumerate(slots)])
        logits[on] = [model.step(cache, [(s, [5 + i + n]) for i, s in enumerate(slots)]) for n in range(4)]
    assert len(ran) == 3 * 4
    model.raise_on_kernel_error()
    for a, b in zip(logits[True], logits[False]):
        assert float((a - b).norm()) < 2e-2 * float(b.norm())


@pytest.mark.parametrize("takes", [True, False])
def test_a_stack_whose_second_mixer_takes_the_sums_or_does_not(takes, monkeypatch):
    """Sums that the next mixer reads, and sums that its block moves into the stream first; an observer sees every layer's stream as two products
    leave it, also after the step."""
    from qwenforge_b200 import ops
    from qwenforge_b200.config import preset_config
    from qwenforge_b200.engine import Model
    model = Model.from_random(preset_config("qwen2.5-0.5b", num_hidden_layers=2, vocab_size=512), 3)
    moved, ran = [], []
    take, forward = ops.take_sums, ops.feed_forward
    monkeypatch.setattr(ops, "take_sums", lambda *a: (moved.append(1), take(*a))[1])
    monkeypatch.setattr(ops, "feed_forward", lambda *a, **k: (ran.append(1), forward(*a, **k))[1])
    if not takes:
        model.blocks[1].mixer.takes_sums = lambda *a: False
    logits, seen = {}, {}
    for on in (True, False):
        if not on:
            monkeypatch.setattr(ops, "feed_forward_takes", lambda *a: False)
        cache = model.new_cache(64 * 3, 3)
        slots = [cache.open() for _ in range(3)]
        model.step(cache, [(s, list(range(1, 20 + 7 * i))) for i, s in enumerate(slots)])
        kept = seen[on] = []
        model.observer = lambda index, hidden, delta: kept.append((hidden.clone(), delta))
        logits[on] = model.step(cache, [(s, [5 + i]) for i, s in enumerate(slots)])
        model.observer = None
    model.raise_on_kernel_error()
    assert len(ran) == 2 and len(moved) == (1 if takes else 2)      # (once at the stack's end)
    streams = {on: [h if d is None else h + d.float() for h, d in kept] for on, kept in seen.items()}
    assert len(streams[True]) == 3 and any(d is not None and bool(d.any()) for _, d in seen[True])
    for a, b in (*zip(streams[True], streams[False]), (logits[True], logits[False])):
        assert float((a - b).norm()) < 2e-2 * float(b.norm())


@pytest.mark.parametrize("rows", [1, 8])
def test_a_layer_that_the_model_does_not_run(rows):
    """A caller of `block.forward` has the feed-forward's output in the stream when the call returns, as with layers beyond the one kernel."""
    import numpy as np
    from qwenforge_b200 import ops
    from qwenforge_b200.cache import SequenceCache
    from qwenforge_b200.config import preset_config
    from qwenforge_b200.engine import Model, build_context
    model = Model.from_random(preset_config("qwen2.5-0.5b", num_hidden_layers=1, vocab_size=128), 5)
    block = model.blocks[0]
    cache = SequenceCache(model.cache_needs(), 64 * rows, rows, model.spec.max_positions, model.dtype, model.device)
    slots = [cache.open() for _ in range(rows)]
    cache.reserve([(s, 1) for s in slots])
    cache.flush()
    ctx = build_context([(s, 0, np.zeros(1, dtype=np.int32)) for s in slots], None, model.err, model.dtype, model.device, model.attention, model.decode_scratch)
    before = torch.randn(rows, 896, generator=torch.Generator(device=DEV).manual_seed(rows), device=DEV)
    ctx.step_memo = {}
    stream = before.clone()
    assert block.forward(stream, None, ctx, cache.site(0), True) is None
    ctx.step_memo = {"model.resolves_sums": True}
    left = before.clone()
    pending = block.forward(left, None, ctx, cache.site(0), True)
    assert ops.feed_forward_takes(rows, block.feed_forward.gate_up_weight, block.feed_forward.down_weight) and pending is not None
    assert float((stream - left).norm()) > 0.1 * float(left.norm())
    pending.add_to(left)
    # both round the normalised rows and the activations to eight bits
    assert float((stream - left).norm()) < 2.0 ** -8 * float(left.norm())


@pytest.mark.parametrize("rows,heads,dim", [(1, 14, 64), (8, 14, 64), (3, 4, 96), (5, 2, 128)])
def test_the_projection_moves_the_sums(rows, heads, dim):
    """With sums the stream is what it is without, plus the sums; zeros stay behind. (96: blocks of 32 inputs; the others of 64.)"""
    from qwenforge_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(rows + dim)
    rnd = lambda *shape: torch.randn(*shape, generator=g, device=DEV)
    width, splits = 272, 3
    scratch = ops.DecodeScratch(torch.device(DEV))
    scratch.part_o = rnd(rows * heads * splits * dim)
    scratch.part_ml = torch.rand(rows * heads * splits * 2, generator=g, device=DEV) + 0.5
    plan = torch.tensor([1 + i % splits for i in range(8)], dtype=torch.int32, device=DEV)
    weight, hidden, sums = (rnd(width, heads * dim) * 0.05).bfloat16(), rnd(rows, width), rnd(rows, width)
    plain, both, left = hidden.clone(), hidden.clone(), sums.clone()
    ops.fold_project(plan, scratch, weight, plain, heads, dim, splits)
    ops.fold_project(plan, scratch, weight, both, heads, dim, splits, left)
    assert not bool(left.any())
    # the shares of up to 56 blocks are added in any order: 56 roundings of 2^-24 of numbers of size up to about 8
    assert float((both - (plain + sums)).abs().max()) < 57 * 2.0 ** -24 * 8
    left = sums.clone()
    ops.take_sums(plain, left)
    assert not bool(left.any()) and float((both - plain).abs().max()) < 57 * 2.0 ** -24 * 8


@pytest.mark.parametrize("rows,dim,summed", [(1, 64, True), (8, 64, True), (7, 64, False), (16, 64, False), (13, 96, True), (16, 64, True)])
def test_the_projection_reads_the_plan_before_or_behind_its_wait(rows, dim, summed):
    """`settled` or not, up to more rows than a block has threads for at once: the same runs are folded."""
    from qwenforge_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(rows + dim)
    rnd = lambda *shape: torch.randn(*shape, generator=g, device=DEV)
    width, heads, splits = 272, 4, 3
    scratch = ops.DecodeScratch(torch.device(DEV))
    scratch.part_o = rnd(rows * heads * splits * dim)
    scratch.part_ml = torch.rand(rows * heads * splits * 2, generator=g, device=DEV) + 0.5
    plan = torch.tensor([1 + i % splits for i in range(16)], dtype=torch.int32, device=DEV)
    weight, hidden, sums = (rnd(width, heads * dim) * 0.05).bfloat16(), rnd(rows, width), rnd(rows, width) if summed else None
    streams = []
    for settled in (False, True):
        stream = hidden.clone()
        ops.fold_project(plan, scratch, weight, stream, heads, dim, splits, None if sums is None else sums.clone(), settled=settled)
        streams.append(stream)
    n_runs = plan[:rows].long()
    ml = scratch.part_ml.view(rows, heads, splits, 2).double()
    live = (torch.arange(splits, device=DEV)[None] < n_runs[:, None])[:, None]
    share = torch.where(live, 2.0 ** (ml[..., 0] - ml[..., 0].amax(-1, keepdim=True)), 0.0)   # (no more than a factor of 2 between the runs' maxima)
    folded = (share[..., None] * scratch.part_o.view(rows, heads, splits, dim).double()).sum(2) / (share * ml[..., 1]).sum(2)[..., None]
    want = hidden.double() + folded.reshape(rows, -1).bfloat16().double() @ weight.double().T + (0 if sums is None else sums.double())
    for stream in streams:   # folded rows may round to the other of two neighbours in eight bits; shares of up to 12 blocks arrive in any order
        assert float((stream.double() - want).norm()) < 2.0 ** -9 * float(want.norm())


@pytest.mark.parametrize("rows", [1, 2, 4, 7, 8])
def test_the_qkv_product_reads_stream_and_sums(rows):
    from qwenforge_b200 import ops
    from qwenforge_b200.measure import layer_products
    products, state = layer_products(rows, 904, 1024, 14, 2, 64)    # (a K of no whole block of 32)
    t = products[3].tensors
    assert ops.skinny_gemm_reads_pending(rows, products[3].weight, 14, 2, 64, 64)
    products[3].run()
    want_q, want_cache = state["q_out"].clone(), state["cache"].clone()
    part = torch.randn_like(t["hidden"])
    rest = t["hidden"] - part
    ops.skinny_gemm(ops.EPI_QKV, products[3].weight, **{**t, "hidden": rest, "pending": t["hidden"] - rest})
    assert int(state["err"]) == 0
    for got, want in ((state["q_out"], want_q), (state["cache"], want_cache)):
        # (hidden - rest) + rest is hidden to a rounding of 2^-24; results lie one step of eight bits apart at most
        assert float((got.float() - want.float()).abs().max()) <= 2.0 ** -7 * float(want.float().abs().max())
        assert float((got.float() - want.float()).norm()) <= 2.0 ** -9 * float(want.float().norm())


def test_pending_rows_are_refused_where_nothing_reads_them():
    """With x in the place of the stream, with another epilogue, on the kernel of up to 64 rows and in a chain of products."""
    from qwenforge_b200 import ops
    from qwenforge_b200.measure import layer_products
    products, _ = layer_products(2, 896, 1024, 14, 2, 64)
    qkv = next(p for p in products if p.epilogue == ops.EPI_QKV)
    rows = torch.zeros_like(qkv.tensors["hidden"])
    by_x = {name: t for name, t in qkv.tensors.items() if name not in ("hidden", "norm_weight", "eps")}
    by_x["x"] = rows.bfloat16()
    for run in (ops.skinny_gemm, ops.wide_gemm):
        run(ops.EPI_QKV, qkv.weight, **by_x)
        with pytest.raises(ops.KernelError, match="pending"):
            run(ops.EPI_QKV, qkv.weight, **by_x, pending=rows)
    plain = dict(hidden=qkv.tensors["hidden"], norm_weight=qkv.tensors["norm_weight"], eps=1e-6, out=torch.empty(2, qkv.weight.shape[0], device=DEV))
    ops.skinny_gemm(ops.EPI_PLAIN, qkv.weight, **plain)
    with pytest.raises(ops.KernelError, match="pending"):
        ops.skinny_gemm(ops.EPI_PLAIN, qkv.weight, **plain, pending=rows)
    chained = ops.FusedProduct(ops.EPI_QKV, qkv.weight, **qkv.tensors, pending=rows)
    assert not ops.skinny_chain_takes([chained])
    with pytest.raises(ops.KernelError, match="pending"):
        ops.skinny_chain([chained], torch.zeros(2, dtype=torch.int32, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV))


@pytest.mark.parametrize("heads,dim,folds,free", [(14, 64, True, 14), (8, 96, True, 0), (4, 128, True, 8), (14, 64, False, 0)])
def test_a_plan_leaves_slots_for_large_blocks_only(heads, dim, folds, free, monkeypatch):
    """The projection's blocks of 64 inputs; not those of 32 (heads of 96), and nothing where it does not fold the partial results."""
    from qwenforge_b200 import ops
    from qwenforge_b200.config import preset_config
    from qwenforge_b200.engine import Model
    model = Model.from_random(preset_config("qwen2.5-0.5b", num_hidden_layers=2, vocab_size=128, hidden_size=heads * dim, intermediate_size=1184,
                                            num_attention_heads=heads, num_key_value_heads=2, head_dim=dim), 5)
    left, ran = [], []
    plan, forward = ops.attention_decode_plan, ops.feed_forward
    monkeypatch.setattr(ops, "attention_decode_plan", lambda *a: (left.append(a[11] if len(a) > 11 else 0), plan(*a))[1])
    monkeypatch.setattr(ops, "feed_forward", lambda *a, **k: (ran.append(1), forward(*a, **k))[1])
    if not folds:
        monkeypatch.setattr(ops, "fold_project_pays", lambda *a: False)
    cache = model.new_cache(256, 2)
    slots = [cache.open() for _ in range(2)]
    model.step(cache, [(s, list(range(1, 20))) for s in slots])
    model.step(cache, [(s, [5]) for s in slots])
    model.raise_on_kernel_error()
    assert left == [free] and len(ran) == 2


@pytest.mark.parametrize("lengths", [[4100] * 8, [1] * 8, [700], [4100, 64, 65, 3000]])
def test_a_plan_that_leaves_slots(lengths):
    """No more runs than fit beside what is left free (or one a sequence); the attention of either plan."""
    from qwenforge_b200 import ops
    from qwenforge_b200.measure import Pages
    heads, kv, dim, leave, n = 14, 2, 64, 14, len(lengths)
    g = torch.Generator(device=DEV).manual_seed(n)
    pages = Pages(n, max(lengths), kv, dim, DEV)
    pages.storage.normal_(generator=g)
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    q, err = torch.randn(n, heads * dim, generator=g, device=DEV).bfloat16(), ints([0])
    cu, pos, slots, splits = ints(list(range(n + 1))), ints([x - 1 for x in lengths]), ints(list(range(n))), max(1, -(-max(lengths) // 512))
    outs, runs = [], []
    for free in (0, leave):
        scratch, out = ops.DecodeScratch(torch.device(DEV)), torch.empty_like(q)
        plan = ops.attention_decode_plan(cu, pos, slots, kv, dim, heads, n, 0, splits, scratch, leave=free)
        ops.attention_decode(q, out, cu, pos, slots, pages.args(), heads, n, dim ** -0.5, 0, splits, scratch, err, plan)
        runs.append(plan.flatten()[:n].tolist())
        outs.append(out.float())
    assert int(err) == 0
    assert sum(runs[1]) * kv <= max(ops.sm_count(DEV) - leave, n * kv) and all(b <= a for a, b in zip(*runs))
    # both are sums of the same weighted values with weights in bfloat16, rounded to bfloat16
    assert float((outs[0] - outs[1]).norm()) < 2.0 ** -7 * float(outs[0].norm())
