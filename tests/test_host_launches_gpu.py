"""What native code launches (csrc/host.cpp) is what the Python entries launch one by one: the same bits, and their way where it steps aside."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
STRETCHES = ("rms_norm", "prompt_attention", "gated_feed_forward", "matrix_memory", "state_space", "gated_linear_attention")


def _model(preset, layer=None):
    from qwenforge_b200.config import config_from_dict, preset_config
    from qwenforge_b200.engine import Model
    if layer is None:
        return Model.from_random(preset_config(preset, num_hidden_layers=1, vocab_size=128), 5)
    kept = preset_config(preset).to_dict()
    kept["layers"] = [dict(next(entry for entry in kept["layers"] if entry["type"] == layer), mlp=None)]
    kept["vocab"] = 128
    return Model.from_random(config_from_dict(kept), 5)


def _step(model, lengths, before):
    from qwenforge_b200.cache import SequenceCache
    from qwenforge_b200.engine import build_context
    cache = SequenceCache(model.cache_needs(), sum(-(-(n + before) // 64) * 64 for n in lengths), len(lengths), model.spec.max_positions, model.dtype, model.device)
    slots = [cache.open() for _ in lengths]
    cache.reserve([(s, n + before) for s, n in zip(slots, lengths)])
    cache.flush()
    ctx = build_context([(s, before, np.zeros(n, dtype=np.int32)) for s, n in zip(slots, lengths)], None, model.err, model.dtype, model.device,
                        model.attention, model.decode_scratch)
    ctx.step_memo = {}
    return cache.site(0), ctx


def _watch(monkeypatch, on):
    """Which stretches native code took, by name; `on` False: none."""
    from qwenforge_b200 import ops
    took = []
    for name in STRETCHES:
        real = getattr(ops.host, name)

        def watched(*args, name=name, real=real):
            out = real(*args) if on else None
            if out is not None:
                took.append(name)
            return out
        monkeypatch.setattr(ops.host, name, watched)
    return took


# (tokens beyond the 64 of the decode form, too few for gate/up on pairs, the benchmark's, unequal and with a portion before; heads of 128, whose
# queries, keys and values go by the library and the rotation kernel below some size and on pairs of SMs above it)
@pytest.mark.parametrize("preset,lengths,before,attention", [
    ("qwen2.5-0.5b", [65], 0, None), ("qwen2.5-0.5b", [300], 0, True), ("qwen2.5-0.5b", [2048], 0, True), ("qwen2.5-0.5b", [201, 517, 133], 70, True),
    ("qwen2.5-3b", [300], 0, True), ("qwen2.5-3b", [700], 0, True), ("qwen2.5-3b", [150, 200], 1000, True)])
def test_a_layer(preset, lengths, before, attention, monkeypatch):
    model = _model(preset)
    x = torch.randn(sum(lengths), model.blocks[0].mixer.hidden, generator=torch.Generator(device=DEV).manual_seed(1), device=DEV)
    pending = torch.randn(x.shape, generator=torch.Generator(device=DEV).manual_seed(2), device=DEV).bfloat16()
    results = []
    for on in (True, False):
        with monkeypatch.context() as patch:
            took = _watch(patch, on)
            site, ctx = _step(model, lengths, before)
            site.storage.zero_()
            stream = x.clone()
            delta = model.blocks[0].forward(stream, pending, ctx, site, True)
        results.append((stream, delta, site.storage.clone()))
        if on:
            assert {"rms_norm", "gated_feed_forward"} <= set(took) and (attention is None or "prompt_attention" in took)
        else:
            assert not took
    model.raise_on_kernel_error()
    for a, b in zip(*results):
        assert torch.equal(a, b)


@pytest.mark.parametrize("preset,layer,stretch", [("zebovik-0.5b", "mlstm", "matrix_memory"), ("zebovik-0.5b", "mamba2", "state_space"),
                                                  ("zebovik-3b", "mamba2", "state_space"), ("gatosun-0.5b", "gla", "gated_linear_attention")])
@pytest.mark.parametrize("lengths", [[100], [700], [2048], [900, 193, 5]])
def test_a_recurrent_mixer(preset, layer, stretch, lengths, monkeypatch):
    """Two steps, the second one from the state that the first one left."""
    model = _model(preset, layer)
    mixer, results = model.blocks[0].mixer, []
    x = torch.randn(sum(lengths), mixer.hidden, generator=torch.Generator(device=DEV).manual_seed(1), device=DEV).bfloat16()
    for on in (True, False):
        with monkeypatch.context() as patch:
            took = _watch(patch, on)
            site, ctx = _step(model, lengths, 0)
            outs = [mixer.forward(x, ctx, site, True) for _ in range(2)]
        results.append((*outs, site.storage.clone()))
        assert (stretch in took) == (on and max(lengths) >= 700)
    model.raise_on_kernel_error()
    for a, b in zip(*results):
        assert torch.equal(a, b)


@pytest.mark.parametrize("layer", ["mlstm", "mamba2"])
def test_buffers_of_one_allocation_begin_on_whole_lines(layer):
    """Heads x tokens of no whole line: the addresses that the kernels are given (by entries that write them down and launch nothing)."""
    import ctypes

    from qwenforge_b200 import ops
    from qwenforge_b200.csrc import library
    p, i, n, f = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong, ctypes.c_float
    entries = {"qf_stabilized_gates": ("recurrent", (p, i, p, f, p, p, i, p, n, n, i, p, p, p, p), (0, 11, 12, 13)),
               "qf_state_chunks": ("state_chunks", (p, i, p, i, p, i, p, p, p, p, i, p, p, i, i, p, n, n, n, i, i, i, i, f, p, n, i, p, p, p), (24, 27, 28)),
               "qf_gated_group_norm": ("recurrent", (i, p, p, i, p, f, p, i, i, i, i, i, i, p, p, f, p, p, i, p), (1, 6, 13, 14))}
    model = _model("zebovik-0.5b", layer)
    mixer, seen, kept = model.blocks[0].mixer, [], []
    x = torch.randn(701, mixer.hidden, device=DEV).bfloat16()
    site, ctx = _step(model, [701], 0)
    mixer.forward(x, ctx, site, True)
    module = ops.host._host("recurrent", "state_chunks")
    fakes = {}
    for name, (_, types, which) in entries.items():
        def write_down(*args, which=which):
            seen.extend(args[at] for at in which if args[at])
            return 0
        kept.append(ctypes.CFUNCTYPE(i, *types)(write_down))
        fakes[name] = ctypes.cast(kept[-1], p).value
    try:
        module.setup(ops.KernelError, fakes)
        mixer.forward(x, ctx, site, True)
    finally:
        module.setup(ops.KernelError, {name: ctypes.cast(getattr(library(source), name), p).value for name, (source, *_) in entries.items()})
    assert len(seen) >= 4 and all(address % 128 == 0 for address in seen)


def test_whoever_replaces_a_kernel_sees_its_calls():
    from qwenforge_b200.ops.timing import KernelTimer
    model = _model("qwen2.5-0.5b")
    site, ctx = _step(model, [2048], 0)
    with KernelTimer() as timer:
        model.blocks[0].forward(torch.randn(2048, 896, device=DEV), None, ctx, site, True)
    seen = [label.split("[")[0] for label, *_ in timer.records]
    assert sorted(seen) == sorted(["add_rms_norm", "qkv_product", "attention_prefill_tc", "linear", "add_rms_norm", "tc_gemm", "linear"])


def test_what_is_not_taken():
    from qwenforge_b200 import ops
    hidden, weight = torch.randn(8, 64, device=DEV), torch.ones(64, device=DEV).bfloat16()
    assert ops.host.rms_norm(hidden, None, weight, 1e-6) is not None
    assert ops.host.rms_norm(hidden.t().contiguous().t(), None, weight, 1e-6) is None                  # rows that are not contiguous
    assert ops.host.rms_norm(hidden, hidden, weight, 1e-6) is None                                     # a pending output of another type
    assert ops.host.rms_norm(hidden, None, weight.as_subclass(type("Other", (torch.Tensor,), {})), 1e-6) is None   # a subclass of tensor
    assert ops.host.rms_norm(hidden.cpu(), None, weight, 1e-6) is None
    x, gate_up, down = torch.randn(2048, 896, device=DEV).bfloat16(), torch.randn(9728, 896, device=DEV).bfloat16(), torch.randn(896, 4864, device=DEV).bfloat16()
    err = torch.zeros(1, dtype=torch.int32, device=DEV)
    assert ops.host.gated_feed_forward(x, gate_up, down, err) is not None
    assert ops.host.gated_feed_forward(x[:16], gate_up, down, err) is not None
    assert ops.host.gated_feed_forward(x[:, :892], gate_up[:, :892], down, err) is None                # a K of no whole pieces of eight
    assert ops.host.gated_feed_forward(x, gate_up, down[:, :4856], err) is None                        # shapes that do not agree


def test_other_threads_run_while_a_launch_waits():
    """Launches behind a busy stream until the driver's queue is full and one of them waits: another thread's clock goes on."""
    import threading
    import time

    from qwenforge_b200 import ops
    hidden, weight = torch.randn(8, 64, device=DEV), torch.ones(64, device=DEV).bfloat16()
    norm = lambda: ops.host.rms_norm(hidden, None, weight, 1e-6)
    assert norm() is not None
    torch.cuda.synchronize()
    gaps, done = [], threading.Event()

    def clock():
        last = time.perf_counter()
        while not done.is_set():
            time.sleep(1e-3)
            now = time.perf_counter()
            gaps.append(now - last)
            last = now
    watcher = threading.Thread(target=clock)
    torch.cuda._sleep(2_000_000_000)   # about a second
    watcher.start()
    began, longest = time.perf_counter(), 0.0
    while time.perf_counter() - began < 0.2 or longest < 0.1:   # (until a call has waited)
        at = time.perf_counter()
        norm()
        longest = max(longest, time.perf_counter() - at)
        if time.perf_counter() - began > 5:
            break
    done.set()
    watcher.join()
    torch.cuda.synchronize()
    if longest < 0.1:
        pytest.skip("no launch waited on this machine")
    assert max(gaps) < 0.5 * longest
