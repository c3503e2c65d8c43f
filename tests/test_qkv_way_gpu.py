"""Which kernels make a decode step's queries, keys and values, and that every way leaves the same numbers."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("rows", [1, 8, 9, 16, 17, 48, 49, 64])
@pytest.mark.parametrize("width,heads,kv_heads,dim", [(896, 14, 2, 64), (2048, 16, 2, 128), (96, 3, 1, 32)])
def test_ways_agree(rows, width, heads, kv_heads, dim, monkeypatch):
    from qwenforge_b200 import ops
    from qwenforge_b200.cache import SequenceCache
    from qwenforge_b200.config import PartSpec
    from qwenforge_b200.engine import build_context
    from qwenforge_b200.parts import build_part
    from qwenforge_b200.csrc import prepare
    g = torch.Generator(device=DEV).manual_seed(rows + width)
    names = {f"{k}_{p}": f"{k}.{p}" for k in "qkv" for p in ("weight", "bias")} | {"o_weight": "o.weight"}
    part = build_part("mixer", PartSpec("gqa_attention", {
        "hidden_size": width, "num_heads": heads, "num_kv_heads": kv_heads, "head_dim": dim, "qkv_bias": True, "out_bias": False,
        "scale": dim ** -0.5, "window": 0, "position": PartSpec("rotary_half", {"head_dim": dim, "theta": 1e6})}, names))
    draw = lambda *shape: (torch.randn(*shape, generator=g, device=DEV) * shape[-1] ** -0.5).bfloat16()
    tensors = {"o.weight": draw(width, heads * dim)}
    for k, n in (("q", heads), ("k", kv_heads), ("v", kv_heads)):
        tensors[k + ".weight"], tensors[k + ".bias"] = draw(n * dim, width), draw(n * dim)
    prepare({"embed", "norm"} | part.kernel_libraries(torch.bfloat16) | {q for p in part.sub_parts() for q in p.kernel_libraries(torch.bfloat16)})
    for p in (part, *part.sub_parts()):
        p.bind(tensors, torch.bfloat16, torch.device(DEV))
    stream, norm = torch.randn(rows, width, generator=g, device=DEV), (1 + draw(1, width)[0]).contiguous()
    # (the pending output of the part before: skinny adds it by a kernel of its own, the others in the norm)
    delta = draw(rows, width)
    results = []
    for way in ("skinny", "wide", "unfused"):
        cache = SequenceCache([part.cache_need()], rows * 64, rows, 64, torch.bfloat16, torch.device(DEV))
        slots = [cache.open() for _ in range(rows)]
        cache.reserve([(s, 6 + i % 50) for i, s in enumerate(slots)])
        cache.flush()
        err = torch.zeros(1, dtype=torch.int32, device=DEV)
        ctx = build_context([(s, 5 + i % 50, [1]) for i, s in enumerate(slots)], None, err, torch.bfloat16, torch.device(DEV), "auto",
                            ops.DecodeScratch(torch.device(DEV)))
        ctx.step_memo = {}
        chosen = part._ways(ctx)
        takes = {"skinny": rows <= 16 and ops.skinny_gemm_takes(rows, part.qkv_weight, ops.EPI_QKV, True, n_heads=heads, kv_heads=kv_heads,
                                                                head_dim=dim, rot_dim=dim),
                 "wide": ops.wide_gemm_takes_rows(ops.EPI_QKV, rows, part.qkv_weight, n_heads=heads, kv_heads=kv_heads, head_dim=dim, rot_dim=dim),
                 "unfused": True}
        assert takes[chosen[0]]
        if not takes[way]:
            continue
        monkeypatch.setattr(type(part), "_ways", lambda self, c, way=way: (way, chosen[1]))
        hidden = stream.clone()
        part.fused_forward(hidden, (norm, 1e-6), ctx, cache.site(0), True, delta.clone())
        monkeypatch.undo()
        assert int(err) == 0
        results.append((hidden, cache.site(0).storage.clone()))
    for hidden, storage in results[1:]:
        # queries, keys and values are rounded to bfloat16 from sums in another order: neighbours at most in the cache (2^-7 of a
        # number of order one to four), and a few such differences in the attention's output
        assert float((storage.float() - results[0][1].float()).abs().max()) <= 2 ** -5
        assert float((hidden - results[0][0]).norm() / results[0][0].norm()) < 1e-2


def test_the_rule():
    from qwenforge_b200 import ops
    small, middle = (torch.zeros(n, k, dtype=torch.bfloat16, device=DEV) for n, k in ((1152, 896), (2560, 2048)))
    way = lambda m, w, *heads: ops.qkv_product_way(m, w, *heads)
    assert [way(m, small, 14, 2, 64, 64) for m in (1, 8, 9, 16, 17, 64)] == ["skinny", "skinny", "wide", "wide", "wide", "wide"]
    assert [way(m, middle, 16, 2, 128, 128) for m in (1, 8, 9, 64)] == ["wide"] * 4
    assert way(65, small, 14, 2, 64, 64) == "unfused" and way(9, small[:, :895], 14, 2, 64, 64) == "unfused"


def test_the_rule_beyond_its_band():
    """The band in which the tcgen05 streamer is the faster one for few rows ends at 16 MB, for a single row at 12."""
    from qwenforge_b200 import ops
    between, large = (torch.zeros(n, k, dtype=torch.bfloat16, device=DEV) for n, k in ((3072, 2048), (3584, 2560)))
    assert [ops.qkv_product_way(m, between, 32, 8, 64, 64) for m in (1, 2, 8, 9)] == ["skinny", "wide", "wide", "wide"]
    assert [ops.qkv_product_way(m, large, 20, 4, 128, 128) for m in (1, 2, 8, 9)] == ["skinny", "skinny", "skinny", "wide"]
