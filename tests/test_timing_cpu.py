"""The per-kernel times name every call that launches kernels."""
import inspect
import re
from pathlib import Path

import qwenforge_b200
from qwenforge_b200 import ops
from qwenforge_b200.ops.timing import TIMED


def test_every_launching_call_of_the_parts_is_timed():
    folder = Path(qwenforge_b200.__file__).parent
    called = set()
    for path in [p for name in ("parts", "engine", "sampling") for p in (folder / name).rglob("*.py")]:
        called |= set(re.findall(r"\bops\.(\w+)\(", path.read_text()))
    functions = {name: getattr(ops, name) for name in called if inspect.isfunction(getattr(ops, name, None))}
    launching = {name for name, fn in functions.items() if re.search(r"_stream\(\)|\blinear\(|\bskinny_gemm\(|torch\.mm\(", inspect.getsource(fn))}
    assert {"qkv_product", "tc_gemm_tail", "linear", "linear_rows", "gated_rows", "rope_cache_write"} <= launching
    assert sorted(launching - set(TIMED)) == []
    assert all(inspect.isfunction(getattr(ops, name)) for name in TIMED) and len(set(TIMED)) == len(TIMED)
