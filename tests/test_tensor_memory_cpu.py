"""Kernels that take tensor memory: the order of allocation and programmatic launch, read from the sources (getting it wrong would
hang a GPU, so it is not tried on one)."""
import re
from pathlib import Path

import pytest

SOURCES = Path(__file__).resolve().parent.parent / "qwenforge_b200" / "csrc"


def kernels():
    for path in sorted([*SOURCES.glob("*.cu"), *SOURCES.glob("*.cuh")]):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for body in text.split("__global__")[1:]:
            body = body[:body.index("\n}")]
            if "tcgen05.alloc" in body:
                name = re.search(r"(\w+_kernel)\(", body).group(1)
                yield pytest.param(body, id=f"{path.name}:{name}")


def test_the_kernels_are_found():
    files = {p.id.split(":")[0] for p in kernels()}
    assert files == {p.name for p in SOURCES.glob("*.cu*") if "tcgen05.alloc" in re.sub(r"//[^\n]*", "", p.read_text())} and len(files) >= 4


@pytest.mark.parametrize("body", list(kernels()))
def test_tensor_memory_before_the_next_kernel_may_start(body):
    allocated = body.index("tcgen05.alloc")
    for early in ("grid_launch_dependents()", "grid_chain_entry()"):
        if early in body:
            assert body.index("__syncthreads()", allocated) < body.index(early)
    assert body.index("tcgen05.dealloc") > body.rindex("__syncthreads()")


def test_every_kernel_keeps_to_the_rule_of_shared_memory():
    """Each source that allocates holds its launches to `qf_tmem_fits` (when it is compiled) or asks for the least that it allows."""
    for path in SOURCES.glob("*.cu*"):
        text = path.read_text()
        launches = len(re.findall(r"cudaFuncAttributeMaxDynamicSharedMemorySize", text)) if "tcgen05.alloc" in text else 0
        assert launches == 0 or "static_assert(qf_tmem_fits(" in text or "QF_TMEM_SMEM_SHARED" in text, path.name
