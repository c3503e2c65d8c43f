"""Which kernels make the gate and up product of a step of up to 64 token rows, at both sides of every line of the rule."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


# 0.5B's (17 MB) and 3B's (90 MB) weights, one on either side of 100 MB, 7B's (272 MB), and columns that no streamer takes
@pytest.mark.parametrize("rows,k,ways", [
    (9728, 896, {1: "skinny", 8: "skinny", 9: "skinny", 16: "skinny", 17: "unfused", 48: "unfused", 64: "unfused"}),
    (22016, 2048, {1: "skinny", 4: "skinny", 8: "skinny", 9: "unfused", 16: "unfused", 48: "unfused", 64: "unfused"}),
    (24400, 2048, {1: "skinny", 8: "skinny", 9: "unfused", 64: "unfused"}), (24432, 2048, {1: "wide", 16: "wide", 64: "wide"}),
    (37888, 3584, {1: "wide", 8: "wide", 9: "wide", 64: "wide"}), (37888, 1404, {1: "unfused", 64: "unfused"})])
def test_the_rule(rows, k, ways):
    """Below 100 MB the gate is float32's own exponential and division: the tcgen05 streamer, whose gate is the hardware's, is not chosen."""
    from qwenforge_b200 import ops
    weight = torch.empty(rows, k, dtype=torch.bfloat16, device=DEV)
    assert {m: ops.gate_product_way(m, weight) for m in ways} == ways
