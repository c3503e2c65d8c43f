"""What a block leaves pending, on its own."""
import torch

from qwenforge_b200.parts.base import PendingSums


def test_a_value_outlives_the_sums_it_was_taken_from():
    """All layers of a step share the rows of `PendingSums`; the next layer takes them along and leaves zeros."""
    sums = torch.ones(2, 4)
    seen = PendingSums(sums).value()
    sums.zero_()
    assert bool((seen == 1).all())
