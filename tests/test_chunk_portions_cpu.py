"""How much the chunked recurrences keep between their launches, whatever the step."""
import pytest

from qwenforge_b200.ops import kernels


@pytest.mark.parametrize("n,n_seqs", [(200, 1), (4206, 3), (32768, 1), (1 << 20, 1), (131072, 64), (300, 100), (65536, 2)])
@pytest.mark.parametrize("chunk,floats", [(128, 32 * (128 * 128 + 129)), (64, 16 * (64 * 128 + 64)), (128, 7 * (64 * 128 + 65))])
def test_records_have_a_bound(n, n_seqs, chunk, floats):
    records, each = kernels._chunk_portions(n, n_seqs, chunk, floats)
    assert records == (n_seqs * each if each else n // chunk + n_seqs)   # room for every chunk of a portion, or of the step
    assert records * floats * 4 <= max(kernels.CHUNK_SCRATCH_BYTES, 4 * n_seqs * floats * 4)
