"""How much the chunked recurrences keep between their launches, whatever the step."""
import pytest

from qwenforge_b200.ops import kernels


@pytest.mark.parametrize("n,n_seqs", [(200, 1), (4206, 3), (32768, 1), (1 << 20, 1), (131072, 64), (300, 100), (65536, 2)])
@pytest.mark.parametrize("chunk,floats", [(128, 32 * (128 * 128 + 129)), (64, 16 * (64 * 128 + 64)), (128, 7 * (64 * 128 + 65))])
def test_records_have_a_bound(n, n_seqs, chunk, floats):
    records, each = kernels._chunk_portions(n, n_seqs, chunk, floats)
    assert records == (n_seqs * each if each else n // chunk + n_seqs)   # room for every chunk of a portion, or of the step
    assert records * floats * 4 <= max(kernels.CHUNK_SCRATCH_BYTES, 4 * n_seqs * floats * 4)


@pytest.mark.parametrize("lengths,heads,dim,vdim,state,rows", [
    ([2048], 7, 64, 128, True, True), ([2175, 1000, 1031], 32, 128, 128, True, None), ([192] + [1] * 31, 7, 64, 128, False, None),
    ([512] + [1] * 31, 16, 64, 128, False, False), ([1024] + [1] * 31, 16, 64, 128, True, True), ([192] + [1] * 63, 32, 128, 128, False, None),
    ([512] + [1] * 63, 32, 64, 64, False, False), ([1024] * 4, 32, 64, 64, True, True), ([512] * 64, 7, 64, 128, True, True)])
def test_many_short_sequences_beside_a_long_one_keep_the_scan(lengths, heads, dim, vdim, state, rows):
    """Where both forms were measured, the rule names the faster one (None: a size that the form is not made for)."""
    n = sum(lengths)
    pays = lambda chunk, costs: kernels._chunks_pay(n, len(lengths), max(lengths), heads * dim * vdim, chunk, *costs)
    assert pays(kernels.STATE_CHUNK, kernels.STATE_CHUNKS_COSTS) is state
    if rows is not None:
        assert pays(kernels.ROW_CHUNK, kernels.ROW_CHUNKS_COSTS) is rows
