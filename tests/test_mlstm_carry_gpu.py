"""The mLSTM's states from one chunk to the next: spans of more chunks than a block composes at a time, heads of one and of several
blocks, and a matrix that blocks do not divide, against float64 as in test_chunk_scan_gpu."""
import pytest

from test_chunk_scan_gpu import test_mlstm_in_chunks_is_as_near_to_64_bits_as_token_by_token as check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lengths,heads,dim,vdim,forget", [
    ([8300, 70], 1, 8, 64, 6.0),          # 130 chunks and 2; one block a head
    ([64, 129], 3, 32, 48, 2.0),          # three blocks a head
    ([4225, 65], 2, 12, 128, 4.0),        # the first chunk of a third run of 32; key channels that are no power of two
    ([130], 2, 16, 36, 1.0),              # 576 elements: no whole blocks
])
def test_states_are_carried_as_near_to_64_bits(lengths, heads, dim, vdim, forget):
    check(lengths, heads, dim, vdim, forget)
