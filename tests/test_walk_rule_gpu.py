"""The states of the chunked scans by the walk and by sums and carry, as the rule takes them: one span and several, sizes between
the walk's tiles, against float64 as in test_chunk_routes_gpu, which asks the rules what they take."""
import pytest

from test_chunk_routes_gpu import test_walk_and_shared_read_outs as check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,lengths,heads,groups,dim,vdim,columns,share", [
    ("scalar", [600], 64, 8, 128, 64, 64, 4),
    ("scalar", [65, 130], 64, 8, 128, 64, 32, 2),
    ("scalar", [65, 130], 200, 200, 66, 70, 32, 1),             # two tiles along the keys, three of 32 columns, one nearly empty
    ("scalar", [130], 48, 3, 40, 33, 0, 1),                     # sixteen heads share keys
    ("channel", [65, 130], 200, 200, 64, 64, 32, 1), ("channel", [100, 64], 200, 200, 40, 50, 32, 1),
    ("channel", [65, 130], 56, 56, 64, 64, 64, 1),
    ("constant", [65, 130], 200, 200, 64, 66, 32, 1), ("constant", [65, 130], 56, 56, 64, 64, 64, 1),
])
def test_states_by_either_route(kind, lengths, heads, groups, dim, vdim, columns, share):
    check(kind, lengths, heads, groups, dim, vdim, columns, share)
