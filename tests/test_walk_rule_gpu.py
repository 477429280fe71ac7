"""The states of the chunked scans by the walk and by sums and carry, as the rule takes them: one span and several, sizes between
the walk's tiles of 64 x 64, against float64 as in test_chunk_routes_gpu."""
import pytest

from test_chunk_routes_gpu import test_walk_and_shared_read_outs as check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,lengths,heads,groups,dim,vdim,launches", [
    ("scalar", [600], 64, 8, 128, 64, 1),                       # eight heads a block of the read-outs
    ("scalar", [65, 130], 64, 8, 128, 64, 1),
    ("scalar", [65, 130], 200, 200, 66, 70, 1),                 # two tiles each way, one nearly empty
    ("scalar", [130], 48, 3, 40, 33, 2),                        # sixteen heads share keys
    ("channel", [65, 130], 200, 200, 64, 64, 1), ("channel", [100, 64], 200, 200, 40, 50, 1),
    ("channel", [65, 130], 56, 56, 64, 64, 2),
    ("constant", [65, 130], 200, 200, 64, 66, 1), ("constant", [65, 130], 56, 56, 64, 64, 2),
])
def test_states_by_either_route(kind, lengths, heads, groups, dim, vdim, launches):
    from celeg_b200 import kernels
    chunks = 2 * (sum(lengths) // 128 + len(lengths)) if kind == "constant" else sum(lengths) // 64 + len(lengths)
    assert kernels.chunk_state_launches(heads, dim, vdim, len(lengths), chunks) == launches
    tiles = -(-vdim // 32) * -(-dim // 64) * heads * len(lengths)
    check(kind, lengths, heads, groups, dim, vdim, tiles >= 222)
