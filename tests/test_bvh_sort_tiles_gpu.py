"""Device LBVH at the sizes where its sort changes tiles: 1,024 sorted keys a tile up to 151,552 triangles, 2,048 up to
303,104, 4,096 up to 606,208, 8,192 above; at each end, and with a ragged last tile between.  Node arrays, order and
permutation byte-identical to the oracle's."""
import pytest

import lumina
import oracle as O
from test_oracle import soup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [100003, 151552, 151553, 200007, 303104, 303105, 450001, 606208, 606209, 700001])
def test_both_sides_of_each_tile_size(n):
    tris = soup(n, n)
    nodes, out, perm = lumina.build_bvh(tris)
    on, ot, operm, _ = O.oracle_build_bvh(tris)
    assert nodes.tobytes() == on.tobytes()
    assert out.tobytes() == ot.tobytes()
    assert (perm == operm).all()
