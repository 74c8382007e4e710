"""Device LBVH at the sizes where its blocks and sort tiles end (512 sorted
triangles per block, 2,048 keys per tile) and with runs of equal Morton codes
that cross them: node arrays, order and permutation byte-identical to the
oracle's."""
import numpy as np
import pytest

import lumina
import oracle as O
from test_oracle import soup

pytestmark = pytest.mark.gpu


def _same(tris):
    nodes, out, perm = lumina.build_bvh(tris)
    on, ot, operm, _ = O.oracle_build_bvh(tris)
    assert nodes.tobytes() == on.tobytes()
    assert out.tobytes() == ot.tobytes()
    assert (perm == operm).all()


@pytest.mark.parametrize("n", [511, 512, 513, 1023, 1025, 2047, 2048, 2049, 4097, 65535, 65537])
def test_block_and_tile_edges(n):
    _same(soup(n, n))


@pytest.mark.parametrize("n,run,at", [(1200, 5, 509), (1200, 700, 300), (3000, 2500, 100), (2600, 2600, 0)])
def test_equal_codes_across_blocks(n, run, at):
    """A run of triangles at one place in a row of triangles sorted along x: a leaf wider than a block's share."""
    t = soup(n, 3)
    x = np.linspace(-5, 5, n).astype(np.float32)
    x[at:at + run] = x[at]
    shape = np.array([[0, 0, 0], [1e-4, 0, 0], [0, 1e-4, 1e-4]], np.float32)
    t["v"] = shape[None] + np.stack([x, 0 * x, 0 * x], -1)[:, None, :]
    _same(t)
