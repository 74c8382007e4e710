"""Device LBVH with leaves wider than the 512 sorted triangles of a block, whose boxes the block fits together: runs
of equal Morton codes of every place and length, several side by side, and zeros of both signs, whose order in the
run decides the sign in the box.  Byte-identical to the oracle's."""
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
    return nodes


@pytest.mark.parametrize("runs", [[40], [17, 16, 15], [503, 9, 600, 17, 530], [511, 513, 512], [5000, 3], [1, 20000, 1],
                                  [30] * 60, [700, 1400, 2100, 40, 40]])
def test_runs_of_equal_codes(runs):
    """Runs at places along x, the triangles of all runs shuffled."""
    n = sum(runs)
    rng = np.random.default_rng(n)
    t = soup(n, 5)
    x = np.repeat(np.arange(len(runs)), runs).astype(np.float32)
    shape = rng.normal(0, 1e-4, (n, 3, 3))
    t["v"] = shape - shape.mean(1, keepdims=True) + np.stack([x, 0 * x, 0 * x], -1)[:, None, :] + 0.5
    _same(t[rng.permutation(n)])


@pytest.mark.parametrize("n", [513, 1600, 9000])
@pytest.mark.parametrize("positive_at", [0, 1, 300, 512, -1])
def test_signed_zeros_in_a_wide_leaf(n, positive_at):
    """Triangles in the plane x = -0 but for one at +0: the first one's sign is the box's."""
    t = soup(n, 7)
    t["v"] = np.array([[-0.0, 0, 0], [-0.0, 1, 0], [-0.0, 0, 1]], np.float32)
    t["v"][positive_at, :, 0] = 0.0
    nodes = _same(t)
    assert len(nodes) == 1
    assert np.signbit(nodes["bbMin"][0, 0]) == (positive_at != 0)
