"""The render tree at the sizes where its build changes form (4,096 clusters: the rounds move into one block) and
at very small ones: a frame through the traversal records equals the same frame over BuildBVH's own topology."""
import numpy as np
import pytest

import lumina

pytestmark = pytest.mark.gpu


def _scene(n, seed):
    """n small triangles scattered in front of the camera of the box room."""
    base = lumina.box_scene(1, width=96, height=48)
    rng = np.random.default_rng(seed)
    t = np.zeros(n, base.tris.dtype)
    c = rng.uniform([-3, -3.5, 0.2], [3.5, 3.5, 3.8], (n, 3))
    t["v"] = (c[:, None, :] + rng.normal(0, 0.25, (n, 3, 3))).astype(np.float32)
    e1, e2 = t["v"][:, 1] - t["v"][:, 0], t["v"][:, 2] - t["v"][:, 0]
    nrm = np.cross(e1, e2)
    t["n"] = (nrm / np.linalg.norm(nrm, axis=1, keepdims=True))[:, None, :]
    t["material"] = rng.integers(0, len(base.mat_albedo), n)
    return lumina.Scene(base.camera, base.sun, t, base.mat_albedo, base.mat_emissive, base.points)


@pytest.mark.parametrize("n", [1, 2, 3, 33, 1023, 1025, 4095, 4096, 4097, 9000])
def test_frame_does_not_depend_on_the_tree(n):
    with lumina.Renderer(0) as r:
        r.set_scene(_scene(n, n))
        a = r.render(spp=4, bounces=1)["accum"]
        r.set_render_tree("buildbvh")
        b = r.render(spp=4, bounces=1)["accum"]
    # the closest hits are the same up to exact ties in t and hits on a box face
    same = np.isclose(a, b, rtol=1e-3, atol=1e-6).all(axis=2)
    assert same.mean() >= 0.999
