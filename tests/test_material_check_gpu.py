"""Material indices are checked on the device after the upload: the first bad triangle is reported, the renderer is
left without a scene, and a valid scene set afterwards renders, by both set-up calls.  (The tree is the oracle's, so
that this runs where the reference's library is absent.)"""
import pytest

import lumina
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("supplied_tree", [False, True])
def test_bad_material_index_is_rejected(box_scene, supplied_tree):
    nodes, bvh_tris, _, _ = O.oracle_build_bvh(box_scene.tris)
    tris = (bvh_tris if supplied_tree else box_scene.tris).copy()
    tris["material"][5], tris["material"][7] = 99, -1
    bad = lumina.Scene(box_scene.camera, box_scene.sun, tris, box_scene.mat_albedo, box_scene.mat_emissive,
                       box_scene.points)
    with lumina.Renderer(0) as r:
        with pytest.raises(lumina.LuminaError) as e:
            r.set_scene_bvh(bad, nodes) if supplied_tree else r.set_scene(bad)
        assert e.value.code == -1 and "triangle 5 has material 99" in str(e.value)
        assert not r.render(spp=1, bounces=0)["rgb"].any()  # no scene: every pixel misses
        r.set_scene(box_scene)
        assert r.render(spp=1, bounces=0)["rgb"].any()
