"""Shadow rays towards point lights that add exactly zero: lg_render traces none (the reference traces them up to three
radii), the image is the one without such lights, bit for bit, and the statistics count what was traced."""
import numpy as np
import pytest

import lumina
import oracle as O

pytestmark = pytest.mark.gpu


def _render(scene, points, camera, nodes, tris):
    sun = scene.sun.copy()
    sun["intensity"] = 2.0
    sc = lumina.Scene(scene.camera, sun, tris, scene.mat_albedo, scene.mat_emissive, points)
    with lumina.Renderer(0) as r:
        r.set_scene_bvh(sc, nodes)
        r.set_counting(True)
        ours = r.render(camera=camera, spp=8, bounces=2)
    return ours, O.oracle_render(sc, nodes, tris, 8, 2, camera=camera)


@pytest.mark.parametrize("scene", ["box_scene", "small_engine_scene"])
def test_no_ray_and_no_difference(scene, request):
    scene = request.getfixturevalue(scene)
    nodes, tris, _, _ = O.oracle_build_bvh(scene.tris)
    camera = scene.camera.copy()
    camera.width, camera.height = 128, 64
    dark = scene.points.copy()
    dark["intensity"] = 0.0
    with_dark, (want, reference) = _render(scene, np.concatenate([dark, scene.points]), camera, nodes, tris)
    without, (_, fewer) = _render(scene, scene.points, camera, nodes, tris)
    assert without["accum"].any() and np.array_equal(with_dark["accum"], without["accum"])
    for k in ("closest_rays", "shadow_rays"):
        assert with_dark[k] == without[k]
    assert reference["shadow_rays"] > fewer["shadow_rays"]  # the reference traces the dark lights' rays
    assert with_dark["shadow_rays"] <= fewer["shadow_rays"] * 1.001
    assert abs(with_dark["closest_rays"] - reference["closest_rays"]) <= 1e-3 * reference["closest_rays"]
    close = np.abs(with_dark["accum"] - want) <= 1e-3 * np.maximum(np.abs(want), np.abs(with_dark["accum"])) + 1e-6
    assert close.all(axis=2).mean() >= 0.999
