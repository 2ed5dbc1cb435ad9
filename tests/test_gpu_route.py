"""Scenes without media through their own routing kernel against the medium kernel: the same scene with a
region of absorbing medium that no boundary faces."""
import numpy as np
import pytest

import owec_abi as A
import owe_cuda
import scenes

pytestmark = pytest.mark.gpu

SCENES = {"sun": lambda: scenes.glass_sphere_on_floor(48, 33), "sky": lambda: scenes.gradient_sky_scene(48, 33),
          "textures": lambda: scenes.texture_gallery(48, 33), "metals": lambda: scenes.materials_gallery(48, 33, fog_box=False),
          "room": lambda: scenes.bvh_stress_room(48, 33, 64, 32)}


@pytest.mark.parametrize("precision", [A.PRECISION_MIXED, A.PRECISION_FP32, A.PRECISION_FP64])
@pytest.mark.parametrize("name", sorted(SCENES))
def test_routing_without_media_matches_the_medium_kernel(name, precision):
    got = []
    for medium in (False, True):
        sb = SCENES[name]()
        if medium:
            sb.region(sb._medium(A.INDEX_CONSTANT, (1.0,), absorption=sb.spectrum_constant(0.5)))
        with owe_cuda.Context(0) as c:
            c.upload(sb.desc())
            c.set_settings(A.make_settings(seed=4, max_depth=12, rr_depth=4, precision=precision))
            c.run_pass(2)
            got.append((c.resolve()[0], c.stats()))
    (a, sa), (b, sb_) = got
    # the same decisions; the sky's and the sun's sum may round differently (a few ulps of FP32 per event)
    assert sa == sb_
    assert np.linalg.norm(a - b) <= 1e-6 * np.linalg.norm(b)
