"""FP64 rays that start far from what they meet: the same hits as from nearby, and no more of the tree visited than
FP32 slabs of FP32 rays would take."""
import math

import numpy as np
import pytest

import owec_abi as A
import owe_cuda
import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("distance", [1e2, 1e4, 1e6])
def test_node_visits_from_far_away(distance):
    visits = {}
    for precision in (A.PRECISION_MIXED, A.PRECISION_FP64):
        sb = scenes.SceneBuilder()
        v, t = scenes.uv_sphere(256, 128)
        sb.boundary(A.SHAPE_MESH, [], scenes.pose(), 0, 0, sb.diffuse(0.5), -1, sb.mesh(v, t))
        sb.sun((0.5, 0.6, 0.7), 1.0e4)
        sb.observer(64, 64, (0.0, -distance, 0.3 * distance), (0.0, 0.0, 0.0), fov_y_deg=math.degrees(2.0 / distance))
        sb.frame_origin((0.0, 0.0, 0.0))  # at the sphere: the rays start far from it
        with owe_cuda.Context(0) as c:
            c.upload(sb.desc())
            c.set_settings(A.make_settings(max_depth=1, precision=precision))
            c.trace_counters(True)
            c.run_pass(1)
            n = c.trace_counters(False)
        visits[precision] = n[1] / n[0]
    # FP32 rays' slabs are widened by at least what FP64 rays' are (2.4e-7 of the distance)
    assert visits[A.PRECISION_FP64] <= 1.02 * visits[A.PRECISION_MIXED], visits


@pytest.mark.parametrize("full", [False, True])
def test_hits_do_not_depend_on_how_far_back_an_fp64_ray_starts(full):
    sb = scenes.bvh_stress_room(8, 8, 128, 64)
    if full:
        sb.boundary(A.SHAPE_CONE, [0.1, 0.0, 0.05, 0.1], scenes.translate(0.0, 0.0, -50.0), 0, 0, sb.diffuse(0.5))
    # from above the ceiling's height outside the walls, so that nothing but the room lies on the longer rays
    o, d = scenes.random_rays(20001, 3, (-2.5, -2.5, 6.0), (2.5, 2.5, 9.0), (-1.0, -1.0, 0.1), (1.0, 1.0, 3.9))
    with owe_cuda.Context(0) as c:
        c.set_settings(A.make_settings(precision=A.PRECISION_FP64))
        c.upload(sb.desc())
        want = c.cast_rays(o, d)
        for back in (1e1, 1e3, 1e5):
            got = c.cast_rays(o - back * d, d)
            # the origin moves off the ray by its rounding, 1e-16 of the way: a near tie at most
            same = (got[0] == want[0]) & (got[1] == want[1])
            assert same.mean() >= 0.9995
            assert np.abs(got[2] - back - want[2])[same].max() <= 1e-14 * back + 1e-12
