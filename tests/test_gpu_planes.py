"""The lean traversal's plane test and its lazily taken quadric roots against the general analytic path:
the same shapes in a scene that also holds a cone frustum far below them, which runs the Full
instantiations."""
import numpy as np
import pytest

import owec_abi as A
import owe_cuda
import scenes

pytestmark = pytest.mark.gpu


def plane_scene(full, quadrics=False):
    """Rectangles, an annulus, a disk and an ellipse, tilted and axis-parallel, one behind another; or a
    sphere, a flat and two curved sags (one an annulus) and a cylinder."""
    sb = scenes.SceneBuilder()
    grey = sb.diffuse(0.5)
    if quadrics:
        tilt = scenes.pose(scenes.rotate_to((0, 0, 1), (0.3, -0.2, 0.9)), (0.1, 0.0, 0.5))
        for shape, params, xf in ((A.SHAPE_SPHERE, [0.5], scenes.translate(0.6, 0.1, 0.7)),
                                  (A.SHAPE_SAG, [0.0, 0.0, 0.8, 0.2], scenes.translate(0.0, 0.0, 1.6)),
                                  (A.SHAPE_SAG, [1.0, -0.5, 0.7, 0.0], tilt),
                                  (A.SHAPE_SAG, [-0.8, 0.2, 0.9, 0.3], scenes.translate(-0.5, 0.0, 0.2)),
                                  (A.SHAPE_CYLINDER, [0.4, -0.5, 1.0], scenes.translate(-0.8, 0.3, 0.4))):
            sb.boundary(shape, params, xf, 0, 0, grey)
        if full:
            sb.boundary(A.SHAPE_CONE, [0.1, 0.0, 0.05, 0.1], scenes.translate(0.0, 0.0, -50.0), 0, 0, grey)
        sb.observer(8, 8, (0.0, -3.0, 1.0), (0.0, 0.0, 0.5))
        return sb.desc()
    tilt = scenes.pose(scenes.rotate_to((0, 0, 1), (0.3, -0.2, 0.9)), (0.1, 0.0, 0.5))
    side = scenes.pose(scenes.rotate_to((0, 0, 1), (1, 0, 0)), (-1.0, 0.0, 0.7))
    for xf, params in ((scenes.pose(), [A.APERTURE_RECT, 1.5, 1.0]), (tilt, [A.APERTURE_DISK, 0.6, 0.2]),
                       (side, [A.APERTURE_ELLIPSE, 0.5, 0.8]),
                       (scenes.pose(scenes.rotate_to((0, 0, 1), (0, 0, -1)), (0, 0, 1.5)), [A.APERTURE_DISK, 1.2, 0.0])):
        sb.boundary(A.SHAPE_PLANE, params, xf, 0, 0, grey)
    if full:
        sb.boundary(A.SHAPE_CONE, [0.1, 0.0, 0.05, 0.1], scenes.translate(0.0, 0.0, -50.0), 0, 0, grey)
    sb.observer(8, 8, (0.0, -3.0, 1.0), (0.0, 0.0, 0.5))
    return sb.desc()


def rays():
    o, d = scenes.random_rays(20001, 3, (-2, -2, -0.5), (2, 2, 2), (-1, -1, 0), (1, 1, 1.5))
    # along the planes and straight at their edges, centres and rims
    o2 = np.array([[0, 0, 3], [1.5, 1.0, 3], [1.5, 0, 3], [0, 0, 0], [-3, 0, 0.7], [-3, 0.5, 0.7], [0, 0, 1.0], [0.2, 0, 3]], float)
    d2 = np.array([[0, 0, -1], [0, 0, -1], [0, 0, -1], [1, 0, 0], [1, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, -1]], float)
    return np.concatenate([o, o2]), np.concatenate([d, d2])


@pytest.mark.parametrize("quadrics", [False, True])
@pytest.mark.parametrize("precision", [A.PRECISION_MIXED, A.PRECISION_FP32, A.PRECISION_FP64])
def test_lean_shapes_match_the_general_path(precision, quadrics):
    o, d = rays()
    got = []
    for full in (False, True):
        with owe_cuda.Context(0) as c:
            c.set_settings(A.make_settings(precision=precision))
            c.upload(plane_scene(full, quadrics))
            c.build_bvh()
            got.append(c.cast_rays(o, d))
    (b0, p0, t0), (b1, p1, t1) = got
    assert (b0 < 5).sum() > 5000
    # the cone is met by no ray; the boundaries agree but where the two paths round a rim differently
    same = b0 == b1
    assert same.mean() > (0.9995 if precision == A.PRECISION_FP32 else 0.99999)
    assert (p0[same] == p1[same]).all()
    hit = same & (b0 < 5)
    # the same refined roots: a few ulps of the arithmetic
    tol = 1e-5 if precision == A.PRECISION_FP32 else 1e-11
    assert np.abs(t0[hit] - t1[hit]).max() <= tol * np.abs(t1[hit]).max()
