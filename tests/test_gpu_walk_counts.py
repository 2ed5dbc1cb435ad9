"""Forward walks in any split: the bins and counters of walks 0 .. n - 1 do not depend on how many calls,
warps or refills they take."""
import numpy as np
import pytest

import owec_abi as A
import owe_cuda
import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("splat", [A.SPLAT_NEAREST, A.SPLAT_BILINEAR])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 127, 129, 4097, 100003])
def test_walks_do_not_depend_on_their_split(n, splat):
    sb, info = scenes.achromat_scene(film=64)
    w = scenes.achromat_walk(info, seed=3, splat=splat)
    got = []
    with owe_cuda.Context(0) as c:
        c.upload(sb.desc())
        c.build_bvh()
        for cuts in ((0, n), (0, n // 3, n // 2, n)):
            c.walk_reset()
            for a, b in zip(cuts, cuts[1:]):
                c.walk(w, a, b - a)
            got.append(c.walk_resolve())
    (b0, s0), (b1, s1) = got
    assert s0 == s1 and s0["walks"] == n and s0["events"] >= n and s0["faults"] == 0
    assert np.array_equal(b0, b1)
    assert (s0["binned"] > 0) == (b0.sum() > 0)


@pytest.mark.parametrize("precision", [A.PRECISION_MIXED, A.PRECISION_FP32, A.PRECISION_FP64])
@pytest.mark.parametrize("n", [1, 33, 383, 385, 148 * 384 - 1, 148 * 384 + 1])
def test_walks_of_general_scenes_do_not_depend_on_their_split(n, precision):
    """The kernels of scenes with general shapes (a cone that no walk meets), at the edges of their blocks."""
    sb, info = scenes.achromat_scene(film=64)
    sb.boundary(A.SHAPE_CONE, [0.1, 0.0, 0.05, 0.1], scenes.translate(0.0, 0.0, -50.0), 0, 0, sb.diffuse(0.5))
    w = scenes.achromat_walk(info, seed=3)
    got = []
    with owe_cuda.Context(0) as c:
        c.set_settings(A.make_settings(precision=precision))
        c.upload(sb.desc())
        c.build_bvh()
        for cuts in ((0, n), (0, n // 3, n // 2, n)):
            c.walk_reset()
            for a, b in zip(cuts, cuts[1:]):
                c.walk(w, a, b - a)
            got.append(c.walk_resolve())
    (b0, s0), (b1, s1) = got
    assert s0 == s1 and s0["walks"] == n and s0["events"] >= n and s0["faults"] == 0
    assert np.array_equal(b0, b1)
