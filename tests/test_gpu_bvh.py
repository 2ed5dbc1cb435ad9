"""The device BVH build at the edges of its node and level sizes, and heightfields set on the device
against the same meshes uploaded."""
import numpy as np
import pytest

import owec_abi as A
import owe_cuda
import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 2, 3, 8, 9, 17, 64, 65, 513])
def test_every_primitive_of_a_stack_is_found(count):
    """Horizontal sheets one above another: a vertical ray between two of them meets the next one."""
    sb = scenes.SceneBuilder()
    grey = sb.diffuse(0.5)
    for k in range(count):
        sb.sheet(1.0 + 0.25 * (k % 3), 1.0, scenes.translate(0.0, 0.0, float(k)), grey)
    sb.observer(8, 8, (0.0, -3.0, 0.5 * count), (0.0, 0.0, 0.0))
    rng = np.random.default_rng(count)
    n = 4 * count + 64
    o = np.stack([rng.uniform(-0.9, 0.9, n), rng.uniform(-0.9, 0.9, n), rng.uniform(-1.0, count, n)], 1)
    up = rng.integers(0, 2, n)
    d = np.stack([np.zeros(n), np.zeros(n), np.where(up, 1.0, -1.0)], 1)
    with owe_cuda.Context(0) as c:
        c.upload(sb.desc())
        c.build_bvh()
        info = c.bvh_info()
        b, _, t = c.cast_rays(o, d)
    assert info["prims"] == count
    met = np.where(up, np.ceil(o[:, 2]), np.floor(o[:, 2]))
    hit = (met >= 0) & (met < count)
    assert ((b < count) == hit).all()
    assert (b[hit] == met[hit]).all()
    assert np.abs(t[hit] - np.abs(met[hit] - o[hit, 2])).max() <= 1e-9 * count


@pytest.mark.parametrize("precision", [A.PRECISION_MIXED, A.PRECISION_FP32, A.PRECISION_FP64])
@pytest.mark.parametrize("n", [2, 3, 17, 64])
def test_heightfield_set_on_the_device_is_the_mesh_uploaded(n, precision):
    rng = np.random.default_rng(n)
    h = rng.uniform(-2e-4, 2e-4, (n, n))
    h[0] = h[-1] = 0
    h[:, 0] = h[:, -1] = 0
    o, d = scenes.random_rays(20000, n, (-0.06, -0.06, 0.05), (0.06, 0.06, 0.2), (-0.05, -0.05, 0.009), (0.05, 0.05, 0.011))
    got = []
    for uploaded in (True, False):
        sb, info = scenes.caustic_slab_scene(n=n, heights=h if uploaded else None)
        with owe_cuda.Context(0) as c:
            c.set_settings(A.make_settings(precision=precision))
            c.upload(sb.desc())
            c.build_bvh()
            if not uploaded:
                c.set_heightfield(info["heightfield"], info["thickness"], rng.uniform(-1e-3, 1e-3, (n, n)))
                c.set_heightfield(info["heightfield"], info["thickness"], h)
            got.append(c.cast_rays(o, d) + (c.bvh_info()["nodes"],))
    for a, b in zip(*got):
        assert np.array_equal(a, b)
    assert (got[0][0] == info["heightfield"]).sum() > 1000
