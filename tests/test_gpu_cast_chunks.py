"""Host rays at the edges of the chunks they travel in: any batch gives what its rays give in small calls,
also into a film-sized context that renders in between."""
import numpy as np
import pytest

import owec_abi as A
import owe_cuda
import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 255, 4096, 4097, 8193, 16385, 40000, 16 * 4096, 16 * 4096 + 1, 5 * 16384, 300001])
def test_batches_match_their_rays_in_small_calls(n):
    desc = scenes.bvh_stress_room(16, 16, 64, 32).desc()
    o, d = scenes.random_rays(n, 5, (-2.5, -2.5, 0.3), (2.5, 2.5, 3.7), (-1.2, -1.2, 0.1), (1.2, 1.2, 2.4))
    with owe_cuda.Context(0) as c:
        c.upload(desc)
        c.set_settings(A.make_settings(max_depth=4))
        whole = c.cast_rays(o, d)
        c.run_pass(1)
        again = c.cast_rays(o, d)
        parts = [c.cast_rays(o[a:a + 10007], d[a:a + 10007]) for a in range(0, n, 10007)]
    for k in range(3):
        assert np.array_equal(whole[k], again[k])
        assert np.array_equal(whole[k], np.concatenate([p[k] for p in parts]))
    assert (whole[0] < 8).all()


@pytest.mark.parametrize("integrator", ["path", "light"])
def test_a_reset_film_starts_from_nothing(integrator):
    """A cleared film renders what a fresh context's does, whatever it held."""
    desc = scenes.bvh_stress_room(33, 17, 32, 16).desc()
    st = A.make_settings(seed=3, max_depth=5, integrator=integrator)
    images = []
    for passes_before in (0, 2):
        with owe_cuda.Context(0) as c:
            c.upload(desc)
            c.set_settings(st)
            for _ in range(passes_before):
                c.run_pass(3)
            if passes_before:
                c.reset_film()
            c.run_pass(2)
            images.append(c.resolve())
    assert np.array_equal(images[0][0], images[1][0])
    assert np.array_equal(images[0][1], images[1][1])


@pytest.mark.parametrize("n", [65537, 8 * 8192, 9 * 8192 - 1, 9 * 8192 + 1, (1 << 21) - 1, (1 << 21) + 1])
def test_pieces_of_large_batches(n):
    """Batches around the pieces that the staging threads deal out, and around the size whose device memory the
    context keeps: every ray's answer in its own place, whatever thread carried it."""
    desc = scenes.bvh_stress_room(16, 16, 64, 32).desc()
    o, d = scenes.random_rays(4099, 7, (-2.5, -2.5, 0.3), (2.5, 2.5, 3.7), (-1.2, -1.2, 0.1), (1.2, 1.2, 2.4))
    pick = np.arange(n) % 4099  # coprime to the pieces: a piece out of place would show
    with owe_cuda.Context(0) as c:
        c.upload(desc)
        want = c.cast_rays(o, d)
        for _ in range(2):
            got = c.cast_rays(o[pick], d[pick])
            for k in range(3):
                assert np.array_equal(got[k], want[k][pick])


@pytest.mark.parametrize("precision", [A.PRECISION_MIXED, A.PRECISION_FP32, A.PRECISION_FP64])
def test_large_batches_of_general_shapes(precision):
    desc = scenes.wave_pool(16, 16).desc()
    o, d = scenes.random_rays(70001, 3, (-0.2, -0.2, 0.05), (0.2, 0.2, 0.5), (-0.2, -0.2, -0.1), (0.2, 0.2, 0.0))
    with owe_cuda.Context(0) as c:
        c.set_settings(A.make_settings(precision=precision))
        c.upload(desc)
        whole = c.cast_rays(o, d)
        parts = [c.cast_rays(o[a:a + 10007], d[a:a + 10007]) for a in range(0, len(o), 10007)]
    for k in range(3):
        assert np.array_equal(whole[k], np.concatenate([p[k] for p in parts]))


def test_rays_may_be_overwritten_by_their_hits():
    """Distances written over the origins' array: all rays are read before the first answer is written."""
    desc = scenes.bvh_stress_room(16, 16, 64, 32).desc()
    n = 200001
    o, d = scenes.random_rays(n, 9, (-2.5, -2.5, 0.3), (2.5, 2.5, 3.7), (-1.2, -1.2, 0.1), (1.2, 1.2, 2.4))
    with owe_cuda.Context(0) as c:
        c.upload(desc)
        b, p, t = c.cast_rays(o, d)
        flat = o.reshape(-1)
        b2, p2 = np.zeros(n, np.uint32), np.zeros(n, np.uint32)
        owe_cuda._check(c.lib, c.lib.owec_cast_rays(
            c.handle, n, flat.ctypes.data_as(A.c_double_p), d.ctypes.data_as(A.c_double_p), b2.ctypes.data_as(A.c_u32_p),
            p2.ctypes.data_as(A.c_u32_p), flat.ctypes.data_as(A.c_double_p)), "owec_cast_rays")
    assert np.array_equal(flat[:n], t) and np.array_equal(b2, b) and np.array_equal(p2, p)
