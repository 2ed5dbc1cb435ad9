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
