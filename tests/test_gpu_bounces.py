"""The bounce loop at its edges: depths from none to far beyond any path's end, films from one pixel up, passes in
one call and in several, batches of one pass after another, images still being copied when the film is cleared,
and paths through null boundaries that outlive the depth."""
import numpy as np
import pytest

import owec_abi as A
import owe_cuda
import scenes

pytestmark = pytest.mark.gpu


def render(c, passes):
    c.reset_film()
    for spp in passes:
        c.run_pass(spp)
    img, n = c.resolve()
    return img, n, c.stats()


@pytest.mark.parametrize("integrator", ["path", "light"])
@pytest.mark.parametrize("size,spp", [((1, 1), 1), ((8, 8), 1), ((33, 17), 3), ((257, 129), 2)])
@pytest.mark.parametrize("depth", [0, 1, 5, 64, 300])
def test_depths_and_film_sizes(size, spp, depth, integrator):
    desc = scenes.materials_gallery(*size).desc()
    with owe_cuda.Context(0) as c:
        c.upload(desc)
        c.set_settings(A.make_settings(seed=2, max_depth=depth, rr_depth=4, integrator=integrator))
        a = render(c, [spp])
        b = render(c, [1] * spp)  # the same sample streams, a pass at a time
    assert np.isfinite(a[0]).all() and np.isfinite(b[0]).all()
    assert a[2]["device_faults"] == 0 and b[2]["device_faults"] == 0
    if integrator == "path":
        assert a[2] == b[2]
        assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
        assert a[2]["paths"] == size[0] * size[1] * spp
        assert a[2]["segments"] >= a[2]["paths"]
    else:
        # the particles of a pass are numbered within it, so only their count is the same
        assert a[1].sum() == b[1].sum()


@pytest.mark.parametrize("precision", [A.PRECISION_MIXED, A.PRECISION_FP32, A.PRECISION_FP64])
def test_times_of_a_pass(precision):
    desc = scenes.bvh_stress_room(160, 90, 64, 32).desc()
    with owe_cuda.Context(0) as c:
        c.upload(desc)
        c.set_settings(A.make_settings(max_depth=6, rr_depth=3, precision=precision))
        for _ in range(3):
            c.run_pass(2)
            total, intersect, shadow, launches = c.last_pass_timing()
            # the two kinds of kernel overlap each other but not themselves (20 us: the timer's steps)
            assert 0 < intersect < total + 2e-5 and 0 < shadow < total + 2e-5
            assert launches >= 7


@pytest.mark.parametrize("size,spp", [((33, 17), 3), ((64, 64), 1030)])
@pytest.mark.parametrize("precision", [A.PRECISION_MIXED, A.PRECISION_FP32, A.PRECISION_FP64])
def test_light_passes_repeat_to_the_bit(size, spp, precision):
    """Splats are fixed-point sums: a connection lost or counted twice beside the next bounce's closest-hit kernel
    would show in any bit. The larger pass takes three batches of 2^21 particles."""
    desc = scenes.materials_gallery(*size).desc()
    with owe_cuda.Context(0) as c:
        c.upload(desc)
        c.set_settings(A.make_settings(seed=2, max_depth=12, rr_depth=4, precision=precision, integrator="light"))
        a = render(c, [spp])
        b = render(c, [spp])
    assert a[0].max() > 0 and a[2]["device_faults"] == 0
    assert a[2] == b[2]
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])


@pytest.mark.parametrize("integrator", ["path", "light"])
def test_film_cleared_while_its_image_is_copied(integrator):
    desc = scenes.bvh_stress_room(641, 359, 64, 32).desc()
    with owe_cuda.Context(0) as c:
        c.upload(desc)
        c.set_settings(A.make_settings(seed=6, max_depth=5, integrator=integrator))
        want = render(c, [1])
        c.reset_film()
        c.run_pass(1)
        out = np.zeros((359, 641, 3))
        samples = np.zeros((359, 641))
        c.resolve_async(out, samples)
        c.reset_film()
        c.run_pass(1)
        c.resolve_wait()
        again = c.resolve()
    assert np.array_equal(out, want[0]) and np.array_equal(samples, want[1])
    assert np.array_equal(again[0], want[0]) and np.array_equal(again[1], want[1])
