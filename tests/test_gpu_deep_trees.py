"""Trees with more pending levels than the traversal keeps in shared memory: octants nested toward a corner over
twenty octaves, against the oracle and against the same triangles in a shallow tree."""
import numpy as np
import pytest

import owec_abi as A
import owe_cuda
import scenes
from oracle_ref import PortEngine

pytestmark = pytest.mark.gpu

PRECISIONS = [A.PRECISION_MIXED, A.PRECISION_FP32, A.PRECISION_FP64]


def nested_vertices(octaves):
    """Of each octave's cube, the seven octants away from the origin hold four triangles each, two of them toward
    either end of the octant's diagonal: a wide node per octave whose children are wide nodes too, so that a ray
    from the corner outward leaves some of them pending at every level."""
    rng = np.random.default_rng(1)
    v = []
    for k in range(octaves):
        s = 2.0 ** -k
        for octant in range(1, 8):
            lo = np.array([(octant >> a) & 1 for a in range(3)]) * (s / 2)
            for low in (0, 1, 0, 1):
                at = lo + s / 2 * (0.03 if low else 0.92) + s / 2 * rng.uniform(0.0, 0.05, 3)
                inward = s / 2 if low else -s / 2
                v += [at, at + inward * rng.uniform(0.0, 0.3, 3), at + inward * rng.uniform(0.0, 0.3, 3)]
    return np.array(v)


def nested_octants(octaves, null_box=False, size=24, shallow=False):
    """Those triangles under a sun and a sky, seen from just outside the corner. shallow: one more triangle, a metre
    wide and 10,000 km below, takes all but a few of the Morton codes' values, so that the tree over the others is
    split by their order and a few levels deep."""
    v = nested_vertices(octaves)
    if shallow:
        v = np.concatenate([v, np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0]]) - [0.0, 0.0, 1e7]])
    sb = scenes.SceneBuilder()
    sb.boundary(A.SHAPE_MESH, [], scenes.pose(), 0, 0, sb.diffuse(0.5), -1,
                sb.mesh(v, np.arange(len(v), dtype=np.uint32).reshape(-1, 3)))
    if null_box:
        bv, bt = scenes.box_mesh((0.955, 0.955, 0.955), (0.97, 0.97, 0.97))
        fog = sb._medium(A.INDEX_CONSTANT, (1.0,), absorption=sb.spectrum_constant(0.2))
        sb.boundary(A.SHAPE_MESH, [], scenes.pose(), 0, sb.region(fog), sb.optics_(A.SURF_NULL), -1, sb.mesh(bv, bt))
    sb.sun((0.5, 0.6, 0.7), 1.0e4)
    sb.uniform_sky(1.0)
    e = 2.0 ** -octaves
    sb.observer(size, size, (-1.0 * e, -1.1 * e, -0.9 * e), (1.0, 1.0, 1.0), fov_y_deg=50.0)
    sb.frame_origin((0.0, 0.0, 0.0))
    return sb.desc()


def node_visits_per_query(desc, precision):
    with owe_cuda.Context(0) as c:
        c.upload(desc)
        c.set_settings(A.make_settings(max_depth=1, precision=precision))
        c.trace_counters(True)
        c.run_pass(1)
        n = c.trace_counters(False)
        return n[1] / n[0], c.bvh_info()["nodes"]


def rays(n):
    """From near the corner, at every octave's scale, toward the middles of triangles of every octave; half of them
    the other way, from outside into the corner."""
    rng = np.random.default_rng(2)
    near = rng.uniform(-1.0, 0.0, (n, 3)) * 2.0 ** -rng.uniform(4, 20, (n, 1))
    middles = nested_vertices(20).reshape(-1, 3, 3).mean(1)
    target = middles[rng.integers(0, len(middles), n)]
    d = target - near
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    outward = np.arange(n)[:, None] % 2 == 1
    return np.where(outward, near, near + 2.5 * d), np.where(outward, d, -d)


def test_hits_match_the_oracle():
    desc = nested_octants(20)
    o, d = rays(4001)
    rb, rp, rt = PortEngine(desc).cast_rays(o, d)
    with owe_cuda.Context(0) as c:
        c.set_settings(A.make_settings(precision=A.PRECISION_FP64))
        c.upload(desc)
        b, p, t = c.cast_rays(o, d)
    assert (rb == 0).sum() > 500
    same = (b == rb) & (p == rp)
    assert same.mean() >= 0.9999
    hit = same & (rb < 2)
    assert np.abs(t - rt)[hit].max() <= 1e-9 * max(1.0, rt[hit].max())


@pytest.mark.parametrize("precision", PRECISIONS)
def test_hits_do_not_depend_on_the_tree(precision):
    o, d = rays(40001)
    got = []
    for shallow in (False, True):
        with owe_cuda.Context(0) as c:
            c.set_settings(A.make_settings(precision=precision))
            c.upload(nested_octants(20, shallow=shallow))
            got.append(c.cast_rays(o, d))
    (b0, p0, t0), (b1, p1, t1) = got
    assert np.array_equal(b0, b1) and (b0 == 0).sum() > 5000
    # a hit's distance comes from its triangle and the ray alone; which of two triangles at the same FP32 distance
    # is named depends on the order they are met in, and the mixed mode refines the named one's
    if precision != A.PRECISION_MIXED:
        assert np.array_equal(t0, t1)
    if precision == A.PRECISION_FP64:
        assert np.array_equal(p0, p1)
    same = p0 == p1
    assert np.array_equal(t0[same], t1[same])
    # the FP32 distance's error: a few ulps of coordinates up to 2.5
    tied = ~same & (b0 == 0)
    assert (np.abs(t0[tied] - t1[tied]) <= 4 * 2.4e-7 * 2.5).all()


@pytest.mark.parametrize("null_box", [False, True])
@pytest.mark.parametrize("precision", PRECISIONS)
def test_films_do_not_depend_on_the_tree(precision, null_box):
    films = []
    for shallow in (False, True):
        with owe_cuda.Context(0) as c:
            c.upload(nested_octants(20, null_box, shallow=shallow))
            c.set_settings(A.make_settings(seed=5, max_depth=6, rr_depth=3, precision=precision))
            c.run_pass(4)
            films.append((c.resolve()[0], c.stats()))
    assert films[0][1]["device_faults"] == 0 and films[0][1]["segments"] > films[0][1]["paths"]
    assert films[0][1] == films[1][1]
    assert np.array_equal(films[0][0], films[1][0])


@pytest.mark.parametrize("precision", PRECISIONS)
def test_deep_levels_are_not_traversed_twice(precision):
    """Down through ten more octaves and up again: a node and a few pending ones per octave, as through the first
    ten; sixteen visits more where the query starts again at the seventeenth level."""
    shallow, _ = node_visits_per_query(nested_octants(5), precision)
    middle, _ = node_visits_per_query(nested_octants(10), precision)
    deep, nodes = node_visits_per_query(nested_octants(20), precision)
    assert nodes > 100
    assert deep - middle <= 2 * (middle - shallow) + 4, (shallow, middle, deep)


def cell_of_triangles(count, shallow=False):
    """Octants nested over twenty octaves of 10 km, and `count` triangles in a row along the diagonal of the smallest
    one's corner, all within one Morton cell: split by their order, they add six levels of their own."""
    v = 1e4 * nested_vertices(20)
    s = 1e4 * 2.0 ** -23  # about a millimetre: a quarter of a cell
    at = (np.arange(count) + 0.5)[:, None] / count * s * np.ones(3)
    size = 0.3 * s / count
    row = np.stack([at, at + [size, 0.0, -size], at + [-size, size, 0.0]], 1).reshape(-1, 3)
    v = np.concatenate([v, row])
    if shallow:
        v = np.concatenate([v, np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0]]) - [0.0, 0.0, 1e11]])
    sb = scenes.SceneBuilder()
    sb.boundary(A.SHAPE_MESH, [], scenes.pose(), 0, 0, sb.diffuse(0.5), -1,
                sb.mesh(v, np.arange(len(v), dtype=np.uint32).reshape(-1, 3)))
    sb.uniform_sky(1.0)
    e = 1e4 * 2.0 ** -25
    sb.observer(16, 16, (-1.0 * e, -1.1 * e, -0.9 * e), (1e4, 1e4, 1e4), fov_y_deg=4.0)
    sb.frame_origin((0.0, 0.0, 0.0))
    return sb.desc()


@pytest.mark.parametrize("precision", PRECISIONS)
def test_levels_beyond_the_shared_stack(precision):
    """More pending levels than the shared stack ever holds: the query starts again with the deep one."""
    count = 8 ** 6
    rng = np.random.default_rng(3)
    n = 512
    e = 1e4 * 2.0 ** -25
    o = -e * rng.uniform(0.5, 1.5, (n, 3))
    d = 1.0 + 0.02 * rng.uniform(-1.0, 1.0, (n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    got = []
    for shallow in (False, True):
        with owe_cuda.Context(0) as c:
            c.set_settings(A.make_settings(precision=precision))
            c.upload(cell_of_triangles(count, shallow))
            got.append(c.cast_rays(o, d))
    (b0, p0, t0), (b1, p1, t1) = got
    assert np.array_equal(b0, b1) and (b0 < 1).any()
    if precision != A.PRECISION_MIXED:
        assert np.array_equal(t0, t1)
    if precision == A.PRECISION_FP64:
        assert np.array_equal(p0, p1)
    desc = cell_of_triangles(count)
    few, _ = node_visits_per_query(cell_of_triangles(1), precision)
    many, _ = node_visits_per_query(desc, precision)
    print("node visits per query", few, many)
    with owe_cuda.Context(0) as c:
        c.upload(desc)
        c.set_settings(A.make_settings(seed=5, max_depth=3, precision=precision))
        c.run_pass(1)
        assert c.stats()["device_faults"] == 0
