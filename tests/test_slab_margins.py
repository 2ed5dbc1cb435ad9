"""The traversal's node test of an FP64 ray, its FP32 arithmetic restated operation by operation: no box that the
ray meets exactly is refused, and boxes farther off than the FP64 test would let pass are."""
from fractions import Fraction

import numpy as np

F = np.float32


def fma(a, b, c):
    # the product of two FP32 numbers is exact in FP64; the sum's second rounding is far below the margins here
    return F(np.float64(a) * np.float64(b) + np.float64(c))


def slab_test(node_o, exps, qlo, qhi, od, d, tmax):
    """intersectChildren<double> for one child: (near, far) of the three axes together."""
    te, tx = F(0), F(np.inf)
    for k in range(3):
        inv64 = 1.0 / (d[k] if abs(d[k]) > 1e-18 else np.copysign(1e-18, d[k]))
        inv = F(inv64)
        a = F(F(2.0) ** F(exps[k])) * inv
        a8 = a * F(0.00390625)
        b = F((np.float64(node_o[k]) - od[k]) * inv64)
        bx = b - F(32768) * a
        m = F(0.004) * abs(a) + F(2.4e-7) * abs(bx)
        near, far = bx - m, bx + m
        qn, qf = (qhi[k], qlo[k]) if inv < 0 else (qlo[k], qhi[k])
        te = max(te, fma(F(8388608 + 256 * int(qn)), a8, near))
        tx = min(tx, fma(F(8388608 + 256 * int(qf)), a8, far))
    limit = np.nextafter(F(tmax), F(np.inf)) if np.float64(F(tmax)) < tmax else F(tmax)
    return te <= min(tx, limit)


def exact_interval(node_o, exps, qlo, qhi, od, d):
    lo, hi = Fraction(0), None
    for k in range(3):
        s = Fraction(2) ** int(exps[k])
        p0, p1 = Fraction(float(node_o[k])) + s * int(qlo[k]), Fraction(float(node_o[k])) + s * int(qhi[k])
        o, v = Fraction(float(od[k])), Fraction(float(d[k]))
        t0, t1 = (p0 - o) / v, (p1 - o) / v
        lo, hi = max(lo, min(t0, t1)), max(t0, t1) if hi is None else min(hi, max(t0, t1))
    return lo, hi


def draw(rng, offset_quanta):
    """A node at up to 1e6 m, a child box of it, and a ray from up to 1e9 m away toward a corner or an inner point
    of the box, moved sideways by that many quanta plus a share of the distance."""
    node_o = (rng.uniform(-1, 1, 3) * 10.0 ** rng.uniform(-3, 6)).astype(np.float32)
    size = 10.0 ** rng.uniform(-4, 5)
    exps = np.round(np.log2(size / 255)) + rng.integers(-2, 1, 3)
    qlo = rng.integers(0, 255, 3)
    qhi = np.minimum(255, qlo + rng.integers(0, 40, 3))
    s = 2.0 ** exps
    corner = rng.integers(0, 2, 3)
    where = np.where(corner, qhi, qlo) if rng.random() < 0.5 else rng.uniform(qlo, qhi)
    target = node_o.astype(np.float64) + where * s
    d = rng.normal(size=3)
    if rng.random() < 0.3:
        d[rng.integers(0, 3)] *= 10.0 ** -rng.uniform(3, 9)
    d /= np.linalg.norm(d)
    dist = size * 10.0 ** rng.uniform(-2, 9)
    side = np.cross(d, rng.normal(size=3))
    side /= np.linalg.norm(side)
    od = target - d * dist + side * offset_quanta(s, dist)
    return node_o, exps, qlo, qhi, od, d, dist


def test_no_box_the_ray_meets_is_refused():
    rng = np.random.default_rng(3)
    met = 0
    with np.errstate(over="ignore"):
        for _ in range(20000):
            node_o, exps, qlo, qhi, od, d, dist = draw(rng, lambda s, r: 0.0)
            lo, hi = exact_interval(node_o, exps, qlo, qhi, od, d)
            if hi < lo:
                continue
            met += 1
            # the limit: somewhere past the entry, down to the entry itself
            tmax = float(lo) + (float(hi) - float(lo)) * rng.uniform(0, 2) if rng.random() < 0.7 else float(lo)
            if Fraction(tmax) < lo:
                tmax = np.nextafter(tmax, np.inf)
            assert slab_test(node_o, exps, qlo, qhi, od, d, tmax), (node_o, exps, qlo, qhi, od, d, tmax)
    assert met > 8000


def test_boxes_well_off_the_ray_are_refused():
    """A cube beside a ray through space at 45 degrees to every axis: refused once it lies farther off than the
    widening, 2.4e-7 of the distance from the ray's origin to the node and a hundredth of a quantum, however far
    from the frame's origin both are."""
    rng = np.random.default_rng(4)
    for _ in range(5000):
        size = 10.0 ** rng.uniform(-4, 3)
        node_o = (rng.uniform(-1, 1, 3) * 10.0 ** rng.uniform(-3, 6)).astype(np.float32)
        exps = np.full(3, np.round(np.log2(size / 255)))
        s = 2.0 ** exps[0]
        lo = int(rng.integers(0, 200))
        qlo, qhi = np.full(3, lo), np.full(3, lo + 30)
        dist = size * 10.0 ** rng.uniform(0, 7)
        d = np.array([1.0, 1.0, 1.0]) / np.sqrt(3)
        centre = node_o.astype(np.float64) + (lo + 15) * s
        gap = 4 * (0.01 * s + 2.6e-7 * (dist + 500 * s)) + 1e-15 * (dist + np.abs(node_o).max())
        # moved along +x, -y by half the cube and the gap: the x and y intervals no longer overlap
        od = centre - d * dist + np.array([1.0, -1.0, 0.0]) * (15 * s + gap)
        assert not slab_test(node_o, exps, qlo, qhi, od, d, np.inf)
