"""The exact answers for box corners and the bounded-permanent f64 stage of the
device predicates (exact.cuh: orient3d_box, lifted_box, five_box, orient4d_box,
insphere_mid), restated in Python and compared with exact rational
determinants.  The device code itself is checked against the oracle by
tests/test_predicates_gpu.py."""
from fractions import Fraction

import numpy as np
import pytest

EPS = 2.0 ** -53


def det3(m):
    return (m[0][0] * (m[1][1] * m[2][2] - m[1][2] * m[2][1]) - m[0][1] * (m[1][0] * m[2][2] - m[1][2] * m[2][0])
            + m[0][2] * (m[1][0] * m[2][1] - m[1][1] * m[2][0]))


def sign(x):
    return (x > 0) - (x < 0)


def exact(p):
    return [[Fraction(float(c)) for c in q] for q in p]


def orient3d(p):
    q = exact(p)
    return sign(det3([[q[i][k] - q[3][k] for k in range(3)] for i in range(3)]))


def lifted(p):
    q = exact(p)
    w = [sum(c * c for c in r) for r in q]
    return sign(det3([[q[i][0] - q[3][0], q[i][1] - q[3][1], w[i] - w[3]] for i in range(3)]))


def insphere_value(p):
    q = exact(p)
    d = [[q[i][k] - q[4][k] for k in range(3)] for i in range(4)]
    rows = [r + [sum(c * c for c in r)] for r in d]
    total = Fraction(0)
    for i in range(4):  # along the lift column
        minor = det3([rows[j][:3] for j in range(4) if j != i])
        total += (-1) ** (i + 3) * rows[i][3] * minor
    return total


def bits(p, axis):
    v = [float(q[axis]) for q in p]
    lo, hi = min(v), max(v)
    return None if any(x not in (lo, hi) for x in v) else [int(x != lo) for x in v], lo, hi


def det_bits(x, y, z):
    return sign(det3([[x[i] - x[3], y[i] - y[3], z[i] - z[3]] for i in range(3)]))


def corners(r, count, spans):
    lo = r.integers(-60, 60, 3)
    ext = r.integers(0 if spans == "flat" else 1, 9, 3)
    c = r.integers(0, 2, (count, 3))
    return ((lo + c * ext).astype(np.float64) / 71.0).astype(np.float32)


@pytest.mark.parametrize("spans", ["full", "flat"])
def test_box_corners(spans):
    r = np.random.default_rng(5)
    seen = set()
    for _ in range(3000):
        p = corners(r, 5, spans)
        b = [bits(p[:4], k) for k in range(3)]
        s = det_bits(*[x[0] for x in b])
        assert orient3d(p[:4]) == s
        w = b[2][2] + b[2][1]
        assert lifted(p[:4]) == s * sign(w)
        assert insphere_value(p) == 0  # any five corners
        seen.add((s, sign(w)))
        if s == 0:  # every permutation of the lifted terms is 0 too: the cascade goes on to its next point set
            for perm in ((0, 2, 1), (1, 2, 0)):
                assert lifted(p[:4][:, perm]) == 0
    assert len(seen) >= 6 or spans == "flat"


def test_three_values_are_not_a_box():
    p = np.array([[0, 0, 0], [1, 0, 0], [2, 1, 0], [0, 1, 1]], np.float32)
    assert bits(p, 0)[0] is None


def mid(p):
    """insphere_mid's determinant and bound (f64 operations in its order, the r_i in f32)."""
    e = p[4]
    r = [np.max(np.abs(p[i] - e)) for i in range(4)]  # f32 differences
    bound = (((16.0 + 224.0 * EPS) * EPS * 18.0 * (1.0 + 2.0 ** -18)) * (float(r[0]) * float(r[1]))
             * (float(r[2]) * float(r[3]))) * ((float(r[0]) + float(r[1])) + (float(r[2]) + float(r[3])))
    d = [[float(p[i][k]) - float(e[k]) for k in range(3)] for i in range(4)]
    (ax, ay, az), (bx, by, bz), (cx, cy, cz), (dx, dy, dz) = d
    ab, bc, cd = ax * by - bx * ay, bx * cy - cx * by, cx * dy - dx * cy
    da, ac, bd = dx * ay - ax * dy, ax * cy - cx * ay, bx * dy - dx * by
    abc = (az * bc - bz * ac) + cz * ab
    bcd = (bz * cd - cz * bd) + dz * bc
    cda = (cz * da + dz * ac) + az * cd
    dab = (dz * ab + az * bd) + bz * da
    al, bl = (ax * ax + ay * ay) + az * az, (bx * bx + by * by) + bz * bz
    cl, dl = (cx * cx + cy * cy) + cz * cz, (dx * dx + dy * dy) + dz * dz
    return (dl * abc - cl * dab) + (bl * cda - al * bcd), bound


@pytest.mark.parametrize("kind", ["uniform", "sphere", "super", "tiny", "lattice"])
def test_bounded_permanent(kind):
    r = np.random.default_rng(11)
    sup = np.array([[-100, -100, -100], [400, -100, -100], [-100, 400, -100], [-100, -100, 400]], np.float32)
    decided = 0
    for _ in range(600):
        p = r.random((5, 3)).astype(np.float32)
        if kind == "sphere":
            g = r.standard_normal((5, 3))
            p = (0.5 + 0.4 * g / np.linalg.norm(g, axis=1, keepdims=True)).astype(np.float32)
        elif kind == "super":
            k = r.integers(1, 4)
            p[r.choice(4, k, replace=False)] = sup[r.choice(4, k, replace=False)]
        elif kind == "tiny":
            p = (r.random(3) + 1e-6 * r.random((5, 3))).astype(np.float32)
        elif kind == "lattice":
            p = (r.integers(0, 6, (5, 3)) / np.float32(71)).astype(np.float32)
        det, bound = mid(p)
        want = insphere_value(p)
        assert abs(Fraction(det) - want) <= Fraction(bound)
        if abs(det) > bound:
            decided += 1
            assert sign(det) == sign(want)
    assert decided > (50 if kind == "lattice" else 400)


def rough(p):
    """insphere_f32's determinant and its bound on the permanent (f32 operations in its order)."""
    f = np.float32
    e = p[4]
    d = [[f(p[i][k] - e[k]) for k in range(3)] for i in range(4)]
    r = [max(abs(x) for x in q) for q in d]
    factor = f(f(f(16.0) + f(f(224.0) * f(2.0 ** -24))) * f(2.0 ** -24)) * f(18.0) * f(1.0 + 3.0e-5)
    bound = f(f(f(f(f(r[0] * r[1]) * f(factor)) * f(r[2] * r[3])) * f(f(r[0] + r[1]) + f(r[2] + r[3]))) + f(1e-33))
    (ax, ay, az), (bx, by, bz), (cx, cy, cz), (dx, dy, dz) = d
    m = lambda u, v, w, x: f(f(u * v) - f(w * x))  # noqa: E731
    ab, bc, cd = m(ax, by, bx, ay), m(bx, cy, cx, by), m(cx, dy, dx, cy)
    da, ac, bd = m(dx, ay, ax, dy), m(ax, cy, cx, ay), m(bx, dy, dx, by)
    abc = f(f(f(az * bc) - f(bz * ac)) + f(cz * ab))
    bcd = f(f(f(bz * cd) - f(cz * bd)) + f(dz * bc))
    cda = f(f(f(cz * da) + f(dz * ac)) + f(az * cd))
    dab = f(f(f(dz * ab) + f(az * bd)) + f(bz * da))
    lift = [f(f(f(x * x) + f(y * y)) + f(z * z)) for x, y, z in d]
    return f(f(f(lift[3] * abc) - f(lift[2] * dab)) + f(f(lift[1] * cda) - f(lift[0] * bcd))), bound


@pytest.mark.parametrize("kind,scale", [("uniform", 1.0), ("super", 1.0), ("tiny", 1e-4), ("tiny", 1e-8), ("tiny", 1e-12)])
def test_rough_bound(kind, scale):
    r = np.random.default_rng(13)
    sup = np.array([[-100, -100, -100], [400, -100, -100], [-100, 400, -100], [-100, -100, 400]], np.float32)
    decided = 0
    for _ in range(600):
        p = (scale * r.random((5, 3))).astype(np.float32)
        if kind == "super":
            k = r.integers(1, 4)
            p[r.choice(4, k, replace=False)] = sup[r.choice(4, k, replace=False)]
        det, bound = rough(p)
        want = insphere_value(p)
        assert abs(Fraction(float(det)) - want) <= Fraction(float(bound))
        decided += abs(det) > bound
    assert decided > 500 or scale < 1e-4
