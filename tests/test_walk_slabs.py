"""The walk's slab test (traverse.cuh visit_slots) restated in numpy float32: for every child it must pass whenever
the plain form t = fma(q, a, o) with a correctly rounded reciprocal passes, and whenever the exact box does, whatever
the reciprocal's last-place error; and its slack must stay below a thirtieth of a quantisation step."""
import numpy as np

F32 = np.float32


def fma(x, y, z):
    """Correctly rounded float32 a * b + c: the product of two float32 is exact in float64, and the sum's second
    rounding is harmless here except at exact ties, which random operands do not meet."""
    return (np.asarray(x, np.float64) * np.asarray(y, np.float64) + np.asarray(z, np.float64)).astype(F32)


def cases(rng, n):
    """Nodes (corner p, power-of-two scale per axis), child boxes (plane bytes) and rays around them."""
    scale = F32(2.0) ** rng.integers(-12, 6, (n, 3)).astype(F32)
    p = (rng.uniform(-100, 100, (n, 3))).astype(F32)
    lo = rng.integers(0, 250, (n, 3))
    hi = np.minimum(255, lo + rng.integers(1, 120, (n, 3)))
    d = rng.standard_normal((n, 3))
    d[: n // 8, 0] *= 1e-6  # nearly parallel to a slab
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(F32)
    # origins aimed at a point of the box or just beside it, from near and far
    at = p + scale * (lo + (hi - lo) * rng.uniform(-0.02, 1.02, (n, 3)))
    o = (at - d.astype(np.float64) * 10 ** rng.uniform(-3, 3, (n, 1))).astype(F32)
    return p, scale, lo, hi, o, d


def planes(d, lo, hi):
    neg = np.signbit(d)
    return np.where(neg, hi, lo), np.where(neg, lo, hi)


def test_slab_test_passes_every_box_the_plain_and_the_exact_forms_pass():
    rng = np.random.default_rng(11)
    p, scale, lo, hi, o, d = cases(rng, 400000)
    qn, qf = planes(d, lo, hi)
    tmax = F32(2.0) ** 60
    exact_inv = (1.0 / d.astype(np.float64))
    near_x = (p.astype(np.float64) + qn * scale - o) * exact_inv
    far_x = (p.astype(np.float64) + qf * scale - o) * exact_inv
    exact = np.maximum(near_x.max(1), 0) <= far_x.min(1)

    inv = (F32(1) / d).astype(F32)
    a, off = scale * inv, (p - o) * inv
    plain = np.maximum(fma(qn.astype(F32), a, off).max(1), F32(0)) <= np.minimum(fma(qf.astype(F32), a, off).min(1), tmax)
    assert 0.3 < exact.mean() < 0.99

    for ulp in (-1, 0, 1):  # the approximate reciprocal may be off by one unit in the last place
        r = inv if ulp == 0 else np.nextafter(inv, inv * F32(4 if ulp > 0 else 0))
        a, off = scale * r, (p - o) * r
        base = fma(F32(-65536), a, off)
        slack = fma(np.minimum(np.abs(off), F32(2.0) ** 100), F32(2.0) ** -20, np.abs(a) * F32(2.0) ** -6)
        near = fma((65536 + qn).astype(F32), a, base - slack)
        far = fma((65536 + qf).astype(F32), a, base + slack)
        got = np.maximum(near.max(1), F32(0)) <= np.minimum(far.min(1), tmax)
        assert not (plain & ~got).any()
        assert not (exact & ~got).any()
        # never much more than that: boxes a thirtieth of a step (or 2^-18 of the distance) outside still miss
        grow = np.abs(scale / 30 * exact_inv) + np.abs(off.astype(np.float64)) * 2.0 ** -18
        wide = np.maximum((near_x - grow).max(1), 0) <= (far_x + grow).min(1)
        assert not (got & ~wide).any()


def test_degenerate_directions_are_containment_tests():
    """|d| <= FLT_EPSILON on an axis: the stand-in reciprocal 2^92 keeps the sign of (plane - origin)."""
    rng = np.random.default_rng(5)
    p, scale, lo, hi, o, d = cases(rng, 50000)
    s = F32(2.0) ** 92
    inside = p[:, 0].astype(np.float64) + scale[:, 0] * (lo[:, 0] + (hi[:, 0] - lo[:, 0]) * rng.uniform(0.05, 0.95, len(p)))
    outside = p[:, 0].astype(np.float64) + scale[:, 0] * (hi[:, 0] + rng.uniform(0.05, 100, len(p)))
    for org, want in ((inside.astype(F32), True), (outside.astype(F32), False)):
        a, off = scale[:, 0] * s, (p[:, 0] - org) * s
        base = fma(F32(-65536), a, off)
        slack = fma(np.minimum(np.abs(off), F32(2.0) ** 100), F32(2.0) ** -20, np.abs(a) * F32(2.0) ** -6)
        near = fma((65536 + lo[:, 0]).astype(F32), a, base - slack)
        far = fma((65536 + hi[:, 0]).astype(F32), a, base + slack)
        ok = np.maximum(near, F32(0)) <= np.minimum(far, F32(1e6))
        # the origin's own rounding may move it by a few units in the last place of the coordinate
        sure = scale[:, 0] * 0.04 > np.spacing(np.abs(org).astype(F32)) * 4
        assert (ok[sure] == want).all()
        assert sure.mean() > 0.5
