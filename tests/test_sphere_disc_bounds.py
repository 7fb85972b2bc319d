"""The FP32 sphere test's error bounds, checked on the host: D = (c.d / sqrt 2)^2
+ c.o + k with o the ray's point nearest the centre and k = (r^2 - |c|^2) / 2
(trace.cu: setup_ray, sphere_disc, certain_sqrt), replayed in numpy float32 with
fma rounded once, against the discriminant and entry distance of the FP64 ray in
extended precision.  Bounds: Edisc = 48u S^2 on 2 (D - |o|^2 / 2), Ep = 48u S on
t, and the certain-hit interval for a reciprocal square root within 2 ulp."""
import numpy as np
import pytest

U = 2.0 ** -24
F = np.float32


def _f(x):
    return np.asarray(x, dtype=F)


def _fma(a, b, c):
    return (a.astype(np.float64) * b.astype(np.float64) + c.astype(np.float64)).astype(F)


def _rays(n, seed, S):
    """Rays past spheres inside |c| + r <= S, many within rounding of tangency, started up to 3 S away or near the sphere."""
    rng = np.random.default_rng(seed)
    r = rng.uniform(.05, 1., n) * min(3.4, .3 * S)
    c = rng.normal(size=(n, 3))
    c *= (rng.uniform(0., 1., n) ** (1 / 3) * (S - r) / np.linalg.norm(c, axis=1))[:, None]
    d = rng.normal(size=(n, 3))
    axis = rng.random(n) < .1                                  # nearly along an axis
    d[axis] = np.eye(3)[rng.integers(0, 3, axis.sum())] + 1e-7 * d[axis]
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    e = rng.normal(size=(n, 3))
    e -= np.sum(e * d, axis=1, keepdims=True) * d
    e /= np.linalg.norm(e, axis=1, keepdims=True)
    delta = rng.choice([0., 1e-7, -1e-7, 1e-5, -1e-5, 1e-3, -1e-3, .3, -.5, -1.], n)
    o = c + (r * (1 + delta))[:, None] * e - (rng.choice([1e-3, .05, 1., 2.], n) * S)[:, None] * d
    keep = np.linalg.norm(o, axis=1) <= 3. * S
    return o[keep], d[keep], c[keep], r[keep]


def _setup(o, d, S):
    S = F(S)
    tau0 = np.sum(o * d, axis=1)
    near = _f(o - tau0[:, None] * d)
    q = _fma(near[:, 0], near[:, 0], _fma(near[:, 1], near[:, 1], near[:, 2] * near[:, 2]))
    dh = _f(d) * F(.707106781)
    thr = F(.5) * (q - F(48 * U) * S * S)
    bmin = (_f(tau0) - F(48 * U) * S) * F(.707106781)
    return near, dh, thr, bmin, F(48 * U) * S * S, F(48 * U) * S


def _test(o, d, c, r, S):
    near, dh, thr, bmin, Edisc, Ep = _setup(o, d, S)
    c32, k = _f(c), _f(.5 * (r * r - np.sum(c * c, axis=1)))
    b = _fma(c32[:, 0], dh[:, 0], _fma(c32[:, 1], dh[:, 1], c32[:, 2] * dh[:, 2]))
    D = _fma(b, b, _fma(c32[:, 0], near[:, 0], _fma(c32[:, 1], near[:, 1], _fma(c32[:, 2], near[:, 2], k))))
    disc = _fma(np.full_like(D, 2), D - thr, np.full_like(D, -Edisc))
    bt = _fma(b - bmin, np.full_like(b, F(1.41421356)), np.full_like(b, -Ep))
    return D, thr, b, bmin, disc, bt, Edisc, Ep


def _true(o, d, c, r):
    o, d, c, r = (np.asarray(v, dtype=np.longdouble) for v in (o, d, c, r))
    x = c - o
    b = np.sum(x * d, axis=1) / np.sum(d * d, axis=1)
    p = x - b[:, None] * d
    return r * r - np.sum(p * p, axis=1), b


@pytest.mark.parametrize('S', [2., 30., 300., 1e4])
def test_discriminant_and_projection_stay_inside_their_bounds(S):
    o, d, c, r = _rays(200_000, int(S), S)
    D, thr, b, bmin, disc, bt, Edisc, Ep = _test(o, d, c, r, S)
    true, proj = _true(o, d, c, r)
    assert float(np.max(np.abs(disc.astype(np.longdouble) - true) / Edisc)) < 1.
    assert float(np.max(np.abs(bt.astype(np.longdouble) - proj) / Ep)) < 1.
    # a certain miss is one: too far from the line, or its centre behind the start
    assert not np.any((D < thr) & (true >= 0)) and not np.any((b < bmin) & (proj > 0))
    assert np.count_nonzero(np.abs(true) < 2 * Edisc) > 1000   # the band does occur


@pytest.mark.parametrize('S', [2., 30., 300.])
def test_certain_hit_interval_holds_the_entry_distance(S):
    o, d, c, r = _rays(200_000, 7 + int(S), S)
    _, _, _, _, disc, bt, Edisc, Ep = _test(o, d, c, r, S)
    true, proj = _true(o, d, c, r)
    sel = disc >= 2 * Edisc
    t_true = (proj - np.sqrt(np.maximum(true, 0)))[sel]
    for ulps in (-2., 2.):
        y = _f(1. / np.sqrt(disc[sel].astype(np.float64)) * (1. + ulps * 2. ** -23))
        s = disc[sel] * y
        t = bt[sel] - s
        Et = F(2) * (Ep + Edisc * y) + F(12 * U) * (np.abs(bt[sel]) + s)
        assert float(np.max(np.abs(t.astype(np.longdouble) - t_true) / Et)) < 1.


def test_lines_beyond_the_scale_meet_no_sphere():
    """q > 1.00002 S^2 drops every sphere: |o| exceeds S by more than FP32 rounding of o and q."""
    S = 25.
    rng = np.random.default_rng(3)
    d = rng.normal(size=(100_000, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    e = rng.normal(size=(100_000, 3))
    e -= np.sum(e * d, axis=1, keepdims=True) * d
    e /= np.linalg.norm(e, axis=1, keepdims=True)
    o = (S * rng.choice([1., 1. + 1e-9, 1. + 1e-6, 1. + 5e-6], 100_000))[:, None] * e - 2 * S * d
    near, _, _, _, _, _ = _setup(o, d, S)
    q = _fma(near[:, 0], near[:, 0], _fma(near[:, 1], near[:, 1], near[:, 2] * near[:, 2]))
    assert not np.any(q > F(1.00002) * F(S) * F(S))
