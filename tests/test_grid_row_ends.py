"""The FP32 row ends of the adaptive grid (row_ends and exact_ends, pa_grid.cu),
replayed in numpy against extended precision: an end's error stays inside the
bound the kernel decides by, so an end that FP32 decides is the exact one.

Every FP32 operation below rounds once (products and sums of an fma are formed
in extended precision first); the approximate reciprocal square root is moved
by its two units in the last place either way.  The tolerance is the kernel's
own bound e; an end counts as decided where |distance to the nearest pixel
centre| > e and rem >= 4 tol, as in the kernel."""
import numpy as np
import pytest

f, X = np.float32, np.longdouble


def _fma(a, b, c):
    return (X(1) * a * b + c).astype(f)


def _row_ends(fx, fy, r2, r, dy_int, ulps):
    tol = f(2.) ** -23 * _fma(f(4.) * r, r, _fma(f(3.), r, f(2.)))
    dy = dy_int.astype(f) - fy
    rem = _fma(-dy, dy, r2)
    q = (1 / np.sqrt(np.maximum(rem, tol).astype(X)) * (1 + ulps * X(2.) ** -23)).astype(f)
    half = rem * q
    e = _fma(tol, q, _fma(half, f(2.) ** -20, f(2.) ** -20))
    xl, xr = fx - half, fx + half
    kl, kr = np.rint(xl), np.rint(xr)               # adding and taking off 1.5 2^23 rounds to nearest even
    return dict(kl=kl, kr=kr, fl=xl - kl, fr=xr - kr, e=e, rem=rem, tol=tol)


def _disks(kind, n, seed):
    rng = np.random.default_rng(seed)
    if kind == 'ends on pixel centres':              # Pythagorean rows: ends that are whole numbers, and a little off them
        a, b = rng.integers(1, 40, (2, n))
        big, small = np.maximum(a, b) + 1, np.minimum(a, b)
        r, dy = (big * big + small * small).astype(float), (big * big - small * small).astype(float)
        shift = rng.choice([0., 1e-15, -1e-15, 1e-9, -1e-9, 1e-6, -1e-6, 1e-4, -1e-4], n)
        return np.abs(shift), np.zeros(n), r + rng.choice([0., 1e-12, -1e-12, 1e-7, -1e-7], n), dy.astype(int)
    r = 10. ** rng.uniform(np.log10(.05), np.log10(4096.), n)
    fx, fy = rng.random((2, n))
    dy = np.floor(rng.uniform(-r - 1., r + 2.)).astype(int) if kind == 'any row' else \
        np.floor(r * rng.choice([-1., 1.], n) + rng.uniform(-2., 2., n)).astype(int)
    return fx, fy, r, dy


@pytest.mark.parametrize('ulps', [-2, 0, 2])
@pytest.mark.parametrize('kind', ['any row', 'first and last rows', 'ends on pixel centres'])
def test_decided_ends_are_exact(kind, ulps):
    fx, fy, r, dy = _disks(kind, 400000, 3)
    R = _row_ends(fx.astype(f), fy.astype(f), (r * r).astype(f), r.astype(f), dy, ulps)
    exact = X(1) * r * r - (X(1) * dy - fy) ** 2
    # rows that FP32 leaves out have no pixel, rows that it passes to the exact ends are not judged here
    assert np.all(exact[R['rem'] < -R['tol']] < 0)
    judged = R['rem'] >= 4 * R['tol']
    assert np.all(exact[judged] > 0) and judged.sum() > (1000 if kind != 'first and last rows' else 100)
    half = np.sqrt(np.where(judged, exact, 1))
    left, right = fx - half, fx + half
    error = np.maximum(np.abs(R['kl'] + X(1) * R['fl'] - left), np.abs(R['kr'] + X(1) * R['fr'] - right)) / R['e']
    assert error[judged].max() < 1
    for k, frac, end, decided in (('kl', 'fl', left, np.ceil), ('kr', 'fr', right, np.floor)):
        sure = judged & (np.abs(R[frac]) > R['e'])
        pixel = R[k] + (R[frac] > 0) if k == 'kl' else R[k] + (R[frac] >= 0) - 1
        assert np.array_equal(pixel[sure].astype(X), decided(end[sure]))
        if kind == 'ends on pixel centres':
            # ends within FP64 rounding of a pixel centre are never decided in FP32
            assert not np.any(sure & (np.abs(end - np.rint(end)) < 1e-9))
