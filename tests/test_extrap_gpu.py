"""The extrapolated reference map at every band point outside the solid is the
weighted least-squares fit over its window, restated here on the final values:
to the bit where the radius-3 window has a regular fit (the roundings of ExtFit,
each product and sum taken exactly and then rounded)."""
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = {
    "circle": lambda s, L: s.add_circle(0.13 * L, -0.21 * L, 0.3 * L, L * L, 2.0),
    "ellipse": lambda s, L: s.add_ellipse(-0.1 * L, 0.2 * L, 0.35 * L, 0.12 * L, 0.7, L * L, 2.0),
    "corner": lambda s, L: s.add_circle(0.83 * L, 0.85 * L, 0.1 * L, L * L, 2.0),  # windows cut by the grid's edge
}


def fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))


def minor(a, b, c, d):
    return fma(a, b, -(c * d))


def fit(phi, band, X, Y, j, i, r):
    """(determinant, X, Y) of the fit at point (i,j) over its window of radius r."""
    nl, ml = phi.shape
    sw = sx = sy = sxx = sxy = syy = 0.0
    acc = [0.0] * 6
    for dj in range(max(-r, -j), min(r, nl - 1 - j) + 1):
        for di in range(max(-r, -i), min(r, ml - 1 - i) + 1):
            q = j + dj, i + di
            if not band[q] or not phi[q] < phi[j, i]:
                continue
            w = float(phi[j, i] - phi[q])
            wi, wj = w * di, w * dj
            sw += w
            sx += wi
            sy += wj
            sxx = fma(di * di, w, sxx)
            sxy = sxy + wi if dj == 1 else sxy + wj if di == 1 else fma(di * dj, w, sxy)
            syy = fma(dj * dj, w, syy)
            for k, v in ((0, float(X[q])), (3, float(Y[q]))):
                acc[k] = fma(w, v, acc[k])
                acc[k + 1] = fma(wi, v, acc[k + 1])
                acc[k + 2] = fma(wj, v, acc[k + 2])
    a = minor(sxy, sxy, sxx, syy)
    det = fma(sy * sy, sxx, fma(-(2 * sx * sxy), sy, fma(sx * sx, syy, sw * a)))
    if abs(det) < 1e-10:
        return det, None, None
    c = [v * (1 / det) for v in (a, minor(sx, syy, sxy, sy), minor(sxx, sy, sxy, sx))]
    x, y = (fma(acc[k + 2], c[2], fma(acc[k], c[0], acc[k + 1] * c[1])) for k in (0, 3))
    return det, x, y


def extrapolated(m, n, L, shape):
    """phi, status and the reference map of a bent body after one extrapolation;
    no map where it reports a singular fit."""
    from incrmt_b200 import capi
    s = capi.Simulation(m, n, ax=-L, bx=L, ay=-L, by=L, visc=1e-2 * L * L, ntrace=0)
    SHAPES[shape](s, L)
    s.initialize()
    X, Y = s.get("X"), s.get("Y")
    s.set("nX", X + 0.01 * L * np.sin(3 * Y / L))
    s.set("nY", Y + 0.02 * L * np.cos(2 * X / L))
    try:
        s.stage("extrapolate")
    except capi.IncrmtError as e:
        assert e.code == capi.ERR_EXTRAP_SINGULAR
        return s, s.get("phi"), s.get("status"), None, None
    return s, s.get("phi"), s.get("status"), s.get("nX"), s.get("nY")


@pytest.mark.parametrize("shape", list(SHAPES))
@pytest.mark.parametrize("m,n", [(64, 64), (101, 83)])
def test_regular_fits_to_the_bit(gpu, shape, m, n):
    s, phi, st, X, Y = extrapolated(m, n, 1.0, shape)
    band = (st >= 2) & (st <= 5)
    points = np.argwhere((st == 4) | (st == 5))
    assert len(points) > 100
    for j, i in points[::5]:
        det, x, y = fit(phi, band, X, Y, j, i, 3)
        assert abs(det) >= 1e-10
        assert x == X[j, i] and y == Y[j, i], (j, i)
    s.close()


@pytest.mark.parametrize("shape", list(SHAPES))
@pytest.mark.parametrize("m,L,radius", [
    (64, 3.2e-4, 4),     # some radius-3 fits are singular, some are not
    (64, 2.5e-4, 4),
    (64, 1.2e-4, 5),
    (256, 1e-3, 4),      # many tiles
])
def test_singular_fits_widen(gpu, shape, m, L, radius):
    """A grid in small units: its weights are so small that the determinant falls
    below the singular limit at radius 3, and not at a wider one."""
    s, phi, st, X, Y = extrapolated(m, m, L, shape)
    band = (st >= 2) & (st <= 5)
    points = np.argwhere((st == 4) | (st == 5))
    if X is None:  # reported only where a fit is singular at every radius (bands cut by the grid's edge)
        assert any(all(abs(fit(phi, band, phi, phi, j, i, r)[0]) < 1e-10 for r in range(3, 8)) for j, i in points)
        s.close()
        return
    widest = 0
    for j, i in points[::max(len(points) // 60, 1)]:
        r = 3
        while r < 8:
            det, x, y = fit(phi, band, X, Y, j, i, r)
            if abs(det) >= 1e-10:
                break
            r += 1
        widest = max(widest, r)
        assert x == X[j, i] and y == Y[j, i], (j, i, r)
    assert widest >= radius
    s.close()
