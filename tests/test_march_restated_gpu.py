"""Every value that the march assigns in a rebuilt band is the second-order
upwind stencil (heap::calc, heap.cc:177-376) over the points that count as
accepted before it: those at the interface and those of its side with smaller
values. Restated here, on shapes without equal values, within 1e-11 of a cell:
the sweeps settle to 1e-13 and a value follows from some seventy others."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def stencil(at, dx, dy):
    """at(di, dj): the neighbour's value if it counts as accepted, else None."""
    def axis(steps):
        out = []
        for near, far in steps:
            v = at(*near)
            if v is None:
                continue
            w = at(*far)
            out.append((2 * v - 0.5 * w, True) if w is not None and w < v else (v, False))
        return out

    xs, ys = axis([((-1, 0), (-2, 0)), ((1, 0), (2, 0))]), axis([((0, -1), (0, -2)), ((0, 1), (0, 2))])

    def one(v, second, h):  # along one direction alone
        return (v + h) / 1.5 if second else v + h

    if not ys:
        return min(one(*v, dx) for v in xs)
    if not xs:
        return min(one(*v, dy) for v in ys)

    def close(ex, ey):  # a point at the two differences is within a cell of the front
        return max(ex, 0) ** 2 + max(ey, 0) ** 2 * (dx / dy) ** 2 < dx ** 2

    def corner(a, h, b, v):
        # ((ca a' - a)/dx)^2 + ((cb b' - b)/dy)^2 = 1 with c = 3/2 for second order
        ca, cb = (1.5 if h else 1.0), (1.5 if v else 1.0)
        A, B, C = (ca / dx) ** 2 + (cb / dy) ** 2, ca * a / dx ** 2 + cb * b / dy ** 2, (a / dx) ** 2 + (b / dy) ** 2 - 1
        # the reference's condition on the difference of the values (corner(), heap.cc:390-435)
        X, Y = dx * dx, dy * dy
        if h == v:
            limit = 1 + X / Y if X > Y else 1 + Y / X
        elif h:
            limit = 1 + X / Y / 2.25 if X > 2.25 * Y else 1 + 2.25 * Y / X
        else:
            limit = 1 + 2.25 * X / Y if 2.25 * X > Y else 1 + Y / (2.25 * X)
        f = ca * cb * (a / ca - b / cb)
        if f * f * limit < ca * ca * Y + cb * cb * X:
            return (B + math.sqrt(B * B - A * C)) / A
        return min(one(a, h, dx), one(b, v, dy))

    def of_two(pair):  # equal orders: the smaller; else (first order, second order)
        if len(pair) == 1 or pair[0][1] == pair[1][1]:
            return min(pair), None
        return (min(pair, key=lambda p: p[1]), max(pair, key=lambda p: p[1]))

    (a, a2), (b, b2) = of_two(xs), of_two(ys)
    if a2 and b2:
        n, s, m, q = a[0], a2[0], b[0], b2[0]
        e, f = 2 * (s - n), 2 * (q - m)
        if e < f:
            h = close(e - n, e - m)
            v = h and close(1.5 * f - s, f - m)
        else:
            v = close(f - n, f - m)
            h = v and close(e - n, 1.5 * e - q)
        return corner(s if h else n, h, q if v else m, v)
    if a2:
        d = 2 * (a2[0] - a[0])
        h = close(d - a[0], (1.5 if b[1] else 1.0) * d - b[0])
        return corner((a2 if h else a)[0], h, *b)
    if b2:
        d = 2 * (b2[0] - b[0])
        v = close((1.5 if a[1] else 1.0) * d - a[0], d - b[0])
        return corner(*a, (b2 if v else b)[0], v)
    return corner(*a, *b)


@pytest.mark.parametrize("m,n,by", [(83, 101, 1.0), (128, 96, 1.0), (120, 120, 1.7)])
@pytest.mark.parametrize("shape", ["ellipse", "rod", "thin"])
def test_values_are_the_stencil(gpu, m, n, by, shape):
    from incrmt_b200 import capi
    s = capi.Simulation(m, n, by=by, ntrace=0)
    if shape == "ellipse":
        s.add_ellipse(-0.103, 0.217, 0.35, 0.22, 0.71, 1.0, 2.0)
    elif shape == "rod":
        s.add_rounded_rod(0.0123, 0.0517, 0.11, 0.31, 1.0, 2.0)
    else:
        s.add_ellipse(0.113, -0.217, 0.41, 0.083, 0.37, 1.0, 2.0)  # fronts that meet inside
    s.initialize()
    s.step(s.dt_reg, 3)  # an evolved band
    phi, st = s.get("phi"), s.get("status").astype(int)
    dx, dy = 2.0 / m, (by + 1) / n
    nl, ml = phi.shape
    points = np.argwhere((st == 5) | (st == 2))
    assert len(points) > 200
    wrong = 0
    for j, i in points:
        side, sign = ((5, 6, 7), 1.0) if st[j, i] == 5 else ((0, 1, 2), -1.0)

        def at(di, dj):
            q = j + dj, i + di
            if not (0 <= q[0] < nl and 0 <= q[1] < ml):
                return None
            v = sign * float(phi[q])
            return None if st[q] in side and not v < sign * phi[j, i] else v
        if abs(stencil(at, dx, dy) - sign * phi[j, i]) > 1e-11 * dx:
            wrong += 1
    assert wrong == 0
    s.close()
