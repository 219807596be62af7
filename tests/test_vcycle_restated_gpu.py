"""One V-cycle against a restatement with sparse matrices, in none of the
library's kernels: operators, weights of the prolongation P, P^T A P, the
four-colour sweeps in their order and the coarsest solve. In double within 1e-11
of the iterate's largest value: a rounding of 1e-16 through some 1e4 operations,
times a coarsest system's condition of 1e1 to 1e3 (a single-precision correction
within 1e-3, 6e-8 times the fine system's condition). The hierarchies have levels
above and inside the cluster launch of the small ones, on one block and on
strips, semi-coarsening either way, periodic levels of even and odd size."""
import numpy as np
import pytest
import scipy.sparse as sp

from test_tile_indices import hierarchy

pytestmark = pytest.mark.gpu

COLOURS = ((0, 0), (1, 1), (1, 0), (0, 1))  # (i mod 2, j mod 2)
OFFSETS = [(di, dj) for dj in (-1, 0, 1) for di in (-1, 0, 1)]


class Level:
    """A grid's matrix; entry(k) is the stencil entry at offset k of every point."""

    def __init__(self, m, n, px, py):
        self.m, self.n, self.px, self.py = m, n, px, py
        self.j, self.i = (v.ravel() for v in np.mgrid[0:n, 0:m])

    def neighbour(self, di, dj):
        i, j = self.i + di, self.j + dj
        ok = (self.px | (0 <= i) & (i < self.m)) & (self.py | (0 <= j) & (j < self.n))
        return i % self.m + self.m * (j % self.n), ok

    def assemble(self, entries):
        rows, cols, vals = [], [], []
        for (di, dj), e in zip(OFFSETS, entries):
            q, ok = self.neighbour(di, dj)
            rows.append(np.arange(q.size)[ok])
            cols.append(q[ok])
            vals.append(np.broadcast_to(e, (self.n, self.m)).ravel()[ok])
        self.A = sp.csr_matrix((np.concatenate(vals), (np.concatenate(rows), np.concatenate(cols))), shape=(self.m * self.n,) * 2)

    def entry(self, di, dj):
        q, ok = self.neighbour(di, dj)
        return np.where(ok, np.asarray(self.A[np.arange(q.size), q]).ravel(), 0.0)

    def smooth(self, z, b, sweeps):
        d = self.A.diagonal()
        odd = (self.px and self.m % 2) or (self.py and self.n % 2)
        for _ in range(sweeps):
            for pi, pj in COLOURS:
                points = np.flatnonzero((self.i % 2 == pi) & (self.j % 2 == pj))
                # points that meet across the seam of an odd level see the values from
                # before the phase; up to 256 unknowns, from before their group of 32
                step = 32 if odd and self.m * self.n <= 256 else max(points.size, 1)
                for k in range(0, points.size, step):
                    p = points[k:k + step]
                    z[p] = z[p] + (b[p] - self.A[p] @ z) / d[p]

    def prolongation(self, mc, nc, kx, ky):
        a = {o: self.entry(*o) for o in OFFSETS}
        ox, oy = (self.i % 2 == 1) & kx, (self.j % 2 == 1) & ky
        base = lambda qx, qy: (self.i // 2 + qx if kx else self.i) % mc + mc * ((self.j // 2 + qy if ky else self.j) % nc)
        there_x = self.px | ((self.i // 2 + 1 if kx else self.i) < mc)
        there_y = self.py | ((self.j // 2 + 1 if ky else self.j) < nc)
        one, rows = np.ones(self.i.size), np.arange(self.i.size)
        P = sp.csr_matrix((self.m * self.n, mc * nc))
        put = lambda sel, w, qx, qy: sp.csr_matrix((w[sel], (rows[sel], base(qx, qy)[sel])), shape=P.shape)
        P = P + put(~ox & ~oy, one, 0, 0)
        with np.errstate(all="ignore"):
            col = [sum(a[(d, e)] for e in (-1, 0, 1)) for d in (-1, 0, 1)]
            row = [sum(a[(e, d)] for e in (-1, 0, 1)) for d in (-1, 0, 1)]
            P = P + put(ox & ~oy, -col[0] / col[1], 0, 0) + put(ox & ~oy & there_x, -col[2] / col[1], 1, 0)
            P = P + put(~ox & oy, -row[0] / row[1], 0, 0) + put(~ox & oy & there_y, -row[2] / row[1], 0, 1)
        inner = sp.diags(np.where(ox & oy, -1 / self.A.diagonal(), 0.0))
        return (P + inner @ ((self.A - sp.diags(self.A.diagonal())) @ P)).tocsr()


def fine_level(sys_, m, n, px, py, zpr, dx, dy, rho):
    """The MAC or the finite-element system of the ghosted density."""
    ir = 1 / rho
    if sys_ == 0:
        L = Level(m, n, px, py)
        ex = 0.5 * ir[2:n + 2, 2:m + 3] + 0.5 * ir[2:n + 2, 1:m + 2]
        ey = 0.5 * ir[2:n + 3, 2:m + 2] + 0.5 * ir[1:n + 2, 2:m + 2]
        xx, yy = 1 / dx ** 2, 1 / dy ** 2
        l, r, d, u = xx * ex[:, :-1], xx * ex[:, 1:], yy * ey[:-1], yy * ey[1:]
        dl, dr, dd, du = l.copy(), r.copy(), d.copy(), u.copy()
        if not px:
            dl[:, 0] = 0
            dr[:, -1] *= 2 if zpr else 0
        if not py:
            dd[0] = du[-1] = 0
        L.assemble([0, d, 0, l, -(dl + dr + dd + du), r, 0, u, 0])
        return L
    mf, nf = m if px else m + 1, n if py else n + 1
    L = Level(mf, nf, px, py)
    c = np.zeros((nf + 1, mf + 1))  # cell below-left of node (i,j)
    c[:nf, :mf] = ir[1:nf + 1, 1:mf + 1]
    c[:, mf] = c[:, 0] if px else 0
    c[nf] = c[0] if py else 0
    if not px:
        c[:, 0] = c[:, mf] = 0
    if not py:
        c[0] = c[nf] = 0
    dl, dr, ul, ur = c[:-1, :-1], c[:-1, 1:], c[1:, :-1], c[1:, 1:]
    fm, fc = (dx / dy + dy / dx) / 3, -(dx / dy + dy / dx) / 6
    hy, hx = (-2 * dx / dy + dy / dx) / 6, (-2 * dy / dx + dx / dy) / 6
    e = [fc * dl, hy * (dl + dr), fc * dr, hx * (dl + ul), fm * (dl + dr + ul + ur), hx * (dr + ur), fc * ul, hy * (ul + ur), fc * ur]
    if zpr:  # the fixed column
        for k in range(9):
            if k != 4:
                e[k] = e[k].copy()
                e[k][:, -1] = 0
    L.assemble(e)
    return L


def vcycle(levels, z, b, l=0):
    L, P = levels[l]
    if P is None:
        N = z.size
        if l == 0 or N > 96:
            L.smooth(z, b, 64)
            return
        A = L.A.toarray()
        total = np.abs(A.diagonal()).sum()
        if np.abs(A.sum(1)).max() <= 1e-10 * total / N:
            A = A + total / N / N
        z[:] = np.linalg.solve(A, b)
        return
    L.smooth(z, b, 2)
    zc = np.zeros(P.shape[1])
    vcycle(levels, zc, P.T @ (b - L.A @ z), l + 1)
    z += P @ zc
    L.smooth(z, b, 2)


CASES = [
    # sys, m, n, width / height, x periodic, y periodic, zero pressure at the right
    (0, 9, 17, 1.0, 0, 0, 0), (0, 33, 33, 1.0, 0, 0, 1), (0, 64, 64, 1.0, 0, 0, 0), (0, 129, 127, 1.0, 0, 0, 0),
    (0, 300, 257, 1.0, 0, 0, 1), (0, 200, 30, 6.7, 0, 0, 0), (0, 160, 160, 3.0, 0, 0, 1), (0, 160, 160, 0.3, 0, 0, 0),
    (1, 6, 6, 1.0, 0, 0, 0), (1, 64, 64, 1.0, 0, 0, 1), (1, 255, 200, 1.0, 0, 0, 0), (1, 150, 150, 3.0, 0, 0, 1),
    (0, 128, 128, 1.0, 0, 1, 1), (0, 288, 144, 3.0, 0, 1, 1), (1, 193, 144, 3.0, 0, 1, 1), (1, 100, 112, 1.0, 0, 1, 1),
    (0, 90, 80, 1.0, 1, 1, 0), (0, 72, 56, 1.0, 1, 0, 0), (1, 96, 72, 1.0, 1, 1, 0), (1, 80, 208, 1.0, 1, 1, 0),
    (0, 76, 300, 0.25, 1, 1, 0),  # 19 x 75 unknowns swept above the cluster launch's sizes
]


@pytest.mark.parametrize("sys_,m,n,aspect,px,py,zpr", CASES)
def test_vcycle(gpu, sys_, m, n, aspect, px, py, zpr):
    import torch
    from incrmt_b200 import capi
    bx, by = -1 + 2 * max(aspect, 1.0), -1 + 2 * max(1 / aspect, 1.0)
    s = capi.MGSolver(sys_, m, n, bx=bx, by=by, x_prd=bool(px), y_prd=bool(py), zpr=bool(zpr))
    rng = np.random.default_rng(m * 13 + n + sys_)
    rho = np.exp(rng.uniform(-1, 1, (n + 4, m + 4)))
    rho[n // 3:n // 2 + 2, m // 4:m // 2 + 2] *= 5
    if px:
        rho[:, :2], rho[:, m + 2:] = rho[:, m:m + 2].copy(), rho[:, 2:4].copy()
    if py:
        rho[:2], rho[n + 2:] = rho[n:n + 2].copy(), rho[2:4].copy()
    s.set_density(rho)
    fine = fine_level(sys_, m, n, bool(px), bool(py), zpr, (bx + 1) / m, (by + 1) / n, rho)
    levels = []
    L = fine
    for mm, nn, mc, nc, kx, ky in hierarchy(fine.m, fine.n, px, py, (((bx + 1) / m) / ((by + 1) / n)) ** 2):
        P = L.prolongation(mc, nc, kx, ky)
        levels.append((L, P))
        C = Level(mc, nc, bool(px), bool(py))
        C.A = (P.T @ L.A @ P).tocsr()
        L = C
    levels.append((L, None))
    b, z0 = rng.standard_normal((2, fine.n, fine.m))
    if sys_ == 1 and zpr:
        b[:, -1] = 0
    b, z0 = b.ravel(), z0.ravel()
    if not zpr:
        b -= b.mean()
    bd, z = torch.tensor(b, device="cuda"), torch.tensor(z0, device="cuda")
    torch.cuda.synchronize()
    s.vcycle_device(bd.data_ptr(), z.data_ptr())
    torch.cuda.synchronize()
    want = z0.copy()
    vcycle(levels, want, b)
    err = np.abs(z.cpu().numpy() - want).max() / np.abs(want).max()
    assert err <= 1e-11
    # one single-precision correction from zero (made free of its mean where the system is singular)
    zm = torch.zeros(b.size, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    with pytest.raises(capi.IncrmtError) as e:  # the cap of one cycle is its expected end
        s.solve_device(bd.data_ptr(), zm.data_ptr(), rel_tol=1e-15, max_vcycles=1, precision=capi.PREC_MIXED)
    assert e.value.code == capi.ERR_NOCONV
    want = np.zeros(b.size)
    vcycle(levels, want, b)
    got = zm.cpu().numpy()
    if not zpr:
        want -= want.mean()
        got -= got.mean()
    assert np.abs(got - want).max() <= 1e-3 * np.abs(want).max()
    s.close()
