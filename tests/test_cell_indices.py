"""Index safety of the multigrid kernels that work by cells (mg_transfer.cuh,
mg_cells.cuh, mg_tail.cuh, the tiled Galerkin product and the pairs across an odd
seam in mg.cu), replayed on the CPU over every level of a set of hierarchies: what
is read or written lies in its array, and what has to be written is, once. The
sizes of the blocks are read from the sources."""
import os
import re

import numpy as np
import pytest

import test_tile_indices as tiles
from test_tile_indices import hierarchy

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "incrmt_b200", "csrc")


def constant(name, file):
    text = open(os.path.join(CSRC, file)).read()
    return int(re.search(r"constexpr [^;]*\b%s = (\d+)" % name, text).group(1))


PX, PY, RX, RY = (constant(k, "mg_transfer.cuh") for k in ("kPX", "kPY", "kRX", "kRY"))
CELL_X = constant("kCellX", "mg_cells.cuh")
GAL_ROWS, SEAM_UNITS, DIRECT_MAX = (constant(k, "mg.cu") for k in ("kGalRows", "kSeamUnits", "kDirectMax"))
TAIL_THREADS, TAIL_ROOT, TAIL_BLOCKS, TAIL_LEVELS = (
    constant(k, "mg_tail.cuh") for k in ("kTailThreads", "kTailRoot", "kTailBlocks", "kTailMaxLevels"))
TAIL_SMEM = constant("kTailSmemBudget", "mg_tail.cuh") * 1024

GRIDS = [
    # fine unknowns m, n, periodic x, y, (dx/dy)^2
    (64, 64, 0, 0, 1), (65, 63, 0, 0, 1), (1024, 1024, 0, 0, 1), (1025, 1025, 0, 0, 1), (301, 233, 0, 0, 1), (7, 7, 0, 0, 1),
    (513, 40, 0, 0, 0.2), (40, 513, 0, 0, 6), (194, 144, 0, 1, 5), (768, 512, 0, 1, 1), (2048, 2048, 0, 1, 9), (288, 144, 0, 1, 2.2),
    (101, 112, 0, 1, 1), (48, 18, 0, 1, 4), (512, 384, 1, 1, 1), (128, 128, 1, 1, 1), (90, 80, 1, 1, 1), (1100, 904, 0, 1, 1),
    (600, 512, 1, 0, 1), (202, 202, 1, 1, 1), (12, 8, 1, 1, 1), (4, 6, 1, 1, 1), (16384, 17, 0, 0, 1), (2, 300, 0, 0, 1),
]


def cdiv(a, b):
    return -(-a // b)


def cells(m, k):
    return (m + 1) // 2 if k else m


def levels(grid):
    """(m, n, cm, cn, kx, ky) of every level that has a coarser one."""
    return hierarchy(*grid)


def inside(v, n):
    return v.size == 0 or (v.min() >= 0 and v.max() < n)


@pytest.mark.parametrize("grid", GRIDS, ids=str)
def test_build_p(grid):
    px, py = grid[2:4]
    for fm, fn, cm, cn, kx, ky in levels(grid):
        both, cx, cy = kx and ky, cells(fm, kx), cells(fn, ky)
        sx, sy = (PX - 1, PY - 1) if both else (PX, PY)
        Iu, tx = (v.ravel() for v in np.broadcast_arrays(np.arange(cdiv(cx, sx))[:, None] * sx + np.arange(PX), np.arange(PX)))
        Ju, ty = (v.ravel() for v in np.broadcast_arrays(np.arange(cdiv(cy, sy))[:, None] * sy + np.arange(PY), np.arange(PY)))
        I = np.where(px & (Iu >= cx), Iu - cx, Iu)
        J = np.where(py & (Ju >= cy), Ju - cy, Ju)
        i, j = (2 * I if kx else I)[I < cx], (2 * J if ky else J)[J < cy]
        assert inside(i, fm) and inside(j, fn)  # the points read: (i+1, j), (i, j+1), (i+1, j+1) where they exist
        wx = (Iu < cx) & ~(both & (tx == PX - 1))
        wy = (Ju < cy) & ~(both & (ty == PY - 1))
        assert np.array_equal(np.sort(I[wx]), np.arange(cx)) and np.array_equal(np.sort(J[wy]), np.arange(cy))
        if both:  # the cell right of (above) a written one is the next thread's, or beyond a wall
            nx, ny = I[np.minimum(np.flatnonzero(wx) + 1, I.size - 1)], J[np.minimum(np.flatnonzero(wy) + 1, J.size - 1)]
            for own, nxt, c, p in ((I[wx], nx, cx, px), (J[wy], ny, cy, py)):
                assert np.array_equal(nxt[own < c - 1], own[own < c - 1] + 1)
                assert not p or (nxt[own == c - 1] == 0).all()


@pytest.mark.parametrize("grid", GRIDS, ids=str)
def test_plane_weights(grid):
    for fm, fn, cm, cn, kx, ky in levels(grid):
        cx, cy = cells(fm, kx), cells(fn, ky)
        NC, planes = cx * cy, 8 if kx and ky else 2
        j, i = np.mgrid[0:fn, 0:fm]
        pi, pj = (i % 2 == 1) & kx, (j % 2 == 1) & ky
        q = (i // 2 if kx else i) + cx * (j // 2 if ky else j) + np.where(kx & pj, np.where(pi, 4, 2), 0) * NC
        assert inside(q[pi | pj] + NC, planes * NC) and inside(q[pi | pj], planes * NC)
        assert inside(q[pi & pj] + 3 * NC, planes * NC)


@pytest.mark.parametrize("grid", GRIDS, ids=str)
def test_transfers(grid):
    px, py = grid[2:4]
    for fm, fn, cm, cn, kx, ky in levels(grid):
        cx, cy = cells(fm, kx), cells(fn, ky)
        assert (cx, cy) == (cm, cn)  # prolongation: a cell's base coarse point exists
        for c, k, p, f, R, cc in ((cx, kx, px, fm, RX, cm), (cy, ky, py, fn, RY, cn)):
            step, off = (R - 1, 1) if k else (R, 0)
            Iu, t = (v.ravel() for v in np.broadcast_arrays(np.arange(cdiv(cc, step))[:, None] * step + np.arange(R) - off, np.arange(R)))
            own = (Iu >= 0) & (Iu < cc) & (t >= off)
            assert np.array_equal(np.sort(Iu[own]), np.arange(cc))
            I = np.where((Iu < 0) & bool(p), Iu + c, Iu)
            use = (I >= 0) & (I < c)
            for u in range(2 if k else 1):
                x = (2 if k else 1) * I + u
                assert inside(x[use & (x < f)], f)
            if not k:
                continue
            # the upper points of the cell below an own one: staged by the thread before, or a wall
            low = np.flatnonzero(own) - 1
            assert (low >= 0).all() and np.array_equal(I[low][Iu[own] > 0], Iu[own][Iu[own] > 0] - 1)
            assert not p or (I[low][Iu[own] == 0] == c - 1).all()
            assert p or not use[low][Iu[own] == 0].any()
            # their weights' cells
            back = np.where(Iu[own] > 0, Iu[own] - 1, c - 1)
            assert inside(back, c)


@pytest.mark.parametrize("grid", GRIDS, ids=str)
def test_galerkin_tiles(grid, monkeypatch):
    monkeypatch.setattr(tiles, "CTH", GAL_ROWS)
    px, py = grid[2:4]
    for fm, fn, cm, cn, kx, ky in levels(grid):
        if fm > 140 and fn > 40:
            continue  # an index is wrapped once: only levels of about a tile can need it twice
        if fm * fn > 60000:
            continue
        # the supports' stencils are staged by points
        assert tiles.replay_galerkin(fm, fn, cm, cn, kx, ky, px, py) == (0, 0)
        # the weights by cells, each direction by itself
        for f, c, k, p, width in ((fm, cm, kx, px, 32), (fn, cn, ky, py, GAL_ROWS)):
            S = 2 * width + 1 if k else width
            N = S + 2                                   # points of the region
            C = (N + 1) // 2 if k else N                # its cells
            smax, count = (2 * c - 1 if k else c - 1), cells(f, k)
            for x0 in range(0, c, width):
                staged = {}
                for a in range(C):
                    u = x0 - 1 + a
                    I, ok = tiles.wrap(u, count, p)
                    ok = ok and (2 * u if k else u) <= smax + 1
                    assert not ok or 0 <= I < count
                    for v in range(2 if k else 1):
                        x = 2 * a + v if k else a
                        if x < N:
                            staged[x] = 2 * I + v if ok and k else I if ok else None
                assert sorted(staged) == list(range(N))
                first = 2 * x0 - 2 if k else x0 - 1     # the fine point of region index 0
                for I in range(x0, min(x0 + width, c)):
                    lo, hi = (2 * I - 2, 2 * I + 2) if k else (I - 1, I + 1)
                    for g in range(lo, hi + 1):         # supports and their neighbours
                        i, ok = tiles.wrap(g, f, p)
                        if ok:
                            assert staged[g - first] == i
                        else:                           # beyond a wall: no point, or one of weight zero
                            assert staged[g - first] is None or staged[g - first] >= f


def smoother_levels(grid):
    """Levels that the tiled smoother takes: periodic directions of even size."""
    for m, n, *_ in levels(grid):
        if (not grid[2] or m % 2 == 0) and (not grid[3] or n % 2 == 0):
            yield m, n


@pytest.mark.parametrize("ry", [16, 24, 32])
@pytest.mark.parametrize("five", [True, False])
@pytest.mark.parametrize("grid", GRIDS, ids=str)
def test_smoother(grid, five, ry):
    px, py = grid[2:4]
    hx, tx, hy = (2, CELL_X - 4, 2) if five else (3, CELL_X - 5, 4)
    ty = ry - 2 * hy
    for m, n in smoother_levels(grid):
        X, Y = np.arange(cdiv(m, 2 * tx)) * tx - hx, np.arange(cdiv(n, 2 * ty)) * ty - hy
        inner = (X[:, None] > 0) & (2 * (X[:, None] + CELL_X) < m) & (Y > 0) & (2 * (Y + ry) < n)
        # an inner tile's cells, with the coefficients one point further, are on the grid
        bx, by = np.nonzero(inner)
        if bx.size:
            assert X[bx].min() > 0 and 2 * (X[bx].max() + CELL_X - 1) + 2 < m
            assert Y[by].min() > 0 and 2 * (Y[by].max() + ry - 1) + 2 < n
        # other tiles: each direction by itself
        for lo, width, c, size, p in ((X, CELL_X, (m + 1) // 2, m, px), (Y, ry, (n + 1) // 2, n, py)):
            I = (lo[:, None] + np.arange(width)).ravel()
            if p:
                I = I % c
                assert inside(2 * I + 1, size)
            k = 2 * I
            on = (k >= 0) & (k < size)
            assert inside(k[on] // 2, c)
            for g in range(3):  # edges: up to index size; cell densities: wrapped or left out
                e = k[on] + g
                assert inside(e[e <= size], size + 1)
                w = np.where(bool(p) & (e >= size), e - size, e)
                assert inside(w[w < size], size) and (not p or (w < size).all())
        # every cell is written once
        for lo, h, t, c in ((X, hx, tx, (m + 1) // 2), (Y, hy, ty, (n + 1) // 2)):
            out = (lo[:, None] + h + np.arange(t)).ravel()
            assert np.array_equal(np.sort(out[out < c]), np.arange(c))
        # colour-split stencils of the points on the grid
        if not five:
            j, i = np.mgrid[0:n, 0:m]
            m0, m1, n0 = (m + 1) // 2, m // 2, (n + 1) // 2
            base = np.choose(i % 2 + 2 * (j % 2), [0, m0 * n0, m * n0, m * n0 + m0 * (n // 2)])
            q = base + (i // 2) + (j // 2) * np.where(i % 2, m1, m0)
            assert np.array_equal(np.sort(q.ravel()), np.arange(m * n))


@pytest.mark.parametrize("five", [True, False])
@pytest.mark.parametrize("ry", [16, 24, 32])
def test_smoother_shared_memory(five, ry):
    """Neighbours of every cell of the staged planes, those of the tile's edge included."""
    PL, pad = CELL_X * ry, CELL_X + 1
    s = np.arange(PL)
    for pi in (0, 1):
        for pj in (0, 1):
            at = [(1 - pi + 2 * pj) * PL + s + pi - 1, (1 - pi + 2 * pj) * PL + s + pi,
                  (pi + 2 * (1 - pj)) * PL + s + (0 if pj else -CELL_X), (pi + 2 * (1 - pj)) * PL + s + (0 if pj else -CELL_X) + CELL_X]
            c = (1 - pi + 2 * (1 - pj)) * PL + s + (0 if pj else -CELL_X) + pi - 1
            for q in at + [c, c + 1, c + CELL_X, c + CELL_X + 1]:
                assert inside(q + pad, 4 * PL + 2 * CELL_X + 2)


@pytest.mark.parametrize("m,n,px,py", [(m, n, px, py) for m in (5, 8, 75, 257, 301) for n in (5, 9, 12, 259) for px in (0, 1) for py in (0, 1)])
def test_seam_pairs(m, n, px, py):
    """Every point of a colour is updated once, and points of a colour that are
    neighbours by one block, after all its values are computed."""
    for pi, pj in ((0, 0), (1, 1), (1, 0), (0, 1)):
        x, y = px and m % 2 and pi == 0, py and n % 2 and pj == 0
        mc, nc = (m - pi + 1) // 2, (n - pj + 1) // 2
        units = (mc if y else 0) + (nc - (2 if y else 0) if x else 0)
        owner = {(i, j): -1 for j in range(pj, n, 2) for i in range(pi, m, 2)
                 if not ((x and i in (0, m - 1)) or (y and j in (0, n - 1)))}
        gx = cdiv(mc, 32)
        count = len(owner)
        for block in range(cdiv(cdiv(units, SEAM_UNITS), gx) * gx):
            for q in range(2 * SEAM_UNITS):
                t, far = SEAM_UNITS * block + q % SEAM_UNITS, q >= SEAM_UNITS
                if t >= units:
                    continue
                if y and t < mc:
                    i, j = (2 * t + pi if not x else 0 if t == 0 else m - 1 if t == 1 else 2 * (t - 1)), (n - 1 if far else 0)
                else:
                    i, j = (m - 1 if far else 0), 2 * (t - (mc if y else 0) + (1 if y else 0)) + pj
                owner[i, j] = block
                count += 1
        assert count == mc * nc and set(owner) == {(i, j) for j in range(pj, n, 2) for i in range(pi, m, 2)}
        for (i, j), block in owner.items():
            for di in (-1, 0, 1):
                for dj in (-1, 0, 1):
                    o = ((i + di) % m if px else i + di, (j + dj) % n if py else j + dj)
                    if o != (i, j) and o in owner:
                        assert block >= 0 and owner[o] == block


def tail_plan(lev, px, py, blocks_max, size=8):
    """tail_plan of mg.cu: the levels' layouts, or None where one does not fit."""
    if not 1 <= len(lev) <= TAIL_LEVELS:
        return None
    plan = []
    for k, (m, n, kx, ky) in enumerate(lev):
        cx, cy = (m + 1) // 2, (n + 1) // 2
        seq = 2 if px and m % 2 else 1 if py and n % 2 else 0
        dist = cx * cy > TAIL_ROOT
        if dist and (seq or k == len(lev) - 1):
            return None
        plan.append(dict(m=m, n=n, kx=kx, ky=ky, cx=cx, cy=cy, seq=seq, dist=dist, rows=cy))
    nd = max([k + 1 for k, L in enumerate(plan) if L["dist"]], default=0)
    blocks = 1
    if nd:
        step = 1
        for L in plan[:nd - 1]:
            step *= 2 if L["ky"] else 1
        rows = cdiv(cdiv(plan[0]["cy"], blocks_max), step) * step
        blocks = cdiv(plan[0]["cy"], rows)
        for L in plan[:nd]:
            L["rows"] = rows
            if rows * L["cx"] > TAIL_THREADS:
                return None
            if L["ky"]:
                rows //= 2
    o = 0
    for k, L in enumerate(plan):
        L["used"], L["za"] = cdiv(L["cy"], L["rows"]), 4 * (L["rows"] + 1) * (L["cx"] + 2)
        L["zo"], L["ro"] = o, o + L["za"]
        o += L["za"] * (2 if k < len(plan) - 1 else 1)
        L["bo"] = o
        o += 4 * L["rows"] * L["cx"] if k else 0
    if o * size > TAIL_SMEM:
        return None
    return plan, nd, blocks


@pytest.mark.parametrize("blocks_max", [TAIL_BLOCKS, 8, 1])
@pytest.mark.parametrize("grid", GRIDS, ids=str)
def test_tail(grid, blocks_max):
    px, py = grid[2:4]
    steps = levels(grid)
    if not steps:
        return
    lev = [(m, n, kx, ky) for m, n, _, _, kx, ky in steps] + [(steps[-1][2], steps[-1][3], 0, 0)]
    for first in range(1, len(lev)):
        made = tail_plan(lev[first:], px, py, blocks_max)
        if made:
            break
    else:
        return
    plan, nd, blocks = made
    assert blocks <= blocks_max and all(L["dist"] for L in plan[:nd])
    for k, L in enumerate(plan):
        m, n, cx, cy, sr, used = (L[v] for v in ("m", "n", "cx", "cy", "rows", "used"))
        W, W2 = cx + 2, 2 * (cx + 2)
        assert used <= blocks if L["dist"] else used == 1 and L["cy"] == sr
        assert sr * cx <= TAIL_THREADS or L["seq"] == 2
        mul = ((1 << 20) + cx - 1) // cx
        t = np.arange(TAIL_THREADS)
        assert np.array_equal(t * mul >> 20, t // cx)
        at = lambda i, r: (r + 1) * W2 + (i & 1) * W + (i >> 1) + 1
        K = plan[k + 1] if k + 1 < len(plan) else None
        seen = set()
        for rank in range(used if L["dist"] else 1):
            row0 = rank * sr if L["dist"] else 0
            rows = min(cy - row0, sr)
            assert rows > 0
            # the strip's points with a halo of one (columns -1 .. 2 cx, rows -1 .. 2 rows)
            r, i = (v.ravel() for v in np.mgrid[-1:2 * rows + 1, -1:2 * cx + 1])
            assert inside(at(i, r), L["za"]) and np.unique(at(i, r)).size == i.size
            # halo rows in the neighbours' strips, with the periodic images of their ends
            for nb, upper in ((rank - 1 if rank else used - 1 if py else -1, False), (rank + 1 if rank + 1 < used else 0 if py else -1, True)):
                if nb < 0 or (not L["dist"] and not py):
                    continue
                nr = min(cy - nb * sr, sr) if L["dist"] else cy
                row = 0 if upper else (n + 1 if L["seq"] else 2 * nr + 1)
                h = row * W2 + np.arange(cx) + 1
                images = np.array([h[0] + cx, h[-1] + W - cx])  # of an even first column, an odd last one
                assert inside(h, L["za"]) and inside(h + W, L["za"]) and inside(images, L["za"])
                if not upper and not L["seq"]:
                    assert row == 2 * nr + 1  # the row above the strip's last
            if K is None:
                continue
            # restriction: coarse points of the strip's cells, in the strip (or block 0's level) that holds them
            for jl in range(rows):
                for I in range(cx):
                    for q in range(1 if L["kx"] and L["ky"] else 2):
                        Ic, Jc = (I if L["kx"] else 2 * I + q), (row0 + jl if L["ky"] else 2 * (row0 + jl) + q)
                        if Ic >= K["m"] or Jc >= K["n"]:
                            continue
                        c = (1 if Ic & 1 else 3) if Jc & 1 else (2 if Ic & 1 else 0)
                        krow0 = rank * K["rows"] if K["dist"] else 0
                        cell = (Jc // 2 - krow0) * K["cx"] + Ic // 2
                        assert 0 <= cell < K["rows"] * K["cx"] and (Ic, Jc) not in seen
                        seen.add((Ic, Jc))
                        assert 0 <= c * K["rows"] * K["cx"] + cell < 4 * K["rows"] * K["cx"]
            # prolongation: the corners' rows are in the coarse strip with its halo
            if K["dist"]:
                top = (row0 + rows - 1 if L["ky"] else 2 * (row0 + rows) - 1) + (1 if L["ky"] else 0)
                assert row0 * (1 if L["ky"] else 2) >= 2 * rank * K["rows"] and top - 2 * rank * K["rows"] <= 2 * K["rows"]
        if K is not None:
            assert len(seen) == K["m"] * K["n"]
