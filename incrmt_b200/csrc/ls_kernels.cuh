// Narrow-band level-set reinitialisation (levelset::build_band,
// levelset.cc:199-335) and reference-map extrapolation
// (levelset::extrapolate_fields, traverse.hh:169-260) on the GPU.
//
// The level-set grid is the ghosted fluid grid: mL=m+4 by nL=n+4 points,
// origin ax-1.5dx (obj_field.cc:18), stored with the fluid row pitch P, so
// level-set point (i,j) is at j*P+i.
//
// Reinitialisation. The reference (1) classifies each point by the sign of
// phi and of its four neighbours, (2) moves the points next to the interface
// to the signed distance of the closest zero of a bicubic interpolant
// (Newton), and (3) fast-marches outwards on each side with a second-order
// upwind stencil (heap.cc:177-376), accepting points in increasing |phi|
// until the band limit. The march is sequential; here step (3) is the
// fixed point of the same stencil: a point's value is the stencil evaluated
// with "in" neighbours = interface points plus same-side points whose
// current value is smaller, iterated (Jacobi, double-buffered) until no value
// changes. In exact arithmetic this is the value the march assigns, since a
// marched point's final value is the stencil over the points accepted before
// it, which are those with smaller values.
//
// Extrapolation. The reference visits the band in increasing phi and fits
// each point outside the solid by weighted least squares over already-visited
// neighbours with smaller phi; the result depends only on phi, so it is
// computed as a wavefront (Jacobi) iteration over the outside band points
// that stops when no value changes; the dependency depth is ~65 for the
// ~7-cell-wide band, independent of the grid size.
#pragma once
#include <cooperative_groups.h>
#include "sim.cuh"

namespace incrmt {

struct LsGrid {
    int mL, nL, P;
    double axl, ayl, dx, dy, xsp, ysp;
    double phi_up, phi_down;
};

/** Level-set arrays of one object. The batched kernels below take an array
 * of these and treat blockIdx.z as the object index; the cooperative ones
 * take a combined list of tiles whose entries carry their object index, so
 * every object's band is rebuilt (or extrapolated) in the same launches. */
struct LsObj {
    double *phi;             // level set (ghosted grid, pitch P)
    int *s;                  // status
    double *phi_new;         // Newton distances of the interface points
    double *a, *b;           // march values, or extrapolated X (ping-pong)
    double *c, *d;           // extrapolated Y (ping-pong)
    unsigned char *ca, *cb;  // change marks of the previous / current sweep
    int *ia, *ib;            // dilation masks; trial statuses
    double *nX, *nY;         // reference map being extrapolated
};

// Status values (levelset.cc:211-263, heap.cc): 0/7 far negative/positive,
// 1/6 trial, 2/5 accepted by the march, 3/4 next to the interface.

/** Point (i,j) of thread (x,y) in object blockIdx.z's window; false
 * outside it. */
__device__ __forceinline__ bool ls_point(const LsGrid &g, const LsWin *win, int &i, int &j) {
    const LsWin w = win[blockIdx.z];
    i = w.x0 + blockIdx.x * blockDim.x + threadIdx.x;
    j = w.y0 + blockIdx.y * blockDim.y + threadIdx.y;
    return i < w.x1 && j < w.y1 && i < g.mL && j < g.nL;
}

/** Sign classification (levelset.cc:209-263): s=4 for phi>0 with a 4-neighbour
 * phi<=0, s=3 for phi<=0 with a neighbour phi>0, else 7 / 0. */
__global__ void k_ls_scan(LsGrid g, const LsObj *ob, const LsWin *win, int *box) {
    __shared__ int sb[4];
    if (threadIdx.x == 0 && threadIdx.y == 0) sb[0] = sb[1] = sb[2] = sb[3] = 0x7fffffff;
    __syncthreads();
    int i, j;
    const bool live = ls_point(g, win, i, j);
    bool keep = false;
    if (live) {
        const double *phi = ob[blockIdx.z].phi;
        int *s = ob[blockIdx.z].s;
        const int ij = j * g.P + i;
        const bool pos = phi[ij] > 0;
        bool diff = false;
        if (i > 0) diff |= (phi[ij - 1] > 0) != pos;
        if (i < g.mL - 1) diff |= (phi[ij + 1] > 0) != pos;
        if (j > 0) diff |= (phi[ij - g.P] > 0) != pos;
        if (j < g.nL - 1) diff |= (phi[ij + g.P] > 0) != pos;
        const int st = pos ? (diff ? 4 : 7) : (diff ? 3 : 0);
        s[ij] = st;
        keep = st != 7;
    }
    // Bounding box of the points inside the solid or next to its interface:
    // a warp is one row, so its extent comes from the ballot; the block's
    // warps meet in shared memory and one thread updates the object's box
    // (minima of x, y, -x, -y).
    const unsigned bal = __ballot_sync(0xffffffffu, keep);
    if (bal && (threadIdx.x & 31) == 0) {
        const int xb = i - static_cast<int>(threadIdx.x & 31);
        atomicMin(&sb[0], xb + __ffs(bal) - 1);
        atomicMin(&sb[1], j);
        atomicMin(&sb[2], -(xb + 31 - __clz(bal)));
        atomicMin(&sb[3], -j);
    }
    __syncthreads();
    if (threadIdx.x == 0 && threadIdx.y == 0 && sb[0] != 0x7fffffff) {
        int *b = box + 4 * blockIdx.z;
        atomicMin(&b[0], sb[0]);
        atomicMin(&b[1], sb[1]);
        atomicMin(&b[2], sb[2]);
        atomicMin(&b[3], sb[3]);
    }
}

/** One-dimensional Hermite weights of the reference's bicubic
 * (levelset/built/bicubic.cc): value weights for the two nodes (a0,a1) and
 * for their slopes (b0,b1), and their derivatives. kind 1 is the cubic
 * interior patch, 0 the quadratic patch at the low edge (no slope at node 0),
 * 2 the quadratic patch at the high edge (no slope at node 1). */
__device__ __forceinline__ void hermite_w(int kind, double e, double &a0, double &a1, double &b0, double &b1,
                                          double &da0, double &da1, double &db0, double &db1) {
    const double me = 1 - e;
    if (kind == 1) {
        a0 = me * me * (1 + 2 * e); a1 = e * e * (3 - 2 * e); b0 = e * me * me; b1 = -e * e * me;
        da0 = -6 * e * me; da1 = 6 * e * me; db0 = me * (1 - 3 * e); db1 = e * (3 * e - 2);
    } else if (kind == 0) {
        a0 = me * me; a1 = e * (2 - e); b0 = 0; b1 = -e * me;
        da0 = -2 * me; da1 = 2 * me; db0 = 0; db1 = 2 * e - 1;
    } else {
        a0 = 1 - e * e; a1 = e * e; b0 = e * me; b1 = 0;
        da0 = -2 * e; da1 = 2 * e; db0 = 1 - 2 * e; db1 = 0;
    }
}

/** Bicubic interpolation of phi with its gradient (levelset::bicubic,
 * levelset.cc:67-79, built/bicubic.cc): a tensor-product Hermite patch whose
 * nodal slopes are central differences (and the cross slope a central second
 * difference), with quadratic one-sided patches in the first and last cell of
 * each direction. Points outside the grid use the nearest edge patch. */
__device__ double ls_bicubic(const LsGrid &g, const double *phi, double x, double y, double &phix, double &phiy) {
    double e = (x - g.axl) * g.xsp, f = (y - g.ayl) * g.ysp;
    const int i = static_cast<int>(e), j = static_cast<int>(f);
    int kx, ky, ci, cj;
    if (i < 1) { kx = 0; ci = 0; }
    else if (i >= g.mL - 2) { kx = 2; ci = g.mL - 2; e -= static_cast<double>(g.mL - 2); }
    else { kx = 1; ci = i; e -= static_cast<double>(i); }
    if (j < 1) { ky = 0; cj = 0; }
    else if (j >= g.nL - 2) { ky = 2; cj = g.nL - 2; f -= static_cast<double>(g.nL - 2); }
    else { ky = 1; cj = j; f -= static_cast<double>(j); }
    double a0, a1, b0, b1, da0, da1, db0, db1;
    hermite_w(kx, e, a0, a1, b0, b1, da0, da1, db0, db1);
    double c0, c1, d0, d1, dc0, dc1, dd0, dd1;
    hermite_w(ky, f, c0, c1, d0, d1, dc0, dc1, dd0, dd1);
    const int P = g.P;
    // Row values V (and d/de) and row y-slopes W at rows cj, cj+1.
    double V[2], Vd[2], W[2], Wd[2];
    for (int r = 0; r < 2; r++) {
        const int rr = cj + r;
        const bool needW = (r == 0) ? (ky != 0) : (ky != 2);
        const int q0 = rr * P + ci, q1 = q0 + 1;
        double sx0 = 0, sx1 = 0;
        if (kx != 0) sx0 = (phi[q0 + 1] - phi[q0 - 1]) * 0.5;
        if (kx != 2) sx1 = (phi[q1 + 1] - phi[q1 - 1]) * 0.5;
        V[r] = a0 * phi[q0] + a1 * phi[q1] + b0 * sx0 + b1 * sx1;
        Vd[r] = da0 * phi[q0] + da1 * phi[q1] + db0 * sx0 + db1 * sx1;
        W[r] = Wd[r] = 0;
        if (needW) {
            const double sy0 = (phi[q0 + P] - phi[q0 - P]) * 0.5, sy1 = (phi[q1 + P] - phi[q1 - P]) * 0.5;
            double sxy0 = 0, sxy1 = 0;
            if (kx != 0) sxy0 = (phi[q0 + P + 1] - phi[q0 - P + 1] - phi[q0 + P - 1] + phi[q0 - P - 1]) * 0.25;
            if (kx != 2) sxy1 = (phi[q1 + P + 1] - phi[q1 - P + 1] - phi[q1 + P - 1] + phi[q1 - P - 1]) * 0.25;
            W[r] = a0 * sy0 + a1 * sy1 + b0 * sxy0 + b1 * sxy1;
            Wd[r] = da0 * sy0 + da1 * sy1 + db0 * sxy0 + db1 * sxy1;
        }
    }
    phix = g.xsp * (c0 * Vd[0] + c1 * Vd[1] + d0 * Wd[0] + d1 * Wd[1]);
    phiy = g.ysp * (dc0 * V[0] + dc1 * V[1] + dd0 * W[0] + dd1 * W[1]);
    return c0 * V[0] + c1 * V[1] + d0 * W[0] + d1 * W[1];
}

/** First-order fallback closest point (levelset::newton_failsafe,
 * levelset.cc:138-195), from the straight-line zero crossings to the
 * opposite-side interface neighbours. */
__device__ bool ls_failsafe(const LsGrid &g, const double *phi, const int *s, int i, int j, double x0, double y0,
                            double &x, double &y) {
    const int P = g.P, ij = j * P + i, ts = 7 - s[ij];
    const double cphi = phi[ij];
    bool hf, vf;
    double tdis;
    if (i > 0 && s[ij - 1] == ts) {
        x = cphi / (phi[ij - 1] - cphi);
        if (i < g.mL - 1 && s[ij + 1] == ts) {
            tdis = cphi / (cphi - phi[ij + 1]);
            if (tdis < -x) x = tdis;
        }
        hf = true;
    } else {
        if (i < g.mL - 1 && s[ij + 1] == ts) { x = cphi / (cphi - phi[ij + 1]); hf = true; }
        else hf = false;
    }
    if (j > 0 && s[ij - P] == ts) {
        y = cphi / (phi[ij - P] - cphi);
        if (j < g.nL - 1 && s[ij + P] == ts) {
            tdis = cphi / (cphi - phi[ij + P]);
            if (tdis < -y) y = tdis;
        }
        vf = true;
    } else {
        if (j < g.nL - 1 && s[ij + P] == ts) { y = cphi / (cphi - phi[ij + P]); vf = true; }
        else vf = false;
    }
    if (hf) {
        if (vf) {
            y *= g.dy;
            tdis = x * g.dx;
            const double c = tdis * y / (tdis * tdis + y * y);
            x = y * c + x0;
            y = tdis * c + y0;
        } else { x = x * g.dx + x0; y = y0; }
        return true;
    }
    if (vf) { x = x0; y = y * g.dy + y0; return true; }
    return false;
}

/** The reference's |v| as compiled: its unqualified abs() on a double binds to
 * int abs(int) (levelset.cc:124,126), i.e. |trunc(v)|. */
__device__ __forceinline__ double int_abs(double v) {
    int t = static_cast<int>(v);
    return static_cast<double>(t < 0 ? -t : t);
}

/** Closest-point Newton iteration of Chopp (levelset::newton,
 * levelset.cc:107-127) for the points next to the interface. Because of the
 * integer abs the loop ends after eight steps whose |phi| < 1 and the
 * closeness test is |x0-x| < 1, exactly as the reference runs. Writes the
 * signed distance to phi_new; sets *err on a failure (levelset.cc:275). */
__global__ void k_ls_newton(LsGrid g, const LsObj *ob, const LsWin *win, int *err) {
    int i, j;
    if (!ls_point(g, win, i, j)) return;
    const double *phi = ob[blockIdx.z].phi;
    const int *s = ob[blockIdx.z].s;
    double *phi_new = ob[blockIdx.z].phi_new;
    const int ij = j * g.P + i, st = s[ij];
    if (st != 3 && st != 4) return;
    const double dyy = g.dy / static_cast<double>(g.mL), step_limit = sqrt(g.dx * g.dx + g.dy * g.dy);
    const double x0 = g.axl + i * g.dx, y0 = g.ayl + static_cast<double>(j * g.mL) * dyy;
    double x = x0, y = y0, px, py;
    double ph = ls_bicubic(g, phi, x, y, px, py);
    int iter = 0, cutoff = 0;
    bool ok = true, fallback = false;
    do {
        const double delx = x0 - x, dely = y0 - y;
        double m0 = delx * px + dely * py + ph;
        const double m1 = px * px + py * py;
        iter++;
        m0 /= m1;
        if (iter > 100 || !isfinite(m0) || m0 > step_limit) { fallback = true; break; }
        x += delx - m0 * px;
        y += dely - m0 * py;
        ph = ls_bicubic(g, phi, x, y, px, py);
        if (int_abs(ph) < 1e-10) cutoff++; else cutoff = 0;
    } while (cutoff < 8);
    if (!fallback && !(int_abs(x0 - x) < 3 * g.dx && int_abs(y0 - y) < 3 * g.dy)) fallback = true;
    if (fallback) ok = ls_failsafe(g, phi, s, i, j, x0, y0, x, y);
    if (!ok) { atomicExch(err, INCRMT_ERR_NEWTON); phi_new[ij] = phi[ij]; return; }
    x -= x0;
    y -= y0;
    const double d = sqrt(x * x + y * y);
    phi_new[ij] = st == 4 ? d : -d;
}

__global__ void k_ls_copy_interface(LsGrid g, const LsObj *ob, const LsWin *win) {
    int i, j;
    if (!ls_point(g, win, i, j)) return;
    const LsObj &o = ob[blockIdx.z];
    const int ij = j * g.P + i;
    if (o.s[ij] == 3 || o.s[ij] == 4) o.phi[ij] = o.phi_new[ij];
}

/** Grid constants of the march's stencil. */
struct MarchK {
    double dx, dy, dx2, dxbydy, dx2bydy2;
    // corner(h, v): index 2 h + v
    double f2[4], i2[4], lim[4];
    __device__ void set(const LsGrid &g) {
        dx = g.dx; dy = g.dy;
        dx2 = dx * dx;
        const double dy2 = dy * dy;
        dxbydy = dx / dy; dx2bydy2 = dxbydy * dxbydy;
        f2[3] = 2.25 * (dy2 + dx2); f2[2] = 2.25 * dy2 + dx2; f2[1] = dy2 + 2.25 * dx2; f2[0] = dy2 + dx2;
        lim[1] = 2.25 * dx2 > dy2 ? 1 + 2.25 * dx2bydy2 : 1 + dy2 / (2.25 * dx2);
        lim[3] = lim[0] = dx2 > dy2 ? 1 + dx2bydy2 : 1 + dy2 / dx2;
        lim[2] = dx2 > 2.25 * dy2 ? 1 + dx2bydy2 / 2.25 : 1 + 2.25 * dy2 / dx2;
        for (int k = 0; k < 4; k++) i2[k] = dy2 / f2[k];
    }
};

/** The second-order upwind stencil of the fast march (heap<d_option>::calc and
 * its helpers, heap.cc:177-376, 390-435) for one candidate, staged at q of
 * arrays with row pitch P: ph the level set, st the status after the sign
 * scan, cur the candidates' values. A point counts as accepted ("in") if it
 * is not a candidate of this side (whose far status is `far`), or one with a
 * smaller value. The negative side is the positive one with every value
 * negated (sg = -1, exact), so one copy of the code serves both. The case
 * analysis only selects which two neighbour values, with which orders, enter
 * the final quadratic (h, v: second order along x, y; a, b: the values).
 * Returns the point's own value if no neighbour is in. */
__device__ __forceinline__ double march_value(const MarchK &K, int P, const double *ph, const unsigned char *st,
                                              const double *cur, int q, int far, double sg, double own, bool l1, bool l2,
                                              bool r1, bool r2, bool d1, bool d2, bool u1, bool u2) {
    const double pv = sg * own;
    auto val = [&](int k) { return sg * (st[k] == far ? cur[k] : ph[k]); };
    auto in = [&](int k) { return st[k] != far || sg * cur[k] < pv; };
    // The neighbour at offset o: whether it is in, its value, extrapolated to
    // second order where the next one is in and smaller (second).
    auto look = [&](int o, bool one, bool two, double &e, bool &second) {
        second = false;
        e = 0;
        if (!one || !in(q + o)) return false;
        e = val(q + o);
        if (two && in(q + 2 * o)) {
            const double f2 = val(q + 2 * o);
            if (f2 < e) {
                e = 2 * e - 0.5 * f2;
                second = true;
            }
        }
        return true;
    };
    double xl, xr, yd, yu;
    bool hl, hr, vd, vu;
    const bool L = look(-1, l1, l2, xl, hl), R = look(1, r1, r2, xr, hr);
    const bool D = look(-P, d1, d2, yd, vd), U = look(P, u1, u2, yu, vu);
    const double ti = 2.0 / 3.0;
    if (!L && !R && !D && !U) return own;
    if (!D && !U) {
        const double c = hl ? (xl + K.dx) * ti : xl + K.dx, d = hr ? (xr + K.dx) * ti : xr + K.dx;
        return sg * (L && R ? (c < d ? c : d) : (L ? c : d));
    }
    if (!L && !R) {
        const double c = vd ? (yd + K.dy) * ti : yd + K.dy, d = vu ? (yu + K.dy) * ti : yu + K.dy;
        return sg * (D && U ? (c < d ? c : d) : (D ? c : d));
    }
    // Differences below zero count as zero in the tests that follow.
    auto near = [&](double e, double f) {
        if (e < 0) e = 0;
        if (f < 0) f = 0;
        return e * e + f * f * K.dx2bydy2 < K.dx2;
    };
    bool h, v;
    double a, b;
    // Both x neighbours of first and second order n, s (threeway1), or both y
    // ones (threeway2): the second-order one where it is near.
    auto three_x = [&](double n, double s, bool vv, double y) {
        const double d = 2 * (s - n);
        h = near(d - n, (vv ? 1.5 * d : d) - y);
        v = vv;
        a = h ? s : n;
        b = y;
    };
    auto three_y = [&](double n, double s, bool hh, double x) {
        const double d = 2 * (s - n);
        v = near((hh ? 1.5 * d : d) - x, d - n);
        h = hh;
        a = x;
        b = v ? s : n;
    };
    if (L && R && D && U && vd != vu) {
        const double ys = vd ? yd : yu, yn = vd ? yu : yd;
        if (hl == hr) {
            three_y(yn, ys, hl, xl < xr ? xl : xr);
        } else {
            // fourway: first and second order along both axes
            const double xs = hl ? xl : xr, xn = hl ? xr : xl;
            const double e = 2 * (xs - xn), f = 2 * (ys - yn);
            if (e < f) {
                h = near(e - xn, e - yn);
                v = h && near(1.5 * f - xs, f - yn);
            } else {
                v = near(f - xn, f - yn);
                h = v && near(e - xn, 1.5 * e - ys);
            }
            a = h ? xs : xn;
            b = v ? ys : yn;
        }
    } else if (L && R) {
        const double y = D && U ? (yd < yu ? yd : yu) : (D ? yd : yu);
        const bool vv = D ? vd : vu;
        if (hl != hr) {
            three_x(hl ? xr : xl, hl ? xl : xr, vv, y);
        } else {
            h = hl; v = vv;
            a = xl < xr ? xl : xr;
            b = y;
        }
    } else if (D && U) {
        const double x = L ? xl : xr;
        const bool hh = L ? hl : hr;
        if (vd != vu) {
            three_y(vd ? yu : yd, vd ? yd : yu, hh, x);
        } else {
            h = hh; v = vd;
            a = x;
            b = yd < yu ? yd : yu;
        }
    } else {
        h = L ? hl : hr; v = D ? vd : vu;
        a = L ? xl : xr;
        b = D ? yd : yu;
    }
    const int k = 2 * h + v;
    double f0 = h == v ? a - b : (h ? __fma_rn(-1.5, b, a) : __fma_rn(1.5, a, -b));
    if (h && v) f0 = __dmul_rn(1.5, f0);
    const double f = __dmul_rn(f0, f0);
    if (__dmul_rn(f, K.lim[k]) < K.f2[k]) {
        // (roundings written out: a shape aligned with the grid has many equal
        // values, whose order decides which of them others see)
        const double bv = v ? b * 1.5 : b;
        const double e = h ? __fma_rn(a, 1.5, __dmul_rn(bv, K.dx2bydy2)) : __fma_rn(bv, K.dx2bydy2, a);
        return sg * __dmul_rn(__fma_rn(K.dxbydy, sqrt(__dsub_rn(K.f2[k], f)), e), K.i2[k]);
    }
    // the two directions apart (corner_bail)
    const double ht = h ? (a + K.dx) * ti : a + K.dx, vt = v ? (b + K.dy) * ti : b + K.dy;
    return sg * (ht < vt ? ht : vt);
}

constexpr double kUnset = 1e300;

/** Initialises both march buffers (+/-kUnset for this side's far points)
 * and clears both change marks. */
__global__ void k_ls_fim_init(LsGrid g, const LsObj *ob, const LsWin *win) {
    int i, j;
    if (!ls_point(g, win, i, j)) return;
    const LsObj &o = ob[blockIdx.z];
    const int ij = j * g.P + i, st = o.s[ij];
    const double v = st == 7 ? kUnset : (st == 0 ? -kUnset : 0.0);
    o.a[ij] = v;
    o.b[ij] = v;
    o.ca[ij] = 0;
    o.cb[ij] = 0;
}

/** Final values and clean-up (heap::march acceptance, levelset::clean,
 * levelset.cc:408-413): far points whose value fell inside the band limit are
 * accepted (5 / 2); every point outside the band is set to the band limit. */
__global__ void k_ls_finish(LsGrid g, const LsObj *ob, const LsWin *win, bool in_b) {
    int i, j;
    if (!ls_point(g, win, i, j)) return;
    const double *cur = in_b ? ob[blockIdx.z].b : ob[blockIdx.z].a;
    int *s = ob[blockIdx.z].s;
    double *phi = ob[blockIdx.z].phi;
    const int ij = j * g.P + i, st = s[ij];
    const double v = cur[ij];
    if (st == 7) {
        if (v < g.phi_up) { s[ij] = 5; phi[ij] = v; }
        else phi[ij] = g.phi_up;
    } else if (st == 0) {
        if (v > g.phi_down) { s[ij] = 2; phi[ij] = v; }
        else phi[ij] = g.phi_down;
    }
}

/** Trial statuses (heap::check_gridpoint / update, heap.cc:38-44,159-167):
 * a far point next to an interface or accepted point of its side was put on
 * the heap and, not being accepted, stays trial (6 / 1). */
__global__ void k_ls_trial(LsGrid g, const LsObj *ob, const LsWin *win) {
    int i, j;
    if (!ls_point(g, win, i, j)) return;
    const int *s = ob[blockIdx.z].s;
    int *s_out = ob[blockIdx.z].ia;
    const int ij = j * g.P + i, st = s[ij];
    int out = st;
    if (st == 7 || st == 0) {
        const int lo = st == 7 ? 4 : 2, hi = st == 7 ? 5 : 3;
        bool nb = false;
        if (i > 0) nb |= s[ij - 1] >= lo && s[ij - 1] <= hi;
        if (i < g.mL - 1) nb |= s[ij + 1] >= lo && s[ij + 1] <= hi;
        if (j > 0) nb |= s[ij - g.P] >= lo && s[ij - g.P] <= hi;
        if (j < g.nL - 1) nb |= s[ij + g.P] >= lo && s[ij + g.P] <= hi;
        if (nb) out = st == 7 ? 6 : 1;
    }
    s_out[ij] = out;
}

/** Copies the trial statuses back into the status array. */
__global__ void k_ls_store_status(LsGrid g, const LsObj *ob, const LsWin *win) {
    int i, j;
    if (!ls_point(g, win, i, j)) return;
    const int ij = j * g.P + i;
    ob[blockIdx.z].s[ij] = ob[blockIdx.z].ia[ij];
}

/** Weighted least-squares extrapolation of the reference map at a band point
 * outside the solid (traverse::extrapolate, traverse.hh:169-231): a linear fit
 * over the band neighbours with smaller phi in a (2r+1)^2 window, weighted by the
 * phi difference w; the window grows from r = 3 to kExtMaxRadius while the system
 * is singular. Here the sums over the points at offsets (di,dj) with values
 * (vx,vy), and what follows from them. Every
 * rounding is written out: the sweeps stop when no value changes, so all loops
 * that evaluate a point have to give it the same bits. */
constexpr int kExtMaxRadius = 7;
struct ExtFit {
    double sw, sx, sy, sxx, sxy, syy;
    __device__ __forceinline__ void clear() { sw = sx = sy = sxx = sxy = syy = 0; }
    __device__ __forceinline__ void moments(int di, int dj, double w) {
        const double wi = __dmul_rn(w, di), wj = __dmul_rn(w, dj);
        sw = __dadd_rn(sw, w);
        sx = __dadd_rn(sx, wi);
        sy = __dadd_rn(sy, wj);
        sxx = __fma_rn(di * di, w, sxx);
        sxy = dj == 1 ? __dadd_rn(sxy, wi) : (di == 1 ? __dadd_rn(sxy, wj) : __fma_rn(di * dj, w, sxy));
        syy = __fma_rn(dj * dj, w, syy);
    }
    static __device__ __forceinline__ void values(int di, int dj, double w, double vx, double vy, double acc[6]) {
        const double wi = __dmul_rn(w, di), wj = __dmul_rn(w, dj);
        acc[0] = __fma_rn(w, vx, acc[0]);
        acc[1] = __fma_rn(wi, vx, acc[1]);
        acc[2] = __fma_rn(wj, vx, acc[2]);
        acc[3] = __fma_rn(w, vy, acc[3]);
        acc[4] = __fma_rn(wi, vy, acc[4]);
        acc[5] = __fma_rn(wj, vy, acc[5]);
    }
    static __device__ __forceinline__ double minor(double a, double b, double c, double d) {
        return __fma_rn(a, b, -__dmul_rn(c, d));
    }
    __device__ __forceinline__ double det() const {
        double t = __fma_rn(__dmul_rn(sx, sx), syy, __dmul_rn(sw, minor(sxy, sxy, sxx, syy)));
        t = __fma_rn(-__dmul_rn(2 * sx, sxy), sy, t);
        return __fma_rn(__dmul_rn(sy, sy), sxx, t);
    }
    static __device__ __forceinline__ bool singular(double det) { return fabs(det) < 1e-10; }
    /** The coefficients al, be, ga of the fit's value at the point. */
    __device__ __forceinline__ void solve(double det, double c[3]) const {
        const double id = 1 / det;
        c[0] = __dmul_rn(minor(sxy, sxy, sxx, syy), id);
        c[1] = __dmul_rn(minor(sx, syy, sxy, sy), id);
        c[2] = __dmul_rn(minor(sxx, sy, sxy, sx), id);
    }
    static __device__ __forceinline__ double value(const double *acc, const double c[3]) {
        return __fma_rn(acc[2], c[2], __fma_rn(acc[0], c[0], __dmul_rn(acc[1], c[1])));
    }
};

/** Appends (tile, object) to the combined list if it has room; flags an
 * overflow otherwise (the list is sized for every point of every object, so
 * this only guards the bound). */
__device__ __forceinline__ void ls_list_push(int *list, int *list_k, int *count, int cap, int *overflow, int tile,
                                             int k) {
    const int t = atomicAdd(count, 1);
    if (t < cap) { list[t] = tile; list_k[t] = k; }
    else atomicExch(overflow, 1);
}

}  // namespace incrmt

namespace incrmt {

/** Marks the points next to the interface (status 3 or 4) as 1 in mark. */
__global__ void k_ls_mark_interface(LsGrid g, const LsObj *ob, const LsWin *win) {
    int i, j;
    if (!ls_point(g, win, i, j)) return;
    const int ij = j * g.P + i, st = ob[blockIdx.z].s[ij];
    ob[blockIdx.z].ia[ij] = (st == 3 || st == 4) ? 1 : 0;
}

/** One direction of a separable dilation by radius R (max over a window):
 * along x from ia into ib, along y from ib back into ia. */
template <bool ALONG_X>
__global__ void k_ls_dilate(LsGrid g, const LsObj *ob, const LsWin *win, int R) {
    int i, j;
    if (!ls_point(g, win, i, j)) return;
    const int *in = ALONG_X ? ob[blockIdx.z].ia : ob[blockIdx.z].ib;
    int *out = ALONG_X ? ob[blockIdx.z].ib : ob[blockIdx.z].ia;
    // Every marked point lies inside the window, and only the window's
    // marks are current: the reach is clipped to it.
    const LsWin w = win[blockIdx.z];
    int v = 0;
    if (ALONG_X) {
        const int lo = i - R < w.x0 ? w.x0 : i - R, hi = i + R >= w.x1 ? w.x1 - 1 : i + R;
        for (int a = lo; a <= hi && !v; a++) v = in[j * g.P + a];
    } else {
        const int lo = j - R < w.y0 ? w.y0 : j - R, hi = j + R >= w.y1 ? w.y1 - 1 : j + R;
        for (int b = lo; b <= hi && !v; b++) v = in[b * g.P + i];
    }
    out[j * g.P + i] = v;
}

/** Whether a point is a candidate of the march: a far point (status 0 or 7)
 * inside the dilated interface region (ia), the only points the march can
 * reach within the band limit. */
__device__ __forceinline__ bool ls_candidate(const LsObj &o, int ij) {
    const int st = o.s[ij];
    return (st == 0 || st == 7) && o.ia[ij];
}

/** Whether a status is that of a band point outside the solid. */
__device__ __forceinline__ bool ls_outside(int st) { return st == 4 || st == 5; }

/** Lists the tiles (TILE x TILE points of an object's window) that hold
 * candidates (OUTSIDE: points of the band outside the solid) as
 * (x | y << 16, object), one block of 256 threads per tile. */
template <int TILE, bool OUTSIDE>
__global__ void k_ls_collect_tiles(LsGrid g, const LsObj *ob, const LsWin *win, int *list, int *list_k, int *count, int cap,
                                   int *overflow) {
    const LsWin w = win[blockIdx.z];
    const int xe = min(w.x1, g.mL), ye = min(w.y1, g.nL);
    bool any = false;
    for (int t = threadIdx.x; t < TILE * TILE; t += blockDim.x) {
        const int i = w.x0 + blockIdx.x * TILE + t % TILE, j = w.y0 + blockIdx.y * TILE + t / TILE;
        if (i < xe && j < ye && (OUTSIDE ? ls_outside(ob[blockIdx.z].s[j * g.P + i]) : ls_candidate(ob[blockIdx.z], j * g.P + i)))
            any = true;
    }
    if (__syncthreads_or(any) && threadIdx.x == 0)
        ls_list_push(list, list_k, count, cap, overflow, blockIdx.x | blockIdx.y << 16, blockIdx.z);
}

/** Threads per block of the cooperative sweeps: one block per SM (the grid
 * barrier costs more with more blocks). */
constexpr int kFimThreads = 1024;

/** The march's staging: tiles of TILE x TILE points, SWEEPS sweeps between grid
 * barriers, the halo they need (the stencil and its change marks reach two
 * points), and the staged region. */
template <int TILE, int SWEEPS>
struct Fim {
    static constexpr int kHalo = 2 * SWEEPS, kReg = TILE + 2 * kHalo, kPoints = kReg * kReg, kRound = (kPoints + 31) & ~31;
    static constexpr size_t kSmem = kPoints * (3 * sizeof(double) + 2 * sizeof(short) + 3);
};

/** Appends q to a shared-memory list for the lanes that ask for it (all lanes
 * of the warp call). */
__device__ __forceinline__ void fim_push(bool on, int q, unsigned short *list, int *n) {
    const unsigned votes = __ballot_sync(0xffffffffu, on);
    if (!votes) return;
    int base = 0;
    if ((threadIdx.x & 31) == 0) base = atomicAdd(n, __popc(votes));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (on) list[base + __popc(votes & ((1u << (threadIdx.x & 31)) - 1))] = static_cast<unsigned short>(q);
}

/** All sweeps of the march fixed point in one cooperative launch: every
 * sweep evaluates the stencil at the candidates (Jacobi, reading cur, writing
 * nxt) and the loop ends after the first sweep that changed nothing. A
 * candidate whose stencil inputs did not change in the previous sweep keeps
 * its value (its stencil would return it again), so later sweeps only touch
 * the moving front.
 *
 * The blocks take the listed tiles (of every object), stage each with its
 * halo in shared memory and run SWEEPS sweeps there, the halo's points
 * redundantly in every tile that holds them, the region one sweep is valid in
 * shrinking by the stencil's reach; a grid barrier then exchanges the tiles
 * through global memory. The values are those of one barrier per sweep: a
 * sweep costs its evaluations, gathered into full warps and reading shared
 * memory, instead of some six round trips to L2 and a barrier, and the sweeps
 * past the last one of a batch change nothing (no marks are left). o.a/o.b
 * hold the values and o.ca/o.cb the change marks, swapped every batch;
 * k_ls_fim_init sets them where no tile is listed.
 *
 * It is bound by the evaluations of the busiest SM (some 600 instructions per
 * warp, half of them FP64) and their latency: about 2-4 us per sweep against
 * 10 us of a sweep over global memory with a barrier each. Measured (B200, us
 * per call before -> now): rotor 128^2 336 -> 108, 1024^2 457 -> 163; 32 bodies
 * 1024 x 2048 503 -> 395; flag 2048^2 892 -> 316. Lists built by the points that
 * change, instead of the marks' scan, took 185 us where this takes 149.
 *
 * flags[0..2] rotate as per-batch masks of the sweeps that changed something;
 * flags[3] receives the number of sweeps and flags[4] 1 if converged; after
 * ceil(sweeps / SWEEPS) batches the values are in o.b if that is odd. */
template <int TILE, int SWEEPS>
__global__ void __launch_bounds__(kFimThreads, 1) k_ls_fim_coop(LsGrid g, const LsObj *ob, const LsWin *win, const int *list,
                              const int *list_k, const int *countp, int cap, int *flags, int max_sweeps) {
    namespace cg = cooperative_groups;
    cg::grid_group grid = cg::this_grid();
    using F = Fim<TILE, SWEEPS>;
    constexpr int REG = F::kReg, RR = F::kPoints;
    extern __shared__ __align__(16) double fim_smem[];
    double *va = fim_smem, *vb = va + RR, *ph = vb + RR;
    unsigned short *cand = reinterpret_cast<unsigned short *>(ph + RR), *work = cand + RR;
    unsigned char *st = reinterpret_cast<unsigned char *>(work + RR), *ma = st + RR, *mb = ma + RR;
    __shared__ int ncand, nwork;
    __shared__ MarchK mk;
    const int tid = threadIdx.x, count = min(*countp, cap);
    if (tid == 0) mk.set(g);
    bool done = false;
    int it0 = 0;
    for (int batch = 0; it0 < max_sweeps; batch++, it0 += SWEEPS) {
        if (blockIdx.x == 0 && tid == 0) flags[(batch + 1) % 3] = 0;
        const bool odd = batch & 1;
        for (int tile = blockIdx.x; tile < count; tile += gridDim.x) {
            const LsObj &o = ob[list_k[tile]];
            const LsWin w = win[list_k[tile]];
            const double *gin = odd ? o.b : o.a;
            double *gout = odd ? o.a : o.b;
            const unsigned char *cin = odd ? o.cb : o.ca;
            unsigned char *cout = odd ? o.ca : o.cb;
            const int x0 = w.x0 + (list[tile] & 0xffff) * TILE - F::kHalo;
            const int y0 = w.y0 + (list[tile] >> 16) * TILE - F::kHalo;
            const int xe = min(w.x1, g.mL), ye = min(w.y1, g.nL);
            __syncthreads();  // the tile before is written out
            if (tid == 0) ncand = 0;
            __syncthreads();
            for (int t = tid; t < F::kRound; t += kFimThreads) {
                const int i = x0 + t % REG, j = y0 + t / REG;
                double v = 0, p = 0;
                unsigned char s = 4, mark = 0;
                bool c = false;
                // Outside the window nothing is a candidate, and no stencil
                // of one reaches there.
                if (t < RR && i >= w.x0 && i < xe && j >= w.y0 && j < ye) {
                    const int ij = j * g.P + i;
                    s = static_cast<unsigned char>(o.s[ij]);
                    p = o.phi[ij];
                    v = gin[ij];
                    mark = cin[ij];
                    c = (s == 0 || s == 7) && o.ia[ij];
                }
                if (t < RR) {
                    va[t] = vb[t] = v;
                    ph[t] = p;
                    st[t] = s;
                    ma[t] = mark;
                    mb[t] = 0;
                }
                fim_push(c, t, cand, &ncand);
            }
            __syncthreads();
            const int nc = ncand;
            int mask = 0;
#pragma unroll 1
            for (int k = 0; k < SWEEPS; k++) {
                const int it = it0 + k, ring = 2 * (k + 1), span = REG - 2 * ring;
                // Where the second-order stencil is not monotone, the plain sweeps can
                // cycle between two states instead of settling (seen on thin solids at
                // fine grids). After half the sweep budget each value may then only
                // move towards the interface, which settles; flags[12] records it.
                const bool monotone = it >= max_sweeps / 2;
                const double *cur = k & 1 ? vb : va;
                double *nxt = k & 1 ? va : vb;
                const unsigned char *cprev = k & 1 ? mb : ma;
                unsigned char *cnow = k & 1 ? ma : mb;
                // The candidates that keep their values are copied; the others
                // are listed, so that full warps evaluate them.
                if (tid == 0) nwork = 0;
                __syncthreads();
                for (int t = tid; t < ((nc + 31) & ~31); t += kFimThreads) {
                    const int q = t < nc ? cand[t] : 0, lx = q % REG - ring, ly = q / REG - ring;
                    bool eval = false;
                    if (t < nc && lx >= 0 && lx < span && ly >= 0 && ly < span) {
                        const unsigned char *m0 = cprev + q;
                        eval = it == 0 || (m0[0] | m0[-1] | m0[1] | m0[-2] | m0[2] | m0[-REG] | m0[REG] | m0[-2 * REG] |
                                           m0[2 * REG]);
                        if (!eval) {
                            nxt[q] = cur[q];
                            cnow[q] = 0;
                        }
                    }
                    fim_push(eval, q, work, &nwork);
                }
                __syncthreads();
                const int nw = nwork;
                bool ch = false;
                for (int t = tid; t < nw; t += kFimThreads) {
                    const int q = work[t], lx = q % REG, ly = q / REG, i = x0 + lx, j = y0 + ly;
                    const double old = cur[q], sg = st[q] == 7 ? 1.0 : -1.0;
                    double v = march_value(mk, REG, ph, st, cur, q, st[q], sg, old, i > 0, i > 1, i < g.mL - 1, i < g.mL - 2,
                                           j > 0, j > 1, j < g.nL - 1, j < g.nL - 2);
                    if (monotone && sg * v > sg * old) v = old;
                    nxt[q] = v;
                    // Changes in the last bits (the tail of the fixed point) do not
                    // count: the sweeps end once every value is settled to 1e-13.
                    const bool c = fabs(v - old) > 1e-13 * fabs(v);
                    cnow[q] = c;
                    if (c && lx >= F::kHalo && lx < F::kHalo + TILE && ly >= F::kHalo && ly < F::kHalo + TILE) ch = true;
                }
                if (__syncthreads_or(ch)) mask |= 1 << k;
            }
            if (mask && tid == 0) atomicOr(&flags[batch % 3], mask);
            for (int t = tid; t < TILE * TILE; t += kFimThreads) {
                const int lx = F::kHalo + t % TILE, ly = F::kHalo + t / TILE, q = ly * REG + lx;
                const int i = x0 + lx, j = y0 + ly;
                if (i < xe && j < ye) {
                    gout[j * g.P + i] = SWEEPS & 1 ? vb[q] : va[q];
                    cout[j * g.P + i] = SWEEPS & 1 ? mb[q] : ma[q];
                }
            }
        }
        grid.sync();
        const int mask = *reinterpret_cast<volatile int *>(&flags[batch % 3]);
        const int last = __ffs(~mask) - 1;  // the first sweep that changed nothing
        if (last < SWEEPS && it0 + last < max_sweeps) {
            it0 += last + 1;
            done = true;
            break;
        }
    }
    if (blockIdx.x == 0 && tid == 0) {
        flags[3] = done ? it0 : max_sweeps;
        flags[4] = done ? 1 : 0;
        flags[12] = flags[3] > max_sweeps / 2 ? 1 : 0;
    }
}

/** The extrapolation's staging, as Fim: the fit reaches three points. */
template <int TILE, int SWEEPS>
struct Ext {
    static_assert(SWEEPS & 1, "the last sweep writes the second buffer, as a single one does");
    static_assert(3 * SWEEPS >= kExtMaxRadius, "the halo holds the widest window");
    static constexpr int kHalo = 3 * SWEEPS, kReg = TILE + 2 * kHalo, kPoints = kReg * kReg, kRound = (kPoints + 31) & ~31;
    // listed points: those a sweep may evaluate (three from the region's edge)
    static constexpr int kList = (kReg - 6) * (kReg - 6);
    static constexpr size_t kSmem = kPoints * 5 * sizeof(double) + kList * (3 * sizeof(double) + sizeof(short));
};

/** The fit at point q of a staged tile of row length reg, whose window grows
 * while it is singular (points outside the grid or the band hold kUnset); false
 * where it stays so. */
__device__ __forceinline__ bool ext_widen(const double *ph, const double *cx, const double *cy, int q, int reg, double &ox,
                                          double &oy) {
    const double pp = ph[q];
    for (int r = 3; r <= kExtMaxRadius; r++) {
        ExtFit f;
        f.clear();
        double acc[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll 1
        for (int dj = -r; dj <= r; dj++)
#pragma unroll 1
            for (int di = -r; di <= r; di++) {
                const int e = q + dj * reg + di;
                const double p = ph[e];
                if (!(p < pp)) continue;
                f.moments(di, dj, pp - p);
                ExtFit::values(di, dj, pp - p, cx[e], cy[e], acc);
            }
        const double det = f.det();
        if (ExtFit::singular(det)) continue;
        double c[3];
        f.solve(det, c);
        ox = ExtFit::value(acc, c);
        oy = ExtFit::value(acc + 3, c);
        return true;
    }
    return false;
}

/** The batches of k_ls_extrap_tiles: the sweeps made until nothing changed, or
 * minus one if they run out or a fit is singular. */
template <int TILE, int SWEEPS, bool WIDE>
__device__ __forceinline__ int ext_batches(const LsGrid &g, const LsObj *ob, const LsWin *win, const int *list, const int *list_k,
                                           int count, int *flags, int max_sweeps) {
    namespace cg = cooperative_groups;
    cg::grid_group grid = cg::this_grid();
    using E = Ext<TILE, SWEEPS>;
    constexpr int REG = E::kReg, RR = E::kPoints, NL = E::kList, kRun = WIDE ? 1 : SWEEPS;
    extern __shared__ __align__(16) double ext_smem[];
    double *ph = ext_smem, *xa = ph + RR, *ya = xa + RR, *xb = ya + RR, *yb = xb + RR, *fit = yb + RR;
    unsigned short *work = reinterpret_cast<unsigned short *>(fit + 3 * NL);
    __shared__ int nwork;
    const int tid = threadIdx.x;
    constexpr int kFirst = WIDE ? 1 : 0;
    for (int it0 = 0, batch = kFirst; it0 < max_sweeps; batch++, it0 += kRun) {
        if (blockIdx.x == 0 && tid == 0) flags[(batch + 1) % 3] = 0;
        const bool odd = batch & 1;
        for (int tile = blockIdx.x; tile < count; tile += gridDim.x) {
            const LsObj &o = ob[list_k[tile]];
            const LsWin w = win[list_k[tile]];
            const double *gx = batch == kFirst ? o.nX : (odd ? o.b : o.a), *gy = batch == kFirst ? o.nY : (odd ? o.d : o.c);
            const int x0 = w.x0 + (list[tile] & 0xffff) * TILE - E::kHalo;
            const int y0 = w.y0 + (list[tile] >> 16) * TILE - E::kHalo;
            const int xe = min(w.x1, g.mL), ye = min(w.y1, g.nL);
            __syncthreads();  // the tile before is written out
            if (tid == 0) nwork = 0;
            __syncthreads();
            for (int t = tid; t < E::kRound; t += kFimThreads) {
                const int lx = t % REG, ly = t / REG, i = x0 + lx, j = y0 + ly;
                // points outside the band never enter a fit
                double p = kUnset, x = 0, y = 0;
                bool out = false;
                if (t < RR && i >= 0 && i < g.mL && j >= 0 && j < g.nL) {
                    const int ij = j * g.P + i, st = o.s[ij];
                    if (st >= 2 && st <= 5) {
                        out = ls_outside(st);
                        p = o.phi[ij];
                        x = out ? gx[ij] : o.nX[ij];
                        y = out ? gy[ij] : o.nY[ij];
                    }
                }
                if (t < RR) {
                    ph[t] = p;
                    xa[t] = xb[t] = x;
                    ya[t] = yb[t] = y;
                }
                // (outside the window the band has no points of this object)
                constexpr int kEdge = WIDE ? E::kHalo : 3;
                fim_push(out && lx >= kEdge && lx < REG - kEdge && ly >= kEdge && ly < REG - kEdge, t, work, &nwork);
            }
            __syncthreads();
            const int nw = nwork;
            int mask = 0;
#pragma unroll 1
            for (int k = 0; k < kRun; k++) {
                const int ring = 3 * (k + 1);
                const double *cx = k & 1 ? xb : xa, *cy = k & 1 ? yb : ya;
                double *tx = k & 1 ? xa : xb, *ty = k & 1 ? ya : yb;
                bool ch = false;
                for (int t = tid; t < nw; t += kFimThreads) {
                    const int q = work[t], lx = q % REG, ly = q / REG;
                    if (!WIDE && (lx < ring || lx >= REG - ring || ly < ring || ly >= REG - ring)) continue;
                    double ox, oy;
                    if constexpr (WIDE) {
                        if (!ext_widen(ph, cx, cy, q, REG, ox, oy)) {
                            flags[5] = INCRMT_ERR_EXTRAP_SINGULAR;
                            ox = cx[q];
                            oy = cy[q];
                        }
                    } else {
                        const double pp = ph[q];
                        double acc[6] = {0, 0, 0, 0, 0, 0}, c[3];
                        if (k == 0) {
                            ExtFit f;
                            f.clear();
#pragma unroll
                            for (int dj = -3; dj <= 3; dj++)
#pragma unroll
                                for (int di = -3; di <= 3; di++) {
                                    const int e = q + dj * REG + di;
                                    const double p = ph[e];
                                    if (!(p < pp)) continue;
                                    const double ww = pp - p;
                                    f.moments(di, dj, ww);
                                    ExtFit::values(di, dj, ww, cx[e], cy[e], acc);
                                }
                            const double det = f.det();
                            if (ExtFit::singular(det)) flags[11] = 1;
                            f.solve(det, c);
                            fit[t] = c[0];
                            fit[NL + t] = c[1];
                            fit[2 * NL + t] = c[2];
                        } else {
#pragma unroll 1
                            for (int dj = -3; dj <= 3; dj++)
#pragma unroll
                                for (int di = -3; di <= 3; di++) {
                                    const int e = q + dj * REG + di;
                                    const double p = ph[e];
                                    if (!(p < pp)) continue;
                                    ExtFit::values(di, dj, pp - p, cx[e], cy[e], acc);
                                }
                            c[0] = fit[t]; c[1] = fit[NL + t]; c[2] = fit[2 * NL + t];
                        }
                        ox = ExtFit::value(acc, c);
                        oy = ExtFit::value(acc + 3, c);
                    }
                    if ((ox != cx[q] || oy != cy[q]) && lx >= E::kHalo && lx < E::kHalo + TILE && ly >= E::kHalo &&
                        ly < E::kHalo + TILE)
                        ch = true;
                    tx[q] = ox;
                    ty[q] = oy;
                }
                if (__syncthreads_or(ch)) mask |= 1 << k;
            }
            if (mask && tid == 0) atomicOr(&flags[batch % 3], mask);
            double *ox = odd ? o.a : o.b, *oy = odd ? o.c : o.d;
            for (int t = tid; t < nw; t += kFimThreads) {
                const int q = work[t], lx = q % REG, ly = q / REG, i = x0 + lx, j = y0 + ly;
                if (lx >= E::kHalo && lx < E::kHalo + TILE && ly >= E::kHalo && ly < E::kHalo + TILE && i < xe && j < ye) {
                    ox[j * g.P + i] = xb[q];
                    oy[j * g.P + i] = yb[q];
                }
            }
        }
        grid.sync();
        // (a singular fit depends on the level set alone: the first batch raises
        // its flag or none does)
        if (*reinterpret_cast<volatile int *>(&flags[WIDE ? 5 : 11])) return -1;
        const int mask = *reinterpret_cast<volatile int *>(&flags[batch % 3]);
        const int last = __ffs(~mask) - 1;  // the first sweep that changed nothing
        if (last < kRun && it0 + last < max_sweeps) return it0 + last + 1;
    }
    return -1;
}

/** All sweeps of the extrapolation wavefront in one cooperative launch, staged
 * like the march (k_ls_fim_coop): the fit's moments depend on the level set
 * alone and are formed by the first sweep of a batch; the others only sum the
 * values of the 7 x 7 window. The first batch reads the reference map itself. A
 * point whose window of radius 3 gives a singular fit (a grid in small units,
 * where the weights are small) raises flags[11] and ends the launch after its
 * first batch; a WIDE launch then starts over from batch 1 with one sweep per
 * batch, for which the halo holds the widest window, and a fit that stays
 * singular raises flags[5]. (One launch for both took the usual batches 1 to 5
 * per cent longer, for the registers.) flags[0..2], [3] and [4] as in
 * k_ls_fim_coop; the values are in o.b, o.d if the last batch's number is even
 * (ext_in_b).
 *
 * Bound by the window sums of the busiest SM. Measured (B200, us per call, one
 * sweep per barrier over global memory -> here): rotor 128^2 266 -> 108, 1024^2
 * 288 -> 107; 32 bodies 1024 x 2048 377 -> 271; flag 2048^2 469 -> 211. Both
 * launches of a circle with windows of radius 4, 22 sweeps: 256^2 940 -> 524,
 * 1024^2 1245 -> 531. */
template <int TILE, int SWEEPS, bool WIDE>
__global__ void __launch_bounds__(kFimThreads, 1) k_ls_extrap_tiles(LsGrid g, const LsObj *ob, const LsWin *win, const int *list,
                                                                    const int *list_k, const int *countp, int cap, int *flags,
                                                                    int max_sweeps) {
    const int sweeps = ext_batches<TILE, SWEEPS, WIDE>(g, ob, win, list, list_k, min(*countp, cap), flags, max_sweeps);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        flags[3] = sweeps < 0 ? max_sweeps : sweeps;
        flags[4] = sweeps >= 0;
    }
}

/** Whether k_ls_extrap_tiles left its values in o.b, o.d: its batches are the
 * sweeps in groups, or a first batch given up and then one per sweep. */
inline bool ext_in_b(int sweeps, int per_batch, bool wide) { return (wide ? sweeps + 1 : cdiv(sweeps, per_batch)) & 1; }

/** Stores the values of k_ls_extrap_tiles (in o.b, o.d if in_b) into nX, nY. */
__global__ void k_ls_extrap_keep(LsGrid g, const LsObj *ob, const LsWin *win, bool in_b) {
    int i, j;
    if (!ls_point(g, win, i, j)) return;
    const LsObj &o = ob[blockIdx.z];
    const int ij = j * g.P + i;
    if (!ls_outside(o.s[ij])) return;
    o.nX[ij] = in_b ? o.b[ij] : o.a[ij];
    o.nY[ij] = in_b ? o.d[ij] : o.c[ij];
}

}  // namespace incrmt
