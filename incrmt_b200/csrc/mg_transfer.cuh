// Transfers between a level and the next coarser one: the operator-dependent
// prolongation weights (black-box multigrid) and the two kernels a V-cycle
// runs on them, one thread per cell.
//
// A cell is the fine points that share a base coarse point: 2 x 2 where both
// directions are halved, 2 x 1 or 1 x 2 where one is. Its point on the coarse
// point has the single weight 1; the others' weights, eight per 2 x 2 cell
// instead of sixteen with four slots per point, are kept as planes over the
// cells, in each precision:
//   both halved: 0, 1: corners (0,0), (1,0) of point (1,0); 2, 3: corners
//     (0,0), (0,1) of point (0,1); 4-7: the four corners of point (1,1);
//   one halved:  0, 1: corners 0, 1 of the odd point.
// All that needs the weights reads these (plane_weights).
#pragma once
#include "mg_ops.cuh"

namespace incrmt {
namespace {

constexpr int kPX = 32, kPY = 8;  // cells of a block of k_build_p

/** Operator-dependent prolongation of a level (black-box multigrid:
 * Dendy, J. Comput. Phys. 48 (1982) 366-386), a fine point's weights for the
 * coarse points about it, as planes Q. A point on a coarse point takes it with weight
 * 1; a point between two coarse points along x takes L/(-C) and R/(-C), L, C, R
 * its stencil summed over the columns left of, through and right of it (the
 * operator collapsed along y), and along y likewise with the rows; a point
 * between four coarse points takes -(its stencil entries times its eight
 * neighbours' weights)/(its diagonal). Constant coefficients give the bilinear
 * 1, 1/2, 1/4; across a density jump the weights follow the flux; at the
 * zero-pressure edge of the MAC system the last point's weight drops to about
 * 1/3. Weights are formed in double precision so that constants map onto
 * constants exactly and the coarse operators of a pure-Neumann problem keep
 * their null space.
 *
 * One thread per cell; where both directions are halved the blocks overlap by
 * a column and a row, whose cells' edge weights the last points need. Bound by
 * the loads' latency and, on the fine level, by memory (4.1 TB/s). Measured (B200,
 * us, two passes of one thread per point -> here): MAC 4096^2 613 -> 124, its
 * Galerkin levels 37 -> 9 each (251 and 14 while it wrote four weights per point
 * as well). */
template <class Op, bool KX, bool KY>
__global__ void __launch_bounds__(kPX * kPY) k_build_p(Op op, int fm, int fn, int px, int py, int cm, int cn, double *Q) {
    constexpr bool both = KX && KY;
    __shared__ double wx[2][kPY][kPX + 1], wy[2][kPY][kPX + 1];
    const int cx = cells_of(fm, KX), cy = cells_of(fn, KY);
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int Iu = blockIdx.x * (both ? kPX - 1 : kPX) + tx, Ju = blockIdx.y * (both ? kPY - 1 : kPY) + ty;
    // the overlap wraps around a periodic grid (even sizes: whole cells)
    const int I = px && Iu >= cx ? Iu - cx : Iu, J = py && Ju >= cy ? Ju - cy : Ju;
    const bool in = I < cx && J < cy;
    const int i = KX ? 2 * I : I, j = KY ? 2 * J : J;
    const bool v1 = I + 1 < cm || px, v2 = J + 1 < cn || py;  // the corners above the base exist
    double a[9], x0 = 0, x1 = 0, y0 = 0, y1 = 0;
    // (the entries are rounded before they are summed)
    auto sum3 = [](double p, double q, double r) { return add_rn(add_rn(p, q), r); };
    if (KX && in && i + 1 < fm) {
        op.coef9(i + 1, j, a);
        const double L = sum3(a[0], a[3], a[6]), C = sum3(a[1], a[4], a[7]), R = sum3(a[2], a[5], a[8]);
        x0 = L / (-C);
        if (v1) x1 = R / (-C);
    }
    if (KY && in && j + 1 < fn) {
        op.coef9(i, j + 1, a);
        const double D = sum3(a[0], a[1], a[2]), M = sum3(a[3], a[4], a[5]), U = sum3(a[6], a[7], a[8]);
        y0 = D / (-M);
        if (v2) y1 = U / (-M);
    }
    if (both) {
        wx[0][ty][tx] = x0; wx[1][ty][tx] = x1;
        wy[0][ty][tx] = y0; wy[1][ty][tx] = y1;
        __syncthreads();
        if (tx == kPX - 1 || ty == kPY - 1) return;
    }
    if (Iu >= cx || Ju >= cy) return;
    const long NC = static_cast<long>(cx) * cy, q = I + static_cast<long>(cx) * J;
    if (!both) {
        Q[q] = KX ? x0 : y0;
        Q[NC + q] = KX ? x1 : y1;
        return;
    }
    double w[4] = {0, 0, 0, 0};
    if (i + 1 < fm && j + 1 < fn) {
        op.coef9(i + 1, j + 1, a);
        // The neighbours in row order, each with its nonzero weights for the
        // cell's corners; an entry outside the grid is zero.
        double c0 = 0, c1 = 0, c2 = 0, c3 = 0;
        c0 = add_prod(c0, a[0], 1.0);
        c0 = add_prod(c0, a[1], x0);
        c1 = add_prod(c1, a[1], x1);
        c1 = add_prod(c1, a[2], 1.0);
        c0 = add_prod(c0, a[3], y0);
        c2 = add_prod(c2, a[3], y1);
        c1 = add_prod(c1, a[5], wy[0][ty][tx + 1]);
        c3 = add_prod(c3, a[5], wy[1][ty][tx + 1]);
        c2 = add_prod(c2, a[6], 1.0);
        c2 = add_prod(c2, a[7], wx[0][ty + 1][tx]);
        c3 = add_prod(c3, a[7], wx[1][ty + 1][tx]);
        c3 = add_prod(c3, a[8], 1.0);
        w[0] = -c0 / a[4];
        if (v1) w[1] = -c1 / a[4];
        if (v2) w[2] = -c2 / a[4];
        if (v1 && v2) w[3] = -c3 / a[4];
    }
    Q[q] = x0; Q[NC + q] = x1;
    Q[2 * NC + q] = y0; Q[3 * NC + q] = y1;
#pragma unroll
    for (int r = 0; r < 4; r++) Q[(4 + r) * NC + q] = w[r];
}

constexpr int kRX = 32, kRY = 16;  // cells of a block of k_restrict_cells

/** Coarse right-hand side b_c = P^T (b - A z), one
 * thread per cell: it forms the residuals of its fine points into shared
 * memory, then sums its coarse point's support with the weights and in the
 * order of k_restrict: the same values. In a halved direction the blocks
 * overlap by a cell, whose upper points the next block's first supports reach.
 * Bound by bandwidth on the large levels (MAC 4096^2: 56 bytes a point, 940 MB
 * in 169 us) and by the loads' latency below. Measured (B200, us, staging every
 * point and its four FP64 weights -> here): MAC 4096^2 FP64 330 -> 169, 2048^2
 * FP32 56 -> 28; FEM 2048^2 FP32 68 -> 32; Galerkin 2048 x 1024 FP32 54 -> 37, a
 * 4096^2 solve's four levels FP64 58.8 -> 27.6 on average. */
template <class Op, class T, bool KX, bool KY>
__global__ void __launch_bounds__(kRX * kRY) k_restrict_cells(Op op, const T *z, const T *b, int fm, int fn, int px, int py,
                                                              int cm, int cn, T *bc, const T *Q) {
    constexpr int NX = KX ? 2 : 1, NY = KY ? 2 : 1;
    __shared__ T rs[NY][NX][kRY][kRX + 1];
    const int cx = cells_of(fm, KX), cy = cells_of(fn, KY);
    const int tx = threadIdx.x, ty = threadIdx.y;
    int I = blockIdx.x * (KX ? kRX - 1 : kRX) + tx - (KX ? 1 : 0), J = blockIdx.y * (KY ? kRY - 1 : kRY) + ty - (KY ? 1 : 0);
    const bool own = I >= 0 && J >= 0 && I < cm && J < cn && tx >= (KX ? 1 : 0) && ty >= (KY ? 1 : 0);
    // the overlap below a periodic grid wraps (even sizes: whole cells)
    if (I < 0 && px) I += cx;
    if (J < 0 && py) J += cy;
    const bool in = I >= 0 && J >= 0 && I < cx && J < cy;
#pragma unroll
    for (int v = 0; v < NY; v++)
#pragma unroll
        for (int u = 0; u < NX; u++) {
            const int i = NX * I + u, j = NY * J + v;
            // (of the overlap's cells only the points next to the block)
            const bool use = in && i < fm && j < fn && (!KX || tx > 0 || u == 1) && (!KY || ty > 0 || v == 1);
            rs[v][u][ty][tx] = use ? residual_at(op, i, j, z, b[i + static_cast<long>(fm) * j]) : T(0);
        }
    __syncthreads();
    if (!own) return;
    const long NC = static_cast<long>(cx) * cy;
    const T *q = Q + I + static_cast<long>(cx) * J;
    // the cells left of and below this one
    const bool hl = I > 0 || px, hd = J > 0 || py;
    const long ql = I > 0 ? -1 : cx - 1, qd = J > 0 ? -static_cast<long>(cx) : NC - cx;
    T t = 0;
    auto add = [&](T w, T r) { if (w != 0) t = add_prod(t, w, r); };
    if constexpr (KX && KY) {
        const T w0 = hl && hd ? q[7 * NC + ql + qd] : T(0), w1 = hd ? q[3 * NC + qd] : T(0), w2 = hd ? q[6 * NC + qd] : T(0);
        const T w3 = hl ? q[NC + ql] : T(0), w5 = q[0];
        const T w6 = hl ? q[5 * NC + ql] : T(0), w7 = q[2 * NC], w8 = q[4 * NC];
        add(w0, rs[1][1][ty - 1][tx - 1]);
        add(w1, rs[1][0][ty - 1][tx]);
        add(w2, rs[1][1][ty - 1][tx]);
        add(w3, rs[0][1][ty][tx - 1]);
        add(T(1), rs[0][0][ty][tx]);
        add(w5, rs[0][1][ty][tx]);
        add(w6, rs[1][1][ty][tx - 1]);
        add(w7, rs[1][0][ty][tx]);
        add(w8, rs[1][1][ty][tx]);
    } else if constexpr (KX) {
        const T w0 = hl ? q[NC + ql] : T(0), w2 = q[0];
        add(w0, rs[0][1][ty][tx - 1]);
        add(T(1), rs[0][0][ty][tx]);
        add(w2, rs[0][1][ty][tx]);
    } else {
        const T w0 = hd ? q[NC + qd] : T(0), w2 = q[0];
        add(w0, rs[1][0][ty - 1][tx]);
        add(T(1), rs[0][0][ty][tx]);
        add(w2, rs[1][0][ty][tx]);
    }
    bc[I + cm * J] = t;
}

/** Fine correction z += P z_c, one thread per cell; vec: the rows' point pairs
 * are aligned for one access. Bound by bandwidth (34 bytes a point in FP64
 * instead of 50, 17 instead of 41 in FP32). Measured (B200, us, four FP64 weights
 * per point -> here): a 4096^2 solve's five levels FP64 45.1 -> 23.2 on average,
 * the 2048^2 flag's in FP32 14.9 -> 6.0. */
template <class T, bool KX, bool KY>
__global__ void __launch_bounds__(256) k_prolong_cells(T *z, int fm, int fn, int px, int py, const T *zc, int cm, int cn,
                                                       const T *Q, bool vec) {
    using T2 = std::conditional_t<sizeof(T) == 8, double2, float2>;
    const int cx = cells_of(fm, KX), cy = cells_of(fn, KY);
    const int I = blockIdx.x * blockDim.x + threadIdx.x, J = blockIdx.y * blockDim.y + threadIdx.y;
    if (I >= cx || J >= cy) return;
    const int NX = KX ? 2 : 1, NY = KY ? 2 : 1;
    const int i = NX * I, j = NY * J;
    const long NC = static_cast<long>(cx) * cy;
    const T *q = Q + I + static_cast<long>(cx) * J;
    // The corner above the base wraps on a periodic grid; on another one its
    // weight is zero where it does not exist.
    const int I1 = I + 1 < cm ? I + 1 : 0, J1 = J + 1 < cn ? J + 1 : 0;
    const T z00 = zc[I + cm * J], z10 = KX ? zc[I1 + cm * J] : T(0), z01 = KY ? zc[I + cm * J1] : T(0),
            z11 = KX && KY ? zc[I1 + cm * J1] : T(0);
    auto two = [](T w0, T a, T w1, T b) {
        T t = 0;
        if (w0 != 0) t = add_prod(t, w0, a);
        if (w1 != 0) t = add_prod(t, w1, b);
        return t;
    };
    T *row = z + i + static_cast<long>(fm) * j;
    const bool right = KX && i + 1 < fm, up = KY && j + 1 < fn;
    const T d00 = z00;
    T d10 = 0, d01 = 0, d11 = 0;
    if (KX) d10 = two(q[0], z00, q[NC], z10);
    if (KY) d01 = two(q[KX ? 2 * NC : 0], z00, q[KX ? 3 * NC : NC], z01);
    if (KX && KY) {
        const T w0 = q[4 * NC], w1 = q[5 * NC], w2 = q[6 * NC], w3 = q[7 * NC];
        if (w0 != 0) d11 = add_prod(d11, w0, z00);
        if (w1 != 0) d11 = add_prod(d11, w1, z10);
        if (w2 != 0) d11 = add_prod(d11, w2, z01);
        if (w3 != 0) d11 = add_prod(d11, w3, z11);
    }
    auto add = [&](T *p, T a, T b) {
        if (KX && vec) {
            T2 *p2 = reinterpret_cast<T2 *>(p);
            T2 v = *p2;
            v.x += a;
            v.y += b;
            *p2 = v;
        } else {
            p[0] += a;
            if (right) p[1] += b;
        }
    };
    add(row, d00, d10);
    if (up) add(row + fm, d01, d11);
}

}  // namespace
}  // namespace incrmt
