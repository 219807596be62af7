// Geometric multigrid kernels and driver (see mg.cuh for the method).
#include <cmath>
#include <cstring>
#include <type_traits>
#include "mg.cuh"
#include "mg_cells.cuh"
#include "mg_tail.cuh"

namespace incrmt {

namespace {

constexpr int kNu1 = 2, kNu2 = 2, kCoarseSweeps = 64, kCoarsestSize = 16, kMaxLevels = 24;
/** Coupling ratio beyond which only the strongly coupled direction is
 * coarsened (semi-coarsening). */
constexpr double kSemiRatio = 2.0;
/** Largest residual ratio an FP32 defect-correction step may reach before the
 * solve continues in FP64. */
constexpr double kMixedContraction = 0.5;

// ---------------------------------------------------------------------------
// Transfer-operator index helpers (identical rules to the CPU oracle's shim).

__host__ __device__ __forceinline__ int wrap_idx(int i, int m, int p, bool &ok) {
    if (i < 0) { if (p) i += m; else ok = false; }
    else if (i >= m) { if (p) i -= m; else ok = false; }
    return i;
}

/** t + a*b with the product rounded before the sum (no fused multiply-add),
 * as the CPU oracle evaluates it: with the operator-dependent weights the
 * products are not exact, and a fused form would round them differently. The
 * FP32 V-cycles are not compared bit for bit and keep the fused form. */
__device__ __forceinline__ double add_prod(double t, double a, double b) { return __dadd_rn(t, __dmul_rn(a, b)); }
__device__ __forceinline__ float add_prod(float t, float a, float b) { return t + a * b; }

/** Floor of a/2 for any sign of a. */
__host__ __device__ __forceinline__ int half_floor(int a) { return a >= 0 ? a / 2 : -((1 - a) / 2); }

/** Coarse base index of fine index i along a direction: i/2 rounded down
 * when the direction is coarsened, else i. */
__host__ __device__ __forceinline__ int base_of(int i, bool k) { return k ? half_floor(i) : i; }

/** Prolongation weight of fine point (fi,fj) (unwrapped indices) for coarse
 * point (I,J): entry qx+2qy of the point's four weights, with (qx,qy)
 * the coarse point's offset from the point's base; 0 when it is not one of
 * its corners or the point is outside a non-periodic grid. */
__device__ __forceinline__ double pweight(const double *Q, int fm, int fn, int px, int py, bool kx, bool ky, int fi,
                                          int fj, int I, int J) {
    const int qx = I - base_of(fi, kx), qy = J - base_of(fj, ky);
    if (qx < 0 || qx > 1 || qy < 0 || qy > 1) return 0;
    bool ok = true;
    const int i = wrap_idx(fi, fm, px, ok), j = wrap_idx(fj, fn, py, ok);
    if (!ok) return 0;
    double w[4];
    plane_weights(Q, cells_of(fm, kx), cells_of(fn, ky), kx, ky, i, j, w);
    return w[qx + 2 * qy];
}

}  // namespace
}  // namespace incrmt

#include "mg_transfer.cuh"

namespace incrmt {

namespace {

inline bool can_coarsen(int m, int p) { return p ? (m % 2 == 0 && m / 2 >= 4) : m >= 5; }

// ---------------------------------------------------------------------------
// Coefficient set-up kernels.

/** Edge reciprocal densities of the MAC system from the ghosted cell density
 * (fluid_2d::set_edge_irho, fluid_2d.cc:1140-1160). */
__global__ void k_mac_coef(const double *rho, int ml, int cm, int cn, double *ex, double *ey,
                           float *exf, float *eyf) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y;
    if (j < cn && i <= cm) {
        const int q = (i + 2) + ml * (j + 2);
        double v = 0.5 / rho[q] + 0.5 / rho[q - 1];
        ex[j * (cm + 1) + i] = v;
        exf[j * (cm + 1) + i] = static_cast<float>(v);
    }
    if (j <= cn && i < cm) {
        const int q = (i + 2) + ml * (j + 2);
        double v = 0.5 / rho[q] + 0.5 / rho[q - ml];
        ey[j * cm + i] = v;
        eyf[j * cm + i] = static_cast<float>(v);
    }
}

/** Cell reciprocal density at each FEM node, the cell below-left of the node
 * (fluid_2d::set_corner_irho, fluid_2d.cc:1163-1170). */
__global__ void k_fem_coef(const double *rho, int ml, int mf, int nf, double *c, float *cf) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= mf || j >= nf) return;
    double v = 1. / rho[(i + 1) + ml * (j + 1)];
    c[j * mf + i] = v;
    cf[j * mf + i] = static_cast<float>(v);
}


/** Galerkin coarse stencil A_c = P^T A P, one thread per coarse unknown
 * (I,J): over the fine points f of its support (the 3 x 3 fine points about
 * (2I,2J)) and the stencil neighbours g of f, P(f,(I,J)) A(f,g) P(g,K) is
 * added to the entry of K - (I,J), K running over g's corners. */
template <class Op>
__global__ void k_galerkin(Op op, int fm, int fn, int px, int py, bool kx, bool ky, int cm, int cn, double *st,
                           const double *Q) {
    const int I = blockIdx.x * blockDim.x + threadIdx.x, J = blockIdx.y * blockDim.y + threadIdx.y;
    if (I >= cm || J >= cn) return;
    double q[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    const int x0 = kx ? 2 * I - 1 : I, x1 = kx ? 2 * I + 1 : I, y0 = ky ? 2 * J - 1 : J, y1 = ky ? 2 * J + 1 : J;
    for (int fj = y0; fj <= y1; fj++)
        for (int fi = x0; fi <= x1; fi++) {
            const double w = pweight(Q, fm, fn, px, py, kx, ky, fi, fj, I, J);
            if (w == 0) continue;
            bool ok = true;
            const int i = wrap_idx(fi, fm, px, ok), j = wrap_idx(fj, fn, py, ok);
            double a[9];
            op.coef9(i, j, a);
            for (int dj = -1; dj <= 1; dj++)
                for (int di = -1; di <= 1; di++) {
                    const double av = a[3 * (dj + 1) + di + 1];
                    if (av == 0) continue;
                    bool okg = true;
                    const int gi = wrap_idx(fi + di, fm, px, okg), gj = wrap_idx(fj + dj, fn, py, okg);
                    if (!okg) continue;
                    double g[4];
                    plane_weights(Q, cells_of(fm, kx), cells_of(fn, ky), kx, ky, gi, gj, g);
                    const int ox = base_of(fi + di, kx) - I, oy = base_of(fj + dj, ky) - J;
                    for (int r = 0; r < 4; r++) {
                        const int kx_ = ox + (r & 1), ky_ = oy + (r >> 1);
                        if (g[r] == 0 || kx_ < -1 || kx_ > 1 || ky_ < -1 || ky_ > 1) continue;
                        double &qe = q[3 * (ky_ + 1) + kx_ + 1];
                        qe = add_prod(qe, __dmul_rn(w, av), g[r]);
                    }
                }
        }
    const long N = static_cast<long>(cm) * cn;
    for (int e = 0; e < 9; e++) st[e * N + colour_index(cm, cn, I, J)] = q[e];
}

constexpr int kGalRows = 4;  // coarse rows of a tile

/** k_galerkin for a 32 x kGalRows tile of coarse unknowns per block,
 * with every input staged in shared memory first: the nine stencil entries
 * of the fine points of the tile's supports (coef9; the fine region
 * 2X0-1 .. 2(X0+31)+1 in a coarsened direction, X0 .. X0+31 otherwise) and
 * the four prolongation weights of that region grown by one point (the
 * stencil neighbours), zero outside a non-periodic grid. The sums then run
 * exactly as in k_galerkin, in the same order: the same values, without
 * each thread re-reading some four hundred entries from global memory.
 * Dynamic shared memory: galerkin_tile_smem(kx, ky) bytes.
 *
 * Bound by the sums' shared-memory reads and FP64 latency. Four rows leave room
 * for three blocks per SM, and the sums have no branches: a point's zero
 * weights are known from its parities. Measured (B200, us; 8 rows, tests of
 * every weight -> here): MAC 4096^2 1782 -> 660 (8 rows 1163, 2 rows 1044), the
 * 2048^2 flag's Galerkin levels 42.1 -> 15.5, FEM 1024 x 2048 94. Weights staged by
 * points take 920 from the planes and 850 from an array with four per point
 * (4096^2). */
template <class Op, bool KX, bool KY>
__global__ void __launch_bounds__(32 * kGalRows) k_galerkin_tile(Op op, int fm, int fn, int px, int py, int cm, int cn,
                                                       double *st, const double *Q) {
    // The coarsening flags are template parameters: with them every loop
    // below has fixed bounds and every offset of a support point or stencil
    // neighbour relative to the coarse point is a constant, so the nine sums
    // stay in registers (indexed at run time they would live in local memory).
    extern __shared__ __align__(16) double gal_smem[];
    constexpr int CTW = 32, CTH = kGalRows;
    constexpr bool kx = KX, ky = KY;
    const int X0 = blockIdx.x * CTW, Y0 = blockIdx.y * CTH;
    const int SX0 = kx ? 2 * X0 - 1 : X0, SY0 = ky ? 2 * Y0 - 1 : Y0;
    constexpr int SW = kx ? 2 * CTW + 1 : CTW, SH = ky ? 2 * CTH + 1 : CTH, SA = SW * SH;
    constexpr int NW = SW + 2, NH = SH + 2;
    double *Ps = gal_smem;             // weights of region point t at Ps[4 * t .. 4 * t + 3]
    double *As = Ps + 4 * (NW * NH);  // entry k of support point t at As[k * SA + t]
    // Only the supports of coarse points I < cm, J < cn (fine x up to sxmax)
    // and their stencil neighbours (one further) are read below. Beyond them
    // the region of a level smaller than the tile would reach more than one
    // period past a periodic grid, where one wrap does not bring an index
    // back inside it: such points are not staged.
    const int sxmax = kx ? 2 * cm - 1 : cm - 1, symax = ky ? 2 * cn - 1 : cn - 1;
    // The weights by cells (the region starts on one; a periodic direction has
    // whole ones): all of a cell's planes are loaded together.
    constexpr int CW = KX ? (NW + 1) / 2 : NW, CH = KY ? (NH + 1) / 2 : NH;
    const int cx = cells_of(fm, kx), cy = cells_of(fn, ky);
    const long NC = static_cast<long>(cx) * cy;
    for (int t = threadIdx.x; t < CW * CH; t += blockDim.x) {
        const int a = t % CW, b = t / CW, Iu = X0 - 1 + a, Ju = Y0 - 1 + b;
        bool ok = (kx ? 2 * Iu : Iu) <= sxmax + 1 && (ky ? 2 * Ju : Ju) <= symax + 1;
        const int I = wrap_idx(Iu, cx, px, ok), J = wrap_idx(Ju, cy, py, ok);
        constexpr int kPlanes = KX && KY ? 8 : 2;
        double w[kPlanes];
        const double *q = Q + I + static_cast<long>(cx) * J;
#pragma unroll
        for (int e = 0; e < kPlanes; e++) w[e] = ok ? q[e * NC] : 0.0;
        auto put = [&](int u, int v, double w0, double w1, double w2, double w3) {
            const int x = kx ? 2 * a + u : a, y = ky ? 2 * b + v : b;
            if (x >= NW || y >= NH) return;
            double2 *p = reinterpret_cast<double2 *>(Ps + 4 * (x + NW * y));
            p[0] = make_double2(w0, w1);
            p[1] = make_double2(w2, w3);
        };
        put(0, 0, ok ? 1.0 : 0.0, 0, 0, 0);
        if constexpr (KX && KY) {
            put(1, 0, w[0], w[1], 0, 0);
            put(0, 1, w[2], 0, w[3], 0);
            put(1, 1, w[4], w[5], w[6], w[7]);
        } else if constexpr (KX) {
            put(1, 0, w[0], w[1], 0, 0);
        } else {
            put(0, 1, w[0], 0, w[1], 0);
        }
    }
    for (int t = threadIdx.x; t < SA; t += blockDim.x) {
        const int xu = SX0 + t % SW, yu = SY0 + t / SW;
        bool ok = xu <= sxmax && yu <= symax;
        const int i = wrap_idx(xu, fm, px, ok), j = wrap_idx(yu, fn, py, ok);
        // outside the grid (weight zero) or no support of the tile: zero
        double a[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
        if (ok) op.coef9(i, j, a);
#pragma unroll
        for (int k = 0; k < 9; k++) As[k * SA + t] = a[k];
    }
    __syncthreads();
    const int I = X0 + (threadIdx.x & 31), J = Y0 + (threadIdx.x >> 5);
    if (I >= cm || J >= cn) return;
    double q[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    // Support points fi = 2I-1+u (u = 0..2) in a coarsened direction, fi = I
    // otherwise; visited in the order of k_galerkin (rows, then columns).
    // Which of a point's weights can differ from zero is known from its
    // parities (a point on a coarse point has the single weight 1), so the sums
    // run without a branch; a weight or entry that is zero all the same adds
    // zero.
    const double *ac = As + (kx ? 2 : 1) * (threadIdx.x & 31) + SW * (ky ? 2 : 1) * (threadIdx.x >> 5);
    const double *pc = Ps + 4 * (1 + (kx ? 2 : 1) * (threadIdx.x & 31) + NW * (1 + (ky ? 2 : 1) * (threadIdx.x >> 5)));
#pragma unroll
    for (int v = 0; v <= (ky ? 2 : 0); v++)
#pragma unroll
        for (int u = 0; u <= (kx ? 2 : 0); u++) {
            // this support point's weight for the coarse point
            const int qx = kx && u == 0, qy = ky && v == 0;
            const bool on_x = !kx || u == 1, on_y = !ky || v == 1;  // on the coarse point's column / row
            const double w = on_x && on_y ? 1.0 : pc[4 * (u + NW * v) + qx + 2 * qy];
#pragma unroll
            for (int dj = -1; dj <= 1; dj++)
#pragma unroll
                for (int di = -1; di <= 1; di++) {
                    if (Op::kFivePoint && di != 0 && dj != 0) continue;
                    const double wa = __dmul_rn(w, ac[(3 * (dj + 1) + di + 1) * SA + u + SW * v]);
                    const double *g = pc + 4 * (u + di + NW * (v + dj));
                    const int ox = kx ? ((u - 1 + di) >> 1) : di, oy = ky ? ((v - 1 + dj) >> 1) : dj;
                    const bool gx = kx && ((u - 1 + di) & 1), gy = ky && ((v - 1 + dj) & 1);  // between coarse columns / rows
#pragma unroll
                    for (int r = 0; r < 4; r++) {
                        const int kx_ = ox + (r & 1), ky_ = oy + (r >> 1);
                        if (((r & 1) && !gx) || ((r >> 1) && !gy)) continue;
                        if (kx_ < -1 || kx_ > 1 || ky_ < -1 || ky_ > 1) continue;
                        double &qe = q[3 * (ky_ + 1) + kx_ + 1];
                        // (outside a non-periodic grid the staged weight is 0)
                        qe = add_prod(qe, wa, g[r]);
                    }
                }
        }
    const long N = static_cast<long>(cm) * cn;
    const long qi = colour_index(cm, cn, I, J);
#pragma unroll
    for (int e = 0; e < 9; e++) st[e * N + qi] = q[e];
}

/** The shared-memory limit of every k_galerkin_tile instance of Op. */
template <class Op>
cudaError_t set_galerkin_attr(int bytes) {
    cudaError_t e = cudaFuncSetAttribute(k_galerkin_tile<Op, true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         bytes);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_galerkin_tile<Op, true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_galerkin_tile<Op, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    return e;
}

/** Shared memory of k_galerkin_tile for the coarsening flags. */
inline size_t galerkin_tile_smem(bool kx, bool ky) {
    const int SW = kx ? 65 : 32, SH = ky ? 2 * kGalRows + 1 : kGalRows;
    return sizeof(double) * (9 * SW * SH + 4 * (SW + 2) * (SH + 2));
}

/** One array to round to single precision: a level's Galerkin stencils (entry
 * k of unknown q at k*N+q) or the weight planes of a transfer, by `blocks`
 * blocks from `first` on. */
struct CastJob {
    const double *src;
    float *dst;
    long N;
    int stencil, first, blocks;
};
constexpr int kCastJobs = 32;
struct CastPlan {
    int count;
    CastJob job[kCastJobs];
};

/** Single-precision copies for the centred FP32 cycles, all levels in one
 * launch. Entry 4 of a stencil holds the row sum of the FP64 entries, summed in
 * FP64, instead of the diagonal. Bound by memory: a point's nine loads go out
 * together (a store between them kept each waiting for the last). The two
 * systems of a 2048^2 flag: 182 us each in eleven launches for the stencils alone,
 * 79 us now with the planes; 1024^2, sixteen launches of 3.6 us before. */
__global__ void __launch_bounds__(256) k_cast_levels(const __grid_constant__ CastPlan p) {
    int l = 0;
    while (l + 1 < p.count && static_cast<int>(blockIdx.x) >= p.job[l + 1].first) l++;
    const double *__restrict__ src = p.job[l].src;
    float *__restrict__ dst = p.job[l].dst;
    const long N = p.job[l].N, step = p.job[l].blocks * 256L;
    const long q0 = (blockIdx.x - p.job[l].first) * 256L + threadIdx.x;
    if (p.job[l].stencil) {
        for (long q = q0; q < N; q += step) {
            double v[9], rs = 0;
#pragma unroll
            for (int k = 0; k < 9; k++) v[k] = src[k * N + q];
#pragma unroll
            for (int k = 0; k < 9; k++) rs += v[k];
#pragma unroll
            for (int k = 0; k < 9; k++) dst[k * N + q] = static_cast<float>(k == 4 ? rs : v[k]);
        }
    } else {
#pragma unroll 4
        for (long q = q0; q < N; q += step) dst[q] = static_cast<float>(src[q]);
    }
}

// ---------------------------------------------------------------------------
// V-cycle kernels.

// On a periodic level of odd size the first and last columns (rows) have one
// colour and are neighbours across the seam. Updated in place by unrelated
// threads each would see the other's value from before or after at random, so
// the points of such pairs are updated by one block, which computes all its
// values before it writes any: every point of a colour sees the values from
// before the phase, as in the tail. The other points run beside them.

constexpr int kSeamUnits = 128;  // pairs of a block of 256 threads

/** Whether colour (pi,pj) meets itself across the x seam and the y seam. */
struct Seam {
    bool x, y;
    __host__ __device__ Seam(int m, int n, int px, int py, int pi, int pj)
        : x(px && (m & 1) && pi == 0), y(py && (n & 1) && pj == 0) {}
    /** Pairs: those of the y seam, then those of the x seam in the rows between. */
    __host__ __device__ int units(int m, int n, int pi, int pj) const {
        return (y ? (m - pi + 1) / 2 : 0) + (x ? (n - pj + 1) / 2 - (y ? 2 : 0) : 0);
    }
    __device__ bool on(int m, int n, int i, int j) const { return (x && (i == 0 || i == m - 1)) || (y && (j == 0 || j == n - 1)); }
};

/** The pairs from number t0 on, by a block of 2 kSeamUnits threads. The four
 * corners of a level odd in both directions are all neighbours: pairs 0 and 1. */
template <class Op, class T>
__device__ void seam_update(const Op &op, const Seam &e, T *z, const T *b, int pi, int pj, int t0) {
    const int m = op.m, n = op.n, q = threadIdx.x + blockDim.x * threadIdx.y;
    const int t = t0 + q % kSeamUnits, ny = e.y ? (m - pi + 1) / 2 : 0;
    const bool far = q >= kSeamUnits, in = t < e.units(m, n, pi, pj);
    int i, j;
    if (t < ny) {
        i = !e.x ? 2 * t + pi : (t == 0 ? 0 : (t == 1 ? m - 1 : 2 * (t - 1)));
        j = far ? n - 1 : 0;
    } else {
        i = far ? m - 1 : 0;
        j = 2 * (t - ny + (e.y ? 1 : 0)) + pj;
    }
    T v = 0;
    if (in) v = gs_update(op, i, j, z, b[i + m * j]);
    __syncthreads();
    if (in) z[i + m * j] = v;
}

/** One colour (pi,pj) of a Gauss-Seidel sweep: z = (b - offdiag)/diag. Rows of
 * blocks beyond the grid update the pairs across the seams. */
template <class Op, class T>
__global__ void k_smooth(Op op, T *z, const T *b, int m, int n, int pi, int pj) {
    const Seam e(m, n, op.px, op.py, pi, pj);
    const int rows = (n - pj + 2 * blockDim.y - 1) / (2 * blockDim.y);
    if (static_cast<int>(blockIdx.y) >= rows) {
        seam_update(op, e, z, b, pi, pj, kSeamUnits * ((blockIdx.y - rows) * gridDim.x + blockIdx.x));
        return;
    }
    const int i = 2 * (blockIdx.x * blockDim.x + threadIdx.x) + pi;
    const int j = 2 * (blockIdx.y * blockDim.y + threadIdx.y) + pj;
    if (i >= m || j >= n || e.on(m, n, i, j)) return;
    const int ij = i + m * j;
    z[ij] = gs_update(op, i, j, z, b[ij]);
}

/** Coarse right-hand side b_c = P^T (b - A z), the fine residual formed on
 * the fly. */
template <class Op, class T>
__global__ void k_restrict(Op op, const T *z, const T *b, int fm, int fn, int px, int py,
                           bool kx, bool ky, int cm, int cn, T *bc, const double *Q) {
    const int I = blockIdx.x * blockDim.x + threadIdx.x, J = blockIdx.y * blockDim.y + threadIdx.y;
    if (I >= cm || J >= cn) return;
    const int x0 = kx ? 2 * I - 1 : I, x1 = kx ? 2 * I + 1 : I, y0 = ky ? 2 * J - 1 : J, y1 = ky ? 2 * J + 1 : J;
    T t = 0;
    for (int fj = y0; fj <= y1; fj++)
        for (int fi = x0; fi <= x1; fi++) {
            const T w = static_cast<T>(pweight(Q, fm, fn, px, py, kx, ky, fi, fj, I, J));
            if (w == 0) continue;
            bool ok = true;
            const int i = wrap_idx(fi, fm, px, ok), j = wrap_idx(fj, fn, py, ok);
            const int f = i + fm * j;
            t = add_prod(t, w, residual_at(op, i, j, z, b[f]));
        }
    bc[I + cm * J] = t;
}

/** Coarsest-level solve: `sweeps` four-colour Gauss-Seidel sweeps by one
 * block of 256 threads, with a block barrier between colours. */
template <class Op, class T>
__global__ void k_coarse(Op op, T *z, const T *b, int m, int n, int sweeps) {
    const int pis[4] = {0, 1, 1, 0}, pjs[4] = {0, 1, 0, 1};
    for (int s = 0; s < sweeps; s++) {
        for (int c = 0; c < 4; c++) {
            const int mc = (m - pis[c] + 1) / 2, nc = (n - pjs[c] + 1) / 2;
            const Seam e(m, n, op.px, op.py, pis[c], pjs[c]);
            for (int p = threadIdx.x; p < mc * nc; p += blockDim.x) {
                const int i = 2 * (p % mc) + pis[c], j = 2 * (p / mc) + pjs[c];
                if (!e.on(m, n, i, j)) z[i + m * j] = gs_update(op, i, j, z, b[i + m * j]);
            }
            for (int t = 0; t < e.units(m, n, pis[c], pjs[c]); t += kSeamUnits) seam_update(op, e, z, b, pis[c], pjs[c], t);
            __syncthreads();
        }
    }
}

/** Coarse levels with at most this many unknowns are solved exactly. */
constexpr int kDirectMax = 96;

/** Dense inverse of the coarsest Galerkin operator, one block, Gauss-Jordan
 * with partial pivoting on [A | I] in shared memory. The singular
 * pure-Neumann operator (zero row sums) is regularised by c e e^T, c the
 * mean |diagonal| / N, which gives the zero-mean solution of a compatible
 * system. Writes the FP64 inverse and an FP32 copy. */
__global__ void k_coarse_inverse(const double *st, int m, int n, int px, int py, double *ginv, float *ginvf) {
    extern __shared__ __align__(16) double gj[];
    const int N = m * n, W = 2 * N;
    double *a = gj, *f = gj + static_cast<long>(N) * W;
    __shared__ double red[32];
    __shared__ int piv;
    __shared__ bool singular;
    __shared__ double creg;
    for (int q = threadIdx.x; q < N * W; q += blockDim.x) a[q] = 0;
    __syncthreads();
    double rsmax = 0, dsum = 0;
    for (int r = threadIdx.x; r < N; r += blockDim.x) {
        const int i = r % m, j = r / m;
        double rs = 0;
        for (int dj = -1; dj <= 1; dj++) {
            bool oky = true;
            const int jj = wrap_idx(j + dj, n, py, oky);
            if (!oky) continue;
            for (int di = -1; di <= 1; di++) {
                bool okx = true;
                const int ii = wrap_idx(i + di, m, px, okx);
                if (!okx) continue;
                const double v = st[(3 * (dj + 1) + di + 1) * static_cast<long>(N) + colour_index(m, n, i, j)];
                a[static_cast<long>(r) * W + ii + m * jj] += v;
                rs += v;
            }
        }
        rsmax = fmax(rsmax, fabs(rs));
        dsum += fabs(st[4 * static_cast<long>(N) + colour_index(m, n, i, j)]);
        a[static_cast<long>(r) * W + N + r] = 1;
    }
    // block max / sum (1024 threads = 32 warps)
    for (int o = 16; o > 0; o >>= 1) {
        rsmax = fmax(rsmax, __shfl_down_sync(0xffffffffu, rsmax, o));
        dsum += __shfl_down_sync(0xffffffffu, dsum, o);
    }
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    if (lane == 0) red[wp] = rsmax;
    __syncthreads();
    if (threadIdx.x == 0) {
        double mx = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) mx = fmax(mx, red[w]);
        creg = mx;
    }
    __syncthreads();
    if (lane == 0) red[wp] = dsum;
    __syncthreads();
    if (threadIdx.x == 0) {
        double sm = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) sm += red[w];
        singular = creg <= 1e-10 * sm / N;
        creg = sm / N / N;
    }
    __syncthreads();
    if (singular)
        for (int q = threadIdx.x; q < N * N; q += blockDim.x) a[static_cast<long>(q / N) * W + q % N] += creg;
    __syncthreads();
    for (int k = 0; k < N; k++) {
        if (threadIdx.x < 32) {
            // warp argmax of |a(r,k)|, r >= k; ties go to the lower row
            int p = -1;
            double best = -1;
            for (int r = k + threadIdx.x; r < N; r += 32) {
                const double v = fabs(a[static_cast<long>(r) * W + k]);
                if (v > best) { best = v; p = r; }
            }
            for (int o = 16; o > 0; o >>= 1) {
                const double ob = __shfl_down_sync(0xffffffffu, best, o);
                const int op_ = __shfl_down_sync(0xffffffffu, p, o);
                if (ob > best || (ob == best && op_ >= 0 && (p < 0 || op_ < p))) { best = ob; p = op_; }
            }
            // no candidate compares (a NaN column): keep row k, so the
            // inverse comes out NaN and the solve reports it, and no row
            // outside the matrix is touched
            if (threadIdx.x == 0) piv = p < 0 ? k : p;
        }
        __syncthreads();
        const int p = piv;
        if (p != k)
            for (int q = threadIdx.x; q < W; q += blockDim.x) {
                const double t = a[static_cast<long>(k) * W + q];
                a[static_cast<long>(k) * W + q] = a[static_cast<long>(p) * W + q];
                a[static_cast<long>(p) * W + q] = t;
            }
        __syncthreads();
        const double iv = 1.0 / a[static_cast<long>(k) * W + k];
        __syncthreads();
        for (int q = threadIdx.x; q < W; q += blockDim.x) a[static_cast<long>(k) * W + q] *= iv;
        for (int r = threadIdx.x; r < N; r += blockDim.x) f[r] = a[static_cast<long>(r) * W + k];
        __syncthreads();
        for (long q = threadIdx.x; q < static_cast<long>(N) * W; q += blockDim.x) {
            const int r = static_cast<int>(q / W);
            if (r == k || f[r] == 0) continue;
            a[q] -= f[r] * a[static_cast<long>(k) * W + q % W];
        }
        __syncthreads();
    }
    for (int q = threadIdx.x; q < N * N; q += blockDim.x) {
        const double v = a[static_cast<long>(q / N) * W + N + q % N];
        ginv[q] = v;
        ginvf[q] = static_cast<float>(v);
    }
}

/** The total of the blocks' sums acc (256 threads each), in the order of the
 * blocks whichever finishes last: that one adds the partials up, so the sum
 * needs no launch of its own. True in its first thread, with the total in acc.
 * *ticket is zero before and after. */
__device__ __forceinline__ bool grid_sum_256(double &acc, double *partial, unsigned *ticket) {
    __shared__ bool last;
    acc = block_sum_256(acc);
    if (threadIdx.x == 0) {
        partial[blockIdx.x] = acc;
        __threadfence();
        last = atomicInc(ticket, gridDim.x - 1) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return false;
    __threadfence();
    acc = 0;
    for (int q = threadIdx.x; q < gridDim.x; q += 256) acc += __ldcg(partial + q);
    acc = block_sum_256(acc);
    return threadIdx.x == 0;
}

/** What the residual at a point reads; load() takes everything without a
 * branch, so that the loads of several points are in flight together. */
template <class Op>
struct ResPoint;
template <>
struct ResPoint<MacOp<double>> {
    double off, diag, zc, b;
    __device__ __forceinline__ void load(const MacOp<double> &op, const double *__restrict__ z, const double *__restrict__ rhs, int i,
                                         int j) {
        const int q = i + op.m * j;
        off = op.offdiag(i, j, z, diag);
        zc = z[q];
        b = rhs[q];
    }
    __device__ __forceinline__ double residual(const MacOp<double> &, int, int) const { return fma_rn(-diag, zc, sub_rn(b, off)); }
};
template <>
struct ResPoint<FemOp<double>> {
    double w[9], cdl, cdr, cul, cur, b;
    __device__ __forceinline__ void load(const FemOp<double> &op, const double *__restrict__ z, const double *__restrict__ rhs, int i,
                                         int j) {
        const int m = op.m, n = op.n, q = i + m * j;
        const int il = i > 0 ? -1 : m - 1, ir = i < m - 1 ? 1 : 1 - m;
        const int jd = j > 0 ? -m : m * (n - 1), ju = j < n - 1 ? m : -m * (n - 1);
        const double *v = z + q;
        w[0] = v[jd + il]; w[1] = v[jd]; w[2] = v[jd + ir];
        w[3] = v[il];      w[4] = v[0];  w[5] = v[ir];
        w[6] = v[ju + il]; w[7] = v[ju]; w[8] = v[ju + ir];
        op.cells(i, j, cdl, cdr, cul, cur);
        b = rhs[q];
    }
    __device__ __forceinline__ double residual(const FemOp<double> &op, int i, int j) const {
        double diag, off;
        if (i > 0 && i < op.m - 1 && j > 0 && j < op.n - 1) off = op.offdiag_int(cdl, cdr, cul, cur, w, 4, 3, diag);
        else off = op.offdiag_cells(i, j, cdl, cdr, cul, cur, w, 4, 3, diag);
        return fma_rn(-diag, w[4], sub_rn(b, off));
    }
};

/** FP64 residual r = b - A z, optionally stored in FP32, and the sum of r^2 in
 * the host's host[0]. Each block takes every gridDim.x-th row, its threads the
 * row's unknowns (coalesced, no index division). Bound by memory once the loads
 * of a point, or of two five-point ones, are in flight together: 4096^2 MAC 144
 * -> 101 us (four points 107), FEM 140 -> 108 (two points spill: 187), of 82 and
 * 61 us for the bytes. The total and its way to the host are this launch's too
 * (small grids: 2.1 us, 1.9 for the sum and 3.3 for the copy before, 4.5 now).
 * Solves: MAC 64^2 603 -> 547 us, FEM 193 x 144 1688 -> 1531. A loop inside the
 * graph, left by this kernel, took as long as a graph launch per cycle (MAC 64^2
 * on the device 411 us and 410) and 0.05 ms more on a solve's first buffers. */
template <class Op>
__global__ void __launch_bounds__(256, 4) k_resnorm(Op op, const double *__restrict__ z, const double *__restrict__ b, int m, int n,
                                                    float *__restrict__ rf, double *partial, unsigned *ticket, double *host) {
    constexpr int U = Op::kFivePoint ? 2 : 1;
    double acc = 0;
    for (int j = blockIdx.x; j < n; j += gridDim.x)
        for (int i = threadIdx.x; i < m; i += U * 256) {
            ResPoint<Op> p[U];
#pragma unroll
            for (int u = 0; u < U; u++) p[u].load(op, z, b, min(i + 256 * u, m - 1), j);
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int k = i + 256 * u;
                if (k < m) {
                    const double r = p[u].residual(op, k, j);
                    if (rf) rf[k + static_cast<long>(m) * j] = static_cast<float>(r);
                    acc += r * r;
                }
            }
        }
    if (grid_sum_256(acc, partial, ticket)) *host = acc;
}

/** out = A z. */
template <class Op>
__global__ void k_apply(Op op, const double *z, double *out, int m, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= m || j >= n) return;
    double diag;
    const double off = op.offdiag(i, j, z, diag);
    out[i + m * j] = fma_rn(diag, z[i + m * j], off);
}

__global__ void k_sumsq(const double *b, long N, double *partial) {
    double acc = 0;
    for (long q = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; q < N;
         q += static_cast<long>(gridDim.x) * blockDim.x)
        acc += b[q] * b[q];
    acc = block_sum_256(acc);
    if (threadIdx.x == 0) partial[blockIdx.x] = acc;
}

/** Sums nb partials in a fixed order (one block), so results are reproducible. */
__global__ void k_reduce(const double *partial, int nb, double *out) {
    double acc = 0;
    for (int q = threadIdx.x; q < nb; q += blockDim.x) acc += partial[q];
    acc = block_sum_256(acc);
    if (threadIdx.x == 0) *out = acc;
}

/** Sum of an FP32 array, accumulated in FP64. */
__global__ void k_sum_f32(const float *a, long N, double *partial, unsigned *ticket, double *out) {
    double acc = 0;
    for (long q = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; q < N;
         q += static_cast<long>(gridDim.x) * blockDim.x)
        acc += static_cast<double>(a[q]);
    if (grid_sum_256(acc, partial, ticket)) *out = acc;
}

/** z += e - mean(e), the mean from the sum in *sum (a correction of a
 * singular system, defined up to a constant). */
__global__ void k_add_f32_centred(double *z, const float *e, long N, const double *sum) {
    const double mean = *sum / static_cast<double>(N);
    for (long q = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; q < N;
         q += static_cast<long>(gridDim.x) * blockDim.x)
        z[q] += static_cast<double>(e[q]) - mean;
}

__global__ void k_add_f32(double *z, const float *e, long N) {
    for (long q = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; q < N;
         q += static_cast<long>(gridDim.x) * blockDim.x)
        z[q] += static_cast<double>(e[q]);
}

template <class T>
__global__ void k_fill(T *a, long N, T v) {
    for (long q = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; q < N;
         q += static_cast<long>(gridDim.x) * blockDim.x)
        a[q] = v;
}

/** Zeroes the right-hand side on the fixed right column (mgs_fem.cc:112). */
__global__ void k_zero_column(double *b, int m, int n) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j < n) b[m - 1 + m * j] = 0;
}

// ---------------------------------------------------------------------------
// Flexible conjugate gradients (FCG(1), Notay, SIAM J. Sci. Comput. 22 (2000)
// 1444-1460) with one V-cycle as the preconditioner e = M r:
//   p_k = e_k - (e_k . q_{k-1} / p_{k-1} . q_{k-1}) p_{k-1},  q_k = A p_k,
//   alpha_k = p_k . r_k / p_k . q_k,  z += alpha_k p_k,  r -= alpha_k q_k.
// The explicit orthogonalisation against the previous direction keeps the
// iteration convergent although the V-cycle (the same colour order before and
// after the coarse correction, FP32 in mixed precision) is not a symmetric
// linear operator. The scalars live on the device (ks), so an iteration needs
// no host round trip besides the residual norm. For the singular systems (no
// zero-pressure edge) e is made mean-free, so every direction, and the
// iterate's mean, stay in the range of A.

/** Per-block sums of e, e.q and q (part[b], part[nb + b], part[2 nb + b]). */
template <class Te>
__global__ void k_cg_dots(const Te *e, const double *q, long N, double *part) {
    double s0 = 0, s1 = 0, s2 = 0;
    for (long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; i < N;
         i += static_cast<long>(gridDim.x) * blockDim.x) {
        const double ev = static_cast<double>(e[i]), qv = q[i];
        s0 += ev;
        s1 += ev * qv;
        s2 += qv;
    }
    s0 = block_sum_256(s0);
    s1 = block_sum_256(s1);
    s2 = block_sum_256(s2);
    if (threadIdx.x == 0) {
        part[blockIdx.x] = s0;
        part[gridDim.x + blockIdx.x] = s1;
        part[2 * gridDim.x + blockIdx.x] = s2;
    }
}

/** out[k] = sum of part[k nb .. k nb + nb - 1] for k < K, in a fixed order. */
template <int K>
__global__ void k_reduce_n(const double *part, int nb, double *out) {
#pragma unroll 1
    for (int k = 0; k < K; k++) {
        double acc = 0;
        for (int q = threadIdx.x; q < nb; q += blockDim.x) acc += part[k * nb + q];
        acc = block_sum_256(acc);
        if (threadIdx.x == 0) out[k] = acc;
    }
}

/** The new direction p = (e - mu) - beta p, mu the mean of e on a singular
 * system (else 0), beta = (e - mu).q / p.q of the previous direction (0 for
 * the first direction, ks[3] == 0, when p is not read). */
template <class Te>
__global__ void k_cg_direction(const Te *e, double *p, long N, const double *ks, int singular) {
    const double mu = singular ? ks[0] / static_cast<double>(N) : 0.0;
    const double pq = ks[3];
    const double beta = pq != 0 ? (ks[1] - mu * ks[2]) / pq : 0.0;
    for (long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; i < N;
         i += static_cast<long>(gridDim.x) * blockDim.x) {
        const double em = static_cast<double>(e[i]) - mu;
        p[i] = beta != 0 ? em - beta * p[i] : em;
    }
}

/** q = A p with per-block sums of p.q and p.r (part[b], part[nb + b]); rows
 * strided over the blocks as in k_resnorm. */
template <class Op>
__global__ void k_cg_apply(Op op, const double *p, double *q, const double *r, int m, int n, double *part) {
    double s0 = 0, s1 = 0;
    for (int j = blockIdx.x; j < n; j += gridDim.x)
        for (int i = threadIdx.x; i < m; i += blockDim.x) {
            const long k = i + static_cast<long>(m) * j;
            double diag;
            const double off = op.offdiag(i, j, p, diag);
            const double pv = p[k], qv = fma_rn(diag, pv, off);
            q[k] = qv;
            s0 += pv * qv;
            s1 += pv * r[k];
        }
    s0 = block_sum_256(s0);
    s1 = block_sum_256(s1);
    if (threadIdx.x == 0) {
        part[blockIdx.x] = s0;
        part[gridDim.x + blockIdx.x] = s1;
    }
}

/** z += alpha p, r -= alpha q (alpha = p.r / p.q from ks[5], ks[4]), the
 * FP32 copy of r for the next mixed cycle, per-block sums of r^2. */
__global__ void k_cg_update(double *z, double *r, const double *p, const double *q, float *rf, long N,
                            const double *ks, double *part) {
    const double pq = ks[4], alpha = pq != 0 ? ks[5] / pq : 0.0;
    double acc = 0;
    for (long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; i < N;
         i += static_cast<long>(gridDim.x) * blockDim.x) {
        z[i] = fma_rn(alpha, p[i], z[i]);
        const double rn = fma_rn(-alpha, q[i], r[i]);
        r[i] = rn;
        if (rf) rf[i] = static_cast<float>(rn);
        acc += rn * rn;
    }
    acc = block_sum_256(acc);
    if (threadIdx.x == 0) part[blockIdx.x] = acc;
}

/** ||r||^2 into *norm from the update's partials; the direction's p.q
 * becomes the previous one for the next iteration. */
__global__ void k_cg_finish(const double *part, int nb, double *norm, double *ks) {
    double acc = 0;
    for (int q = threadIdx.x; q < nb; q += blockDim.x) acc += part[q];
    acc = block_sum_256(acc);
    if (threadIdx.x == 0) {
        *norm = acc;
        ks[3] = ks[4];
    }
}

/** r = b - A z in FP64 (and FP32 into rf if given), per-block sums of r^2. */
template <class Op>
__global__ void k_cg_residual(Op op, const double *z, const double *b, int m, int n, double *r, float *rf,
                              double *part) {
    double acc = 0;
    for (int j = blockIdx.x; j < n; j += gridDim.x)
        for (int i = threadIdx.x; i < m; i += blockDim.x) {
            const long k = i + static_cast<long>(m) * j;
            double diag;
            const double off = op.offdiag(i, j, z, diag);
            const double rv = fma_rn(-diag, z[k], sub_rn(b[k], off));
            r[k] = rv;
            if (rf) rf[k] = static_cast<float>(rv);
            acc += rv * rv;
        }
    acc = block_sum_256(acc);
    if (threadIdx.x == 0) part[blockIdx.x] = acc;
}

constexpr int kRedBlocks = 4 * kB200SMs;  // reduction grid: 4 x 148 blocks of 256

inline dim3 grid2(int m, int n) { return dim3(cdiv(m, 32), cdiv(n, 8)); }
const dim3 kBlk2(32, 8);

/** The attributes a launch of k_tail needs. */
template <class T, bool SEQ>
cudaError_t set_tail_attr() {
    const cudaError_t e = cudaFuncSetAttribute(k_tail<T, SEQ>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               static_cast<int>(kTailSmemBudget));
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(k_tail<T, SEQ>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
}

/** Runs `sweeps` four-colour sweeps on the iterate z. Two sweeps on a grid
 * whose periodic directions have even sizes run as one tile-fused launch that
 * reads z and writes zalt (*res = zalt); otherwise one launch per colour
 * updates z in place (*res = z). zero: the sweeps start from 0 and z need not
 * hold it (tiles then read no iterate). When prof is given, each launch is bracketed
 * by CUDA events and credited with the bytes it cannot do without: its operands
 * read and its result written once, bytes_per_unit for each unknown it updates. */
template <class Op, class T>
int smooth(Op op, T *z, T *zalt, const T *b, int m, int n, int sweeps, cudaStream_t s, long long &nl, T **res,
           bool zero = false, Multigrid *prof = nullptr, double bytes_per_unit = 0) {
    *res = z;
    if (sweeps == 2 && zalt && (!op.px || m % 2 == 0) && (!op.py || n % 2 == 0)) {
        const double words = zero ? sizeof(T) : 0;  // not read
        if (prof) { int r = prof->prof_begin(static_cast<double>(m) * n * (bytes_per_unit - words)); if (r) return r; }
        smooth_cells(op, zero ? static_cast<const T *>(nullptr) : z, zalt, b, m, n, s);
        nl++;
        if (prof) { int r = prof->prof_end(); if (r) return r; }
        INCRMT_CKL("k_smooth_cells");
        *res = zalt;
        return INCRMT_OK;
    }
    if (zero) INCRMT_CK(cudaMemsetAsync(z, 0, sizeof(T) * m * n, s));
    const int pis[4] = {0, 1, 1, 0}, pjs[4] = {0, 1, 0, 1};
    for (int q = 0; q < sweeps; q++)
        for (int c = 0; c < 4; c++) {
            const int mc = (m - pis[c] + 1) / 2, nc = (n - pjs[c] + 1) / 2;
            if (mc <= 0 || nc <= 0) continue;
            if (prof) { int r = prof->prof_begin(static_cast<double>(mc) * nc * bytes_per_unit); if (r) return r; }
            dim3 grid = grid2(mc, nc);
            grid.y += cdiv(cdiv(Seam(m, n, op.px, op.py, pis[c], pjs[c]).units(m, n, pis[c], pjs[c]), kSeamUnits), grid.x);
            k_smooth<Op, T><<<grid, kBlk2, 0, s>>>(op, z, b, m, n, pis[c], pjs[c]);
            nl++;
            if (prof) { int r = prof->prof_end(); if (r) return r; }
        }
    INCRMT_CKL("k_smooth");
    return INCRMT_OK;
}

/** Coarse right-hand side: the restriction by
 * cells, or k_restrict when tiles are off (the identity check of
 * incrmt_mg_set_tiles covers both). */
template <class Op, class T>
void restrict_launch(bool tiles, Op op, cudaStream_t s, const T *z, const T *b, int px, int py, const MgLevel &L,
                     const MgLevel &C, T *bc, const T *Q) {
    const int fm = L.m, fn = L.n, cm = C.m, cn = C.n;
    if (!tiles) {
        k_restrict<<<grid2(cm, cn), kBlk2, 0, s>>>(op, z, b, fm, fn, px, py, L.kx, L.ky, cm, cn, bc, L.Q);
        return;
    }
    const dim3 g(cdiv(cm, L.kx ? kRX - 1 : kRX), cdiv(cn, L.ky ? kRY - 1 : kRY)), t(kRX, kRY);
    if (L.kx && L.ky) k_restrict_cells<Op, T, true, true><<<g, t, 0, s>>>(op, z, b, fm, fn, px, py, cm, cn, bc, Q);
    else if (L.kx) k_restrict_cells<Op, T, true, false><<<g, t, 0, s>>>(op, z, b, fm, fn, px, py, cm, cn, bc, Q);
    else k_restrict_cells<Op, T, false, true><<<g, t, 0, s>>>(op, z, b, fm, fn, px, py, cm, cn, bc, Q);
}

/** z += P z_c. */
template <class T>
void prolong_launch(cudaStream_t s, T *z, int px, int py, const MgLevel &L, const MgLevel &C, const T *zc, const T *Q) {
    const dim3 g = grid2(cells_of(L.m, L.kx), cells_of(L.n, L.ky));
    const bool vec = L.m % 2 == 0 && reinterpret_cast<uintptr_t>(z) % (2 * sizeof(T)) == 0;
    if (L.kx && L.ky) k_prolong_cells<T, true, true><<<g, kBlk2, 0, s>>>(z, L.m, L.n, px, py, zc, C.m, C.n, Q, vec);
    else if (L.kx) k_prolong_cells<T, true, false><<<g, kBlk2, 0, s>>>(z, L.m, L.n, px, py, zc, C.m, C.n, Q, vec);
    else k_prolong_cells<T, false, true><<<g, kBlk2, 0, s>>>(z, L.m, L.n, px, py, zc, C.m, C.n, Q, vec);
}

}  // namespace

MacOp<double> Multigrid::mac64() const {
    MacOp<double> o; o.m = m; o.n = n; o.px = px; o.py = py; o.zpr = zpr;
    o.xxsp = xxsp; o.yysp = yysp; o.ex = ex; o.ey = ey; return o;
}
MacOp<float> Multigrid::mac32() const {
    MacOp<float> o; o.m = m; o.n = n; o.px = px; o.py = py; o.zpr = zpr;
    o.xxsp = static_cast<float>(xxsp); o.yysp = static_cast<float>(yysp); o.ex = exf; o.ey = eyf; return o;
}
FemOp<double> Multigrid::fem64() const {
    FemOp<double> o; o.m = m; o.n = n; o.px = px; o.py = py; o.zpr = zpr;
    o.fm = fm; o.fc = fc; o.hex = hex; o.hey = hey; o.c = c; return o;
}
FemOp<float> Multigrid::fem32() const {
    FemOp<float> o; o.m = m; o.n = n; o.px = px; o.py = py; o.zpr = zpr;
    o.fm = static_cast<float>(fm); o.fc = static_cast<float>(fc);
    o.hex = static_cast<float>(hex); o.hey = static_cast<float>(hey); o.c = cf; return o;
}

int Multigrid::create(int sys_, int cm_, int cn_, double ax, double bx, double ay, double by,
                      int px_, int py_, int zpr_, cudaStream_t ext) {
    if (sys_ != INCRMT_SYS_MAC && sys_ != INCRMT_SYS_FEM) { set_error("unknown system %d", sys_); return INCRMT_ERR_BADARG; }
    if (cm_ < 2 || cn_ < 2 || !(bx > ax) || !(by > ay)) { set_error("bad grid %dx%d", cm_, cn_); return INCRMT_ERR_BADARG; }
    sys = sys_; cm = cm_; cn = cn_; px = px_ ? 1 : 0; py = py_ ? 1 : 0; zpr = zpr_ ? 1 : 0;
    dx = (bx - ax) / cm; dy = (by - ay) / cn;
    const double xsp = 1 / dx, ysp = 1 / dy;
    xxsp = xsp * xsp; yysp = ysp * ysp;
    if (sys == INCRMT_SYS_MAC) { m = cm; n = cn; }
    else { m = px ? cm : cm + 1; n = py ? cn : cn + 1; }
    if ((px && m % 2) || (py && n % 2)) {
        set_error("a periodic direction needs an even number of unknowns (got %dx%d)", m, n);
        return INCRMT_ERR_BADARG;
    }
    // Finite-element stencil constants (mgs_fem.cc:12-21).
    const double dydx = dy / dx, dxdy = dx / dy;
    fm = 1. / 3. * (dxdy + dydx);
    const double fey = 1. / 3. * (-2 * dxdy + dydx), fex = 1. / 3. * (-2 * dydx + dxdy);
    hey = 0.5 * fey; hex = 0.5 * fex;
    fc = -1. / 6. * (dxdy + dydx);
    if (ext) { stream = ext; own_stream = false; }
    else INCRMT_CK(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking));
    INCRMT_CK(cudaEventCreate(&ev0));
    INCRMT_CK(cudaEventCreate(&ev1));
    const long N = static_cast<long>(m) * n;
    if (sys == INCRMT_SYS_MAC) {
        INCRMT_CK(cudaMalloc(&ex, sizeof(double) * (cm + 1) * cn));
        INCRMT_CK(cudaMalloc(&ey, sizeof(double) * cm * (cn + 1)));
        INCRMT_CK(cudaMalloc(&exf, sizeof(float) * (cm + 1) * cn));
        INCRMT_CK(cudaMalloc(&eyf, sizeof(float) * cm * (cn + 1)));
    } else {
        INCRMT_CK(cudaMalloc(&c, sizeof(double) * N));
        INCRMT_CK(cudaMalloc(&cf, sizeof(float) * N));
    }
    INCRMT_CK(cudaMalloc(&rho, sizeof(double) * (cm + 4) * (cn + 4)));
    INCRMT_CK(cudaMalloc(&bbuf, sizeof(double) * N));
    INCRMT_CK(cudaMalloc(&zbuf, sizeof(double) * N));
    INCRMT_CK(cudaMalloc(&partial, sizeof(double) * kRedBlocks));
    INCRMT_CK(cudaMalloc(&dnorm, sizeof(double) * 5));
    ticket = reinterpret_cast<unsigned *>(dnorm + 4);
    INCRMT_CK(cudaMemsetAsync(ticket, 0, sizeof(unsigned), stream));
    INCRMT_CK(cudaMallocHost(&hnorm, sizeof(double) * 4));
    return build_hierarchy();
}

int Multigrid::build_hierarchy() {
    lev.clear();
    MgLevel L0; L0.m = m; L0.n = n; L0.N = static_cast<long>(m) * n;
    INCRMT_CK(cudaMalloc(&L0.zf, sizeof(float) * L0.N));
    INCRMT_CK(cudaMalloc(&L0.bf, sizeof(float) * L0.N));
    INCRMT_CK(cudaMalloc(&L0.z2, sizeof(double) * L0.N));
    INCRMT_CK(cudaMalloc(&L0.zf2, sizeof(float) * L0.N));
    lev.push_back(L0);
    int mm = m, nn = n;
    // Semi-coarsening on anisotropic grids: r is the ratio of the operator's
    // y coupling to its x coupling, (dx/dy)^2 on the fine level of both
    // systems. Point Gauss-Seidel smooths only along the strong direction, so
    // while one direction's coupling is more than twice the other's only
    // that direction is halved, which divides (or multiplies) r by 4.
    double r = yysp / xxsp;
    while (static_cast<int>(lev.size()) < kMaxLevels && mm * nn > kCoarsestSize) {
        bool kx = can_coarsen(mm, px), ky = can_coarsen(nn, py);
        if (kx && ky) {
            if (r > kSemiRatio) kx = false;
            else if (r < 1 / kSemiRatio) ky = false;
        }
        if (!kx && !ky) break;
        if (kx && !ky) r *= 4;
        else if (ky && !kx) r /= 4;
        const int mc = kx ? (px ? mm / 2 : (mm + 1) / 2) : mm, nc = ky ? (py ? nn / 2 : (nn + 1) / 2) : nn;
        lev.back().kx = kx; lev.back().ky = ky;
        MgLevel L; L.m = mc; L.n = nc; L.N = static_cast<long>(mc) * nc;
        INCRMT_CK(cudaMalloc(&L.z, sizeof(double) * L.N));
        INCRMT_CK(cudaMalloc(&L.b, sizeof(double) * L.N));
        INCRMT_CK(cudaMalloc(&L.st, sizeof(double) * 9 * L.N));
        INCRMT_CK(cudaMalloc(&L.zf, sizeof(float) * L.N));
        INCRMT_CK(cudaMalloc(&L.bf, sizeof(float) * L.N));
        INCRMT_CK(cudaMalloc(&L.stf, sizeof(float) * 9 * L.N));
        INCRMT_CK(cudaMalloc(&L.z2, sizeof(double) * L.N));
        INCRMT_CK(cudaMalloc(&L.zf2, sizeof(float) * L.N));
        lev.push_back(L);
        mm = mc; nn = nc;
    }
    // Prolongation weights of every level but the coarsest (k_build_p).
    for (size_t l = 0; l + 1 < lev.size(); l++) {
        // the planes in both precisions
        INCRMT_CK(cudaMalloc(&lev[l].Q, (sizeof(double) + sizeof(float)) * lev[l].planes()));
        lev[l].Qf = reinterpret_cast<float *>(lev[l].Q + lev[l].planes());
    }
    if (lev.size() > 1 && lev.back().N <= kDirectMax) {
        const long N = lev.back().N;
        INCRMT_CK(cudaMalloc(&ginv, sizeof(double) * N * N));
        INCRMT_CK(cudaMalloc(&ginvf, sizeof(float) * N * N));
        // The attribute is per kernel, shared by every solver: set the maximum.
        INCRMT_CK(cudaFuncSetAttribute(k_coarse_inverse, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       static_cast<int>(sizeof(double) * (2 * kDirectMax * kDirectMax + kDirectMax))));
    }
    INCRMT_CK((set_tail_attr<double, false>()));
    INCRMT_CK((set_tail_attr<double, true>()));
    INCRMT_CK((set_tail_attr<float, false>()));
    INCRMT_CK((set_tail_attr<float, true>()));
    const int gal_smem = static_cast<int>(galerkin_tile_smem(true, true));
    INCRMT_CK(set_galerkin_attr<MacOp<double>>(gal_smem));
    INCRMT_CK(set_galerkin_attr<FemOp<double>>(gal_smem));
    INCRMT_CK(set_galerkin_attr<GenOp<double>>(gal_smem));
    return choose_tail();
}

void Multigrid::destroy() {
    for (auto &L : lev) {
        cudaFree(L.z); cudaFree(L.b); cudaFree(L.st); cudaFree(L.zf); cudaFree(L.bf); cudaFree(L.stf);
        cudaFree(L.z2); cudaFree(L.zf2); cudaFree(L.Q);
    }
    lev.clear();
    cudaFree(ex); cudaFree(ey); cudaFree(exf); cudaFree(eyf); cudaFree(c); cudaFree(cf);
    cudaFree(rho); cudaFree(bbuf); cudaFree(zbuf); cudaFree(partial); cudaFree(dnorm);
    cudaFree(ginv); cudaFree(ginvf); ginv = nullptr; ginvf = nullptr;
    cudaFree(tail_pk); tail_pk = nullptr;

    if (hnorm) cudaFreeHost(hnorm);
    if (gexec) { cudaGraphExecDestroy(gexec); gexec = nullptr; }
    if (setup_exec) { cudaGraphExecDestroy(setup_exec); setup_exec = nullptr; }
    if (kexec) { cudaGraphExecDestroy(kexec); kexec = nullptr; }
    cudaFree(kr); cudaFree(kp); cudaFree(kq); cudaFree(ke); cudaFree(kpart); cudaFree(ks);
    kr = kp = kq = ke = kpart = ks = nullptr;
    for (auto e : prof_ev) cudaEventDestroy(e);
    prof_ev.clear();
    if (ev0) cudaEventDestroy(ev0);
    if (ev1) cudaEventDestroy(ev1);
    if (stream && own_stream) cudaStreamDestroy(stream);
    stream = nullptr;
}

int Multigrid::set_density_device(const double *d_rho, int ld) {
    if (ld <= 0) ld = cm + 4;
    if (sys == INCRMT_SYS_MAC) {
        k_mac_coef<<<grid2(cm + 1, cn + 1), kBlk2, 0, stream>>>(d_rho, ld, cm, cn, ex, ey, exf, eyf);
    } else {
        k_fem_coef<<<grid2(m, n), kBlk2, 0, stream>>>(d_rho, ld, m, n, c, cf);
    }
    launches++;
    INCRMT_CKL("coefficients");
    int r = galerkin_graph();
    if (r == INCRMT_OK) ready = true;
    coarse_builds++;
    coarse_age = 0;
    coarse_vc0 = -1;
    coarse_stale = false;
    return r;
}

int Multigrid::set_density_lagged(const double *d_rho, int ld) {
    lag_rho = d_rho;
    lag_ld = ld;
    if (!ready || coarse_stale || coarse_every <= 1 || coarse_age + 1 >= coarse_every)
        return set_density_device(d_rho, ld);
    if (ld <= 0) ld = cm + 4;
    if (sys == INCRMT_SYS_MAC) {
        k_mac_coef<<<grid2(cm + 1, cn + 1), kBlk2, 0, stream>>>(d_rho, ld, cm, cn, ex, ey, exf, eyf);
    } else {
        k_fem_coef<<<grid2(m, n), kBlk2, 0, stream>>>(d_rho, ld, m, n, c, cf);
    }
    launches++;
    INCRMT_CKL("coefficients");
    coarse_age++;
    return INCRMT_OK;
}

void Multigrid::note_vcycles(int vc) {
    if (coarse_vc0 < 0) coarse_vc0 = vc;
    else if (vc > coarse_vc0 + 1) coarse_stale = true;
}

int Multigrid::solve_lagged(const double *d_b, double *d_z, const incrmt_mg_opts *o, incrmt_mg_stats *st,
                            bool time_it) {
    incrmt_mg_stats s1{};
    int r = solve_device(d_b, d_z, o, &s1, time_it);
    if (r == INCRMT_OK) {
        note_vcycles(s1.vcycles);
        if (st) *st = s1;
        return r;
    }
    coarse_stale = true;
    if ((r == INCRMT_ERR_NOCONV || r == INCRMT_ERR_NONFINITE) && coarse_age > 0 && lag_rho) {
        if (r == INCRMT_ERR_NONFINITE)
            INCRMT_CK(cudaMemsetAsync(d_z, 0, sizeof(double) * static_cast<size_t>(m) * n, stream));
        int rr = set_density_device(lag_rho, lag_ld);
        if (rr) return rr;
        coarse_retries++;
        incrmt_mg_stats s2{};
        r = solve_device(d_b, d_z, o, &s2, time_it);
        s1.vcycles += s2.vcycles;
        s1.rel_res = s2.rel_res;
        s1.device_ms += s2.device_ms;
        if (r == INCRMT_OK) note_vcycles(s2.vcycles);
        else coarse_stale = true;
    }
    if (st) *st = s1;
    return r;
}

int Multigrid::set_unit_density() {
    const long N = static_cast<long>(cm + 4) * (cn + 4);
    double *ones = nullptr;
    INCRMT_CK(cudaMalloc(&ones, sizeof(double) * N));
    k_fill<<<cdiv(N, 256) < kRedBlocks ? cdiv(N, 256) : kRedBlocks, 256, 0, stream>>>(ones, N, 1.0);
    launches++;
    int r = set_density_device(ones, cm + 4);
    cudaError_t e = cudaStreamSynchronize(stream);
    cudaFree(ones);
    if (r) return r;
    INCRMT_CK(e);
    return INCRMT_OK;
}

int Multigrid::galerkin_all() {
    for (size_t l = 1; l < lev.size(); l++) {
        MgLevel &F = lev[l - 1], &C = lev[l];
        const dim3 gc = grid2(C.m, C.n), gt(cdiv(C.m, 32), cdiv(C.n, kGalRows));
        const size_t gsm = galerkin_tile_smem(F.kx, F.ky);
        auto build = [&](auto op) {
            using OpT = decltype(op);
            const int cx = cells_of(F.m, F.kx), cy = cells_of(F.n, F.ky);
            const bool both = F.kx && F.ky;
            const dim3 gb(cdiv(cx, both ? kPX - 1 : kPX), cdiv(cy, both ? kPY - 1 : kPY)), tb(kPX, kPY);
            if (both) k_build_p<OpT, true, true><<<gb, tb, 0, stream>>>(op, F.m, F.n, px, py, C.m, C.n, F.Q);
            else if (F.kx) k_build_p<OpT, true, false><<<gb, tb, 0, stream>>>(op, F.m, F.n, px, py, C.m, C.n, F.Q);
            else k_build_p<OpT, false, true><<<gb, tb, 0, stream>>>(op, F.m, F.n, px, py, C.m, C.n, F.Q);
            if (tiles && F.kx && F.ky)
                k_galerkin_tile<OpT, true, true><<<gt, 32 * kGalRows, gsm, stream>>>(op, F.m, F.n, px, py, C.m, C.n, C.st, F.Q);
            else if (tiles && F.kx)
                k_galerkin_tile<OpT, true, false><<<gt, 32 * kGalRows, gsm, stream>>>(op, F.m, F.n, px, py, C.m, C.n, C.st, F.Q);
            else if (tiles)
                k_galerkin_tile<OpT, false, true><<<gt, 32 * kGalRows, gsm, stream>>>(op, F.m, F.n, px, py, C.m, C.n, C.st, F.Q);
            else
                k_galerkin<<<gc, kBlk2, 0, stream>>>(op, F.m, F.n, px, py, F.kx, F.ky, C.m, C.n, C.st, F.Q);
        };
        if (l == 1 && sys == INCRMT_SYS_MAC) {
            build(mac64());
        } else if (l == 1) {
            build(fem64());
        } else {
            GenOp<double> g; g.m = F.m; g.n = F.n; g.px = px; g.py = py; g.N = F.N; g.st = F.st;
            build(g);
        }
        launches += 2;
        INCRMT_CKL("galerkin");
    }
    f32_stale = true;
    if (ginv) {
        const MgLevel &C = lev.back();
        const size_t sm = sizeof(double) * (2 * C.N * C.N + C.N);
        k_coarse_inverse<<<1, 1024, sm, stream>>>(C.st, C.m, C.n, px, py, ginv, ginvf);
        launches++;
        INCRMT_CKL("k_coarse_inverse");
    }
    return tail_pack<double>();
}

int Multigrid::galerkin_graph() {
    // The hierarchy's arrays never move, so the whole rebuild (weights,
    // Galerkin products, the coarsest inverse: dozens of launches, most on
    // small levels) is captured once and replayed; profiling runs it
    // directly.
    if (prof) return galerkin_all();
    if (!setup_exec) {
        const long long l0 = launches;
        cudaGraph_t graph = nullptr;
        INCRMT_CK(cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal));
        int rc = galerkin_all();
        cudaError_t ce = cudaStreamEndCapture(stream, &graph);
        if (rc == INCRMT_OK && ce == cudaSuccess) ce = cudaGraphInstantiate(&setup_exec, graph, 0);
        if (graph) cudaGraphDestroy(graph);
        if (rc != INCRMT_OK || ce != cudaSuccess) {
            setup_exec = nullptr;
            cudaGetLastError();
            launches = l0;
            return galerkin_all();
        }
        setup_launches = launches - l0;
        launches = l0;
    }
    INCRMT_CK(cudaGraphLaunch(setup_exec, stream));
    launches += setup_launches;
    f32_stale = true;
    return INCRMT_OK;
}

int Multigrid::cast_levels() {
    if (!f32_stale) return INCRMT_OK;
    CastPlan p{};
    int blocks = 0;
    const auto flush = [&]() {
        if (!p.count) return;
        k_cast_levels<<<blocks, 256, 0, stream>>>(p);
        launches++;
        p.count = blocks = 0;
    };
    const auto add = [&](const double *src, float *dst, long N, int stencil) {
        const int nb = cdiv(N, 256) < 2 * kRedBlocks ? cdiv(N, 256) : 2 * kRedBlocks;
        p.job[p.count++] = CastJob{src, dst, N, stencil, blocks, nb};
        blocks += nb;
        if (p.count == kCastJobs) flush();
    };
    for (size_t l = 1; l < lev.size(); l++) add(lev[l].st, lev[l].stf, lev[l].N, 1);
    for (size_t l = 0; l + 1 < lev.size(); l++) add(lev[l].Q, lev[l].Qf, lev[l].planes(), 0);
    flush();
    INCRMT_CKL("k_cast_levels");
    int r = tail_pack<float>();
    if (r) return r;
    f32_stale = false;
    return INCRMT_OK;
}

int Multigrid::cycle64(int l, const double *b0, double *z0, bool zero) {
    if (l > 0 && l == tail_level) return tail64();
    const MgLevel &L = lev[l];
    const double *b = l == 0 ? b0 : L.b;
    double *z = l == 0 ? z0 : L.z;
    GenOp<double> g; g.m = L.m; g.n = L.n; g.px = px; g.py = py; g.N = L.N; g.st = L.st;
    const bool last = l == static_cast<int>(lev.size()) - 1;
    if (last) {
        if (zero) INCRMT_CK(cudaMemsetAsync(z, 0, sizeof(double) * L.N, stream));
        if (l == 0) {
            if (sys == INCRMT_SYS_MAC) k_coarse<<<1, 256, 0, stream>>>(mac64(), z, b, L.m, L.n, kCoarseSweeps);
            else k_coarse<<<1, 256, 0, stream>>>(fem64(), z, b, L.m, L.n, kCoarseSweeps);
        } else k_coarse<<<1, 256, 0, stream>>>(g, z, b, L.m, L.n, kCoarseSweeps);
        launches++;
        INCRMT_CKL("k_coarse");
        return INCRMT_OK;
    }
    const MgLevel &C = lev[l + 1];
    int r;
    Multigrid *pf = prof ? this : nullptr;
    // Bytes per unknown of a fine FP64 smoothing launch: read z, b and the
    // coefficient words, write z (3+c words; c=2 MAC, c=1 FEM).
    const double bpu = 8.0 * (sys == INCRMT_SYS_MAC ? 5 : 4);
    // Pre-smoothing may leave the iterate in the level's second buffer; the
    // restriction, prolongation and post-smoothing follow it, and the
    // post-smoothing brings it back (both smoothings use the same kind of
    // launch, so the two moves cancel).
    double *cur = z;
    if (l == 0 && sys == INCRMT_SYS_MAC) {
        auto op = mac64();
        if ((r = smooth(op, z, tiles ? L.z2 : nullptr, b, L.m, L.n, kNu1, stream, launches, &cur, zero, pf, bpu))) return r;
        restrict_launch(tiles, op, stream, cur, b, px, py, L, C, C.b, L.Q);
    } else if (l == 0) {
        auto op = fem64();
        if ((r = smooth(op, z, tiles ? L.z2 : nullptr, b, L.m, L.n, kNu1, stream, launches, &cur, zero, pf, bpu))) return r;
        restrict_launch(tiles, op, stream, cur, b, px, py, L, C, C.b, L.Q);
    } else {
        if ((r = smooth(g, z, tiles ? L.z2 : nullptr, b, L.m, L.n, kNu1, stream, launches, &cur, zero))) return r;
        restrict_launch(tiles, g, stream, cur, b, px, py, L, C, C.b, L.Q);
    }
    launches++;
    INCRMT_CKL("k_restrict");
    if ((r = cycle64(l + 1, b0, z0, true))) return r;
    prolong_launch<double>(stream, cur, px, py, L, C, C.z, L.Q);
    launches++;
    INCRMT_CKL("k_prolong");
    double *alt = !tiles ? nullptr : cur == z ? L.z2 : z, *out = cur;
    if (l == 0 && sys == INCRMT_SYS_MAC) r = smooth(mac64(), cur, alt, b, L.m, L.n, kNu2, stream, launches, &out, false, pf, bpu);
    else if (l == 0) r = smooth(fem64(), cur, alt, b, L.m, L.n, kNu2, stream, launches, &out, false, pf, bpu);
    else r = smooth(g, cur, alt, b, L.m, L.n, kNu2, stream, launches, &out);
    if (r) return r;
    if (out != z) INCRMT_CK(cudaMemcpyAsync(z, out, sizeof(double) * L.N, cudaMemcpyDeviceToDevice, stream));
    return INCRMT_OK;
}

int Multigrid::prof_begin(double bytes) {
    constexpr int kMaxEvents = 4096;
    if (prof_used + 2 > kMaxEvents) {
        int r = prof_collect();
        if (r) return r;
    }
    while (prof_used + 2 > static_cast<int>(prof_ev.size())) {
        cudaEvent_t e;
        INCRMT_CK(cudaEventCreate(&e));
        prof_ev.push_back(e);
    }
    INCRMT_CK(cudaEventRecord(prof_ev[prof_used], stream));
    pending_bytes = bytes;
    prof_bytes += bytes;
    return INCRMT_OK;
}

int Multigrid::prof_end() {
    INCRMT_CK(cudaEventRecord(prof_ev[prof_used + 1], stream));
    prof_used += 2;
    prof_launches++;
    return INCRMT_OK;
}

/** Folds the recorded event pairs into prof_ms (synchronises the stream).
 * \return 0 (the number of pairs still pending) or an error status. */
int Multigrid::prof_collect() {
    if (prof_used == 0) return 0;
    INCRMT_CK(cudaStreamSynchronize(stream));
    for (int k = 0; k + 1 < prof_used; k += 2) {
        float ms = 0;
        INCRMT_CK(cudaEventElapsedTime(&ms, prof_ev[k], prof_ev[k + 1]));
        prof_ms += ms;
    }
    prof_used = 0;
    return 0;
}

int Multigrid::cycle32(int l) {
    if (l > 0 && l == tail_level) return tail32();
    const MgLevel &L = lev[l];
    const float *b = L.bf;
    float *z = L.zf;
    GenOp<float> g; g.m = L.m; g.n = L.n; g.px = px; g.py = py; g.N = L.N; g.st = L.stf;
    const bool last = l == static_cast<int>(lev.size()) - 1;
    if (last) {
        INCRMT_CK(cudaMemsetAsync(z, 0, sizeof(float) * L.N, stream));
        if (l == 0) {
            if (sys == INCRMT_SYS_MAC) k_coarse<<<1, 256, 0, stream>>>(mac32(), z, b, L.m, L.n, kCoarseSweeps);
            else k_coarse<<<1, 256, 0, stream>>>(fem32(), z, b, L.m, L.n, kCoarseSweeps);
        } else k_coarse<<<1, 256, 0, stream>>>(g, z, b, L.m, L.n, kCoarseSweeps);
        launches++;
        INCRMT_CKL("k_coarse");
        return INCRMT_OK;
    }
    const MgLevel &C = lev[l + 1];
    int r;
    float *cur = z;  // as in cycle64
    Multigrid *pf = prof ? this : nullptr;
    const double bpu = 4.0 * (sys == INCRMT_SYS_MAC ? 5 : 4);  // FP32 words: z, b, coefficients in; z out
    if (l == 0 && sys == INCRMT_SYS_MAC) {
        auto op = mac32();
        if ((r = smooth(op, z, tiles ? L.zf2 : nullptr, b, L.m, L.n, kNu1, stream, launches, &cur, true, pf, bpu))) return r;
        restrict_launch(tiles, op, stream, static_cast<const float *>(cur), b, px, py, L, C, C.bf, L.Qf);
    } else if (l == 0) {
        auto op = fem32();
        if ((r = smooth(op, z, tiles ? L.zf2 : nullptr, b, L.m, L.n, kNu1, stream, launches, &cur, true, pf, bpu))) return r;
        restrict_launch(tiles, op, stream, static_cast<const float *>(cur), b, px, py, L, C, C.bf, L.Qf);
    } else {
        if ((r = smooth(g, z, tiles ? L.zf2 : nullptr, b, L.m, L.n, kNu1, stream, launches, &cur, true))) return r;
        restrict_launch(tiles, g, stream, static_cast<const float *>(cur), b, px, py, L, C, C.bf, L.Qf);
    }
    launches++;
    INCRMT_CKL("k_restrict");
    if ((r = cycle32(l + 1))) return r;
    prolong_launch<float>(stream, cur, px, py, L, C, C.zf, L.Qf);
    launches++;
    INCRMT_CKL("k_prolong");
    float *alt = !tiles ? nullptr : cur == z ? L.zf2 : z, *out = cur;
    if (l == 0 && sys == INCRMT_SYS_MAC) r = smooth(mac32(), cur, alt, b, L.m, L.n, kNu2, stream, launches, &out, false, pf, bpu);
    else if (l == 0) r = smooth(fem32(), cur, alt, b, L.m, L.n, kNu2, stream, launches, &out, false, pf, bpu);
    else r = smooth(g, cur, alt, b, L.m, L.n, kNu2, stream, launches, &out);
    if (r) return r;
    if (out != z) INCRMT_CK(cudaMemcpyAsync(z, out, sizeof(float) * L.N, cudaMemcpyDeviceToDevice, stream));
    return INCRMT_OK;
}

namespace {

/** The tail's plan from level `first` down (see mg_tail.cuh), over at most
 * max_blocks blocks; false if some level does not fit. Levels of more than
 * kTailRoot cells are cut into strips over the cluster. */
template <class T>
bool tail_plan(const std::vector<MgLevel> &lev, int first, int px, int py, const T *ginv, int max_blocks,
               TailPlan<T> &p, int &blocks, int &threads, size_t &smem) {
    p = TailPlan<T>{};
    p.count = static_cast<int>(lev.size()) - first;
    if (p.count < 1 || p.count > kTailMaxLevels) return false;
    p.px = px; p.py = py; p.nu1 = kNu1; p.nu2 = kNu2; p.coarse_sweeps = kCoarseSweeps;
    p.ginv = ginv;
    for (int k = 0; k < p.count; k++) {
        const MgLevel &L = lev[first + k];
        TailLevel<T> &t = p.lev[k];
        t.m = L.m; t.n = L.n; t.cx = (L.m + 1) / 2; t.cy = (L.n + 1) / 2;
        t.kx = L.kx; t.ky = L.ky;
        if constexpr (sizeof(T) == 8) t.pk = L.pk;
        else t.pk = L.pkf;
        t.seq = px && L.m % 2 ? 2 : (py && L.n % 2 ? 1 : 0);
        t.dist = static_cast<long>(t.cx) * t.cy > kTailRoot;
        t.rows = t.cy;
        if (t.dist && (t.seq || k == p.count - 1)) return false;
        if (t.dist) p.ndist = k + 1;
    }
    // A strip's cell rows halve with the level, so the first level's are a
    // multiple of 2 for every such step between strip levels.
    blocks = 1;
    if (p.ndist) {
        int step = 1;
        for (int k = 0; k + 1 < p.ndist; k++)
            if (p.lev[k].ky) step *= 2;
        int rows = cdiv(cdiv(p.lev[0].cy, max_blocks), step) * step;
        blocks = cdiv(p.lev[0].cy, rows);
        for (int k = 0; k < p.ndist; k++) {
            p.lev[k].rows = rows;
            if (static_cast<long>(rows) * p.lev[k].cx > kTailThreads) return false;
            if (p.lev[k].ky) rows /= 2;
        }
    }
    threads = 96;  // the coarsest solve's rows
    long o = 0;
    for (int k = 0; k < p.count; k++) {
        TailLevel<T> &t = p.lev[k];
        if (t.rows * t.cx > threads) threads = t.rows * t.cx;
        t.used = cdiv(t.cy, t.rows);
        t.mul = ((1 << 20) + t.cx - 1) / t.cx;
        const long za = 4L * (t.rows + 1) * (t.cx + 2);
        t.zo = static_cast<int>(o); o += za;
        t.ro = static_cast<int>(o); o += k < p.count - 1 ? za : 0;
        t.bo = static_cast<int>(o); o += k ? 4L * t.rows * t.cx : 0;
    }
    threads = (threads + 31) / 32 * 32;
    p.zeroed = static_cast<int>(o);
    const long budget = static_cast<long>(kTailSmemBudget / sizeof(T));
    if (o > budget) return false;
    p.go = -1;
    const long Nc = lev.back().N;
    if (ginv) {
        if (o + Nc * Nc > budget) return false;
        p.go = static_cast<int>(o);
        o += Nc * Nc;
    }
    // Staged from the coarsest level up while they fit: all slots, else the
    // stencils alone.
    for (int k = p.count - 1; k >= 0; k--) {
        if (k == p.count - 1 && ginv) continue;  // solved by the inverse alone
        const long np = static_cast<long>(p.lev[k].rows) * p.lev[k].cx;
        int slots = kTailSlots<T>;
        if (o + slots * np > budget) slots = kTailRw<T>;
        if (o + slots * np > budget) break;
        p.lev[k].co = static_cast<int>(o);
        p.lev[k].staged = slots;
        o += slots * np;
    }
    smem = static_cast<size_t>(o) * sizeof(T);
    return true;
}

cudaLaunchConfig_t tail_config(int blocks, int threads, size_t smem, cudaStream_t s, cudaLaunchAttribute *at) {
    cudaLaunchConfig_t c{};
    c.gridDim = dim3(blocks);
    c.blockDim = dim3(threads);
    c.dynamicSmemBytes = smem;
    c.stream = s;
    at->id = cudaLaunchAttributeClusterDimension;
    at->val.clusterDim.x = blocks;
    at->val.clusterDim.y = at->val.clusterDim.z = 1;
    c.attrs = at;
    c.numAttrs = 1;
    return c;
}

}  // namespace

int Multigrid::choose_tail() {
    // The first level (never level 0) from which on everything fits, at the
    // largest cluster size that the device grants.
    tail_level = -1;
    for (int mb = kTailBlocks; mb >= 1 && tail_level < 0; mb /= 2)
        for (int l = 1; l < static_cast<int>(lev.size()); l++) {
            TailPlan<double> p;
            int blocks, threads;
            size_t smem;
            if (!tail_plan<double>(lev, l, px, py, ginv, mb, p, blocks, threads, smem)) continue;
            cudaLaunchAttribute at[1];
            cudaLaunchConfig_t c = tail_config(blocks, threads, smem, stream, at);
            int active = 0;
            if (cudaOccupancyMaxActiveClusters(&active, k_tail<double, true>, &c) != cudaSuccess) cudaGetLastError();
            if (active < 1) break;
            tail_level = l;
            tail_max_blocks = mb;
            break;
        }
    if (tail_level < 0) return INCRMT_OK;
    auto cells = [](const MgLevel &L) { return static_cast<size_t>((L.m + 1) / 2) * ((L.n + 1) / 2); };
    size_t total = 0;
    for (size_t l = tail_level; l < lev.size(); l++) total += cells(lev[l]);
    INCRMT_CK(cudaMalloc(&tail_pk, (sizeof(double) * kTailSlots<double> + sizeof(float) * kTailSlots<float>) * total));
    double *d = static_cast<double *>(tail_pk);
    float *f = reinterpret_cast<float *>(d + kTailSlots<double> * total);
    for (size_t l = tail_level; l < lev.size(); l++) {
        lev[l].pk = d;
        lev[l].pkf = f;
        d += kTailSlots<double> * cells(lev[l]);
        f += kTailSlots<float> * cells(lev[l]);
    }
    return INCRMT_OK;
}

template <class T>
int Multigrid::tail_pack() {
    if (tail_level < 0) return INCRMT_OK;
    TailPack<T> p{};
    p.count = static_cast<int>(lev.size()) - tail_level;
    p.px = px; p.py = py;
    int most = 0;
    for (int k = 0; k < p.count; k++) {
        const MgLevel &L = lev[tail_level + k];
        TailPackLevel<T> &t = p.lev[k];
        t.m = L.m; t.n = L.n; t.kx = L.kx; t.ky = L.ky; t.Q = L.Q;
        t.cells = ((L.m + 1) / 2) * ((L.n + 1) / 2);
        if constexpr (sizeof(T) == 8) { t.st = L.st; t.pk = L.pk; }
        else { t.st = L.stf; t.pk = L.pkf; }
        if (t.cells > most) most = t.cells;
    }
    k_tail_pack<T><<<dim3(cdiv(most, 64), p.count, 6), 64, 0, stream>>>(p);
    launches++;
    INCRMT_CKL("k_tail_pack");
    return INCRMT_OK;
}

template <class T>
int Multigrid::tail_launch() {
    TailPlan<T> p;
    int blocks, threads;
    size_t smem;
    const T *gi;
    if constexpr (sizeof(T) == 8) gi = ginv;
    else gi = ginvf;
    if (!tail_plan<T>(lev, tail_level, px, py, gi, tail_max_blocks, p, blocks, threads, smem)) {
        set_error("tail levels do not fit");
        return INCRMT_ERR_CUDA;
    }
    if constexpr (sizeof(T) == 8) { p.z = lev[tail_level].z; p.b = lev[tail_level].b; }
    else { p.z = lev[tail_level].zf; p.b = lev[tail_level].bf; }
    cudaLaunchAttribute at[1];
    cudaLaunchConfig_t c = tail_config(blocks, threads, smem, stream, at);
    bool seq = false;
    for (int k = 0; k < p.count; k++) seq = seq || p.lev[k].seq;
    if (seq) INCRMT_CK(cudaLaunchKernelEx(&c, k_tail<T, true>, p));
    else INCRMT_CK(cudaLaunchKernelEx(&c, k_tail<T, false>, p));
    launches++;
    INCRMT_CKL("k_tail");
    return INCRMT_OK;
}

int Multigrid::tail64() { return tail_launch<double>(); }
int Multigrid::tail32() { return tail_launch<float>(); }

int Multigrid::norm2_rhs(const double *b, double *out_dev) {
    const long N = static_cast<long>(m) * n;
    const int nb = cdiv(N, 256) < kRedBlocks ? cdiv(N, 256) : kRedBlocks;
    k_sumsq<<<nb, 256, 0, stream>>>(b, N, partial);
    k_reduce<<<1, 256, 0, stream>>>(partial, nb, out_dev);
    launches += 2;
    INCRMT_CKL("norm");
    return INCRMT_OK;
}

int Multigrid::residual_norm(const double *b, const double *z, float *rf) {
    const int nb = n < kRedBlocks ? n : kRedBlocks;  // blocks over the rows
    if (sys == INCRMT_SYS_MAC) k_resnorm<<<nb, 256, 0, stream>>>(mac64(), z, b, m, n, rf, partial, ticket, hnorm);
    else k_resnorm<<<nb, 256, 0, stream>>>(fem64(), z, b, m, n, rf, partial, ticket, hnorm);
    launches++;
    INCRMT_CKL("residual norm");
    return INCRMT_OK;
}

int Multigrid::fetch_norm(double *v) {
    INCRMT_CK(cudaMemcpyAsync(hnorm, dnorm, sizeof(double), cudaMemcpyDeviceToHost, stream));
    INCRMT_CK(cudaStreamSynchronize(stream));
    *v = hnorm[0];
    return INCRMT_OK;
}

/** One V-cycle (FP64, or one FP32 defect-correction step in mixed mode),
 * the FP64 residual norm of the new iterate in hnorm[0]. */
int Multigrid::vcycle_and_norm(int prec, const double *b, double *d_z, long N) {
    int r;
    const long long l0 = launches;
    if (prec == INCRMT_PREC_FP64) {
        if ((r = cycle64(0, b, d_z))) return r;
        if ((r = residual_norm(b, d_z, nullptr))) return r;
    } else {
        const int nbk = cdiv(N, 256) < kRedBlocks ? cdiv(N, 256) : kRedBlocks;
        if ((r = cycle32(0))) return r;
        if (zpr) {
            k_add_f32<<<nbk, 256, 0, stream>>>(d_z, lev[0].zf, N);
            launches++;
        } else {
            // Without the zero-pressure edge both systems are singular (the
            // constants): the FP32 cycle's correction comes back with a
            // constant part thousands of times its variation on the finest
            // grids, which the iterate would accumulate; it is removed.
            k_sum_f32<<<nbk, 256, 0, stream>>>(lev[0].zf, N, partial, ticket, dnorm + 1);
            k_add_f32_centred<<<nbk, 256, 0, stream>>>(d_z, lev[0].zf, N, dnorm + 1);
            launches += 2;
        }
        INCRMT_CKL("defect correction");
        if ((r = residual_norm(b, d_z, lev[0].bf))) return r;
    }
    graph_launches = launches - l0;
    return INCRMT_OK;
}

int Multigrid::krylov_alloc() {
    if (kr) return INCRMT_OK;
    const size_t N = static_cast<size_t>(m) * n;
    INCRMT_CK(cudaMalloc(&kr, sizeof(double) * N));
    INCRMT_CK(cudaMalloc(&kp, sizeof(double) * N));
    INCRMT_CK(cudaMalloc(&kq, sizeof(double) * N));
    INCRMT_CK(cudaMalloc(&ke, sizeof(double) * N));
    INCRMT_CK(cudaMalloc(&kpart, sizeof(double) * 3 * kRedBlocks));
    INCRMT_CK(cudaMalloc(&ks, sizeof(double) * 8));
    // q enters the first iteration's dot products (whose results the first
    // direction does not use): keep it finite
    INCRMT_CK(cudaMemsetAsync(kq, 0, sizeof(double) * N, stream));
    INCRMT_CK(cudaMemsetAsync(kp, 0, sizeof(double) * N, stream));
    INCRMT_CK(cudaMemsetAsync(ks, 0, sizeof(double) * 8, stream));
    return INCRMT_OK;
}

int Multigrid::krylov_residual(int prec, const double *b, const double *d_z) {
    const int nb = n < kRedBlocks ? n : kRedBlocks;  // blocks over the rows
    float *rf = prec == INCRMT_PREC_MIXED ? lev[0].bf : nullptr;
    if (sys == INCRMT_SYS_MAC) k_cg_residual<<<nb, 256, 0, stream>>>(mac64(), d_z, b, m, n, kr, rf, kpart);
    else k_cg_residual<<<nb, 256, 0, stream>>>(fem64(), d_z, b, m, n, kr, rf, kpart);
    k_reduce<<<1, 256, 0, stream>>>(kpart, nb, dnorm);
    launches += 2;
    INCRMT_CKL("krylov residual");
    return INCRMT_OK;
}

int Multigrid::krylov_iteration(int prec, double *d_z, long N) {
    int r;
    const long long l0 = launches;
    const int nbk = cdiv(N, 256) < kRedBlocks ? cdiv(N, 256) : kRedBlocks;
    const int nbr = n < kRedBlocks ? n : kRedBlocks;
    const int singular = zpr ? 0 : 1;
    if (prec == INCRMT_PREC_FP64) {
        if ((r = cycle64(0, kr, ke, true))) return r;
        k_cg_dots<double><<<nbk, 256, 0, stream>>>(ke, kq, N, kpart);
        k_reduce_n<3><<<1, 256, 0, stream>>>(kpart, nbk, ks);
        k_cg_direction<double><<<nbk, 256, 0, stream>>>(ke, kp, N, ks, singular);
    } else {
        if ((r = cycle32(0))) return r;
        k_cg_dots<float><<<nbk, 256, 0, stream>>>(lev[0].zf, kq, N, kpart);
        k_reduce_n<3><<<1, 256, 0, stream>>>(kpart, nbk, ks);
        k_cg_direction<float><<<nbk, 256, 0, stream>>>(lev[0].zf, kp, N, ks, singular);
    }
    if (sys == INCRMT_SYS_MAC) k_cg_apply<<<nbr, 256, 0, stream>>>(mac64(), kp, kq, kr, m, n, kpart);
    else k_cg_apply<<<nbr, 256, 0, stream>>>(fem64(), kp, kq, kr, m, n, kpart);
    k_reduce_n<2><<<1, 256, 0, stream>>>(kpart, nbr, ks + 4);
    k_cg_update<<<nbk, 256, 0, stream>>>(d_z, kr, kp, kq, prec == INCRMT_PREC_MIXED ? lev[0].bf : nullptr, N, ks,
                                         kpart);
    k_cg_finish<<<1, 256, 0, stream>>>(kpart, nbk, dnorm, ks);
    launches += 7;
    INCRMT_CKL("krylov iteration");
    INCRMT_CK(cudaMemcpyAsync(hnorm, dnorm, sizeof(double), cudaMemcpyDeviceToHost, stream));
    kexec_launches = launches - l0;
    return INCRMT_OK;
}

int Multigrid::krylov_solve(int prec, const double *b, double *d_z, long N, double tol, int maxc, int &k,
                            double &rn2, bool &conv, bool &finite, bool &fell) {
    int r;
    conv = false;
    finite = true;
    fell = false;
    if ((r = krylov_alloc())) return r;
    if (prec == INCRMT_PREC_MIXED && (r = cast_levels())) return r;
    // The fixed column's rows of the FEM system with the zero-pressure edge
    // hold the diagonal alone and a zero right-hand side: their solution is
    // 0, set here, so that the iteration stays on the symmetric remainder.
    if (sys == INCRMT_SYS_FEM && zpr) {
        k_zero_column<<<cdiv(n, 256), 256, 0, stream>>>(d_z, m, n);
        launches++;
        INCRMT_CKL("zero column");
    }
    if ((r = krylov_residual(prec, b, d_z))) return r;
    if ((r = fetch_norm(&rn2))) return r;
    double rn_prev = std::sqrt(rn2);
    if (!std::isfinite(rn_prev)) { finite = false; return INCRMT_OK; }
    if (rn_prev <= tol) { conv = true; return INCRMT_OK; }
    INCRMT_CK(cudaMemsetAsync(ks, 0, sizeof(double) * 8, stream));
    const bool use_graph = !prof;
    if (use_graph && (!kexec || kkey_prec != prec || kkey_b != b || kkey_z != d_z)) {
        if (kexec) { cudaGraphExecDestroy(kexec); kexec = nullptr; }
        cudaGraph_t graph = nullptr;
        INCRMT_CK(cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal));
        const int rc = krylov_iteration(prec, d_z, N);
        cudaError_t ce = cudaStreamEndCapture(stream, &graph);
        if (rc || ce != cudaSuccess) {
            if (ce == cudaSuccess && graph) cudaGraphDestroy(graph);
            if (rc) return rc;
            return cuda_status(ce, "capture", __FILE__, __LINE__);
        }
        ce = cudaGraphInstantiate(&kexec, graph, 0);
        cudaGraphDestroy(graph);
        if (ce != cudaSuccess) { kexec = nullptr; return cuda_status(ce, "instantiate", __FILE__, __LINE__); }
        kkey_prec = prec; kkey_b = b; kkey_z = d_z;
    }
    while (k < maxc) {
        if (use_graph) {
            INCRMT_CK(cudaGraphLaunch(kexec, stream));
            launches += kexec_launches;
        } else if ((r = krylov_iteration(prec, d_z, N))) {
            return r;
        }
        INCRMT_CK(cudaStreamSynchronize(stream));
        rn2 = hnorm[0];
        k++;
        const double rn = std::sqrt(rn2);
        if (!std::isfinite(rn)) { finite = false; return INCRMT_OK; }
        if (rn <= tol) {
            // The recurrence's residual has converged: confirm it on b - A z
            // itself, else restart from that residual.
            if ((r = krylov_residual(prec, b, d_z))) return r;
            if ((r = fetch_norm(&rn2))) return r;
            const double rt = std::sqrt(rn2);
            if (!std::isfinite(rt)) { finite = false; return INCRMT_OK; }
            if (rt <= tol) { conv = true; return INCRMT_OK; }
            INCRMT_CK(cudaMemsetAsync(ks, 0, sizeof(double) * 8, stream));
            rn_prev = rt;
            continue;
        }
        // An iteration that does not halve the residual: the preconditioned
        // iteration is not working on this system; the caller finishes with
        // plain FP64 V-cycles from the current iterate.
        if (rn > kMixedContraction * rn_prev) {
            fell = true;
            krylov_fallbacks++;
            return INCRMT_OK;
        }
        rn_prev = rn;
    }
    return INCRMT_OK;
}

int Multigrid::vcycle64(const double *d_b, double *d_z) {
    if (!ready) { set_error("density not set"); return INCRMT_ERR_BADARG; }
    return cycle64(0, d_b, d_z);
}

int Multigrid::effective_rhs(const double *d_b, const double **out) {
    *out = d_b;
    if (sys != INCRMT_SYS_FEM || !zpr) return INCRMT_OK;
    const long N = static_cast<long>(m) * n;
    if (d_b != bbuf) INCRMT_CK(cudaMemcpyAsync(bbuf, d_b, sizeof(double) * N, cudaMemcpyDeviceToDevice, stream));
    k_zero_column<<<cdiv(n, 256), 256, 0, stream>>>(bbuf, m, n);
    launches++;
    INCRMT_CKL("zero column");
    *out = bbuf;
    return INCRMT_OK;
}

int Multigrid::apply_device(const double *d_z, double *d_out) {
    if (!ready) { set_error("density not set"); return INCRMT_ERR_BADARG; }
    if (sys == INCRMT_SYS_MAC) k_apply<<<grid2(m, n), kBlk2, 0, stream>>>(mac64(), d_z, d_out, m, n);
    else k_apply<<<grid2(m, n), kBlk2, 0, stream>>>(fem64(), d_z, d_out, m, n);
    launches++;
    INCRMT_CKL("k_apply");
    return INCRMT_OK;
}

int Multigrid::solve_device(const double *d_b, double *d_z, const incrmt_mg_opts *o,
                            incrmt_mg_stats *st, bool time_it) {
    if (!ready) { set_error("density not set"); return INCRMT_ERR_BADARG; }
    const double rtol = (o && o->rel_tol > 0) ? o->rel_tol : 1e-9;
    const int maxc = (o && o->max_vcycles > 0) ? o->max_vcycles : 200;
    int prec = o ? o->precision : INCRMT_PREC_FP64;
    if (prec != INCRMT_PREC_FP64 && prec != INCRMT_PREC_MIXED) { set_error("bad precision %d", prec); return INCRMT_ERR_BADARG; }
    // After kMixedStrikes consecutive mixed solves that fell back to FP64,
    // the next kMixedRest solves run FP64 from the start (the FP32 cycle
    // only cost time on this system), then mixed precision is tried again.
    if (prec == INCRMT_PREC_MIXED && mixed_rest > 0) {
        mixed_rest--;
        mixed_rested++;
        prec = INCRMT_PREC_FP64;
    }
    const long N = static_cast<long>(m) * n;
    // The solve reads a residual norm back to the host after every V-cycle,
    // which a stream under capture cannot do.
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    INCRMT_CK(cudaStreamIsCapturing(stream, &cap));
    if (cap != cudaStreamCaptureStatusNone) {
        set_error("a solve cannot run while its stream is being captured into a CUDA graph");
        return INCRMT_ERR_BADARG;
    }
    if (time_it) INCRMT_CK(cudaEventRecord(ev0, stream));
    const double *b = d_b;
    if (sys == INCRMT_SYS_FEM && zpr) {
        if (d_b != bbuf) INCRMT_CK(cudaMemcpyAsync(bbuf, d_b, sizeof(double) * N, cudaMemcpyDeviceToDevice, stream));
        k_zero_column<<<cdiv(n, 256), 256, 0, stream>>>(bbuf, m, n);
        launches++;
        INCRMT_CKL("zero column");
        b = bbuf;
    }
    int r;
    double nb2, rn2 = 0;
    if ((r = norm2_rhs(b, dnorm))) return r;
    if ((r = fetch_norm(&nb2))) return r;
    const double nb = std::sqrt(nb2), tol = rtol * nb;
    int k = 0;
    if (nb == 0) {
        // A zero right-hand side: z = 0 solves A z = 0 exactly (for the
        // singular pure-Neumann systems it is the zero-mean solution), and the
        // warm start need not, so the iterate is cleared.
        INCRMT_CK(cudaMemsetAsync(d_z, 0, sizeof(double) * N, stream));
        if (time_it) {
            INCRMT_CK(cudaEventRecord(ev1, stream));
            INCRMT_CK(cudaEventSynchronize(ev1));
        }
        if (st) {
            st->vcycles = 0;
            st->rel_res = 0;
            float ms = 0;
            if (time_it) cudaEventElapsedTime(&ms, ev0, ev1);
            st->device_ms = ms;
        }
        return INCRMT_OK;
    }
    bool conv = false, finite = true, plain = true;
    double rn_prev = 0;
    int cur = prec;
    if (krylov) {
        // Flexible CG around the V-cycle; plain FP64 V-cycles finish the
        // solve only if an iteration fails to halve the residual.
        bool fell = false;
        if ((r = krylov_solve(prec, b, d_z, N, tol, maxc, k, rn2, conv, finite, fell))) return r;
        plain = fell;
        if (fell) {
            cur = INCRMT_PREC_FP64;
            if (prec == INCRMT_PREC_MIXED) mixed_fallbacks++;
        }
    } else if (prec == INCRMT_PREC_MIXED) {
        if ((r = cast_levels())) return r;
        if ((r = residual_norm(b, d_z, lev[0].bf))) return r;
        INCRMT_CK(cudaStreamSynchronize(stream));
        rn2 = hnorm[0];
        rn_prev = std::sqrt(rn2);
    }
    // One V-cycle and its residual norm, captured once into a CUDA graph per
    // (precision, b, z) and replayed per cycle.
    const bool use_graph = !prof;
    auto capture = [&]() -> int {
        if (gexec) { cudaGraphExecDestroy(gexec); gexec = nullptr; }
        cudaGraph_t graph = nullptr;
        INCRMT_CK(cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal));
        int rc = vcycle_and_norm(cur, b, d_z, N);
        cudaError_t ce = cudaStreamEndCapture(stream, &graph);
        if (rc || ce != cudaSuccess) {
            if (ce == cudaSuccess && graph) cudaGraphDestroy(graph);
            if (rc) return rc;
            return cuda_status(ce, "capture", __FILE__, __LINE__);
        }
        ce = cudaGraphInstantiate(&gexec, graph, 0);
        cudaGraphDestroy(graph);
        if (ce != cudaSuccess) { gexec = nullptr; return cuda_status(ce, "instantiate", __FILE__, __LINE__); }
        gkey_prec = cur; gkey_b = b; gkey_z = d_z;
        return INCRMT_OK;
    };
    if (plain && use_graph && (!gexec || gkey_prec != cur || gkey_b != b || gkey_z != d_z) && (r = capture()))
        return r;
    while (plain && k < maxc) {
        if (use_graph) {
            INCRMT_CK(cudaGraphLaunch(gexec, stream));
            launches += graph_launches;
        } else if ((r = vcycle_and_norm(cur, b, d_z, N))) {
            return r;
        }
        INCRMT_CK(cudaStreamSynchronize(stream));
        rn2 = hnorm[0];
        k++;
        const double rn = std::sqrt(rn2);
        if (!std::isfinite(rn)) { finite = false; break; }
        if (rn <= tol) { conv = true; break; }
        // An FP32 correction that does not halve the FP64 residual means the
        // single-precision cycle no longer approximates the system's inverse
        // well enough for defect correction to converge: the rest of the
        // solve runs FP64 V-cycles from the current iterate.
        if (cur == INCRMT_PREC_MIXED && rn > kMixedContraction * rn_prev) {
            cur = INCRMT_PREC_FP64;
            mixed_fallbacks++;
            if (use_graph && (r = capture())) return r;
        }
        rn_prev = rn;
    }
    if (prec == INCRMT_PREC_MIXED) {
        if (cur != prec) {
            if (++mixed_streak >= kMixedStrikes) {
                mixed_streak = 0;
                mixed_rest = kMixedRest;
            }
        } else {
            mixed_streak = 0;
        }
    }
    if (time_it) {
        INCRMT_CK(cudaEventRecord(ev1, stream));
        INCRMT_CK(cudaEventSynchronize(ev1));
    }
    if (prof && (r = prof_collect())) return r;
    if (st) {
        st->vcycles = k;
        st->rel_res = nb > 0 ? std::sqrt(rn2) / nb : std::sqrt(rn2);
        float ms = 0;
        if (time_it) cudaEventElapsedTime(&ms, ev0, ev1);
        st->device_ms = ms;
    }
    if (!finite) { set_error("non-finite residual after %d V-cycles", k); return INCRMT_ERR_NONFINITE; }
    if (!conv && nb > 0) { set_error("V-cycle failed to converge in %d cycles", k); return INCRMT_ERR_NOCONV; }
    return INCRMT_OK;
}

}  // namespace incrmt
