// Two four-colour Gauss-Seidel sweeps in tiles, one thread per 2 x 2 cell of
// unknowns with the cell's coefficients in registers.
//
// A colour phase is a few shared-memory reads, a chain of up to fourteen fused
// operations and a division, so what decides the time is how the operands get
// there. With the coefficients in registers they cross L2 once per launch, not
// once per sweep, all of a thread's loads (up to 44) are in flight together
// before the first phase, and the phases need no index arithmetic: lanes run
// along x, warps along y, edges are flags set once. A tile pays for this with
// its halo, which is why its height is as large as the registers allow
// (40 doubles of stencil and right-hand side per thread: 512 threads; four cell
// densities in FEM or edges in MAC shared between a cell's points: 1024).
//
// Large MAC levels in double are bound by L1 and shared memory (75% busy, DRAM at
// 39%, loads the first stall), the single-precision ones by issue (53 to 60%),
// Galerkin levels in double by the phases' latency (one block of 16 warps per
// SM); small levels by one load latency and eight phases, 4 to 5 us. Measured
// (B200, two sweeps, us; the former kernels first: a pipeline along y for the
// large fine levels, a 64 x 32 or 32 x 16 tile of unknowns that read its
// coefficients from L2 in every phase otherwise):
//
//                MAC                 FEM                 Galerkin
//   size      FP64      FP32      FP64      FP32      FP64      FP32
//   4096^2  234->173  215->137  405->281  234->170
//   2048^2   66->47    61->36   118->79    79->49   163->160  110->83
//   1024^2   24->14    23->12    38->24    30->18    49->41    38->21
//   512^2    13->5.9   13->5.3   17->11.5  14->8.8   19->14    17->8.5
//   256^2   7.4->4.1  7.3->4.1   10->6.0  9.4->5.4   12->5.8   10->4.4
#pragma once
#include <type_traits>
#include "mg_ops.cuh"

namespace incrmt {
namespace {

constexpr int kCellX = 32;  // cells of a tile along x with its halo: one warp

/** Output cells of a tile: what two sweeps reach inward from its edges. Both
 * reds of a five-point sweep (and both blacks) update at once. */
template <class Op>
struct CellCfg {
    static constexpr bool kFive = Op::kFivePoint;
    static constexpr int kOffX = kFive ? 2 : 3, kOutX = kFive ? kCellX - 4 : kCellX - 5;
    static constexpr int kOffY = kFive ? 2 : 4;
    __host__ __device__ static constexpr int out_y(int ry) { return ry - 2 * kOffY; }
};

template <class T>
struct CellPair;
template <>
struct CellPair<double> { using type = double2; };
template <>
struct CellPair<float> { using type = float2; };

/** p[0] and p[1], in one load where the rows allow it (PAIR). */
template <bool PAIR, class T>
__device__ __forceinline__ void cell_pair(const T *__restrict__ p, T &a, T &b) {
    if constexpr (PAIR) {
        const typename CellPair<T>::type v = *reinterpret_cast<const typename CellPair<T>::type *>(p);
        a = v.x;
        b = v.y;
    } else {
        a = p[0];
        b = p[1];
    }
}

/** Neighbour values of point (PI, PJ) of cell s in the tile (planes of PL). */
template <class T, int PI, int PJ, int PL>
struct CellHood {
    static constexpr int RX = kCellX;
    T *own;
    const T *side, *vert, *corner;
    __device__ __forceinline__ CellHood(T *zs, int s)
        : own(zs + (PI + 2 * PJ) * PL + s), side(zs + (1 - PI + 2 * PJ) * PL + s + PI - 1),
          vert(zs + (PI + 2 * (1 - PJ)) * PL + s + (PJ ? 0 : -RX)),
          corner(zs + (1 - PI + 2 * (1 - PJ)) * PL + s + (PJ ? 0 : -RX) + PI - 1) {}
};

/** Where a cell lies: grid indices of its (0,0) point and which of its points
 * are on the grid and inside it. */
struct CellPos {
    int i, j;
    bool on0, on1, vn0, vn1;  // columns i, i+1 and rows j, j+1 are on the grid
    bool l, r, r1, d, u, u1;  // neighbours of column i (left, right), i+1 (right), row j (below, above), j+1 (above)
    template <int PI, int PJ>
    __device__ __forceinline__ bool on() const { return (PI ? on1 : on0) && (PJ ? vn1 : vn0); }
    /** The cell's four values of array f, point (PI, PJ) to v[PI + 2 PJ], zero off the grid. */
    template <bool INNER, bool PAIR, class T>
    __device__ __forceinline__ void four(const T *__restrict__ f, int m, T v[4]) const {
        f += i + static_cast<long>(m) * j;
        if constexpr (INNER) {
            cell_pair<PAIR>(f, v[0], v[1]);
            cell_pair<PAIR>(f + m, v[2], v[3]);
        } else {
            v[0] = on0 && vn0 ? f[0] : T(0);
            v[1] = on1 && vn0 ? f[1] : T(0);
            v[2] = on0 && vn1 ? f[m] : T(0);
            v[3] = on1 && vn1 ? f[m + 1] : T(0);
        }
    }
};

template <class Op, class T, bool INNER, bool PAIR>
struct CellData;

template <class T, bool INNER, bool PAIR>
struct CellData<GenOp<T>, T, INNER, PAIR> {
    T k[4][9], b[4];
    template <int PI, int PJ>
    __device__ __forceinline__ void point(const GenOp<T> &op, const CellPos &p, bool need, unsigned q) {
        constexpr int C = PI + 2 * PJ;
        if (!need || (!INNER && !p.template on<PI, PJ>())) return;
#pragma unroll
        for (int e = 0; e < 9; e++) k[C][e] = op.st[e * op.N + q];
    }
    __device__ __forceinline__ void load(const GenOp<T> &op, const T *__restrict__ rhs, const CellPos &p, int y, int ry) {
        const int m = op.m, n = op.n, m0 = (m + 1) >> 1, m1 = m >> 1, n0 = (n + 1) >> 1, n1 = n >> 1, I = p.i >> 1, J = p.j >> 1;
        p.template four<INNER, PAIR>(rhs, m, b);
        point<0, 0>(op, p, y >= 1, I + J * m0);
        point<1, 1>(op, p, y >= 1 && y <= ry - 2, m * n0 + m0 * n1 + I + J * m1);
        point<1, 0>(op, p, y >= 2 && y <= ry - 2, m0 * n0 + I + J * m1);
        point<0, 1>(op, p, y >= 2 && y <= ry - 3, m * n0 + I + J * m0);
    }
    template <int PI, int PJ, int PL>
    __device__ __forceinline__ void update(const GenOp<T> &, T *zs, int s, const CellPos &p) const {
        constexpr bool CEN = sizeof(T) == 4;
        constexpr int C = PI + 2 * PJ, RX = kCellX;
        if (!INNER && !p.template on<PI, PJ>()) return;
        const CellHood<T, PI, PJ, PL> h(zs, s);
        const T *a = k[C];
        const T zc = CEN ? h.own[0] : T(0);
        T diag = a[4];
        const bool l = PI ? true : p.l, r = PI ? p.r1 : p.r, d = PJ ? true : p.d, u = PJ ? p.u1 : p.u;
        const T off = GenOp<T>::template gen_terms<CEN>(l, r, d, u, a[0], a[1], a[2], a[3], a[5], a[6], a[7], a[8], h.corner[0],
                                                        h.vert[0], h.corner[1], h.side[0], h.side[1], h.corner[RX], h.vert[RX],
                                                        h.corner[RX + 1], zc, diag);
        h.own[0] = gs_value(b[C], off, diag, zc, a[4]);
    }
};

template <class T, bool INNER, bool PAIR>
struct CellData<FemOp<T>, T, INNER, PAIR> {
    T c[3][3], b[4];  // reciprocal densities of the cells around the four nodes
    __device__ __forceinline__ void load(const FemOp<T> &op, const T *__restrict__ rhs, const CellPos &p, int y, int ry) {
        const int m = op.m, n = op.n;
#pragma unroll
        for (int e = 0; e < 3; e++)
#pragma unroll
            for (int g = 0; g < 3; g++) {
                int i = p.i + g, j = p.j + e;
                bool in = true;
                if (!INNER) {
                    if (op.px && i >= m) i -= m;
                    if (op.py && j >= n) j -= n;
                    in = i >= 0 && i < m && j >= 0 && j < n;
                }
                c[e][g] = in ? op.c[i + m * j] : T(0);
            }
        p.template four<INNER, PAIR>(rhs, m, b);
    }
    template <int PI, int PJ, int PL>
    __device__ __forceinline__ void update(const FemOp<T> &op, T *zs, int s, const CellPos &p) const {
        constexpr bool CEN = sizeof(T) == 4;
        constexpr int RX = kCellX;
        if (!INNER && !p.template on<PI, PJ>()) return;
        const CellHood<T, PI, PJ, PL> h(zs, s);
        const T w[9] = {h.corner[0], h.vert[0], h.corner[1], h.side[0], h.own[0], h.side[1], h.corner[RX], h.vert[RX], h.corner[RX + 1]};
        const T cdl = c[PJ][PI], cdr = c[PJ][PI + 1], cul = c[PJ + 1][PI], cur = c[PJ + 1][PI + 1];
        const int i = p.i + PI, j = p.j + PJ;
        T diag, off, rs = T(0);
        if (INNER || (i > 0 && i < op.m - 1 && j > 0 && j < op.n - 1)) {
            off = op.template offdiag_int<CEN>(cdl, cdr, cul, cur, w, 4, 3, diag);
        } else {
            off = op.template offdiag_cells<CEN>(i, j, cdl, cdr, cul, cur, w, 4, 3, diag);
            if (op.zpr && i == op.m - 1) rs = diag;
        }
        h.own[0] = gs_value(b[PI + 2 * PJ], off, diag, CEN ? w[4] : T(0), rs);
    }
};

template <class T, bool INNER, bool PAIR>
struct CellData<MacOp<T>, T, INNER, PAIR> {
    T ex[2][3], ey[3][2], b[4];
    __device__ __forceinline__ void load(const MacOp<T> &op, const T *__restrict__ rhs, const CellPos &p, int y, int ry) {
        const int m = op.m, n = op.n;
#pragma unroll
        for (int e = 0; e < 2; e++)
#pragma unroll
            for (int g = 0; g < 3; g++) {
                const bool in = INNER || (p.on0 && p.i + g <= m && (e ? p.vn1 : p.vn0));
                ex[e][g] = in ? op.ex[(p.j + e) * (m + 1) + p.i + g] : T(0);
                const bool jn = INNER || (p.vn0 && p.j + g <= n && (e ? p.on1 : p.on0));
                ey[g][e] = jn ? op.ey[(p.j + g) * m + p.i + e] : T(0);
            }
        p.template four<INNER, PAIR>(rhs, m, b);
    }
    template <int PI, int PJ, int PL>
    __device__ __forceinline__ void update(const MacOp<T> &op, T *zs, int s, const CellPos &p) const {
        constexpr bool CEN = sizeof(T) == 4;
        constexpr int RX = kCellX;
        if (!INNER && !p.template on<PI, PJ>()) return;
        const CellHood<T, PI, PJ, PL> h(zs, s);
        const bool l = PI ? true : p.l, r = PI ? p.r1 : p.r, d = PJ ? true : p.d, u = PJ ? p.u1 : p.u;
        const T el = ex[PJ][PI], er = ex[PJ][PI + 1], ed = ey[PJ][PI], eu = ey[PJ + 1][PI];
        const T zc = CEN ? h.own[0] : T(0);
        const int i = INNER ? 0 : p.i + PI;
        T diag, rs = T(0);
        if (INNER) diag = mac_diag(mul_rn(-op.xxsp, add_rn(el, er)), op.yysp, add_rn(ed, eu));
        else diag = op.diag_of(i, l, r, d, u, el, er, ed, eu);
        const T off = op.template mac_terms<CEN>(l, r, d, u, el, er, ed, eu, h.side[0], h.side[1], h.vert[0], h.vert[RX], zc);
        if (CEN && !INNER && op.zpr && !op.px && i == op.m - 1) rs = -2 * op.xxsp * er;
        h.own[0] = gs_value(b[PI + 2 * PJ], off, diag, zc, rs);
    }
};

template <class Op, class T, int RY, bool INNER, bool PAIR>
__device__ __forceinline__ void cell_sweeps(const Op &op, T *zs, const T *__restrict__ zin, const T *__restrict__ b, int m, int n,
                                            int X, int Y) {
    constexpr int RX = kCellX, PL = RX * RY;
    const int x = threadIdx.x & 31, y = threadIdx.x >> 5, s = y * RX + x;
    const bool px = op.px, py = op.py;
    const int m0 = (m + 1) >> 1, n0 = (n + 1) >> 1;
    int I = X + x, J = Y + y;
    if (!INNER && px) { I %= m0; I = I < 0 ? I + m0 : I; }
    if (!INNER && py) { J %= n0; J = J < 0 ? J + n0 : J; }
    CellPos p;
    p.i = 2 * I;
    p.j = 2 * J;
    p.on0 = INNER || (p.i >= 0 && p.i < m);
    p.on1 = INNER || (p.i >= 0 && p.i + 1 < m);
    p.vn0 = INNER || (p.j >= 0 && p.j < n);
    p.vn1 = INNER || (p.j >= 0 && p.j + 1 < n);
    p.l = INNER || px || p.i > 0;
    p.r = INNER || px || p.i < m - 1;
    p.r1 = INNER || px || p.i + 1 < m - 1;
    p.d = INNER || py || p.j > 0;
    p.u = INNER || py || p.j < n - 1;
    p.u1 = INNER || py || p.j + 1 < n - 1;
    CellData<Op, T, INNER, PAIR> a;
    a.load(op, b, p, y, RY);
    T z[4] = {};
    if (zin) p.template four<INNER, PAIR>(zin, m, z);
#pragma unroll
    for (int q = 0; q < 4; q++) zs[q * PL + s] = z[q];
    __syncthreads();
    // A phase leaves out the rows of cells whose neighbours are not final; the
    // columns beyond are computed and never read.
    if constexpr (Op::kFivePoint) {
#pragma unroll 1
        for (int g = 0; g < 2; g++) {
            if (y >= 1 + g && y <= RY - 1 - g) a.template update<0, 0, PL>(op, zs, s, p);
            if (y >= g && y <= RY - 2 - g) a.template update<1, 1, PL>(op, zs, s, p);
            __syncthreads();
            if (y >= 1 + g && y <= RY - 2 - g) {
                a.template update<1, 0, PL>(op, zs, s, p);
                a.template update<0, 1, PL>(op, zs, s, p);
            }
            __syncthreads();
        }
    } else {
#pragma unroll 1
        for (int g = 0; g < 4; g += 2) {
            if (y >= 1 + g && y <= RY - 1 - g) a.template update<0, 0, PL>(op, zs, s, p);
            __syncthreads();
            if (y >= 1 + g && y <= RY - 2 - g) a.template update<1, 1, PL>(op, zs, s, p);
            __syncthreads();
            if (y >= 2 + g && y <= RY - 2 - g) a.template update<1, 0, PL>(op, zs, s, p);
            __syncthreads();
            if (y >= 2 + g && y <= RY - 3 - g) a.template update<0, 1, PL>(op, zs, s, p);
            __syncthreads();
        }
    }
}

/** zin is not written, so every point sees the neighbour values of the
 * one-launch-per-colour schedule: the result is identical to it. In a periodic
 * direction (even size) the halo holds periodic images, updated like the points
 * they copy. */
template <class Op, class T, int RY, int MINB, bool PAIR>
__global__ void __launch_bounds__(32 * RY, MINB) k_smooth_cells(Op op, const T *__restrict__ zin, T *__restrict__ zout,
                                                                const T *__restrict__ b, int m, int n) {
    using C = CellCfg<Op>;
    constexpr int RX = kCellX, PL = RX * RY, HX = C::kOffX, HY = C::kOffY, TX = C::kOutX, TY = C::out_y(RY);
    __shared__ T zpad[4 * PL + 2 * RX + 2];
    T *zs = zpad + RX + 1;  // point (pi, pj) of cell (x, y): [(pi + 2 pj) * PL + y * RX + x]
    const int X = blockIdx.x * TX - HX, Y = blockIdx.y * TY - HY;
    if (X > 0 && Y > 0 && 2 * (X + RX) < m && 2 * (Y + RY) < n) cell_sweeps<Op, T, RY, true, PAIR>(op, zs, zin, b, m, n, X, Y);
    else cell_sweeps<Op, T, RY, false, PAIR>(op, zs, zin, b, m, n, X, Y);
    if constexpr (PAIR) {
        const int x = threadIdx.x & 31, y = threadIdx.x >> 5, i = 2 * (X + x), j = 2 * (Y + y);
        if (x < HX || x >= HX + TX || y < HY || y >= HY + TY || i >= m || j >= n) return;
        const T *src = zs + y * RX + x;
        using V = typename CellPair<T>::type;
        T *dst = zout + i + static_cast<long>(m) * j;
        *reinterpret_cast<V *>(dst) = V{src[0], src[PL]};
        if (j + 1 < n) *reinterpret_cast<V *>(dst + m) = V{src[2 * PL], src[3 * PL]};
    } else {
        for (int r = 2 * HY + (threadIdx.x >> 5); r < 2 * (HY + TY); r += RY) {
            const int j = 2 * Y + r;
            if (j >= n) break;
            const T *src = zs + (r & 1) * 2 * PL + (r >> 1) * RX;
            for (int t = 2 * HX + (threadIdx.x & 31); t < 2 * (HX + TX); t += 32) {
                const int i = 2 * X + t;
                if (i < m) zout[i + static_cast<long>(m) * j] = src[(t & 1) * PL + (t >> 1)];
            }
        }
    }
}

template <class Op, class T, int RY, int MINB>
void smooth_cells_launch(bool pair, const Op &op, const T *z, T *zout, const T *b, int m, int n, cudaStream_t s) {
    using C = CellCfg<Op>;
    const dim3 grid((m + 2 * C::kOutX - 1) / (2 * C::kOutX), (n + 2 * C::out_y(RY) - 1) / (2 * C::out_y(RY)));
    if constexpr (C::kFive)
        if (pair) {
            k_smooth_cells<Op, T, RY, MINB, true><<<grid, 32 * RY, 0, s>>>(op, z, zout, b, m, n);
            return;
        }
    k_smooth_cells<Op, T, RY, MINB, false><<<grid, 32 * RY, 0, s>>>(op, z, zout, b, m, n);
}

/** Two sweeps of z into zout; z null: from zero, as every coarse level's first
 * smoothing and a defect correction's start (clearing and reading it took 1 to
 * 3 per cent of a solve: MAC 1024^2 mixed 1.69 -> 1.64 ms, FEM 2048^2 4.70 -> 4.56).
 *
 * Rows of even length whose arrays allow it are read and written by pairs in
 * the five-point system (4096^2 FP64 210 -> 194 us at the same tile); the
 * nine-point ones gain nothing (Galerkin 2048^2 FP32 81 -> 83).
 *
 * Tile heights, from sweeps over 10 to 32: MAC 16 (FP64 4096^2: 12 rows 194,
 * 16 rows 173, 32 rows 188 us); Galerkin 16 (FP64 2048^2: 14 rows 180, 16 rows
 * 160, 18 rows, spilling, 161; FP32, mean of a 4096^2 MAC system's four levels: 12
 * rows 41, 16 rows, two blocks per SM, 27, 24 rows, one block, 33). FEM: the tallest that fits (FP64 4096^2: 16 rows
 * 464, 24 rows 331, 32 rows 281; FP32: 16 rows 190, 24 rows 170), except where
 * 16 rows make a grid that all runs at once: fewer warps per tile then shorten
 * the phases (FP64 257^2: 16 rows 6.0, 32 rows 11.3; FP32 513^2: 16 rows 8.8, 24
 * rows 10.4, equal at 1025^2). */
template <class Op, class T>
void smooth_cells(const Op &op, const T *z, T *zout, const T *b, int m, int n, cudaStream_t s) {
    constexpr bool kDouble = sizeof(T) == 8;
    const auto addr = [](const void *p) { return reinterpret_cast<unsigned long long>(p); };
    const bool pair = m % 2 == 0 && (addr(z) | addr(zout) | addr(b)) % (2 * sizeof(T)) == 0;
    if constexpr (Op::kFivePoint) {
        smooth_cells_launch<Op, T, 16, kDouble ? 2 : 3>(pair, op, z, zout, b, m, n, s);
    } else if constexpr (std::is_same<Op, GenOp<T>>::value) {
        smooth_cells_launch<Op, T, 16, kDouble ? 1 : 2>(pair, op, z, zout, b, m, n, s);
    } else {
        constexpr int kPerSm = kDouble ? 1 : 3;  // blocks of 16 rows that an SM holds
        using C = CellCfg<Op>;
        const long tiles = static_cast<long>((m + 2 * C::kOutX - 1) / (2 * C::kOutX)) * ((n + 2 * C::out_y(16) - 1) / (2 * C::out_y(16)));
        if (tiles <= (kDouble ? 1 : 2) * kPerSm * kB200SMs)
            smooth_cells_launch<Op, T, 16, kPerSm>(pair, op, z, zout, b, m, n, s);
        else
            smooth_cells_launch<Op, T, kDouble ? 32 : 24, kDouble ? 1 : 2>(pair, op, z, zout, b, m, n, s);
    }
}

}  // namespace
}  // namespace incrmt
