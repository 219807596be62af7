// The V-cycle below its large levels as one launch: smoothing, transfers and
// the coarsest solve of every level that fits a thread-block cluster.
//
// Below some 180 x 180 unknowns a level is bound by latency alone: a
// smoothing, restriction or prolongation launch costs 3-10 us however small
// it is, and a level needs four of them per V-cycle. Here one cluster of up to
// 16 thread blocks holds the levels on chip for the whole cycle. A thread owns
// one 2 x 2 cell of unknowns, one of each Gauss-Seidel colour, with their
// stencils in registers, so that a colour phase is eight shared-memory reads,
// a chain of fourteen fused operations and a barrier. The larger levels are
// cut into strips of cell rows, one strip per block, with one halo row on
// either side that the neighbouring block writes over distributed shared
// memory as it updates its edge row; a cluster barrier ends each phase. From
// the first level of at most kTailRoot cells on, the first block works alone,
// with barriers over the warps that hold cells.
//
// What decides the time is the latency of one phase (DFMA 8 cycles, shared
// read 30, block barrier 38, cluster barrier 415), so all that a phase needs
// is computed once per level: addresses, edge flags, and the reciprocals of the
// diagonals. The stencils and transfer weights are packed by cell once per
// density (k_tail_pack). All levels and both smoothings run the same copy of
// the code, in registers throughout: with the shared memory in use nothing is
// left of L1, and a version that spilled a few hundred bytes (one thread per
// unknown, 64 registers) took 56 us instead of 22.
//
// Every update, residual and transfer evaluates the expressions of the
// launch-per-level kernels in the same order (the quotient included, see
// quotient()), so the results are the same to the last bit.
//
// Measured (B200, FP64, one V-cycle): 32 x 32 and below 69.7 us with one block
// reading the stencils from L2 and dividing in every update, 21.6 us here;
// 128 x 128 and below (two more levels, four launches each: 58 us on top)
// 39 us; in single precision 74.9 + 58 us and 44.8 us.
#pragma once
#include <cooperative_groups.h>
#include "mg_ops.cuh"

namespace incrmt {
namespace {

constexpr int kTailThreads = 384;      // cells a block can hold
constexpr int kTailRegs = 168;         // registers a thread may use: 12 warps x 32 x 168 fit an SM's 65536
constexpr int kTailRoot = 300;         // cells of the first level that one block takes alone (33 x 33 unknowns: 289)
constexpr int kTailBlocks = 16;        // blocks of the cluster (above 8: a non-portable size)
constexpr int kTailMaxLevels = 14;
constexpr size_t kTailSmemBudget = 220 * 1024;
/** Largest level with an odd periodic size that one warp sweeps. */
constexpr int kTailSeq = 256;

/** Packed values of a cell, slot q of a level's cell t at pk[q * cells + t]:
 * eight off-diagonal stencil entries, the diagonal, its reciprocal and (single
 * precision) the row sum of each colour; then the nine restriction weights of
 * the cell's coarse points, then the prolongation weights. */
template <class T>
constexpr int kTailCoef = sizeof(T) == 8 ? 10 : 11;
template <class T>
constexpr int kTailRw = 4 * kTailCoef<T>;
template <class T>
constexpr int kTailPw = kTailRw<T> + 9;
template <class T>
constexpr int kTailSlots = kTailPw<T> + 8;

/** One level of the launch. */
template <class T>
struct TailLevel {
    int m, n;          // unknowns
    int cx, cy;        // 2 x 2 cells
    int rows;          // cell rows of a block's strip (cy on the first block's own levels)
    int dist;          // cut into strips over the cluster
    int kx, ky;        // whether the next level halves x / y
    int seq;           // odd periodic size, where colours touch across the seam: 1 in y only, 2 in x
    int used;          // strips that hold cell rows
    int mul;           // 2^20 / cx, rounded up: t / cx = t * mul >> 20 for t < kTailThreads
    int zo, ro, bo;    // offsets (elements) of the iterate, the residual and the right-hand side
    int co, staged;    // offset of the staged slots, and how many are staged: none, the stencils, or all
    const T *pk;       // packed stencils and weights
};

template <class T>
struct TailPlan {
    int count, ndist, px, py;
    int nu1, nu2, coarse_sweeps;
    int go;            // offset of the staged coarsest inverse, or -1
    int zeroed;        // elements cleared at the start (the staged entries follow)
    T *z;              // first level's iterate (written) and right-hand side (read), global memory
    const T *b;
    const T *ginv;     // dense inverse of the coarsest level, or null
    TailLevel<T> lev[kTailMaxLevels];
};

/** What k_tail_pack reads of a level. */
template <class T>
struct TailPackLevel {
    int m, n, kx, ky, cells;
    const T *st;       // Galerkin stencils (single precision: entry 4 the row sum)
    const double *Q;   // prolongation weights (planes), null on the coarsest level
    T *pk;
};
template <class T>
struct TailPack {
    int count, px, py;
    TailPackLevel<T> lev[kTailMaxLevels];
};

/** n / d from r = 1/d rounded to nearest, by two residual corrections of
 * n * r: the first leaves a quotient within one unit in the last place, from
 * which the second gives the correctly rounded one (P. W. Markstein, IBM J.
 * Res. Dev. 34 (1990) 111-119), the same value as the division. Five dependent
 * operations instead of a division (40 cycles against 145 in double). Where n or
 * the quotient nears the subnormal range the last bits may differ, an infinite n
 * gives NaN (a solve stops at either), and d needs a normal reciprocal: a level
 * whose diagonals have none in single precision (cells of 2^64 units) has no
 * finite coarsest inverse either. Testing for such d took k_tail 0.9 to 2.9 us. */
template <class T>
__device__ __forceinline__ T quotient(T n, T d, T r) {
    T q = mul_rn(n, r);
    q = fma_rn(fma_rn(-q, d, n), r, q);
    return fma_rn(fma_rn(-q, d, n), r, q);
}

/** Colours in sweep order: (0,0), (1,1), (1,0), (0,1). */
__host__ __device__ constexpr int tail_pi(int c) { return c == 1 || c == 2; }
__host__ __device__ constexpr int tail_pj(int c) { return c & 1; }
__host__ __device__ constexpr int tail_colour(int pi, int pj) { return pj ? (pi ? 1 : 3) : (pi ? 2 : 0); }

/** Prolongation weight e of fine point (i,j), unwrapped; 0 outside. */
template <class T>
__device__ __forceinline__ double tail_weight(const TailPackLevel<T> &L, int px, int py, int i, int j, int e) {
    if (i < 0 || i >= L.m) { if (!px) return 0; i += i < 0 ? L.m : -L.m; }
    if (j < 0 || j >= L.n) { if (!py) return 0; j += j < 0 ? L.n : -L.n; }
    double w[4];
    plane_weights(L.Q, cells_of(L.m, L.kx), cells_of(L.n, L.ky), L.kx, L.ky, i, j, w);
    return w[e];
}

/** Packs the levels' stencils and transfer weights by cell, one thread per
 * cell and slot (blockIdx.y: the level). A point outside the grid gets zero
 * entries and a unit diagonal, so that its value stays zero. */
template <class T>
__global__ void k_tail_pack(const __grid_constant__ TailPack<T> p) {
    const TailPackLevel<T> L = p.lev[blockIdx.y];
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= L.cells) return;
    const int cx = (L.m + 1) / 2, I = t % cx, J = t / cx;
    const long N = static_cast<long>(L.m) * L.n;
    const int part = blockIdx.z;  // colours 0..3, restriction, prolongation
    T *pk = L.pk + t;
    if (part < 4) {
        const int i = 2 * I + tail_pi(part), j = 2 * J + tail_pj(part);
        const bool in = i < L.m && j < L.n;
        const long q = in ? colour_index(L.m, L.n, i, j) : 0;
        T d = in ? L.st[4 * N + q] : T(1), a = 0;
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const T v = in ? L.st[(k < 4 ? k : k + 1) * N + q] : T(0);
            a = add_rn(a, v);
            pk[(kTailCoef<T> * part + k) * L.cells] = v;
        }
        if constexpr (sizeof(T) == 4) {
            pk[(kTailCoef<T> * part + 10) * L.cells] = in ? d : T(0);
            d = sub_rn(d, a);  // entry 4 is the row sum
        }
        pk[(kTailCoef<T> * part + 8) * L.cells] = d;
        pk[(kTailCoef<T> * part + 9) * L.cells] = T(1) / d;
        return;
    }
    if (!L.Q) return;
    if (part == 4) {
        // Weights of the fine points (x0+u, y0+v) of a coarse point's
        // support: slot 3v+u with both directions halved; with one halved the
        // cell has two coarse points, q the second, slots 3q+u (or 3q+v).
        for (int e = 0; e < 9; e++) {
            double w = 0;
            if (L.kx && L.ky) {
                const int u = e % 3, v = e / 3;
                w = tail_weight(L, p.px, p.py, 2 * I - 1 + u, 2 * J - 1 + v, (u == 0) + 2 * (v == 0));
            } else if (e < 6) {
                const int q = e / 3, u = e % 3;
                if (L.kx && 2 * J + q < L.n)
                    w = tail_weight(L, p.px, p.py, 2 * I - 1 + u, 2 * J + q, u == 0);
                if (L.ky && 2 * I + q < L.m)
                    w = tail_weight(L, p.px, p.py, 2 * I + q, 2 * J - 1 + u, 2 * (u == 0));
            }
            pk[(kTailRw<T> + e) * L.cells] = static_cast<T>(w);
        }
        return;
    }
    // Prolongation weights: colour (1,0): corners 0, 1; (0,1): 0, 2; (1,1): 0-3.
    for (int e = 0; e < 8; e++) {
        const int c = e < 2 ? 2 : (e < 4 ? 3 : 1), r = e < 2 ? e : (e < 4 ? 2 * (e - 2) : e - 4);
        const int i = 2 * I + tail_pi(c), j = 2 * J + tail_pj(c);
        pk[(kTailPw<T> + e) * L.cells] = i < L.m && j < L.n ? static_cast<T>(tail_weight(L, p.px, p.py, i, j, r)) : T(0);
    }
}

__device__ __forceinline__ void tail_copy_async(void *dst, const double *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(static_cast<unsigned>(__cvta_generic_to_shared(dst))),
                 "l"(src) : "memory");
}
__device__ __forceinline__ void tail_copy_async(void *dst, const float *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(static_cast<unsigned>(__cvta_generic_to_shared(dst))),
                 "l"(src) : "memory");
}

/** Barrier over the first `threads` threads of the block (a multiple of 32). */
__device__ __forceinline__ void tail_bar(int threads) {
    if (threads == 32) __syncwarp();
    else asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory");
}

/** The stencils of one cell: entries, diagonal, reciprocal, row sum. */
template <class T>
struct TailCell {
    T c[4][kTailCoef<T>];
};

/** One block's view of one level, everything a phase needs in registers. */
template <class T, bool SEQ>
struct TailView {
    T *s;              // shared memory
    int m, n, cx, cells, stride, px, py, kx, ky, dist, seq;
    int zo, ro, bo, co, staged;
    const T *pk;
    int W, W2;         // row layout: W even columns, then W odd ones, one pad on either side
    int rows;          // cell rows of this block's strip
    int row0;          // its first cell row
    int I, jl;         // this thread's cell
    bool on;
    int own;           // offset of the cell's (0,0) point in an array
    int edge;          // 1, 2: periodic image of an even / odd column; 4, 8: row of the strip's lower / upper edge
    T *lo, *hi;        // where the edge rows' values go in the neighbouring strips' iterates

    __device__ int at(int i, int r) const { return (r + 1) * W2 + (i & 1) * W + (i >> 1) + 1; }

    __device__ TailView(const TailPlan<T> &p, int l, T *smem, int rank) {
        const TailLevel<T> &L = p.lev[l];
        s = smem;
        m = L.m; n = L.n; cx = L.cx; px = p.px; py = p.py; kx = L.kx; ky = L.ky; dist = L.dist; seq = L.seq;
        zo = L.zo; ro = L.ro; bo = L.bo; co = L.co; pk = L.pk;
        staged = L.staged;
        const int cy = L.cy, sr = L.rows;
        cells = cx * cy;
        stride = cx * sr;
        W = cx + 2; W2 = 2 * W;
        row0 = dist ? rank * sr : 0;
        rows = min(cy - row0, sr);
        jl = static_cast<int>(threadIdx.x) * L.mul >> 20;
        I = threadIdx.x - jl * cx;
        on = jl < rows;
        own = (2 * jl + 1) * W2 + I + 1;
        edge = 0;
        lo = hi = nullptr;
        if ((px || py || dist) && on && (!SEQ || seq < 2)) {
            const int used = L.used;
            if (px) edge = (I == 0) + 2 * (2 * I + 1 == m - 1);
            int nb = !dist ? (py ? 0 : -1) : (rank > 0 ? rank - 1 : (py ? used - 1 : -1));
            if (jl == 0 && nb >= 0) {
                // the row above the lower strip's last one (row n if n is odd)
                const int nr = min(cy - nb * sr, sr);
                lo = s + zo + (SEQ && seq ? n + 1 : 2 * nr + 1) * W2 + I + 1;
                if (dist && nb != rank) lo = cooperative_groups::this_cluster().map_shared_rank(lo, nb);
                edge |= 4;
            }
            nb = !dist ? (py ? 0 : -1) : (rank + 1 < used ? rank + 1 : (py ? 0 : -1));
            if (jl == rows - 1 && nb >= 0) {
                hi = s + zo + I + 1;
                if (dist && nb != rank) hi = cooperative_groups::this_cluster().map_shared_rank(hi, nb);
                edge |= 8;
            }
        }
    }

    __device__ bool inside(int c) const { return 2 * I + tail_pi(c) < m && 2 * (row0 + jl) + tail_pj(c) < n; }
    /** Packed slot q of the cell. */
    __device__ T slot(int q) const {
        return q < staged ? s[co + q * stride + threadIdx.x] : pk[q * cells + row0 * cx + threadIdx.x];
    }

    __device__ void load(TailCell<T> &w) const {
        const T *src = staged ? s + co + threadIdx.x : pk + row0 * cx + threadIdx.x;
        const int ld = staged ? stride : cells;
#pragma unroll
        for (int q = 0; q < kTailRw<T>; q++) w.c[q / kTailCoef<T>][q % kTailCoef<T>] = src[q * ld];
    }

    /** Starts copying the cell's slots to shared memory. */
    __device__ void stage() const {
        if (!on) return;
        T *dst = s + co + threadIdx.x;
        const T *src = pk + row0 * cx + threadIdx.x;
#pragma unroll 4
        for (int q = 0; q < staged; q++) tail_copy_async(dst + q * stride, src + q * cells);
    }

    /** Off-diagonal sum of colour C of the cell (gen_terms of GenOp). */
    template <int C>
    __device__ T offdiag(const TailCell<T> &w, T zc) const {
        constexpr int pi = tail_pi(C), pj = tail_pj(C);
        constexpr bool CEN = sizeof(T) == 4;
        // x: the point's own column; y: the other parity, left neighbour first
        const T *x = s + zo + own + pj * W2 + (pi ? W : 0);
        const T *y = s + zo + own + pj * W2 + (pi ? 0 : W - 1);
        const T z0 = y[-W2], z1 = x[-W2], z2 = y[1 - W2], z3 = y[0], z5 = y[1], z6 = y[W2], z7 = x[W2], z8 = y[1 + W2];
        const T *c = w.c[C];
        T t = mul_rn(c[0], cen<CEN>(z0, zc));
        t = acc_rn(t, c[1], cen<CEN>(z1, zc));
        t = acc_rn(t, c[2], cen<CEN>(z2, zc));
        t = acc_rn(t, c[3], cen<CEN>(z3, zc));
        t = acc_rn(t, c[4], cen<CEN>(z5, zc));
        t = acc_rn(t, c[5], cen<CEN>(z6, zc));
        t = acc_rn(t, c[6], cen<CEN>(z7, zc));
        return acc_rn(t, c[7], cen<CEN>(z8, zc));
    }

    /** Writes a point of the iterate (or of the residual, `to` = ro - zo),
     * its periodic image, and the halo row of the strip it borders. */
    template <int C>
    __device__ void put(T v, int to = 0) const {
        constexpr int pi = tail_pi(C), pj = tail_pj(C);
        T *a = s + zo + to + own + pj * W2 + (pi ? W : 0);
        *a = v;
        constexpr int xbit = pi ? 2 : 1;
        if (edge) {
            const int im = pi ? -cx : cx;
            if (edge & xbit) a[im] = v;
            // the lower edge row is the strip's first (even) row; the upper
            // one its last: odd, or even where n is odd
            const bool up = SEQ && seq ? pj == 0 : pj == 1;
            T *h = nullptr;
            if (pj == 0 && (edge & 4)) h = lo;
            if (up && (edge & 8)) h = hi;  // (never both: a periodic level has several rows)
            if (h) {
                h += to + (pi ? W : 0);
                *h = v;
                if (edge & xbit) h[im] = v;
            }
        }
    }

    __device__ T center(int C) const { return s[zo + own + tail_pj(C) * W2 + (tail_pi(C) ? W : 0)]; }

    template <int C>
    __device__ T value(const TailCell<T> &w, T b) const {
        const T zc = sizeof(T) == 4 ? center(C) : T(0);
        const T off = offdiag<C>(w, zc);
        if constexpr (sizeof(T) == 8) return quotient(sub_rn(b, off), w.c[C][8], w.c[C][9]);
        else return add_rn(zc, quotient(fma_rn(-w.c[C][10], zc, sub_rn(b, off)), w.c[C][8], w.c[C][9]));
    }

    /** A colour phase. With n odd and periodic, rows 0 and n-1 hold the same
     * colours and meet across the seam: a point of the last row sees the new
     * value of row 0 where it comes in a later group of 32 points (in row
     * order) than its partner on a level of at most kTailSeq unknowns; all
     * other points see the values from before the phase. */
    template <int C>
    __device__ void phase(const TailCell<T> &w, T b, int threads) const {
        constexpr int pi = tail_pi(C), pj = tail_pj(C);
        if (SEQ && seq) {
            const bool in = on && inside(C);
            const int mc = (m - pi + 1) / 2;
            const bool late = pj == 0 && jl == rows - 1 && m * n <= kTailSeq && (jl * mc + I) / 32 > I / 32;
#pragma unroll 1
            for (int pass = 0; pass < (pj == 0 ? 2 : 1); pass++) {
                const bool now = in && late == (pass != 0);
                T v = 0;
                if (now) v = value<C>(w, b);
                if (pj == 0) tail_bar(threads);
                if (now) put<C>(v);
                tail_bar(threads);
            }
            return;
        }
        if (on) put<C>(value<C>(w, b));
        if (dist) cooperative_groups::this_cluster().sync();
        else tail_bar(threads);
    }

    template <int C>
    __device__ void residual(const TailCell<T> &w, T b) const {
        const T zc = center(C);
        const T off = offdiag<C>(w, zc);
        put<C>(fma_rn(-w.c[C][sizeof(T) == 8 ? 8 : 10], zc, sub_rn(b, off)), ro - zo);
    }

    /** `sweeps` four-colour sweeps; with `res` the residual then goes to the
     * residual array. b0: the right-hand side in global memory, or null. */
    __device__ void smooth(const T *b0, int sweeps, bool res) const {
        const int threads = dist ? blockDim.x : (cells + 31) & ~31;
        if (dist || threadIdx.x < threads) {
            TailCell<T> w;
            T b[4] = {0, 0, 0, 0};
            if (on) {
                load(w);
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    if (!b0) b[c] = s[bo + c * stride + threadIdx.x];
                    else if (inside(c)) b[c] = b0[2 * I + tail_pi(c) + m * (2 * (row0 + jl) + tail_pj(c))];
                }
            }
#pragma unroll 1
            for (int k = 0; k < sweeps; k++) {
                phase<0>(w, b[0], threads);
                phase<1>(w, b[1], threads);
                phase<2>(w, b[2], threads);
                phase<3>(w, b[3], threads);
            }
            if (res && on) {
                residual<0>(w, b[0]);
                if (!SEQ || inside(1)) residual<1>(w, b[1]);
                residual<2>(w, b[2]);
                if (!SEQ || inside(3)) residual<3>(w, b[3]);
            }
        }
        if (!dist) __syncthreads();
        else if (res) cooperative_groups::this_cluster().sync();
    }

    /** Gauss-Seidel value (or residual) of a point of a level with an odd
     * periodic x size, its neighbours by wrapped index. */
    template <bool RES>
    __device__ T seq_value(const T *b0, int i, int j) const {
        const bool l = px || i > 0, r = px || i < m - 1, d = py || j > 0, u = py || j < n - 1;
        const int il = i > 0 ? i - 1 : m - 1, ir = i < m - 1 ? i + 1 : 0;
        const int jd = j > 0 ? j - 1 : n - 1, ju = j < n - 1 ? j + 1 : 0;
        const T *z = s + zo;
        const int c = tail_colour(i & 1, j & 1), t = (j >> 1) * cx + (i >> 1);
        const T *src = (staged ? s + co : pk) + kTailCoef<T> * c * cells + t;  // (such a level is not cut)
        T k[kTailCoef<T>];
#pragma unroll
        for (int e = 0; e < kTailCoef<T>; e++) k[e] = src[e * cells];
        const T zc = z[at(i, j)];
        constexpr bool CEN = sizeof(T) == 4;
        T diag = 0;
        const T off = GenOp<T>::template gen_terms<CEN>(
            l, r, d, u, k[0], k[1], k[2], k[3], k[4], k[5], k[6], k[7], z[at(il, jd)], z[at(i, jd)], z[at(ir, jd)],
            z[at(il, j)], z[at(ir, j)], z[at(il, ju)], z[at(i, ju)], z[at(ir, ju)], CEN ? zc : T(0), diag);
        const T b = b0 ? b0[i + m * j] : s[bo + c * stride + t];
        if (RES) return fma_rn(-k[CEN ? kTailCoef<T> - 1 : 8], zc, sub_rn(b, off));
        if (!CEN) return quotient(sub_rn(b, off), k[8], k[9]);
        return add_rn(zc, quotient(fma_rn(-k[kTailCoef<T> - 1], zc, sub_rn(b, off)), k[8], k[9]));
    }

    /** smooth() of a level with an odd periodic x size: at most kTailSeq
     * unknowns are swept by the first warp, 32 points at a time in row order;
     * on larger levels every point of a colour sees the values from before
     * the phase. */
    __device__ void smooth_seq(const T *b0, int sweeps, bool res) const {
        const int threads = m * n <= kTailSeq ? 32 : blockDim.x;
        if (threadIdx.x < threads) {
#pragma unroll 1
            for (int k = 0; k < 4 * sweeps; k++) {
                const int c = k & 3, mc = (m - tail_pi(c) + 1) / 2, nc = (n - tail_pj(c) + 1) / 2;
#pragma unroll 1
                for (int q0 = 0; q0 < mc * nc; q0 += threads) {
                    const int q = q0 + threadIdx.x, i = 2 * (q % mc) + tail_pi(c), j = 2 * (q / mc) + tail_pj(c);
                    const bool in = q < mc * nc;
                    T v = 0;
                    if (in) v = seq_value<false>(b0, i, j);
                    tail_bar(threads);
                    if (in) s[zo + at(i, j)] = v;
                    tail_bar(threads);
                }
            }
        }
        __syncthreads();
        if (res) {
            for (int q = threadIdx.x; q < m * n; q += blockDim.x)
                s[ro + at(q % m, q / m)] = seq_value<true>(b0, q % m, q / m);
            __syncthreads();
        }
    }

    __device__ static double add(double t, double a, double b) { return __dadd_rn(t, __dmul_rn(a, b)); }
    __device__ static float add(float t, float a, float b) { return __fmaf_rn(a, b, t); }

    /** Residual at (i, row r), wrapped on a level that keeps no images. */
    __device__ T res_at(int i, int r) const {
        if (SEQ && seq == 2) {
            if (i < 0 && px) i += m;
            if (r < 0 && py) r += n;
        }
        return s[ro + at(i, r)];
    }

    /** Right-hand side of the next level C, P^T r in k_restrict's order. */
    __device__ void restrict_to(const TailView &C) const {
        if (on) {
            T *bc = s + C.bo;
            if (dist && !C.dist) bc = cooperative_groups::this_cluster().map_shared_rank(bc, 0);
            T w[9];
#pragma unroll
            for (int e = 0; e < 9; e++) w[e] = slot(kTailRw<T> + e);
            const int r = 2 * jl, i = 2 * I;
            T t0 = 0, t1 = 0;
            if (kx && ky) {
#pragma unroll
                for (int e = 0; e < 9; e++) t0 = add(t0, w[e], res_at(i - 1 + e % 3, r - 1 + e / 3));
            } else if (kx) {
#pragma unroll
                for (int e = 0; e < 3; e++) {
                    t0 = add(t0, w[e], res_at(i - 1 + e, r));
                    t1 = add(t1, w[3 + e], res_at(i - 1 + e, r + 1));
                }
            } else {
#pragma unroll
                for (int e = 0; e < 3; e++) {
                    t0 = add(t0, w[e], res_at(i, r - 1 + e));
                    t1 = add(t1, w[3 + e], res_at(i + 1, r - 1 + e));
                }
            }
            const int J = row0 + jl;
#pragma unroll
            for (int q = 0; q < 2; q++) {
                if (q == 1 && kx && ky) break;
                const int Ic = kx ? I : 2 * I + q, Jc = ky ? J : 2 * J + q;
                if (Ic < C.m && Jc < C.n)
                    bc[tail_colour(Ic & 1, Jc & 1) * C.stride + ((Jc >> 1) - C.row0) * C.cx + (Ic >> 1)] = q ? t1 : t0;
            }
        }
        if (dist) cooperative_groups::this_cluster().sync();
        else __syncthreads();
    }

    /** Value of the coarse level K at (Ic, Jc) for the prolongation. */
    __device__ T coarse_at(const TailView &K, const T *zc, int Ic, int Jc) const {
        if (Ic >= K.m) Ic -= K.m;             // only periodic grids weigh such a corner
        if (!K.dist && Jc >= K.n) Jc -= K.n;  // (a strip's upper halo row holds it)
        return zc[K.at(Ic, Jc - 2 * K.row0)];
    }

    /** z += P z_c of colour C, corners q of weights w (zero weights skipped). */
    template <int C>
    __device__ void prolong_point(const TailView &K, const T *zc, const T *w) const {
        constexpr int pi = tail_pi(C), pj = tail_pj(C);
        if (!inside(C)) return;
        const int J = row0 + jl, bx = kx ? I : 2 * I + pi, by = ky ? J : 2 * J + pj;
        T t = 0;
        if (C == 0) {
            t = coarse_at(K, zc, bx, by);
        } else {
#pragma unroll
            for (int r = 0; r < 4; r++) {
                if ((r & 1) > pi || (r >> 1) > pj) continue;
                const T wt = w[pi && pj ? r : (pi ? r & 1 : r >> 1)];
                if (wt != 0) t = add(t, wt, coarse_at(K, zc, bx + (r & 1), by + (r >> 1)));
            }
        }
        put<C>(center(C) + t);
    }

    /** z += P z_c from the next level K. */
    __device__ void prolong_from(const TailView &K) const {
        if (on) {
            const T *zc = s + K.zo;
            if (dist && !K.dist) zc = cooperative_groups::this_cluster().map_shared_rank(s + K.zo, 0);
            T w[8];
#pragma unroll
            for (int e = 0; e < 8; e++) w[e] = slot(kTailPw<T> + e);
            prolong_point<0>(K, zc, w);
            prolong_point<1>(K, zc, w + 4);
            prolong_point<2>(K, zc, w);
            prolong_point<3>(K, zc, w + 2);
        }
        if (dist) cooperative_groups::this_cluster().sync();
        else __syncthreads();
    }
};

/** The coarsest solve by the dense inverse, staged transposed at go. */
template <class T, bool SEQ>
__device__ void tail_direct(const TailView<T, SEQ> &L, int go, const T *b0) {
    const int N = L.m * L.n;
    for (int r = threadIdx.x; r < N; r += blockDim.x) {
        T t = 0;
        int i = 0, j = 0;
        for (int q = 0; q < N; q++) {
            const T b = b0 ? b0[q] : L.s[L.bo + tail_colour(i & 1, j & 1) * L.cells + (j >> 1) * L.cx + (i >> 1)];
            t = fma_rn(L.s[go + q * N + r], b, t);
            if (++i == L.m) { i = 0; j++; }
        }
        L.s[L.zo + L.at(r % L.m, r / L.m)] = t;
    }
    __syncthreads();
}

/** One V-cycle over the plan's levels from a zero iterate of the first. SEQ:
 * some level has an odd periodic size. */
template <class T, bool SEQ>
__global__ void __maxnreg__(kTailRegs) k_tail(const __grid_constant__ TailPlan<T> p) {
    extern __shared__ __align__(16) unsigned char tail_smem[];
    T *s = reinterpret_cast<T *>(tail_smem);
    const int rank = blockIdx.x, last = p.count - 1;
    const bool many = gridDim.x > 1;
    // Iterates, halos and the right-hand sides of points outside the grid
    // start at zero.
    for (int q = threadIdx.x; q < p.zeroed; q += blockDim.x) s[q] = T(0);
    for (int l = 0; l < p.count; l++)
        if (l < p.ndist || rank == 0) TailView<T, SEQ>(p, l, s, rank).stage();
    if (p.go >= 0 && rank == 0) {
        const int N = p.lev[last].m * p.lev[last].n;
        for (int q = threadIdx.x; q < N * N; q += blockDim.x) tail_copy_async(s + p.go + (q % N) * N + q / N, p.ginv + q);
    }
    // A first level that is not staged does not wait for the others.
    if (p.lev[0].staged || last == 0) asm volatile("cp.async.wait_all;" ::: "memory");
    if (many) cooperative_groups::this_cluster().sync();
    else __syncthreads();

    // Down to the coarsest level and back up: one copy of the code for every
    // level and both smoothings, which is fetched once.
#pragma unroll 1
    for (int v = 0; v <= 2 * last; v++) {
        const int l = v <= last ? v : 2 * last - v;
        if (l >= p.ndist && rank != 0) continue;
        if (many && v > last && l == p.ndist - 1) cooperative_groups::this_cluster().sync();  // block 0 is done
        const TailView<T, SEQ> L(p, l, s, rank);
        const T *b0 = l == 0 ? p.b : nullptr;
        if (v > last) L.prolong_from(TailView<T, SEQ>(p, l + 1, s, rank));
        if (l == last && p.go >= 0) {
            tail_direct(L, p.go, b0);
        } else {
            const int sweeps = l == last ? p.coarse_sweeps : (v < last ? p.nu1 : p.nu2);
            if (SEQ && L.seq == 2) L.smooth_seq(b0, sweeps, v < last);
            else L.smooth(b0, sweeps, v < last);
        }
        if (v == 0) asm volatile("cp.async.wait_all;" ::: "memory");
        if (v < last) L.restrict_to(TailView<T, SEQ>(p, l + 1, s, rank));
        if (v == 2 * last && L.on) {
#pragma unroll
            for (int c = 0; c < 4; c++)
                if (L.inside(c)) p.z[2 * L.I + tail_pi(c) + L.m * (2 * (L.row0 + L.jl) + tail_pj(c))] = L.center(c);
        }
    }
}

}  // namespace
}  // namespace incrmt
