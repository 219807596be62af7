// Two four-colour Gauss-Seidel sweeps of a large fine level in one pass over memory:
// the eight colour phases run as a pipeline along y.
//
// A block owns a strip of 64 columns of 2 x 2 cells (points A = (0,0),
// B = (1,1), C = (1,0), D = (0,1), the colours in sweep order) and walks a
// chunk of cell rows upwards. Its eight warps are the eight phases: in
// step t phase p updates cell row t - skew(p), the skews chosen so that all a
// phase reads was written in an earlier step and none of it is overwritten
// before it is read, so that the phases of a step are independent and one
// block barrier ends the step. Iterate, right-hand side and coefficients go
// through rings of rows in shared memory, filled by cp.async a few steps
// ahead; every value is fetched once per sweep pair, apart from the halo (as
// many cells on either side as the phases reach, computed redundantly).
//
// Each point sees exactly the neighbour values of the one-launch-per-colour
// schedule and the arithmetic is that of mg_ops.cuh, so the results are the
// same to the last bit. Periodic directions (even sizes) wrap in the loads;
// their images are updated like the points they copy.
//
// What bounds it is instruction issue and latency, not memory: about 140
// instructions per 32 updates in double (26 of them FP64), half what the tiled
// kernels need, at 16-24 warps per SM. Measured (B200, two sweeps; tiled kernel
// -> this one): MAC 4096^2 FP64 321 -> 232 us (its 671 MB alone: 102 us),
// 2048^2 91.5 -> 65.6, 1024^2 32.5 -> 23.7, 512^2 14.1 -> 13.1, 384^2 10.2 ->
// 10.9; FP32 2048^2 71.6 -> 48.7, 1024^2 28.8 -> 22.9; FEM FP32 3000^2 163 ->
// 130, 2048^2 85.5 -> 79.8, 1024^2 29.8 -> 36.0; FEM FP64 3000^2 224 -> 222.
// Two columns per thread and eight warps took 237 instructions down to 142;
// preloading ones instead of zeros as the coefficients of columns outside the
// grid took MAC 4096^2 from 314 to 232 us (its edge strips divided by zero).
// The same pipeline for the Galerkin levels (36 ring rows of stencils, one
// block per SM) was slower than the tiles: 331 against 234 us per V-cycle
// smoothing from 2048^2 down in FP64.
#pragma once
#include "mg_ops.cuh"

namespace incrmt {
namespace {

constexpr int kStrW = 64;  // cell columns of a strip, halo included

/** The pipeline of an operator: halo cells, the phases' skews (ascending),
 * ring rows and prefetch distance in steps. A nine-point phase A needs B, C, D
 * of the sweep before; B then A of its row and the next; C then B of its row
 * and the one below; D then C of its row and the next. */
template <class Op>
struct StreamCfg {
    static constexpr int kHalo = 4, kRing = 16, kPf = 2, kLast = 11, kNat = 3;
    static __device__ __forceinline__ int skew(int p) { return ((p & 3) * 2 - ((p & 3) > 1)) + (p > 3 ? 6 : 0); }
};
/** Five points: A and B (red) do not touch, nor do C and D; the reach is that
 * of four phases. */
template <class T>
struct StreamCfg<MacOp<T>> {
    static constexpr int kHalo = 2, kRing = 10, kPf = 3, kLast = 5, kNat = 5;
    static __device__ __forceinline__ int skew(int p) { return min(p & 3, 2) + (p > 3 ? 3 : 0); }
};

/** Shared memory elements: kNat arrays of the four points of a cell. */
template <class Op>
__host__ __device__ constexpr int stream_elems() {
    return 4 * StreamCfg<Op>::kNat * StreamCfg<Op>::kRing * (kStrW + 2);
}

/** Blocks per SM that registers and shared memory allow. */
template <class T>
__host__ __device__ constexpr int stream_per_sm() {
    return sizeof(T) == 8 ? 2 : 3;
}

__device__ __forceinline__ void stream_copy(double *dst, const double *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(static_cast<unsigned>(__cvta_generic_to_shared(dst))),
                 "l"(src) : "memory");
}
__device__ __forceinline__ void stream_copy(float *dst, const float *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(static_cast<unsigned>(__cvta_generic_to_shared(dst))),
                 "l"(src) : "memory");
}

/** Off-diagonal sum, diagonal and row sum of a point from its neighbours'
 * values (low0..2, zl, zr, up0..2) and its staged coefficients. */
template <class Op, class T>
struct StreamPoint {
    T low0, low1, low2, zl, zr, up0, up1, up2, zc;
    static constexpr bool CEN = sizeof(T) == 4;

    __device__ __forceinline__ T mac(const Op &op, int i, bool l, bool r, bool d, bool u, bool fix, T el, T er, T ed, T eu,
                                     T bv) const {
        const T diag = op.diag_of(i, l, r, d, u, el, er, ed, eu);
        const T off = op.template mac_terms<CEN>(l, r, d, u, el, er, ed, eu, zl, zr, low1, up1, zc);
        return gs_value(bv, off, diag, zc, CEN && fix ? -2 * op.xxsp * er : T(0));
    }
    __device__ __forceinline__ T fem(const Op &op, T cdl, T cdr, T cul, T cur, T bv) const {
        const T w[9] = {low0, low1, low2, zl, zc, zr, up0, up1, up2};
        T diag;
        const T off = op.template offdiag_int<CEN>(cdl, cdr, cul, cur, w, 4, 3, diag);
        return gs_value(bv, off, diag, zc, T(0));
    }
    __device__ __forceinline__ T fem_edge(const Op &op, int i, int j, T cdl, T cdr, T cul, T cur, T bv) const {
        const T w[9] = {low0, low1, low2, zl, zc, zr, up0, up1, up2};
        T diag;
        const T off = op.template offdiag_cells<CEN>(i, j, cdl, cdr, cul, cur, w, 4, 3, diag);
        return gs_value(bv, off, diag, zc, op.zpr && i == op.m - 1 ? diag : T(0));
    }
};

/** One warp per phase, two columns (32 apart) per thread: what a step costs
 * besides its updates (ring and row arithmetic, addresses of the loads, the
 * barrier) is shared by both. */
template <class Op, class T>
__global__ void __launch_bounds__(256, stream_per_sm<T>())
    k_smooth_stream(Op op, const T *__restrict__ zin, T *__restrict__ zout, const T *__restrict__ b, int m, int n, int chunk) {
    using C = StreamCfg<Op>;
    constexpr bool kFive = Op::kFivePoint;
    constexpr int W = kStrW + 2, R = C::kRing, RW = R * W, H = C::kHalo, PF = C::kPf;
    constexpr bool CEN = sizeof(T) == 4;
    extern __shared__ __align__(16) unsigned char stream_smem[];
    T *zs = reinterpret_cast<T *>(stream_smem);  // point (pi, pj) of ring row r, column X: [(pi + 2 pj) * RW + r * W + X + 1]
    const int tid = threadIdx.x, g = tid >> 5, X = tid & 31, c = g & 3;
    const int pi = c == 1 || c == 2, pj = c & 1;
    const bool px = op.px, py = op.py;
    const int cx = (m + 1) >> 1, cy = (n + 1) >> 1;
    const int I0 = blockIdx.x * (kStrW - 2 * H) - H;
    const int J0 = blockIdx.y * chunk, J1 = min(J0 + chunk, cy);
    const int Js = py ? J0 - H : max(J0 - H, 0), Je = py ? J1 + H : min(J1 + H, cy);
    auto wrap = [](int i, int s) { i %= s; return i < 0 ? i + s : i; };
    // This thread's phase: its columns and the arrays it reads.
    int ci[2];
    bool col[2];
#pragma unroll
    for (int q = 0; q < 2; q++) {
        const int I = px ? wrap(I0 + X + 32 * q, cx) : I0 + X + 32 * q;
        ci[q] = 2 * I + pi;
        col[q] = I >= 0 && ci[q] < m;
    }
    // (a warp away from the grid's left and right edges skips their cases)
    const bool inner = __all_sync(0xffffffffu, ((ci[0] > 0 && ci[0] < m - 1) || !col[0]) && ((ci[1] > 0 && ci[1] < m - 1) || !col[1]));
    T *own = zs + (pi + 2 * pj) * RW + X + 1;
    const T *side = zs + (1 - pi + 2 * pj) * RW + X + pi;          // left neighbour; the right one next to it
    const T *corner = zs + (1 - pi + 2 * (1 - pj)) * RW + X + pi;  // row above, left; right one next to it
    const T *vert = zs + (pi + 2 * (1 - pj)) * RW + X + 1;         // row above
    const T *right = pi ? zs + (16 + pj) * RW + X + 1 : side + 8 * RW + 1;  // MAC: edges right of and above the point
    const T *above = pj ? zs + (18 + pi) * RW + X + 1 : vert + 12 * RW;
    // And its share of the loads: one point of a cell row.
    const int ne = tid & 127, nj = tid >> 7;
    const int ni = px ? wrap(2 * I0 + ne, m) : 2 * I0 + ne;
    const bool ncol = ni >= 0 && ni < m;
    T *nat = zs + ((ne & 1) + 2 * nj) * RW + (ne >> 1) + 1;
    T *natx = zs + (16 + nj) * RW + (ne >> 1) + 1, *naty = zs + (18 + (ne & 1)) * RW + (ne >> 1) + 1;
    // Columns outside the grid are never loaded: their values stay zero and
    // their coefficients one (a zero diagonal would send the quotients of their
    // lanes, whose results are not used, down the division's slow path).
    for (int q = tid; q < stream_elems<Op>(); q += 256) zs[q] = T(q >= 4 * RW);
    __syncthreads();

    int lt = Js, lw = py ? wrap(Js, cy) : Js, lslot = 0;
    long lq = ni + static_cast<long>(m) * (2 * lw + nj), lx = lq + 2 * lw + nj;
    const long lwrap = static_cast<long>(m) * n;
    // Loads of a step: cell row lt.
    auto fetch = [&]() {
        if (lt < Je) {
            if (ncol && 2 * lw + nj < n) {
                stream_copy(nat + lslot, zin + lq);
                stream_copy(nat + lslot + 4 * RW, b + lq);
                if constexpr (kFive) {
                    // edges below and (further down) left of the point; for the
                    // odd column and row also the ones right of and above it
                    stream_copy(nat + lslot + 12 * RW, op.ey + lq);
                    if (ne & 1) stream_copy(natx + lslot, op.ex + lx + 1);
                    if (nj) stream_copy(naty + lslot, op.ey + lq + m);
                } else {
                    stream_copy(nat + lslot + 8 * RW, op.c + lq);
                }
            }
            if constexpr (kFive) {  // (the right boundary edge belongs to no point)
                if (ni >= 0 && ni <= m && 2 * lw + nj < n) stream_copy(nat + lslot + 8 * RW, op.ex + lx);
            }
            lt++;
            lslot = lslot + W == RW ? 0 : lslot + W;
            lq += 2 * m;
            lx += 2 * m + 2;
            if (++lw == cy && py) { lw = 0; lq -= lwrap; lx -= lwrap + n; }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int q = 0; q < PF; q++) fetch();

    StreamPoint<Op, T> p[2];  // (the row below: what was the row above a step ago)
    int J = Js - C::skew(g), j = 2 * (py ? wrap(Js, cy) : Js) + pj;  // the phase's cell row (its first is Js) and row
    int so = 0, su = pj ? W : 0;          // ring slots: the phase's row, the row above
    int Jo = Js - C::kLast - 1, sz = 0;   // the row that goes out
    const bool outc = (ne >> 1) >= H && (ne >> 1) < kStrW - H && 2 * I0 + ne < m;
    T *zo = zout + 2 * I0 + ne + static_cast<long>(m) * (2 * J0 + nj);
#pragma unroll 1
    for (int t = Js; t <= Je + C::kLast; t++, J++, Jo++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(PF - 1) : "memory");
        __syncthreads();
        fetch();
        // the row finished in the last step goes out
        if (Jo >= Js) {
            if (Jo >= J0 && Jo < J1) {
                if (outc && 2 * Jo + nj < n) *zo = nat[sz];
                zo += 2 * m;
            }
            sz = sz + W == RW ? 0 : sz + W;
        }
        if (J < Js || J >= Je) continue;
        T v[2];
#pragma unroll
        for (int q = 0; q < 2; q++) {
            p[q].zl = side[so + 32 * q];
            p[q].zr = side[so + 32 * q + 1];
            if constexpr (!kFive) {
                p[q].up0 = corner[su + 32 * q];
                p[q].up2 = corner[su + 32 * q + 1];
            }
            p[q].up1 = vert[su + 32 * q];
            p[q].zc = CEN ? own[so + 32 * q] : T(0);
        }
        if (pj && J == Js) {  // no step before this one: the cell's own even row
#pragma unroll
            for (int q = 0; q < 2; q++) {
                p[q].low1 = vert[so + 32 * q];
                if constexpr (!kFive) {
                    p[q].low0 = corner[so + 32 * q];
                    p[q].low2 = corner[so + 32 * q + 1];
                }
            }
        }
        if (inner && j > 0 && j < n - 1) {
#pragma unroll
            for (int q = 0; q < 2; q++) {
                const int x = 32 * q;
                if constexpr (kFive)
                    v[q] = p[q].mac(op, 1, true, true, true, true, false, own[so + x + 8 * RW], right[so + x],
                                    own[so + x + 12 * RW], above[so + x], own[so + x + 4 * RW]);
                else
                    v[q] = p[q].fem(op, own[so + x + 8 * RW], side[so + x + 8 * RW + 1], vert[su + x + 8 * RW],
                                    corner[su + x + 8 * RW + 1], own[so + x + 4 * RW]);
            }
        } else {
#pragma unroll
            for (int q = 0; q < 2; q++) {
                const int x = 32 * q, i = ci[q];
                const bool l = px || i > 0, r = px || i < m - 1, d = py || j > 0, u = py || j < n - 1;
                if constexpr (kFive) {
                    v[q] = p[q].mac(op, i, l, r, d, u, op.zpr && !px && i == m - 1, own[so + x + 8 * RW], right[so + x],
                                    own[so + x + 12 * RW], above[so + x], own[so + x + 4 * RW]);
                } else {
                    const T bv = own[so + x + 4 * RW], cdl = own[so + x + 8 * RW];
                    const T cdr = r ? side[so + x + 8 * RW + 1] : T(0), cul = u ? vert[su + x + 8 * RW] : T(0),
                            cur = r && u ? corner[su + x + 8 * RW + 1] : T(0);
                    if (i > 0 && i < m - 1 && j > 0 && j < n - 1) v[q] = p[q].fem(op, cdl, cdr, cul, cur, bv);
                    else v[q] = p[q].fem_edge(op, i, j, cdl, cdr, cul, cur, bv);
                }
            }
        }
        if (j < n) {
            if (col[0]) own[so] = v[0];
            if (col[1]) own[so + 32] = v[1];
        }
#pragma unroll
        for (int q = 0; q < 2; q++) {
            p[q].low0 = p[q].up0;
            p[q].low1 = p[q].up1;
            p[q].low2 = p[q].up2;
        }
        so = so + W == RW ? 0 : so + W;
        su = so;
        if (pj) su = so + W == RW ? 0 : so + W;
        j += 2;
        if (py && j >= n) j -= n;
    }
}

/** Chunks of a launch: one wave of the blocks that fit the chip. */
template <class Op, class T>
struct StreamGrid {
    dim3 grid;
    int chunk;
    StreamGrid(int m, int n) {
        const int per_sm = stream_per_sm<T>();
        const int cx = (m + 1) / 2, cy = (n + 1) / 2;
        const int strips = cdiv(cx, kStrW - 2 * StreamCfg<Op>::kHalo);
        int chunks = kB200SMs * per_sm / strips;
        if (chunks < 1) chunks = 1;
        chunk = cdiv(cy, chunks < cy ? chunks : cy);
        grid = dim3(strips, cdiv(cy, chunk));
    }
};

template <class Op, class T>
cudaError_t set_stream_attr() {
    return cudaFuncSetAttribute(k_smooth_stream<Op, T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                static_cast<int>(stream_elems<Op>() * sizeof(T)));
}

}  // namespace
}  // namespace incrmt
