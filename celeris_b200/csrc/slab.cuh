// One uniform-in-z layer as a two-port, without an eigendecomposition.
//
// Inside a layer the tangential fields follow g'' = -M g with g = W q^-1 (a - b) (the
// amplitude vector of e = kp g) and i h = g' (h = W (a + b)), M = ep2 kp - kk^T the
// matrix whose eigenvalues are q^2. A slab of thickness x therefore maps the two
// boundary values of g to the two of i h by functions of M alone:
//     i h(0) = -A g(0) + B g(x),   i h(x) = -B g(0) + A g(x),
//     A = Q cot(Q x),  B = Q / sin(Q x),  Q = M^(1/2),
// both even in Q, so no square root and no eigenvector is needed:
//   * C = cos(Q y), S = sin(Q y) / Q by their Taylor series in M y^2 (degree 11 in
//     groups of four, Paterson and Stockmeyer's scheme, Higham, Functions of Matrices,
//     sec. 4.2) at a y where the spectral radius of Q y is at most 2.2; up to two
//     double-angle steps (while no propagating mode reaches the zero of sin at pi);
//     B = S^-1, A = S^-1 C. A smaller y loses digits of the slow modes in I - M y^2 / 2
//     (radius 1.1: five times the error), a larger one to cosh of the evanescent ones;
//   * the slab is then put together with itself until it has the layer's thickness
//     (the doubling of layer theory): X = A^-1 B, B <- B X / 2, A <- A - B.
// Everything is matrix products and Gauss-Jordan solves, which run on the FP64 tensor
// cores; for a layer with real M (real permittivities, real in-plane wavevector) in
// real arithmetic. The evanescent orders decay in B multiplicatively, so nothing
// overflows however thick the layer is.
//
// A doubling is ill conditioned where A has a small eigenvalue, i.e. where a mode has
// cos(q x) ~ 0; max |X| ~ 1 / |cos(q x)| shows it, and the error of the result grows as
// eps max |X|. The last doublings (q x of a propagating mode reaches pi / 2 only there)
// are then left out: the slab of h / 2^r is used 2^r times in the caller's recursion
// from the substrate up, whose systems A + load are damped by the radiation and have
// no such poles. Each step of that recursion is a complex solve, so it costs about
// four times the real doubling it replaces.
//
// One thread block per matrix. Matrices are row-major in global memory (the working
// set of a block stays in L1 / L2); panels of the Gauss-Jordan steps live in registers.
#pragma once

#include "cblas_block.cuh"

namespace cb {
namespace slab {

constexpr int kMaxOrder = 512;        // largest order of the routines here
constexpr int kNB = 16;               // Gauss-Jordan panel width
// Row stride of the staged panel: 64 bytes mod 128, so that the fragment reads (16 bytes a
// lane, two rows per quarter-warp) do not conflict.
constexpr int kGs = 20, kGsReal = 24;
constexpr double kSpectral = 2.2;     // largest spectral radius of Q y of the series
constexpr double kPhaseMax = 2.5;     // largest q x of a propagating mode at S^-1 (sin q x = 0 at pi)
constexpr int kMaxAngles = 2;         // double-angle steps
constexpr int kMaxDoublings = 40;
constexpr unsigned kFlagPolls = 1u << 22;  // bound of a panel's wait for a column
// Largest max |X| of a doubling: beyond it the doublings stop where at most kMaxRest are left
// (1 << kMaxRest slabs), or the layer is given up. The error grows as eps |X|^2. Largest
// difference from the eigendecomposition over 6000 mirror-symmetric cells M = 1 .. 3 and 1000
// oblique cells M = 1: 6e-11 and 3.4e-9 at a limit of 1000, 2e-12 and 6e-11 at 100, 2e-12 and
// 6e-12 at 30, what is left being resonances of both. A stop costs complex solves that
// hold up the batch (limit 1000 -> 30: 64 cells M = 3 0.33 -> 0.40 ms, 512 rasterised cells 6.3 ->
// 10.7 ms with the buckets one after another, 6.0 side by side, 96 oblique cells M = 4 5.0 -> 7.2 ms, 64 stacks 2.5 -> 3.8 ms); that is the price of the digits.
constexpr int kMaxRest = 4;
constexpr double kGrowthLimit = 30.0;

// ---- scalars: double or complex ---------------------------------------------------------
__device__ __forceinline__ double zero_of(double) { return 0.0; }
__device__ __forceinline__ cplx zero_of(cplx) { return C(0.0, 0.0); }
__device__ __forceinline__ double mul(double a, double b) { return a * b; }
__device__ __forceinline__ cplx mul(cplx a, cplx b) { return cmul(a, b); }
__device__ __forceinline__ double fms(double a, double b, double c) { return fma(-a, b, c); }  // c - a b
__device__ __forceinline__ cplx fms(cplx a, cplx b, cplx c) { return cfms(a, b, c); }
__device__ __forceinline__ double add(double a, double b) { return a + b; }
__device__ __forceinline__ cplx add(cplx a, cplx b) { return cadd(a, b); }
__device__ __forceinline__ double sub(double a, double b) { return a - b; }
__device__ __forceinline__ cplx sub(cplx a, cplx b) { return csub(a, b); }
__device__ __forceinline__ double scale(double a, double s) { return a * s; }
__device__ __forceinline__ cplx scale(cplx a, double s) { return cscale(a, s); }
__device__ __forceinline__ double neg(double a) { return -a; }
__device__ __forceinline__ cplx neg(cplx a) { return cneg(a); }
__device__ __forceinline__ double recip(double a) { return 1.0 / a; }
__device__ __forceinline__ cplx recip(cplx a) {
    const double s = 1.0 / cnorm2(a);
    return C(a.x * s, -a.y * s);
}
__device__ __forceinline__ double size1(double a) { return fabs(a); }
__device__ __forceinline__ double size1(cplx a) { return cabs1(a); }
// A size whose high word (sign aside) ranks pivots: |a|, or |re| + |im|.
__device__ __forceinline__ double pivot_size(double a) { return a; }
__device__ __forceinline__ double pivot_size(cplx a) { return cabs1(a); }
__device__ __forceinline__ double real_part(double a) { return a; }
__device__ __forceinline__ double real_part(cplx a) { return a.x; }
__device__ __forceinline__ double plus_real(double a, double r) { return a + r; }
__device__ __forceinline__ cplx plus_real(cplx a, double r) { return C(a.x + r, a.y); }
__device__ __forceinline__ double shfl_of(double a, int l) { return __shfl_sync(0xffffffffu, a, l); }
__device__ __forceinline__ cplx shfl_of(cplx a, int l) {
    return C(__shfl_sync(0xffffffffu, a.x, l), __shfl_sync(0xffffffffu, a.y, l));
}
__device__ __forceinline__ cplx as_cplx(double a) { return C(a, 0.0); }
__device__ __forceinline__ cplx as_cplx(cplx a) { return a; }

// Accumulator of one 8 x 8 tile: the lane's two entries (rows g, columns 2 t, 2 t + 1).
template <bool CPLX>
struct Acc {
    double r[2], i[CPLX ? 2 : 1];
    __device__ void clear() {
        r[0] = r[1] = 0.0;
        i[0] = 0.0;
        if constexpr (CPLX) i[1] = 0.0;
    }
    __device__ void set(int h, double v) { r[h] = v; }
    __device__ void set(int h, cplx v) {
        r[h] = v.x;
        if constexpr (CPLX) i[h] = v.y;
    }
    __device__ __forceinline__ void get(int h, double& v) const { v = r[h]; }
    __device__ __forceinline__ void get(int h, cplx& v) const { v = C(r[h], CPLX ? i[CPLX ? h : 0] : 0.0); }
};
__device__ __forceinline__ void mma(Acc<false>& c, double a, double b) { dmma(c.r[0], c.r[1], a, b); }
__device__ __forceinline__ void mma(Acc<true>& c, double a, cplx b) {
    dmma(c.r[0], c.r[1], a, b.x);
    dmma(c.i[0], c.i[1], a, b.y);
}
__device__ __forceinline__ void mma(Acc<true>& c, cplx a, cplx b) {
    dmma(c.r[0], c.r[1], a.x, b.x);
    dmma(c.i[0], c.i[1], a.x, b.y);
    dmma(c.r[0], c.r[1], -a.y, b.y);
    dmma(c.i[0], c.i[1], a.y, b.x);
}
template <class TA, class TB>
struct Prod {
    typedef cplx type;
};
template <>
struct Prod<double, double> {
    typedef double type;
};

// ---- product: epi(row, col, (A B)[row][col]) for every entry, A m x k, B k x n -----------------
// Fragments come straight from memory (L1 holds the rows the warps share), so no
// staging and no barrier inside; what bounds the real products is L1's throughput
// (8-byte fragments: 56 % of L1 and 25 % of the tensor pipe busy at order 162), so they
// load 16 bytes per lane: two k of A at a time (the order of k within a step of 8
// is free) and two columns of B, and a warp's unit is 8 R x 8 W with the R, W that leave
// the least to the busiest warp (96 oblique cells of order 162: 7.0 -> 5.6 ms a call when doublings
// stopped at a growth of 1000, 30 today). Real operands have even leading dimensions and
// 16-byte-aligned bases. bmap (shared, may be NULL): row r of B is stored at row bmap[r].
template <class TB, int R, int W, class Epi>
__device__ __forceinline__ void gemm_units_real(int m, int n, int k, const double* A, int lda, const TB* B, int ldb,
                                                const int* bmap, const Epi& epi) {
    constexpr bool CP = sizeof(TB) == sizeof(cplx);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarp = blockDim.x >> 5;
    const int g = lane >> 2, t4 = lane & 3;
    const int rt = (m + 8 * R - 1) / (8 * R), units = rt * ((n + 8 * W - 1) / (8 * W));
    for (int u = warp; u < units; u += nwarp) {
        const int i0 = (u % rt) * (8 * R), j0 = (u / rt) * (8 * W);
        const double* ap[R];
#pragma unroll
        for (int r = 0; r < R; ++r) ap[r] = A + (size_t)min(i0 + 8 * r + g, m - 1) * lda + 2 * t4;
        Acc<CP> acc[R][W];
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
            for (int j = 0; j < W; ++j) acc[r][j].clear();
        // real B: columns j0 + 16 q + 2 g (+ 1) feed tiles 2 q (+ 1); complex B: column j0 + 8 j + g
        constexpr int NB = CP ? W : W / 2;
        int col[NB];
#pragma unroll
        for (int q = 0; q < NB; ++q)
            col[q] = CP ? min(j0 + 8 * q + g, n - 1) : min(j0 + 16 * q + 2 * g, (n - 1) & ~1);
        struct Step {
            double2 a[R], b[2][NB];
        };
        auto load = [&](int k0, Step& st) {
            const int kk = k0 + 2 * t4;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                double2 v = make_double2(0.0, 0.0);
                if (kk < k) {
                    v = *reinterpret_cast<const double2*>(ap[r] + k0);
                    if (kk + 1 >= k) v.y = 0.0;
                }
                st.a[r] = v;
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int kc = min(kk + h, k - 1);
                const TB* bp = B + (size_t)(bmap ? bmap[kc] : kc) * ldb;
#pragma unroll
                for (int q = 0; q < NB; ++q) st.b[h][q] = *reinterpret_cast<const double2*>(bp + col[q]);
            }
        };
        auto product = [&](const Step& st) {
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const double a = h == 0 ? st.a[r].x : st.a[r].y;
#pragma unroll
                    for (int q = 0; q < NB; ++q) {
                        if constexpr (CP) {
                            mma(acc[r][q], a, st.b[h][q]);
                        } else {
                            mma(acc[r][2 * q], a, st.b[h][q].x);
                            mma(acc[r][2 * q + 1], a, st.b[h][q].y);
                        }
                    }
                }
        };
        Step s0, s1;
        load(0, s0);
        int k0 = 0;
        for (; k0 + 8 < k; k0 += 16) {
            load(k0 + 8, s1);
            product(s0);
            if (k0 + 16 < k) load(k0 + 16, s0);
            product(s1);
        }
        if (k0 < k) product(s0);
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int row = i0 + 8 * r + g;
            if (row >= m) continue;
#pragma unroll
            for (int j = 0; j < W; ++j)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int c = CP ? j0 + 8 * j + 2 * t4 + h : j0 + 16 * (j >> 1) + 4 * t4 + 2 * h + (j & 1);
                    if (c < n) {
                        typename Prod<double, TB>::type v;
                        acc[r][j].get(h, v);
                        epi(row, c, v);
                    }
                }
        }
    }
}
// Complex A: units of 8 rows x 8 W columns, W in {1, 2, 4}.
template <class TA, class TB, int W, class Epi>
__device__ __forceinline__ void gemm_units(int m, int n, int k, const TA* A, int lda, const TB* B, int ldb,
                                           const int* bmap, const Epi& epi) {
    typedef typename Prod<TA, TB>::type TC;
    constexpr bool CP = sizeof(TC) == sizeof(cplx);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarp = blockDim.x >> 5;
    const int g = lane >> 2, t4 = lane & 3;
    const int rt = (m + 7) >> 3, units = rt * ((n + 8 * W - 1) / (8 * W));
    for (int u = warp; u < units; u += nwarp) {
        const int i0 = (u % rt) * 8, j0 = (u / rt) * (8 * W);
        const TA* ap = A + (size_t)min(i0 + g, m - 1) * lda;
        int col[W];
#pragma unroll
        for (int j = 0; j < W; ++j) col[j] = min(j0 + 8 * j + g, n - 1);
        Acc<CP> acc[W];
#pragma unroll
        for (int j = 0; j < W; ++j) acc[j].clear();
        auto load = [&](int k0, TA& a, TB (&b)[W]) {
            const int kk = k0 + t4, kc = min(kk, k - 1);
            a = ap[kc];
            if (kk >= k) a = zero_of(TA());
            const TB* bp = B + (size_t)(bmap ? bmap[kc] : kc) * ldb;
#pragma unroll
            for (int j = 0; j < W; ++j) b[j] = bp[col[j]];
        };
        TA a0, a1;
        TB b0[W], b1[W];
        load(0, a0, b0);
        int k0 = 0;
        for (; k0 + 4 < k; k0 += 8) {  // two steps per round, the next step's loads ahead of the products
            load(k0 + 4, a1, b1);
#pragma unroll
            for (int j = 0; j < W; ++j) mma(acc[j], a0, b0[j]);
            if (k0 + 8 < k) load(k0 + 8, a0, b0);
#pragma unroll
            for (int j = 0; j < W; ++j) mma(acc[j], a1, b1[j]);
        }
        if (k0 < k) {
#pragma unroll
            for (int j = 0; j < W; ++j) mma(acc[j], a0, b0[j]);
        }
        const int row = i0 + g;
        if (row < m) {
#pragma unroll
            for (int j = 0; j < W; ++j)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int c = j0 + 8 * j + 2 * t4 + h;
                    if (c < n) {
                        TC v;
                        acc[j].get(h, v);
                        epi(row, c, v);
                    }
                }
        }
    }
}
// Column width (in 8-column tiles) of the warps' units for `rt` row tiles and `ct` column tiles.
__device__ __forceinline__ int unit_width(int rt, int ct) {
    const int nwarp = blockDim.x >> 5;
    int best = 1, cost = 1 << 30;
#pragma unroll
    for (int w = 1; w <= 4; w *= 2) {
        const int rounds = (rt * ((ct + w - 1) / w) + nwarp - 1) / nwarp;
        const int c = rounds * (4 * w + 1);
        if (c <= cost) {
            cost = c;
            best = w;
        }
    }
    return best;
}
// Cost of the busiest warp with units of 8 r x 8 w: tensor work and fragment loads.
__device__ __forceinline__ int unit_cost(int m, int n, int r, int w) {
    const int units = ((m + 8 * r - 1) / (8 * r)) * ((n + 8 * w - 1) / (8 * w)), nwarp = blockDim.x >> 5;
    return ((units + nwarp - 1) / nwarp) * (2 * r * w + r + w);
}
template <class TB, class Epi>
__device__ void gemm(int m, int n, int k, const double* A, int lda, const TB* B, int ldb, const int* bmap,
                     const Epi& epi) {
    const int c12 = unit_cost(m, n, 1, 2), c14 = unit_cost(m, n, 1, 4), c22 = unit_cost(m, n, 2, 2),
              c24 = unit_cost(m, n, 2, 4);
    const int best = min(min(c12, c14), min(c22, c24));
    if (((m + 7) >> 3) * ((n + 7) >> 3) <= (int)(blockDim.x >> 5)) {  // one 8 x 8 tile per warp
        gemm_units<double, TB, 1>(m, n, k, A, lda, B, ldb, bmap, epi);
        return;
    }
    if (sizeof(TB) == sizeof(double) && best == c24) gemm_units_real<TB, 2, 4>(m, n, k, A, lda, B, ldb, bmap, epi);
    else if (best == c22 || best == c24) gemm_units_real<TB, 2, 2>(m, n, k, A, lda, B, ldb, bmap, epi);
    else if (best == c14) gemm_units_real<TB, 1, 4>(m, n, k, A, lda, B, ldb, bmap, epi);
    else gemm_units_real<TB, 1, 2>(m, n, k, A, lda, B, ldb, bmap, epi);
}
template <class Epi>
__device__ void gemm(int m, int n, int k, const cplx* A, int lda, const cplx* B, int ldb, const int* bmap,
                     const Epi& epi) {
    const int w = unit_width((m + 7) >> 3, (n + 7) >> 3);
    if (w == 4) gemm_units<cplx, cplx, 4>(m, n, k, A, lda, B, ldb, bmap, epi);
    else if (w == 2) gemm_units<cplx, cplx, 2>(m, n, k, A, lda, B, ldb, bmap, epi);
    else gemm_units<cplx, cplx, 1>(m, n, k, A, lda, B, ldb, bmap, epi);
}

// ---- Gauss-Jordan ------------------------------------------------------------------------
// Shared memory of the routines (dynamic): see carve().
struct Shared {
    cplx* pan;    // staged panel [n][kGs]; during a panel its columns [kNB][rows_of(n)]
    cplx* prow;   // staged pivot rows [kNB][chunk + pad]
    int* perm;    // [n] row that holds variable k
    int* pos;     // [n] variable of row r, -1 while it has none
    int* perm2;   // [n] a kept copy of perm
    int* flag;    // [kNB] of a panel's columns: 0, or 1 + the pivot's row, or -1 (no pivot)
    int* bad;     // set when a column had no pivot, or a warp's wait for one ran out
    double* red;  // [32]
    int chunk;    // columns staged at a time
    int lost;     // a warp whose waits for a column count as run out (tests; -1: none)
    long long* prof;  // optional clock64 sums: [0] panels, [1] updates of the other columns, [2] whole kernel
};
__host__ __device__ inline size_t pad16(size_t b) { return (b + 15) & ~size_t(15); }
// Rows the panel's lanes cover: 32 times a power of two.
__host__ __device__ inline int rows_of(int n) { return n <= 32 ? 32 : n <= 64 ? 64 : n <= 128 ? 128 : n <= 256 ? 256 : 512; }
// Columns of a staged chunk of pivot rows: as wide as 64 KB allows, and the whole
// augmented matrix when it is narrower.
__host__ __device__ inline int chunk_of(int n) {
    const int all = (2 * n + 31) & ~31;
    const int cap = n <= 256 ? 256 : 64;
    return all < cap ? all : cap;
}
__host__ __device__ inline size_t panel_elems(int n) {
    const size_t g = (size_t)n * kGs, c = (size_t)kNB * rows_of(n);
    return g > c ? g : c;
}
__host__ __device__ inline size_t shared_bytes(int n) {
    return panel_elems(n) * 16 + pad16((size_t)kNB * (chunk_of(n) + 4) * 16) + 3 * pad16((size_t)n * 4) + 64 + 16 + 256;
}
__device__ __forceinline__ Shared carve(unsigned char* p, int n) {
    Shared s;
    s.prof = nullptr;
    s.chunk = chunk_of(n);
    s.lost = -1;
    s.pan = reinterpret_cast<cplx*>(p);
    p += panel_elems(n) * 16;
    s.prow = reinterpret_cast<cplx*>(p);
    p += pad16((size_t)kNB * (s.chunk + 4) * 16);
    s.perm = reinterpret_cast<int*>(p);
    p += pad16((size_t)n * 4);
    s.pos = reinterpret_cast<int*>(p);
    p += pad16((size_t)n * 4);
    s.perm2 = reinterpret_cast<int*>(p);
    p += pad16((size_t)n * 4);
    s.flag = reinterpret_cast<int*>(p);
    p += 64;
    s.bad = reinterpret_cast<int*>(p);
    p += 16;
    s.red = reinterpret_cast<double*>(p);
    return s;
}
template <class T>
__device__ __forceinline__ T* as(cplx* p) {
    return reinterpret_cast<T*>(p);
}

// The larger of m and v, NaN if either is (fmax would drop it).
__device__ __forceinline__ double nan_max(double m, double v) { return v > m || v != v ? v : m; }
// Largest value over the block, the same in every thread; NaN if any is.
__device__ __forceinline__ double block_max(double v, double* red) {
    for (int o = 16; o > 0; o >>= 1) v = nan_max(v, __shfl_xor_sync(0xffffffffu, v, o));
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    double m = red[0];
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) m = nan_max(m, red[w]);
    return m;
}

// One panel of kb <= kNB columns (k0 ..) of the n-row matrix Wm, in registers of the
// first PW = kNB / CPW warps: lane l holds rows l + 32 r, warp w columns w + PW q. In-place
// Gauss-Jordan with partial pivoting over the rows that have no variable yet (rows are
// not moved: perm / pos record which row serves which variable). What bounds a panel is
// the chain from one pivot to the next, so a column is handed over without a barrier:
// its owner stores the raw column in a buffer of its own, finds the pivot with one warp
// reduction over the magnitudes' high words (the row in the low bits: a pivot within
// 0.1 % of the largest) and raises the column's flag with the row; every warp then
// forms the reciprocal itself. The owner of the next column brings that one up to date and
// hands it over before it touches its others. Cycles per column at 25 / 61 / 113 / 162
// rows, real: 646, 740, 950, 1396 (complex 865, 960, 1330, 2240); one column per warp
// behind block-wide barriers took 830, 1109, 1537, 2065 (1006, 1477, 2166, 2926). The
// finished panel G goes to s.pan (over the column buffers): the update of every other
// column is row <- row + G (old pivot rows), with the pivot rows themselves replaced
// (trailing()).
template <class T>
__host__ __device__ constexpr int panel_stride() {
    return sizeof(T) == sizeof(double) ? kGsReal : kGs;
}
__device__ __forceinline__ int wait_column(const int* flag) {
    const unsigned a = (unsigned)__cvta_generic_to_shared(flag);
    int v = 0;
    for (unsigned i = 0; i < kFlagPolls && v == 0; ++i)
        asm volatile("ld.acquire.cta.shared.s32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v == 0 ? -1 : v;
}
__device__ __forceinline__ void raise_column(int* flag, int v) {
    asm volatile("st.release.cta.shared.s32 [%0], %1;" ::"r"((unsigned)__cvta_generic_to_shared(flag)), "r"(v) : "memory");
}
template <int THREADS>
__device__ __forceinline__ void panel_barrier() {
    asm volatile("bar.sync 1, %0;" ::"n"(THREADS) : "memory");
}
template <class T, int RA, int CPW>
__device__ __noinline__ void panel(int n, int k0, int kb, const T* Wm, int ld, const Shared& s, unsigned& used) {
    constexpr int PW = kNB / CPW, nr = 32 * RA;
    constexpr unsigned kRow = kMaxOrder - 1;  // row bits of a pivot key
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp >= PW) return;
    T* col = as<T>(s.pan);  // [kNB][nr]
    int* flag = s.flag;
    int *perm = s.perm + k0, *pos = s.pos;
    T a[CPW][RA];
#pragma unroll
    for (int q = 0; q < CPW; ++q) {
        const int c = warp + PW * q;
#pragma unroll
        for (int r = 0; r < RA; ++r) {
            const int row = lane + 32 * r;
            a[q][r] = (c < kb && row < n) ? Wm[(size_t)row * ld + k0 + c] : zero_of(T());
        }
    }
    // row candidates: the sign and the row bits cleared from a magnitude's high word, all
    // of it once the row has a variable (or past the matrix)
    unsigned mask = used, keep[RA];
#pragma unroll
    for (int r = 0; r < RA; ++r) keep[r] = (lane + 32 * r < n && !((mask >> r) & 1u)) ? 0x7fffffffu & ~kRow : 0u;
    auto hand_over = [&](const T(&c)[RA], int j) {
        unsigned key = 0u;
#pragma unroll
        for (int r = 0; r < RA; ++r) {
            const int row = lane + 32 * r;
            col[j * nr + row] = c[r];
            key = max(key, ((unsigned)__double2hiint(pivot_size(c[r])) & keep[r]) | (unsigned)row);
        }
        key = __reduce_max_sync(0xffffffffu, key);
        // a warp reduction does not order memory: without this, lane 0's release would cover
        // its own rows of the column only
        __syncwarp();
        if (lane == 0) {
            const int p = (int)(key & kRow);
            // zero (or denormal), infinite and NaN pivots: the high word's exponent field
            const unsigned e = (key >> 20) & 0x7ffu;
            const bool none = e == 0u || e == 0x7ffu;
            raise_column(flag + j, none ? -1 : p + 1);
            if (!none) {  // else p may be a lane's row past the matrix
                perm[j] = p;
                pos[p] = k0 + j;
            }
        }
    };
    if (warp == 0) hand_over(a[0], 0);
    bool ok = warp != s.lost;
#pragma unroll
    for (int qo = 0; qo < CPW; ++qo) {
        if (!ok) break;
        for (int wo = 0; wo < PW; ++wo) {
            const int j = qo * PW + wo;
            if (j >= kb) break;
            const int got = wait_column(flag + j);
            if (got < 0) {
                ok = false;
                break;
            }
            const int p = got - 1, pl = p & 31, pr = p >> 5;
            const T* cj = col + j * nr;
            const T d = recip(cj[p]);
            if (lane == pl) mask |= 1u << pr;
#pragma unroll
            for (int r = 0; r < RA; ++r)
                if (lane == pl && r == pr) keep[r] = 0u;
            // column j + 1's slot in its owner: qo, or qo + 1 after the last warp
            const bool wrap = wo == PW - 1;
            const bool next = warp == (wrap ? 0 : wo + 1) && j + 1 < kb;
            auto update = [&](T(&c)[RA]) {
                T v = c[0];
#pragma unroll
                for (int r = 1; r < RA; ++r)
                    if (r == pr) v = c[r];
                v = mul(shfl_of(v, pl), d);  // the scaled pivot row's entry in this column
#pragma unroll
                for (int r = 0; r < RA; ++r) {
                    const T e = fms(cj[lane + 32 * r], v, c[r]);
                    c[r] = (lane == pl && r == pr) ? v : e;
                }
            };
            if (next) {
                if (!wrap) {
                    update(a[qo]);
                    hand_over(a[qo], j + 1);
                } else if (qo + 1 < CPW) {
                    update(a[qo + 1 < CPW ? qo + 1 : qo]);
                    hand_over(a[qo + 1 < CPW ? qo + 1 : qo], j + 1);
                }
            }
#pragma unroll
            for (int q = 0; q < CPW; ++q) {
                if (next && q == (wrap ? qo + 1 : qo)) continue;
                if (warp == wo && q == qo) {
#pragma unroll
                    for (int r = 0; r < RA; ++r) {
                        const T e = neg(mul(a[q][r], d));
                        a[q][r] = (lane == pl && r == pr) ? d : e;
                    }
                } else {
                    update(a[q]);
                }
            }
        }
    }
    used = mask;
    panel_barrier<PW * 32>();  // the column buffers are read; G overlays them
    if (!ok) {
        if (lane == 0) *s.bad = 1;  // any warp's: its columns of G are missing
        return;
    }
    T* pan = as<T>(s.pan);
#pragma unroll
    for (int q = 0; q < CPW; ++q)
#pragma unroll
        for (int r = 0; r < RA; ++r) {
            const int row = lane + 32 * r;
            if (row < n) pan[row * panel_stride<T>() + warp + PW * q] = a[q][r];  // zero in the columns past kb
        }
}

// Columns [c0, c0 + cn) of Wm after a panel: row i <- (pivot row of this panel ? 0 : row i) + G[i] . old
// pivot rows (staged in s.prow from c0). K = kNB, on the tensor cores.
template <class T, int W>
__device__ __forceinline__ void trailing_units(int n, int c0, int cn, T* Wm, int ld, const Shared& s, int k0, int ldp) {
    constexpr bool CP = sizeof(T) == sizeof(cplx);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarp = blockDim.x >> 5;
    const int g = lane >> 2, t4 = lane & 3;
    const T* pan = as<T>(s.pan);
    const T* pr = as<T>(s.prow);
    const int rt = (n + 7) >> 3, units = rt * ((cn + 8 * W - 1) / (8 * W));
    for (int u = warp; u < units; u += nwarp) {
        const int row = (u % rt) * 8 + g, j0 = (u / rt) * (8 * W);
        const int rowc = min(row, n - 1);
        const bool keep = row < n && s.pos[rowc] < k0;  // pos >= k0: a pivot row of this panel
        T* wrow = Wm + (size_t)rowc * ld + c0;
        Acc<CP> acc[W];
#pragma unroll
        for (int j = 0; j < W; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int c = j0 + 8 * j + 2 * t4 + h;
                acc[j].set(h, (keep && c < cn) ? wrow[c] : zero_of(T()));
            }
#pragma unroll
        for (int ks = 0; ks < kNB; ks += 4) {
            const T av = pan[rowc * kGs + ks + t4];
#pragma unroll
            for (int j = 0; j < W; ++j) mma(acc[j], av, pr[(ks + t4) * ldp + j0 + 8 * j + g]);
        }
        if (row < n) {
#pragma unroll
            for (int j = 0; j < W; ++j)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int c = j0 + 8 * j + 2 * t4 + h;
                    if (c < cn) {
                        T v;
                        acc[j].get(h, v);
                        wrow[c] = v;
                    }
                }
        }
    }
}
// The same in real arithmetic with 16-byte accesses throughout (36 instead of 16 shared and
// global accesses per 16 tensor instructions otherwise; 64 cells M = 3: 0.345 -> 0.333 ms a call when
// doublings stopped at a growth of 1000, 30 today): units of 8 R x 32, two k of G and two columns of the pivot rows
// and of Wm per access, as in gemm_units_real. c0 and ld are even.
template <int R>
__device__ __forceinline__ void trailing_units_real(int n, int c0, int cn, double* Wm, int ld, const Shared& s, int k0,
                                                    int ldp) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarp = blockDim.x >> 5;
    const int g = lane >> 2, t4 = lane & 3;
    const double* pan = as<double>(s.pan) + 2 * t4;
    const double* pr = as<double>(s.prow);
    const int rt = (n + 8 * R - 1) / (8 * R), units = rt * ((cn + 31) >> 5);
    for (int u = warp; u < units; u += nwarp) {
        const int i0 = (u % rt) * (8 * R), j0 = (u / rt) * 32;
        Acc<false> acc[R][4];
        double* wrow[R];
        const double* grow[R];
        bool live[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int row = i0 + 8 * r + g, rowc = min(row, n - 1);
            live[r] = row < n;
            const bool keep = live[r] && s.pos[rowc] < k0;  // pos >= k0: a pivot row of this panel
            wrow[r] = Wm + (size_t)rowc * ld + c0 + j0 + 4 * t4;
            grow[r] = pan + rowc * kGsReal;
#pragma unroll
            for (int q = 0; q < 2; ++q) {  // columns j0 + 16 q + 4 t4 .. + 3: tiles 2 q, 2 q + 1
                const int c = j0 + 16 * q + 4 * t4;
                double2 lo = make_double2(0.0, 0.0), hi = lo;
                if (keep && c < cn) lo = *reinterpret_cast<const double2*>(wrow[r] + 16 * q);
                if (keep && c + 2 < cn) hi = *reinterpret_cast<const double2*>(wrow[r] + 16 * q + 2);
                acc[r][2 * q].r[0] = lo.x;
                acc[r][2 * q + 1].r[0] = lo.y;
                acc[r][2 * q].r[1] = hi.x;
                acc[r][2 * q + 1].r[1] = hi.y;
            }
        }
#pragma unroll
        for (int ks = 0; ks < kNB; ks += 8) {
            double2 av[R], bv[2][2];
#pragma unroll
            for (int r = 0; r < R; ++r) av[r] = *reinterpret_cast<const double2*>(grow[r] + ks);
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int q = 0; q < 2; ++q)
                    bv[h][q] = *reinterpret_cast<const double2*>(pr + (ks + 2 * t4 + h) * ldp + j0 + 16 * q + 2 * g);
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const double a = h == 0 ? av[r].x : av[r].y;
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        mma(acc[r][2 * q], a, bv[h][q].x);
                        mma(acc[r][2 * q + 1], a, bv[h][q].y);
                    }
                }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (!live[r]) continue;
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int c = j0 + 16 * q + 4 * t4;
                if (c < cn)
                    *reinterpret_cast<double2*>(wrow[r] + 16 * q) =
                        make_double2(acc[r][2 * q].r[0], acc[r][2 * q + 1].r[0]);
                if (c + 2 < cn)
                    *reinterpret_cast<double2*>(wrow[r] + 16 * q + 2) =
                        make_double2(acc[r][2 * q].r[1], acc[r][2 * q + 1].r[1]);
            }
        }
    }
}

template <class T>
__device__ void trailing(int n, int c0, int c1, T* Wm, int ld, const Shared& s, int k0, int kb) {
    constexpr bool CP = sizeof(T) == sizeof(cplx);
    T* pr = as<T>(s.prow);
    const int cmax = CP ? s.chunk : 2 * s.chunk;  // staged columns
    for (int c = c0; c < c1; c += cmax) {
        const int cn = min(cmax, c1 - c);
        const int ldp = cmax + 2;  // fragment reads of the staged rows do not conflict
        for (int e = threadIdx.x; e < kNB * cn; e += blockDim.x) {
            const int l = e / cn, j = e - l * cn;
            pr[l * ldp + j] = l < kb ? Wm[(size_t)s.perm[k0 + l] * ld + c + j] : zero_of(T());
        }
        __syncthreads();
        if constexpr (!CP) {
            if (unit_cost(n, cn, 2, 4) < unit_cost(n, cn, 1, 4)) trailing_units_real<2>(n, c, cn, Wm, ld, s, k0, ldp);
            else trailing_units_real<1>(n, c, cn, Wm, ld, s, k0, ldp);
            __syncthreads();
            continue;
        }
        const int w = unit_width((n + 7) >> 3, (cn + 7) >> 3);
        if (w == 4) trailing_units<T, 4>(n, c, cn, Wm, ld, s, k0, ldp);
        else if (w == 2) trailing_units<T, 2>(n, c, cn, Wm, ld, s, k0, ldp);
        else trailing_units<T, 1>(n, c, cn, Wm, ld, s, k0, ldp);
        __syncthreads();
    }
}

// Gauss-Jordan on the n x ncol matrix Wm = [A | R] (A its first n columns, in real
// arithmetic R from the next even column, ld even): afterwards row
// s.perm[k] of the right part holds row k of A^-1 R. inverse: A's part becomes A^-1 in
// place, its entry (k, perm[l]) stored at (row perm[k], column l). Returns false (in
// every thread) at a zero or non-finite pivot. Starts and ends on a barrier.
template <class T>
__device__ bool gauss_jordan(int n, int ncol, T* Wm, int ld, bool inverse, const Shared& s) {
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x) s.pos[i] = -1;
    if (threadIdx.x < kNB) s.flag[threadIdx.x] = 0;
    if (threadIdx.x == 0) *s.bad = 0;
    __syncthreads();
    unsigned used = 0u;
    for (int k0 = 0; k0 < n; k0 += kNB) {
        const int kb = min(kNB, n - k0);
        const long long t0 = clock64();
        if (n <= 32) panel<T, 1, 2>(n, k0, kb, Wm, ld, s, used);
        else if (n <= 64) panel<T, 2, 2>(n, k0, kb, Wm, ld, s, used);
        else if (n <= 128) panel<T, 4, 2>(n, k0, kb, Wm, ld, s, used);
        else if (n <= 256) panel<T, 8, 2>(n, k0, kb, Wm, ld, s, used);
        else panel<T, 16, 1>(n, k0, kb, Wm, ld, s, used);
        __syncthreads();
        if (*s.bad) return false;
        if (threadIdx.x < kNB) s.flag[threadIdx.x] = 0;  // a barrier follows before the next panel
        const long long t1 = clock64();
        const int c1 = sizeof(T) == sizeof(double) ? (k0 + kb + 1) & ~1 : k0 + kb;
        if (inverse) {
            if (k0 > 0) trailing(n, 0, k0, Wm, ld, s, k0, kb);
            const T* pan = as<T>(s.pan);
            for (int e = threadIdx.x; e < n * kb; e += blockDim.x) {
                const int i = e / kb, j = e - i * kb;
                Wm[(size_t)i * ld + k0 + j] = pan[i * panel_stride<T>() + j];
            }
        }
        if (c1 < ncol) trailing(n, c1, ncol, Wm, ld, s, k0, kb);
        __syncthreads();
        if (s.prof && threadIdx.x == 0) {
            s.prof[0] += t1 - t0;
            s.prof[1] += clock64() - t1;
        }
    }
    return true;
}

// ---- the layer's two-port ------------------------------------------------------------------
// Work area of one matrix: kAreas buffers of order x ld_of(order) complex plus 12 order (the
// padding of q and e[0] takes right-hand-side columns; four vectors of two columns). In real
// arithmetic the same buffers hold doubles. Routines share buffers by lifetime:
//   two_port       e[2] M, w1 M^2 and then a B, e[0..1] [M^3 | M^4], p and q the series and
//                  [S | C], p then A | B, q the doublings' systems
//   slab_port      q [A + L | B], e[0] the load L and at last the incident system, e[1], e[2] the
//                  product of the slabs' X (A and B stay in p and w1)
constexpr int kAreas = 8;
// Leading dimension of the n x n matrices in the work area (real products load pairs).
__host__ __device__ inline int ld_of(int n) { return (n + 1) & ~1; }
__host__ __device__ inline size_t work_size(int n) { return (size_t)kAreas * n * ld_of(n) + 12 * (size_t)n; }
struct Work {
    cplx *w1, *p, *q, *v;  // p: 2 n^2, q: 2 n (n + 1); v: 8 n
    cplx* e[3];            // n^2 each, e[0]: n (n + 2)
};
__host__ __device__ inline size_t work_q(int n) { return 3 * (size_t)n * ld_of(n); }                        // q
__host__ __device__ inline size_t work_e(int n) { return 5 * (size_t)n * ld_of(n) + 2 * (size_t)n; }  // e[0]
__device__ __forceinline__ Work carve_work(cplx* base, int n) {
    const size_t nn = (size_t)n * ld_of(n);
    Work w;
    w.w1 = base;
    w.p = w.w1 + nn;
    w.q = base + work_q(n);
    w.e[0] = base + work_e(n);
    w.e[1] = w.e[0] + nn + 2 * (size_t)n;
    w.e[2] = w.e[1] + nn;
    w.v = w.e[2] + nn;
    return w;
}

// max |.|_inf (row sums of |re| + |im|) of an n x n matrix.
template <class T>
__device__ double norm_inf(int n, const T* A, int ld, double* red) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarp = blockDim.x >> 5;
    double best = 0.0;
    for (int i = warp; i < n; i += nwarp) {
        double t = 0.0;
        for (int j = lane; j < n; j += 32) t += size1(A[(size_t)i * ld + j]);
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        best = nan_max(best, t);
    }
    return block_max(best, red);
}

// max |re| + |im| of the entries (row i < n, column c0 + j, j < n).
template <class T>
__device__ double max_entry(int n, const T* A, int ld, int c0, double* red) {
    double best = 0.0;
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
        const int i = e / n, j = e - i * n;
        best = nan_max(best, size1(A[(size_t)i * ld + c0 + j]));
    }
    return block_max(best, red);
}

// A, B of the slab of thickness h / 2^*rest from M (n x n), *rest = 0 unless the last
// doublings are ill conditioned. In real arithmetic (T double) M's real part is used.
// qmax bounds the propagating modes' q. Returns false (in every thread) when S or an earlier
// doubling is ill conditioned too. A and B point into the work area (w.q and w.e free). M may lie in w.q.
template <class T>
__device__ __noinline__ bool two_port(int n, cplx* Mc, double h, double qmax, const Work& w, const Shared& s, T** Aout, T** Bout,
                                      int* rest) {
    // matrices of leading dimension ln; pairs [. | .] side by side, the right one from column ln
    const int tid = threadIdx.x, nt = blockDim.x, ln = ld_of(n), n2 = 2 * ln, nw = ln + n;
    T* M1 = as<T>(w.e[2]);
    for (int e = tid; e < n * n; e += nt) {
        if constexpr (sizeof(T) == sizeof(double)) M1[(e / n) * ln + e % n] = Mc[e].x;
        else M1[(e / n) * ln + e % n] = Mc[e];
    }
    T *M2 = as<T>(w.w1), *M34 = as<T>(w.e[0]), *P = as<T>(w.p), *Q = as<T>(w.q);
    T* A = P;
    T* B0 = P + (size_t)n * ln;
    __syncthreads();
    // M^2, then [M^3 | M^4] (side by side, ld 2 n)
    gemm(n, n, n, M1, ln, M1, ln, nullptr, [=](int r, int c, T v) { M2[(size_t)r * ln + c] = v; });
    __syncthreads();
    gemm(n, n, n, M2, ln, M1, ln, nullptr, [=](int r, int c, T v) { M34[(size_t)r * n2 + c] = v; });
    gemm(n, n, n, M2, ln, M2, ln, nullptr, [=](int r, int c, T v) { M34[(size_t)r * n2 + ln + c] = v; });
    __syncthreads();
    // spectral radius of Q: from ||M||, or ||M^2||, ||M^4|| (every power's root bounds it)
    const double b1 = norm_inf(n, M1, ln, s.red), b2 = norm_inf(n, M2, ln, s.red),
                 b4 = norm_inf(n, M34 + ln, n2, s.red);
    const double rho = sqrt(fmin(b1, fmin(sqrt(b2), sqrt(sqrt(b4)))));
    if (!isfinite(b1 + b2 + b4) || !(h > 0.0)) return false;
    int ns = 0;  // halvings of h
    double y = h;
    while (rho * y > kSpectral && ns < kMaxDoublings) {
        y *= 0.5;
        ++ns;
    }
    if (rho * y > kSpectral) return false;
    int angles = 0;
    double x = y;
    while (angles < min(kMaxAngles, ns) && 2.0 * qmax * x <= kPhaseMax) {
        x *= 2.0;
        ++angles;
    }
    ns -= angles;
    // S / y and C: sum_k (-M y^2)^k / (2k + 1)!, / (2k)!, k = 0 .. 11, as three groups in
    // M^4; [S | C] side by side
    const double y2 = y * y, y4 = y2 * y2, y6 = y4 * y2, y8 = y4 * y4;
    auto group = [=](int r, int c, double f0, double f1, double f2, double f3) {
        // f0 I + f1 M y^2 + f2 M^2 y^4 + f3 M^3 y^6
        T v = scale(M1[(size_t)r * ln + c], f1 * y2);
        v = add(v, scale(M2[(size_t)r * ln + c], f2 * y4));
        v = add(v, scale(M34[(size_t)r * n2 + c], f3 * y6));
        return r == c ? plus_real(v, f0) : v;
    };
    auto group_s = [=](int r, int c, int k) {
        return k == 0   ? group(r, c, 1.0, -1.0 / 6.0, 1.0 / 120.0, -1.0 / 5040.0)
               : k == 1 ? group(r, c, 1.0 / 362880.0, -1.0 / 39916800.0, 1.0 / 6227020800.0, -1.0 / 1307674368000.0)
                        : group(r, c, 1.0 / 355687428096000.0, -1.0 / 121645100408832000.0,
                                1.0 / 51090942171709440000.0, -1.0 / 25852016738884976640000.0);
    };
    auto group_c = [=](int r, int c, int k) {
        return k == 0   ? group(r, c, 1.0, -0.5, 1.0 / 24.0, -1.0 / 720.0)
               : k == 1 ? group(r, c, 1.0 / 40320.0, -1.0 / 3628800.0, 1.0 / 479001600.0, -1.0 / 87178291200.0)
                        : group(r, c, 1.0 / 20922789888000.0, -1.0 / 6402373705728000.0, 1.0 / 2432902008176640000.0,
                                -1.0 / 1124000727777607680000.0);
    };
    for (int e = tid; e < n * n; e += nt) {
        const int r = e / n, c = e - r * n;
        P[(size_t)r * n2 + c] = group_s(r, c, 2);
        P[(size_t)r * n2 + ln + c] = group_c(r, c, 2);
    }
    __syncthreads();
    // (column n of an odd order is padding: nothing reads what lands there)
    gemm(n, nw, n, M34 + ln, n2, P, n2, nullptr, [=](int r, int c, T v) {
        if (c >= n && c < ln) return;
        const T g = c < n ? group_s(r, c, 1) : group_c(r, c - ln, 1);
        Q[(size_t)r * n2 + c] = add(scale(v, y8), g);
    });
    __syncthreads();
    gemm(n, nw, n, M34 + ln, n2, Q, n2, nullptr, [=](int r, int c, T v) {
        if (c >= n && c < ln) return;
        const T g = add(scale(v, y8), c < n ? group_s(r, c, 0) : group_c(r, c - ln, 0));
        P[(size_t)r * n2 + c] = c < n ? scale(g, y) : g;
    });
    __syncthreads();
    // double angle: S(2y) = 2 C S, C(2y) = 2 C^2 - I
    T *X = P, *Xn = Q;
    for (int a = 0; a < angles; ++a) {
        gemm(n, nw, n, X + ln, n2, X, n2, nullptr, [=](int r, int c, T v) {
            const T d = scale(v, 2.0);
            Xn[(size_t)r * n2 + c] = c == r + ln ? plus_real(d, -1.0) : d;
        });
        __syncthreads();
        T* t = X;
        X = Xn;
        Xn = t;
    }
    if (X != Q) {
        for (size_t e = tid; e < (size_t)n * n2; e += nt) Q[e] = X[e];
        __syncthreads();
    }
    if (!gauss_jordan(n, nw, Q, n2, true, s)) return false;  // [S^-1 | S^-1 C]
    // qmax keeps every mode's q x below 2.5, where max |x S^-1| is at most 3.5 (4400 random cells);
    // a mode beyond it near sin(q x) = 0 would show as a doubling's does
    if (!(x * max_entry(n, Q, n2, 0, s.red) <= kGrowthLimit)) return false;
    for (int e = tid; e < n * n; e += nt) {
        const int k = e / n, c = e - k * n;
        const size_t row = (size_t)s.perm[k] * n2;
        B0[(size_t)k * ln + s.perm[c]] = Q[row + c];
        A[(size_t)k * ln + c] = Q[row + ln + c];
    }
    T *B = B0, *Bn = M2;
    *rest = 0;
    for (int i = 0; i < ns; ++i) {
        __syncthreads();
        for (int e = tid; e < n * n; e += nt) {
            const int r = e / n, c = e - r * n;
            Q[(size_t)r * n2 + c] = A[(size_t)r * ln + c];
            Q[(size_t)r * n2 + ln + c] = B[(size_t)r * ln + c];
        }
        // X = A^-1 B in the right half of Q (rows by s.perm)
        const bool ok = gauss_jordan(n, nw, Q, n2, false, s);
        const int left = ns - 1 - i;
        if (!ok || !(max_entry(n, Q, n2, ln, s.red) <= kGrowthLimit)) {  // NaN too
            if (left + 1 > kMaxRest) return false;
            *rest = left + 1;
            break;
        }
        gemm(n, n, n, B, ln, Q + ln, n2, s.perm, [=](int r, int c, T v) {
            const size_t e = (size_t)r * ln + c;
            const T b = scale(v, 0.5);
            Bn[e] = b;
            A[e] = sub(A[e], b);
        });
        T* t = B;
        B = Bn;
        Bn = t;
    }
    __syncthreads();
    *Aout = A;
    *Bout = B;
    return true;
}

}  // namespace slab
}  // namespace cb
