// Batched 2D vectorial RCWA on sm_100a (FP64 throughout).
//
// Reference: src/celeris/rcwa/rcwa2d.cpp:209-488 (solve_rcwa_2d), 147-205
// (shape_operators), 74-95 (rasterize_eps), src/celeris/design/metalens.cpp:
// 122-163 (library sweep), src/celeris/rcwa/eig.cpp (eig_general).
//
// One unit cell = one patterned layer between the incident and substrate
// half-spaces (the library-sweep stack). Cells are bucketed by (Mx, My, raster
// size, symmetry); a bucket runs as a fixed sequence of kernels with one CTA per cell or
// parity class:
//   rcwa_fourier_rect / rcwa_fourier_laurent  eps operators (analytic Li rule,
//                 or 4x4-supersampled raster -> centred DFT -> Laurent Toeplitz)
//                 and Einv (LU inverse for the Laurent path)
//                 (order basis)
//   rcwa_sym_ops  the same for the excited parity classes of a mirror-symmetric cell:
//                 their blocks of the eps operators, M = ep2 kp - kkT and kp
//   rcwa_slab     the layer as a two-port without an eigendecomposition (slab.cuh),
//                 then the amplitudes between the half-spaces
//   rcwa_sym_expand  class amplitudes into the order basis
//   rcwa_epilogue Poynting flux and order-0 field for each requested excitation
// Stacks run rcwa_slab per layer and rcwa_stack_port (one CTA per stack).
// Measured (one B200, whole calls, against the eigendecomposition's sequence below):
//   one M = 5 cell 4.7 -> 0.55 ms; 64 cells M = 3 0.98 -> 0.40 ms; 512 rasterised cells M = 3..7
//   37 -> 6.0 ms; 96 oblique cells M = 4 26 -> 7.2 ms; 64 two-layer stacks M = 3 15.6 -> 3.8 ms
//
// The eigendecomposition's sequence remains for what the two-port does not take (needs_qr)
// or flags (kInfoRedo), and for celeris_eig_general; it runs in the order basis, or on the
// class operators of a mirror-symmetric cell (hess, schur, vec, then rcwa_sym_smat):
//   rcwa_build_M  M = ep2 kp - kkT using the diagonal Kx, Ky (two N^3 GEMMs)
//   rcwa_hess     Householder reduction to Hessenberg form H = Q^H M Q (in
//                 shared memory for n <= 112, blocked compact-WY panels above)
//   rcwa_schur    multishift QR with aggressive early deflation: Schur form
//                 T = Z^H M Z (schur_aed.cuh)
//   rcwa_vec      triangular back substitution for the eigenvectors of T;
//                 W = Z X; q = branch(sqrt(lambda))
//   rcwa_smat1    A = kp W, T11/T12 of interface 0, S12 and u = T11^{-1} a0
//   rcwa_smat2    W^{-1}, A^{-1}, T11'/T12' of interface 1, B = T11' - D S12 T12',
//                 aN = B^{-1} D u, b0 = T12 u + S22 T12' aN
// Its algebra is that of the reference's grcwa recursion specialised to
// phi = I in the half-spaces and to the two excitation columns actually read
// (a0 has two non-zeros), so only 2 columns of the global S11/S21 are formed.
#include <cuda_runtime.h>
#include <math.h>

#include <atomic>
#include <cmath>

#include <algorithm>
#include <chrono>
#include <complex>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <tuple>
#include <vector>

#include "cblas_block.cuh"
#include "schur_aed.cuh"
#include "slab.cuh"
#include "slab_check.cuh"
#include "runtime.cuh"

namespace {

using namespace cb;
using celeris_rt::count_launch;
using celeris_rt::set_error;
using celeris_rt::Workspace;

constexpr double PI = 3.14159265358979323846;
constexpr int kRT = 256;            // threads per CTA
constexpr int kDbgSlots = 16;       // diagnostic counters per cell
constexpr int kSmemEigMaxN = 116;   // Hessenberg reduction in shared memory up to this n ((n^2 + 2n) 16 B <= 227 KB)

struct CellDev {
    double omega;  // k0 = 2 pi / lambda (c = 1 units, omega = k0)
    double px, py, h, theta;
    double fill_x, fill_y, shape_param, rot;
    cplx kx0, ky0;
    cplx eps_p, eps_b;
    cplx n_inc, n_sub;
    cplx ex0, ey0;  // excitation of result slot 0 (batch: X = (1, 0))
    int shape, nexc;
    int real_mat;  // M is real in exact arithmetic (real permittivities and in-plane wavevector)
    int pad1;
};

struct Bucket {
    int Mx, My, N, n, ng, ncell;
    const CellDev* cells;
    cplx *H, *Z, *X, *W, *A, *T11, *T11lu, *T12, *S12;
    cplx *Einv, *Exx, *Eyy;
    cplx* q1;
    int* piv;
    cplx* vec;  // per cell [10n]: aN_X, aN_Y, b0_X, b0_Y | x [n x 2] | y [n x 2] | z [n x 2]
    int* info;
    celeris_rcwa_result* res;  // per cell: nexc results
    size_t s_nn, s_ns, s_NN, s_n;
    const cplx* phx;  // [(4Mx+1) x ng] centred DFT phase table (x)
    const cplx* phy;  // [(4My+1) x ng]
    const cplx* pcx;  // class path: [(2Mx+1) x (ng+1)] prefix sums of phx (there phx, phy hold m >= 0)
    cplx* G1;         // class path, per cell s_g1: the raster's row transform, or the 1D inverses
    size_t s_g1;
    long long* dbg;   // optional per-cell counters, kDbgSlots each (CELERIS_RCWA_STAGE_CLOCKS=1), else NULL
    double* ord;      // optional per-order efficiencies: per cell and excitation [N][2] = (de_t, de_r), else NULL
    // mirror-symmetric cells (sym != 0): the layer problem in its excited parity
    // classes
    int sym;         // 0: full path; 1: both excited classes; 2: also C4-symmetric (one class)
    int ncls, cls0;  // excited classes solved per cell (2, or 1 = class 1 only) and the first one
    double sym_tol;  // largest asymmetry of M (relative to max |M|) the class split accepts
    int m;           // order of a class
    // per solved class (matrix ncls * cell + class): M and kp in the class basis,
    // and the amplitudes aN | b0 (2 m)
    cplx *cM, *cKp, *cvec;
    // QR path in the classes: eigen-stage buffers (m^2 each), q and the eigensolve's info
    cplx *sZ, *sX, *sW, *sA, *sq;
    int* sinfo;
    // the layer two-port (slab.cuh): work area of a full-order cell (s_w complex), kp. The
    // Fourier operators (s_NN = s_w) and the scratch of their LU lie in parts of the work area
    // that the two-port has not reached when they are read
    cplx *slab, *Kp, *lu;
    size_t s_w;
    // layers of a stack: A, B and kp of cell i go to slot lslot[i] (s_nn each; no Kp)
    cplx *lA, *lB, *lK;
    const int* lslot;
    int* lrest;  // log2 of the slabs (A, B) the layer consists of
};

__device__ __forceinline__ cplx* at(cplx* base, size_t stride, int c) { return base + stride * c; }

// Mirror-symmetric cells (Bucket::sym != 0): per-cell info code of a cell found
// not symmetric to the tolerance, which is solved again by the full path.
constexpr int kInfoAsym = 1 << 29;
// A cell whose two-port was ill conditioned (slab.cuh), which is solved again
// through the eigendecomposition.
constexpr int kInfoRedo = 1 << 28;

// Parity classes under the two mirrors p -> -p, q -> -q.
// class c: 0 = (+,+), 1 = (-,-), 2 = (+,-), 3 = (-,+)
__host__ __device__ __forceinline__ int sym_class_a(int c) { return (c == 0 || c == 2) ? 1 : -1; }
__host__ __device__ __forceinline__ int sym_class_b(int c) { return (c == 0 || c == 3) ? 1 : -1; }
__host__ __device__ __forceinline__ int sym_count(int M, int parity) { return parity > 0 ? M + 1 : M; }

__device__ __forceinline__ void order_pq(const Bucket& b, int i, int& p, int& q) {
    const int ny = 2 * b.My + 1;
    p = i / ny - b.Mx;
    q = i % ny - b.My;
}
__device__ __forceinline__ cplx kx_of(const Bucket& b, const CellDev& c, int i) {
    int p, q;
    order_pq(b, i, p, q);
    return csub(c.kx0, C(2.0 * PI * (double)p / c.px, 0.0));  // rcwa2d.cpp:240
}
__device__ __forceinline__ cplx ky_of(const Bucket& b, const CellDev& c, int i) {
    int p, q;
    order_pq(b, i, p, q);
    return csub(c.ky0, C(2.0 * PI * (double)q / c.py, 0.0));  // rcwa2d.cpp:241
}
__device__ __forceinline__ double rect1d(int m, double fill) {
    return m == 0 ? fill : sin(PI * m * fill) / (PI * m);  // rcwa2d.cpp:108-110
}
// kz of a homogeneous region (rcwa2d.cpp:259-261): grazing guard, then branch
__device__ __forceinline__ cplx kz_uniform(cplx er, double omega, cplx kx, cplx ky) {
    cplx v = csub(csub(cscale(er, omega * omega), cmul(kx, kx)), cmul(ky, ky));
    cplx kz = csqrt_p(v);
    if (cabs(kz) < 1e-8) kz = C(0.0, 1e-8);
    if (kz.y < 0.0) kz = cneg(kz);
    return kz;
}
// kp block of a homogeneous region for order i (rcwa2d.cpp:265-269)
__device__ __forceinline__ void kp_uniform(cplx ier, double omega, cplx kx, cplx ky, cplx& a, cplx& b, cplx& c,
                                           cplx& d) {
    const cplx w2 = C(omega * omega, 0.0);
    a = csub(w2, cmul(ier, cmul(ky, ky)));
    b = cmul(ier, cmul(ky, kx));
    c = cmul(ier, cmul(kx, ky));
    d = csub(w2, cmul(ier, cmul(kx, kx)));
}

// ---- Fourier operators: analytic rectangle (Li inverse rule) ------------------
// dynamic smem: hx [nx*nx] | ax [nx*nx] | hy [ny*ny] | ay [ny*ny]
__global__ void __launch_bounds__(kRT) rcwa_fourier_rect(Bucket b) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int pv[32];
    __shared__ RedScratch rs;
    const int cell = blockIdx.x;
    const CellDev c = b.cells[cell];
    const int nx = 2 * b.Mx + 1, ny = 2 * b.My + 1, N = b.N;
    cplx* hx = reinterpret_cast<cplx*>(smem);
    cplx* ax = hx + nx * nx;
    cplx* hy = ax + nx * nx;
    cplx* ay = hy + ny * ny;
    cplx* stg = ay + ny * ny;  // LU staging: 2 * max(nx, ny)
    const int tid = threadIdx.x, nt = blockDim.x;
    const cplx ep = c.eps_p, eb = c.eps_b;
    const cplx ipe = cinv(ep), ibe = cinv(eb);
    const cplx dI = csub(ipe, ibe);
    // Hx, Hy: in-band 1D reciprocal Toeplitz (rcwa2d.cpp:299-303, 317-321)
    for (int e = tid; e < nx * nx; e += nt) {
        const int a = e / nx, bb = e % nx;
        cplx v = cscale(dI, rect1d(a - bb, c.fill_x));
        if (a == bb) v = cadd(v, ibe);
        hx[e] = v;
        ax[e] = C(a == bb ? 1.0 : 0.0, 0.0);
    }
    for (int e = tid; e < ny * ny; e += nt) {
        const int a = e / ny, bb = e % ny;
        cplx v = cscale(dI, rect1d(a - bb, c.fill_y));
        if (a == bb) v = cadd(v, ibe);
        hy[e] = v;
        ay[e] = C(a == bb ? 1.0 : 0.0, 0.0);
    }
    __syncthreads();
    blk_lu(nx, hx, nx, pv, &rs, stg);
    blk_lu_solve(nx, hx, nx, pv, nx, ax, nx, stg);  // ax = Hx^{-1}
    blk_lu(ny, hy, ny, pv, &rs, stg);
    blk_lu_solve(ny, hy, ny, pv, ny, ay, ny, stg);  // ay = Hy^{-1}
    cplx* Einv = at(b.Einv, b.s_NN, cell);
    cplx* Exx = at(b.Exx, b.s_NN, cell);
    cplx* Eyy = at(b.Eyy, b.s_NN, cell);
    for (int e = tid; e < N * N; e += nt) {
        const int r = e / N, col = e % N;
        int p, q, pp, qq;
        order_pq(b, r, p, q);
        order_pq(b, col, pp, qq);
        const double sx = rect1d(p - pp, c.fill_x), sy = rect1d(q - qq, c.fill_y);
        // (1/eps)_{pq} (rcwa2d.cpp:25-35, 288-295)
        cplx ei = cscale(dI, sx * sy);
        if (p == pp && q == qq) ei = cadd(ei, ibe);
        Einv[e] = ei;
        // Exx (rcwa2d.cpp:305-315): inverse rule in x, Laurent in y
        cplx vx = cscale(ax[(p + b.Mx) * nx + (pp + b.Mx)], sy);
        if (p == pp) vx = cadd(vx, cscale(eb, (q == qq ? 1.0 : 0.0) - sy));
        Exx[e] = vx;
        // Eyy (rcwa2d.cpp:323-333)
        cplx vy = cscale(ay[(q + b.My) * ny + (qq + b.My)], sx);
        if (q == qq) vy = cadd(vy, cscale(eb, (p == pp ? 1.0 : 0.0) - sx));
        Eyy[e] = vy;
    }
}

// ---- Fourier operators: rasterised shape, Laurent rule --------------------------
__device__ bool inside_shape(const CellDev& c, double xf, double yf) {
    if (c.rot != 0.0) {  // rcwa2d.cpp:41-47
        const double co = cos(c.rot), si = sin(c.rot);
        const double xr = co * xf + si * yf;
        const double yr = -si * xf + co * yf;
        xf = xr;
        yf = yr;
    }
    const double ax = c.fill_x * 0.5, ay = c.fill_y * 0.5;
    switch (c.shape) {
        case CELERIS_SHAPE_RECT:
            return fabs(xf) <= ax && fabs(yf) <= ay;
        case CELERIS_SHAPE_ELLIPSE: {
            if (ax <= 0.0 || ay <= 0.0) return false;
            const double u = xf / ax, v = yf / ay;
            return u * u + v * v <= 1.0;
        }
        case CELERIS_SHAPE_CROSS: {
            const double hx = ax * c.shape_param, hy = ay * c.shape_param;
            const bool vbar = fabs(xf) <= hx && fabs(yf) <= ay;
            const bool hbar = fabs(yf) <= hy && fabs(xf) <= ax;
            return vbar || hbar;
        }
        case CELERIS_SHAPE_RING: {
            if (ax <= 0.0 || ay <= 0.0) return false;
            const double u = xf / ax, v = yf / ay;
            const double r2 = u * u + v * v;
            const double ri = c.shape_param;
            return r2 <= 1.0 && r2 >= ri * ri;
        }
    }
    return false;
}

// phase tables: ph[(m + mmax) * ng + i] = exp(-2 pi i m xf_i) / ng, xf = (i+0.5)/ng - 0.5
__global__ void rcwa_phase_table(int ng, int mmax, cplx* ph) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (2 * mmax + 1) * ng) return;
    const int m = e / ng - mmax, i = e % ng;
    const double xf = (i + 0.5) / ng - 0.5;
    double s, co;
    sincos(-2.0 * PI * m * xf, &s, &co);
    ph[e] = C(co / ng, s / ng);
}

// Rows of G1 in shared memory: at least 4, so that the per-axis sample tables
// of the raster (2 x 4 ng doubles) fit in the same region.
__host__ __device__ __forceinline__ int laurent_g1_rows(int Mx) { return 4 * Mx + 1 > 4 ? 4 * Mx + 1 : 4; }

// The sample coordinate (rcwa2d.cpp:88-89) of subsample s of pixel i.
__device__ __forceinline__ double raster_coord(int i, int s, int ng) { return (i + (s + 0.5) / 4) / ng - 0.5; }

// dynamic smem: G1 [laurent_g1_rows(Mx) * ng] | Ge [(4Mx+1)(4My+1)] | counts [ng*ng] u8,
// counts stored column-major (cnt[ix * ng + iy]) so that the row sums of G1 read
// consecutive bytes across a warp.
__global__ void __launch_bounds__(kRT) rcwa_fourier_laurent(Bucket b) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ RedScratch rs;
    const int cell = blockIdx.x;
    const CellDev c = b.cells[cell];
    const int ng = b.ng, N = b.N;
    const int mx4 = 4 * b.Mx + 1, my4 = 4 * b.My + 1;
    const int tid = threadIdx.x, nt = blockDim.x;
    cplx* G1 = reinterpret_cast<cplx*>(smem);
    cplx* Ge = G1 + (size_t)laurent_g1_rows(b.Mx) * ng;
    unsigned char* cnt = reinterpret_cast<unsigned char*>(Ge + (size_t)mx4 * my4);
    // 4x4 supersampled inside counts (rcwa2d.cpp:74-95). Unrotated, every shape
    // test factors into per-axis terms: the sample coordinates (or their scaled
    // squares) are tabulated once per axis in the G1 region, and each of a
    // pixel's 16 samples combines one entry of each table with the reference's
    // own roundings (u*u and v*v rounded separately, then added).
    const double ax = c.fill_x * 0.5, ay = c.fill_y * 0.5;
    const bool round_shape = c.shape == CELERIS_SHAPE_ELLIPSE || c.shape == CELERIS_SHAPE_RING;
    if (c.rot != 0.0 || (round_shape && (ax <= 0.0 || ay <= 0.0))) {
        for (int e = tid; e < ng * ng; e += nt) {
            const int ix = e / ng, iy = e % ng;
            int hit = 0;
            for (int sy = 0; sy < 4; ++sy)
                for (int sx = 0; sx < 4; ++sx)
                    if (inside_shape(c, raster_coord(ix, sx, ng), raster_coord(iy, sy, ng))) ++hit;
            cnt[e] = (unsigned char)hit;
        }
    } else {
        double* tx = reinterpret_cast<double*>(G1);
        double* ty = tx + 4 * ng;
        const double hx = ax * c.shape_param, hy = ay * c.shape_param;
        for (int t = tid; t < 4 * ng; t += nt) {
            const double xf = raster_coord(t >> 2, t & 3, ng), yf = xf;  // square raster: one coordinate set
            if (round_shape) {
                const double u = xf / ax, v = yf / ay;
                tx[t] = __dmul_rn(u, u);
                ty[t] = __dmul_rn(v, v);
            } else {  // bit 0: within the main half-width, bit 1: within the cross arm's
                tx[t] = (fabs(xf) <= ax ? 1.0 : 0.0) + (fabs(xf) <= hx ? 2.0 : 0.0);
                ty[t] = (fabs(yf) <= ay ? 1.0 : 0.0) + (fabs(yf) <= hy ? 2.0 : 0.0);
            }
        }
        __syncthreads();
        const double ri2 = __dmul_rn(c.shape_param, c.shape_param);
        for (int e = tid; e < ng * ng; e += nt) {
            const int ix = e / ng, iy = e % ng;
            double X[4], Y[4];
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                X[s] = tx[4 * ix + s];
                Y[s] = ty[4 * iy + s];
            }
            int hit = 0;
#pragma unroll
            for (int sy = 0; sy < 4; ++sy)
#pragma unroll
                for (int sx = 0; sx < 4; ++sx) {
                    bool in;
                    if (round_shape) {
                        const double r2 = __dadd_rn(X[sx], Y[sy]);
                        in = r2 <= 1.0 && (c.shape == CELERIS_SHAPE_ELLIPSE || r2 >= ri2);
                    } else {
                        const int bx = (int)X[sx], by = (int)Y[sy];
                        in = c.shape == CELERIS_SHAPE_RECT ? ((bx & by & 1) != 0)
                                                           : (((bx >> 1) & by & 1) != 0 || ((by >> 1) & bx & 1) != 0);
                    }
                    hit += in ? 1 : 0;
                }
            cnt[e] = (unsigned char)hit;
        }
        __syncthreads();  // the tables are dead: G1 overwrites them
    }
    __syncthreads();
    const cplx dE = csub(c.eps_p, c.eps_b);
    // G1[dp][iy] = sum_ix eps[iy][ix] PX[dp][ix]   (rcwa2d.cpp:170-177); four
    // rows dp per thread share the raster reads and give four independent chains
    for (int e = tid; e < ((mx4 + 3) >> 2) * ng; e += nt) {
        const int dp0 = 4 * (e / ng), iy = e % ng;
        const int nd = min(4, mx4 - dp0);
        cplx s[4] = {C(0.0, 0.0), C(0.0, 0.0), C(0.0, 0.0), C(0.0, 0.0)};
        for (int ix = 0; ix < ng; ++ix) {
            const cplx eps = cadd(c.eps_b, cscale(dE, cnt[ix * ng + iy] / 16.0));
#pragma unroll
            for (int d = 0; d < 4; ++d)
                if (d < nd) s[d] = cfma(eps, b.phx[(size_t)(dp0 + d) * ng + ix], s[d]);
        }
        for (int d = 0; d < nd; ++d) G1[(size_t)(dp0 + d) * ng + iy] = s[d];
    }
    __syncthreads();
    // Ge[dp][dq] = sum_iy G1[dp][iy] PY[dq][iy]   (rcwa2d.cpp:179-185)
    for (int e = tid; e < mx4 * my4; e += nt) {
        const int dpi = e / my4, dqi = e % my4;
        const cplx* ph = b.phy + (size_t)dqi * ng;
        cplx s = C(0.0, 0.0);
        for (int iy = 0; iy < ng; ++iy) s = cfma(G1[dpi * ng + iy], ph[iy], s);
        Ge[e] = s;
    }
    __syncthreads();
    // Laurent Toeplitz (rcwa2d.cpp:191-198); Exx = Eyy = epsT
    cplx* Exx = at(b.Exx, b.s_NN, cell);
    cplx* lu = b.lu ? at(b.lu, b.s_w, cell) : at(b.H, b.s_nn, cell);  // scratch for the LU of epsT
    cplx* Einv = at(b.Einv, b.s_NN, cell);
    for (int e = tid; e < N * N; e += nt) {
        const int r = e / N, col = e % N;
        int p, q, pp, qq;
        order_pq(b, r, p, q);
        order_pq(b, col, pp, qq);
        const cplx v = Ge[(p - pp + 2 * b.Mx) * my4 + (q - qq + 2 * b.My)];
        Exx[e] = v;
        lu[e] = v;
        Einv[e] = C(r == col ? 1.0 : 0.0, 0.0);
    }
    __syncthreads();
    // the raster, G1 and Ge are dead: the LU staging and GEMM tiles overlay them
    cplx* stg = reinterpret_cast<cplx*>(smem);
    GemmSmem* gs = reinterpret_cast<GemmSmem*>(stg + 2 * N + LNB * LNB);
    int* piv = b.piv + b.s_n * cell;
    const int info = blk_lu_blocked(N, lu, N, piv, &rs, stg, gs);
    if (info != 0 && tid == 0 && b.info[cell] == 0) b.info[cell] = -info;  // keep an earlier stage's code
    blk_lu_solve_blocked(N, lu, N, piv, N, Einv, N, stg, gs);  // Einv = epsT^{-1} (rcwa2d.cpp:203)
}

// ---- M = ep2 kp - kkT -------------------------------------------------------------
__global__ void __launch_bounds__(kRT) rcwa_build_M(Bucket b, int laurent) {
    __shared__ GemmSmem gs;
    const int cell = blockIdx.x;
    const CellDev c = b.cells[cell];
    const int N = b.N, n = b.n;
    const int tid = threadIdx.x, nt = blockDim.x;
    const cplx* Einv = at(b.Einv, b.s_NN, cell);
    const cplx* Exx = at(b.Exx, b.s_NN, cell);
    const cplx* Eyy = laurent ? Exx : at(b.Eyy, b.s_NN, cell);
    cplx* tmp = at(b.Z, b.s_nn, cell);  // [2N x N]: Eyy diag(-ky) ; Exx diag(kx)
    cplx* Y = at(b.X, b.s_nn, cell);    // [2N x N]: Ytop ; Ybot
    for (int e = tid; e < N * N; e += nt) {
        const int col = e % N;
        tmp[e] = cmul(Eyy[e], cneg(ky_of(b, c, col)));
        tmp[N * N + e] = cmul(Exx[e], kx_of(b, c, col));
    }
    blk_gemm(2 * N, N, N, C(1.0, 0.0), tmp, N, Einv, N, C(0.0, 0.0), Y, N, &gs);
    cplx* H = at(b.H, b.s_nn, cell);
    const double w2 = c.omega * c.omega;
    for (int e = tid; e < n * n; e += nt) {
        const int i = e / n, j = e % n;
        cplx v;
        if (i < N && j < N) {
            v = cfma(Y[i * N + j], ky_of(b, c, j), cscale(Eyy[i * N + j], w2));
            if (i == j) v = csub(v, cmul(kx_of(b, c, i), kx_of(b, c, i)));
        } else if (i < N) {
            const int m = j - N;
            v = cneg(cmul(Y[i * N + m], kx_of(b, c, m)));
            if (i == m) v = csub(v, cmul(kx_of(b, c, i), ky_of(b, c, i)));
        } else if (j < N) {
            const int l = i - N;
            v = cmul(Y[(N + l) * N + j], ky_of(b, c, j));
            if (l == j) v = csub(v, cmul(ky_of(b, c, l), kx_of(b, c, l)));
        } else {
            const int l = i - N, m = j - N;
            v = cfms(Y[(N + l) * N + m], kx_of(b, c, m), cscale(Exx[l * N + m], w2));
            if (l == m) v = csub(v, cmul(ky_of(b, c, l), ky_of(b, c, l)));
        }
        H[e] = v;
    }
}

// ---- eigensolve -----------------------------------------------------------------------
// Three kernels so that each gets its own register budget (the bulge chase
// keeps 16-element row/column segments in registers). SMEM variants (n <= 112)
// stage H in shared memory for the duration of the kernel.
// dynamic smem: SMEM: H [n*n] | v [n] | w [n] (rank-1 updates on the shared
// copy); otherwise the staging of blk_hessenberg_blocked (scratch in X, which
// is free until the eigenvectors).
// The shared-memory variant may run 512 threads: for the larger orders its
// shared block leaves one CTA per SM, and the column steps are latency-bound.
constexpr int kHessBigThreads = 512;
template <bool SMEM>
__global__ void __launch_bounds__(SMEM ? kHessBigThreads : kRT) rcwa_hess(Bucket b) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ RedScratch rs;
    const int cell = blockIdx.x;
    const int n = b.n;
    const int tid = threadIdx.x, nt = blockDim.x;
    cplx* Hg = at(b.H, b.s_nn, cell);
    if constexpr (SMEM) {
        // reduce H in shared memory recording the reflectors in X (free until
        // the eigenvectors), write H back, then form Z = Q in the same shared
        // buffer
        cplx* H = reinterpret_cast<cplx*>(smem);
        cplx* v = H + (size_t)n * n;
        cplx* refl = at(b.X, b.s_nn, cell);
        for (int e = tid; e < n * n; e += nt) H[e] = Hg[e];
        __syncthreads();
        blk_hessenberg_refl(n, H, n, refl, v, v + n, &rs);
        __syncthreads();
        for (int e = tid; e < n * n; e += nt) Hg[e] = H[e];
        __syncthreads();
        blk_form_q(n, H, n, refl, v, v + n);
        __syncthreads();
        cplx* Zg = at(b.Z, b.s_nn, cell);
        for (int e = tid; e < n * n; e += nt) Zg[e] = H[e];
    } else {
        __shared__ GemmSmem gs;
        blk_hessenberg_blocked(n, Hg, n, at(b.Z, b.s_nn, cell), n, at(b.X, b.s_nn, cell),
                               reinterpret_cast<cplx*>(smem), &rs, &gs,
                               b.dbg ? b.dbg + kDbgSlots * (size_t)cell + 9 : nullptr);
    }
}

// Schur form by multishift QR with aggressive early deflation (schur_aed.cuh).
// dynamic smem: AedShared.
// QR iteration cap for failure-path tests (0: the solver's own cap); set by
// celeris_debug_qr_iteration_cap.
__device__ int g_qr_iter_cap;

__global__ void __launch_bounds__(kSchurThreads, 2) rcwa_schur(Bucket b) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int cell = blockIdx.x;
    const int n = b.n;
    const int tid = threadIdx.x, nt = blockDim.x;
    cplx* H = at(b.H, b.s_nn, cell);
    AedShared* sh = reinterpret_cast<AedShared*>(smem);
    const int info = blk_schur_aed(n, H, n, at(b.Z, b.s_nn, cell), n, sh,
                                   b.dbg ? b.dbg + kDbgSlots * (size_t)cell : nullptr, g_qr_iter_cap);
    if (tid == 0) {
        if (info != 0) b.info[cell] = info;
        if (b.dbg) b.dbg[kDbgSlots * (size_t)cell + 6] = sh->nsweep;
    }
    // eigenvalues -> q = branch(sqrt(lambda)) (rcwa2d.cpp:364)
    cplx* q1 = at(b.q1, b.s_n, cell);
    for (int i = tid; i < n; i += nt) {
        cplx q = csqrt_p(H[(size_t)i * n + i]);
        if (q.y < 0.0) q = cneg(q);
        q1[i] = q;
    }
}

// eigenvectors of T, then W = Z X
__global__ void __launch_bounds__(kRT) rcwa_vec(Bucket b) {
    __shared__ GemmSmem gs;
    const int cell = blockIdx.x;
    const int n = b.n;
    cplx* X = at(b.X, b.s_nn, cell);
    blk_trevc(n, at(b.H, b.s_nn, cell), n, X, n, at(b.A, b.s_nn, cell), &gs);  // A is free until smat1
    blk_gemm(n, n, n, C(1.0, 0.0), at(b.Z, b.s_nn, cell), n, X, n, C(0.0, 0.0), at(b.W, b.s_nn, cell), n, &gs);
}

// ---- S-matrix, interface 0 --------------------------------------------------------------
// dynamic smem: LU staging (2n + LNB^2 complex)
__global__ void __launch_bounds__(kRT) rcwa_smat1(Bucket b) {
    extern __shared__ __align__(16) unsigned char smem[];
    cplx* stg = reinterpret_cast<cplx*>(smem);
    __shared__ GemmSmem gs;
    __shared__ RedScratch rs;
    const int cell = blockIdx.x;
    const CellDev c = b.cells[cell];
    const int N = b.N, n = b.n;
    const int tid = threadIdx.x, nt = blockDim.x;
    const double w2 = c.omega * c.omega;
    const cplx* W = at(b.W, b.s_nn, cell);
    const cplx* Einv = at(b.Einv, b.s_NN, cell);
    const cplx* q1 = at(b.q1, b.s_n, cell);
    cplx* V = at(b.Z, b.s_nn, cell);  // [N x n]
    cplx* U = at(b.X, b.s_nn, cell);  // [N x n]
    cplx* A = at(b.A, b.s_nn, cell);
    // A = kp W = w^2 W - Jk Einv (Jk^T W), Jk = [-Ky; Kx]
    for (int e = tid; e < N * n; e += nt) {
        const int i = e / n, j = e % n;
        V[e] = cfma(kx_of(b, c, i), W[(size_t)(N + i) * n + j], cneg(cmul(ky_of(b, c, i), W[(size_t)i * n + j])));
    }
    blk_gemm(N, n, N, C(1.0, 0.0), Einv, N, V, n, C(0.0, 0.0), U, n, &gs);
    for (int e = tid; e < N * n; e += nt) {
        const int i = e / n;
        A[e] = cfma(ky_of(b, c, i), U[e], cscale(W[e], w2));
        A[(size_t)N * n + e] = cfms(kx_of(b, c, i), U[e], cscale(W[(size_t)N * n + e], w2));
    }
    __syncthreads();
    // P = diag(q0) kp0^{-1} A diag(1/q1); T11 = (W + P)/2, T12 = (W - P)/2
    cplx* T11 = at(b.T11, b.s_nn, cell);
    cplx* T11lu = at(b.T11lu, b.s_nn, cell);
    cplx* T12 = at(b.T12, b.s_nn, cell);
    const cplx ier = cinv(cmul(c.n_inc, c.n_inc));
    const cplx er = cmul(c.n_inc, c.n_inc);
    for (int e = tid; e < N * n; e += nt) {
        const int i = e / n, j = e % n;
        const cplx kx = kx_of(b, c, i), ky = ky_of(b, c, i);
        cplx ka, kb, kc, kd;
        kp_uniform(ier, c.omega, kx, ky, ka, kb, kc, kd);
        const cplx kz = kz_uniform(er, c.omega, kx, ky);
        const cplx idet = cinv(csub(cmul(ka, kd), cmul(kb, kc)));
        const cplx c00 = cmul(kz, cmul(kd, idet)), c01 = cneg(cmul(kz, cmul(kb, idet)));
        const cplx c10 = cneg(cmul(kz, cmul(kc, idet))), c11 = cmul(kz, cmul(ka, idet));
        const cplx iq = cinv(q1[j]);
        const cplx a0 = A[(size_t)i * n + j], a1 = A[(size_t)(N + i) * n + j];
        const cplx p0 = cmul(cfma(c00, a0, cmul(c01, a1)), iq);
        const cplx p1 = cmul(cfma(c10, a0, cmul(c11, a1)), iq);
        const cplx w0 = W[(size_t)i * n + j], w1 = W[(size_t)(N + i) * n + j];
        const cplx t0 = cscale(cadd(w0, p0), 0.5), t1 = cscale(cadd(w1, p1), 0.5);
        T11[(size_t)i * n + j] = t0;
        T11[(size_t)(N + i) * n + j] = t1;
        T11lu[(size_t)i * n + j] = t0;
        T11lu[(size_t)(N + i) * n + j] = t1;
        T12[(size_t)i * n + j] = cscale(csub(w0, p0), 0.5);
        T12[(size_t)(N + i) * n + j] = cscale(csub(w1, p1), 0.5);
    }
    __syncthreads();
    // RHS [ -T12 D | a0_X | a0_Y ], D = diag(exp(i q1 h))
    cplx* S = at(b.S12, b.s_ns, cell);
    const int ld = n + 2;
    const int i0 = b.Mx * (2 * b.My + 1) + b.My;  // order (0, 0)
    for (int e = tid; e < n * ld; e += nt) {
        const int i = e / ld, j = e % ld;
        cplx v;
        if (j < n)
            v = cneg(cmul(T12[(size_t)i * n + j], cexpi(cscale(q1[j], c.h))));
        else if (j == n)
            v = C(i == N + i0 ? 1.0 : 0.0, 0.0);  // X: Ex0 = 1
        else
            v = C(i == i0 ? -1.0 : 0.0, 0.0);     // Y: Ey0 = 1 -> a0[i0] = -1
        S[e] = v;
    }
    __syncthreads();
    int* piv = b.piv + b.s_n * cell;
    const int info = blk_lu_blocked(n, T11lu, n, piv, &rs, stg, &gs);
    if (info != 0 && tid == 0 && b.info[cell] == 0) b.info[cell] = -info;  // keep an earlier stage's code
    blk_lu_solve_blocked(n, T11lu, n, piv, ld, S, ld, stg, &gs);  // [S12 | u_X | u_Y]
}

// ---- S-matrix, interface 1 + exterior amplitudes --------------------------------------------
// The layer -> substrate interface in the reference's form (rcwa2d.cpp:394-410) is
// T11' = (W^-1 + P')/2, T12' = (W^-1 - P')/2 with P' = diag(q1) A^-1 K, K the
// substrate kp diag(1/kz) blocks; the exterior amplitudes solve
// (T11' - D S12 T12') aN = D u, D = diag(exp(i q1 h)). With aN = W y the
// inverse of W drops out: T11' aN = (y + Q y)/2, T12' aN = (y - Q y)/2 with
// Q = diag(q1) A^-1 K W, so
//     (I + Q - D S12 + D S12 Q) y = 2 D u,   aN = W y,   y2 = T12' aN = (y - Q y)/2,
//     b0 = T12 (u + S12 y2) + T11 D y2.
// One LU of A with n right-hand sides, one GEMM and one LU of the combined
// matrix (instead of two inverses, a GEMM and an LU).
// dynamic smem: staging (2n + LNB^2 complex)
__global__ void __launch_bounds__(kRT) rcwa_smat2(Bucket b) {
    extern __shared__ __align__(16) unsigned char smem[];
    cplx* stg = reinterpret_cast<cplx*>(smem);
    __shared__ GemmSmem gs;
    __shared__ RedScratch rs;
    const int cell = blockIdx.x;
    const CellDev c = b.cells[cell];
    const int N = b.N, n = b.n;
    const int tid = threadIdx.x, nt = blockDim.x;
    const cplx* W = at(b.W, b.s_nn, cell);
    cplx* A = at(b.A, b.s_nn, cell);
    cplx* Q = at(b.H, b.s_nn, cell);   // K W, then Q (H, Z, X are dead after the eigenvectors)
    cplx* SQ = at(b.Z, b.s_nn, cell);  // S12 Q
    cplx* Cm = at(b.X, b.s_nn, cell);  // I + Q - D S12 + D S12 Q, then its LU
    const cplx* q1 = at(b.q1, b.s_n, cell);
    int* piv = b.piv + b.s_n * cell;
    // K W: rows m and N+m mix through the substrate kp block of order m over kz_m
    const cplx ier = cinv(cmul(c.n_sub, c.n_sub));
    const cplx er = cmul(c.n_sub, c.n_sub);
    for (int e = tid; e < N * n; e += nt) {
        const int m = e / n, j = e % n;
        const cplx kx = kx_of(b, c, m), ky = ky_of(b, c, m);
        cplx ka, kb, kc, kd;
        kp_uniform(ier, c.omega, kx, ky, ka, kb, kc, kd);
        const cplx iq2 = cinv(kz_uniform(er, c.omega, kx, ky));
        const cplx w0 = W[(size_t)m * n + j], w1 = W[(size_t)(N + m) * n + j];
        Q[(size_t)m * n + j] = cmul(cfma(ka, w0, cmul(kb, w1)), iq2);
        Q[(size_t)(N + m) * n + j] = cmul(cfma(kc, w0, cmul(kd, w1)), iq2);
    }
    int info = blk_lu_blocked(n, A, n, piv, &rs, stg, &gs);
    blk_lu_solve_blocked(n, A, n, piv, n, Q, n, stg, &gs);  // A^-1 K W
    if (tid == 0 && info && b.info[cell] == 0) b.info[cell] = -info;
    for (int e = tid; e < n * n; e += nt) Q[e] = cmul(q1[e / n], Q[e]);
    cplx* S = at(b.S12, b.s_ns, cell);
    const int ld = n + 2;
    blk_gemm(n, n, n, C(1.0, 0.0), S, ld, Q, n, C(0.0, 0.0), SQ, n, &gs);
    for (int e = tid; e < n * n; e += nt) {
        const int i = e / n, j = e % n;
        const cplx d = cexpi(cscale(q1[i], c.h));
        cplx v = cadd(Q[e], cmul(d, csub(SQ[e], S[(size_t)i * ld + j])));
        if (i == j) v.x += 1.0;
        Cm[e] = v;
    }
    // rhs = 2 D u (2 columns) into vec scratch [n x 2]
    cplx* vec = at(b.vec, 10 * b.s_n, cell);
    cplx* x = vec + 4 * (size_t)b.s_n;    // [n x 2] row-major: y
    cplx* y2 = vec + 6 * (size_t)b.s_n;   // [n x 2]: Q y, then y2
    cplx* zz = vec + 8 * (size_t)b.s_n;   // [n x 2]: u + S12 y2
    for (int e = tid; e < 2 * n; e += nt) {
        const int i = e / 2, r = e % 2;
        x[e] = cscale(cmul(cexpi(cscale(q1[i], c.h)), S[(size_t)i * ld + n + r]), 2.0);
    }
    info = blk_lu_blocked(n, Cm, n, piv, &rs, stg, &gs);
    if (tid == 0 && info && b.info[cell] == 0) b.info[cell] = -info;
    blk_lu_solve_blocked(n, Cm, n, piv, 2, x, 2, stg, &gs);  // x = y (X, Y)
    cplx* aN = vec;                      // [2][n]
    cplx* b0 = vec + 2 * (size_t)b.s_n;  // [2][n]
    for (int e = tid; e < 2 * n; e += nt) stg[e] = x[e];
    __syncthreads();
    blk_matvec2(n, n, W, n, stg, aN, 1, b.s_n, false);  // aN = W y
    blk_matvec2(n, n, Q, n, stg, y2, 2, 1, false);      // Q y
    __syncthreads();
    for (int e = tid; e < 2 * n; e += nt) {
        const cplx v = cscale(csub(stg[e], y2[e]), 0.5);
        y2[e] = v;
        zz[e] = S[(size_t)(e / 2) * ld + n + (e % 2)];  // u
    }
    __syncthreads();
    for (int e = tid; e < 2 * n; e += nt) stg[e] = y2[e];
    __syncthreads();
    blk_matvec2(n, n, S, ld, stg, zz, 2, 1, true);  // u + S12 y2
    __syncthreads();
    // b0 = T12 zz + T11 (D y2)
    const cplx* T11 = at(b.T11, b.s_nn, cell);
    const cplx* T12 = at(b.T12, b.s_nn, cell);
    for (int e = tid; e < 2 * n; e += nt) stg[e] = zz[e];
    __syncthreads();
    blk_matvec2(n, n, T12, n, stg, b0, 1, b.s_n, false);
    __syncthreads();
    for (int e = tid; e < 2 * n; e += nt) stg[e] = cmul(cexpi(cscale(q1[e / 2], c.h)), y2[e]);
    __syncthreads();
    blk_matvec2(n, n, T11, n, stg, b0, 1, b.s_n, true);
}

// ---- multi-layer stacks ----------------------------------------------------------------------
// A stack is its incident half-space, nl patterned layers and the substrate. The
// layers run through the single-layer stages up to the eigenvectors as separate
// cells; rcwa_layer_out keeps each layer's region data (phi = W, kp phi = A,
// q, thickness) in a layer store; rcwa_stack_smat then runs the reference's
// S-matrix recursion over the nl + 1 interfaces (rcwa2d.cpp:376-401) for the two
// excitation columns (bN = 0, so only S11 a0 and S21 a0 are needed, with S12 and
// S22 kept whole for the recursion).
struct StackDev {
    int nl;     // patterned layers
    int slot0;  // first layer's slot in the layer store (layers are consecutive)
};
struct StackBucket {
    int Mx, My, N, n, nstack;
    const CellDev* cells;  // shared parameters of each stack (its first layer's descriptor)
    const StackDev* stacks;
    cplx *LW, *LA, *Lq;    // layer store: W [n*n], A [n*n], q [n] per slot
    const double* Lh;      // thickness per slot
    cplx *S12, *S22, *Q, *P, *X, *Y, *Z1;  // per stack, n*n each
    cplx* vec;             // per stack 10n: aN_X, aN_Y, b0_X, b0_Y | u [n x 2] | w [n x 2] | unused [n x 2]
    int* piv;
    int* info;
    size_t s_nn, s_n;
};

// Region data of one layer for the recursion: A = kp W (the operator of
// rcwa2d.cpp:344-349 applied to the eigenvectors), copied with W, q and the
// thickness into the layer store. Z and X are free after the eigenvectors.
__global__ void __launch_bounds__(kRT) rcwa_layer_out(Bucket b, cplx* LW, cplx* LA, cplx* Lq, double* Lh,
                                                      const int* slot) {
    __shared__ GemmSmem gs;
    const int cell = blockIdx.x;
    const CellDev c = b.cells[cell];
    const int N = b.N, n = b.n;
    const int tid = threadIdx.x, nt = blockDim.x;
    const double w2 = c.omega * c.omega;
    const cplx* W = at(b.W, b.s_nn, cell);
    const cplx* Einv = at(b.Einv, b.s_NN, cell);
    cplx* V = at(b.Z, b.s_nn, cell);
    cplx* U = at(b.X, b.s_nn, cell);
    const int sl = slot[cell];
    cplx* Wo = LW + b.s_nn * sl;
    cplx* Ao = LA + b.s_nn * sl;
    // V = Jk^T W = Kx W_bottom - Ky W_top; U = Einv V
    for (int e = tid; e < N * n; e += nt) {
        const int i = e / n, j = e % n;
        V[e] = cfma(kx_of(b, c, i), W[(size_t)(N + i) * n + j], cneg(cmul(ky_of(b, c, i), W[(size_t)i * n + j])));
    }
    blk_gemm(N, n, N, C(1.0, 0.0), Einv, N, V, n, C(0.0, 0.0), U, n, &gs);
    // kp W = w^2 W + [Ky U; -Kx U]
    for (int e = tid; e < N * n; e += nt) {
        const int i = e / n;
        Ao[e] = cfma(ky_of(b, c, i), U[e], cscale(W[e], w2));
        Ao[(size_t)N * n + e] = cfms(kx_of(b, c, i), U[e], cscale(W[(size_t)N * n + e], w2));
    }
    for (int e = tid; e < n * n; e += nt) Wo[e] = W[e];
    for (int i = tid; i < n; i += nt) Lq[b.s_n * sl + i] = at(b.q1, b.s_n, cell)[i];
    if (tid == 0) Lh[sl] = c.h;
}

// kp block (2 x 2 per order) and kz of a homogeneous half-space (rcwa2d.cpp:254-273)
__device__ __forceinline__ void half_space(const StackBucket& sb, const CellDev& c, cplx nreg, int i, cplx& ka,
                                           cplx& kb, cplx& kc, cplx& kd, cplx& kz) {
    const int p = i / (2 * sb.My + 1) - sb.Mx, q = i % (2 * sb.My + 1) - sb.My;
    const cplx kx = csub(c.kx0, C(2.0 * PI * (double)p / c.px, 0.0));
    const cplx ky = csub(c.ky0, C(2.0 * PI * (double)q / c.py, 0.0));
    const cplx er = cmul(nreg, nreg);
    kp_uniform(cinv(er), c.omega, kx, ky, ka, kb, kc, kd);
    kz = kz_uniform(er, c.omega, kx, ky);
}

// One CTA per stack, two per SM (measured faster than one at 255 registers despite
// the spills at 128). dynamic smem: lu_stage_bytes(n)
__global__ void __launch_bounds__(kRT, 2) rcwa_stack_smat(StackBucket sb) {
    extern __shared__ __align__(16) unsigned char smem[];
    cplx* stg = reinterpret_cast<cplx*>(smem);
    __shared__ GemmSmem gs;
    __shared__ RedScratch rs;
    const int st = blockIdx.x;
    const CellDev c = sb.cells[st];
    const StackDev sd = sb.stacks[st];
    const int N = sb.N, n = sb.n;
    const int tid = threadIdx.x, nt = blockDim.x;
    const size_t nn = sb.s_nn;
    cplx* S12 = sb.S12 + nn * st;
    cplx* S22 = sb.S22 + nn * st;
    cplx* Q = sb.Q + nn * st;
    cplx* P = sb.P + nn * st;
    cplx* X = sb.X + nn * st;
    cplx* Y = sb.Y + nn * st;
    cplx* Z1 = sb.Z1 + nn * st;
    cplx* vec = sb.vec + 10 * sb.s_n * st;
    cplx* u = vec + 4 * sb.s_n;  // S11 a0, [n x 2]
    cplx* w = vec + 6 * sb.s_n;  // T12 u, [n x 2]
    int* piv = sb.piv + sb.s_n * st;
    const int i0 = sb.Mx * (2 * sb.My + 1) + sb.My;
    int status = 0;
    // S11 a0 = a0 (columns X: Ex0 = 1, Y: Ey0 = 1), S21 a0 = 0, S12 = 0, S22 = I
    for (int e = tid; e < 2 * n; e += nt) {
        const int i = e / 2, r = e % 2;
        u[e] = (r == 0) ? C(i == N + i0 ? 1.0 : 0.0, 0.0) : C(i == i0 ? -1.0 : 0.0, 0.0);
        vec[(size_t)r * sb.s_n + i] = C(0.0, 0.0);
        vec[(2 + (size_t)r) * sb.s_n + i] = C(0.0, 0.0);
    }
    for (int e = tid; e < n * n; e += nt) {
        S12[e] = C(0.0, 0.0);
        S22[e] = C(e / n == e % n ? 1.0 : 0.0, 0.0);
    }
    __syncthreads();
    const int NL = sd.nl + 2;  // regions: incident, layers, substrate
    for (int ia = 0; ia + 1 < NL; ++ia) {
        const int ib = ia + 1;
        const bool a_inc = ia == 0, b_sub = ib == NL - 1;
        const int sa = sd.slot0 + ia - 1, sbb = sd.slot0 + ib - 1;
        const cplx* qa = a_inc ? nullptr : sb.Lq + sb.s_n * sa;
        const cplx* qb = b_sub ? nullptr : sb.Lq + sb.s_n * sbb;
        const double ha = a_inc ? 0.0 : sb.Lh[sa], hb = b_sub ? 0.0 : sb.Lh[sbb];
        // Q = phi_a^-1 phi_b ; P = A_a^-1 A_b  (A = kp phi; half-spaces: phi = I, A = kp)
        for (int e = tid; e < n * n; e += nt) {
            const int i = e / n, j = e % n;
            cplx qv, pv;
            if (b_sub) {
                qv = C(i == j ? 1.0 : 0.0, 0.0);
                const int m = i % N;
                cplx ka, kb, kc, kd, kz;
                half_space(sb, c, c.n_sub, m, ka, kb, kc, kd, kz);
                // kp of the substrate: [[ka, kb], [kc, kd]] on rows / columns (m, N + m)
                pv = C(0.0, 0.0);
                if (j == m) pv = i < N ? ka : kc;
                else if (j == N + m) pv = i < N ? kb : kd;
            } else {
                qv = sb.LW[nn * sbb + e];
                pv = sb.LA[nn * sbb + e];
            }
            Q[e] = qv;
            P[e] = pv;
        }
        __syncthreads();
        if (a_inc) {
            // phi_a = I: Q is phi_b already; P <- kp_inc^-1 P by 2 x 2 blocks per order
            for (int e = tid; e < N * n; e += nt) {
                const int m = e / n, j = e % n;
                cplx ka, kb, kc, kd, kz;
                half_space(sb, c, c.n_inc, m, ka, kb, kc, kd, kz);
                const cplx idet = cinv(csub(cmul(ka, kd), cmul(kb, kc)));
                const cplx x0 = P[(size_t)m * n + j], x1 = P[(size_t)(N + m) * n + j];
                P[(size_t)m * n + j] = cmul(idet, csub(cmul(kd, x0), cmul(kb, x1)));
                P[(size_t)(N + m) * n + j] = cmul(idet, csub(cmul(ka, x1), cmul(kc, x0)));
            }
        } else {
            // the layer store's W and A of region a are not needed after this interface
            cplx* Wa = sb.LW + nn * sa;
            cplx* Aa = sb.LA + nn * sa;
            int inf = blk_lu_blocked(n, Wa, n, piv, &rs, stg, &gs);
            blk_lu_solve_blocked(n, Wa, n, piv, n, Q, n, stg, &gs);
            if (inf) status = inf;
            inf = blk_lu_blocked(n, Aa, n, piv, &rs, stg, &gs);
            blk_lu_solve_blocked(n, Aa, n, piv, n, P, n, stg, &gs);
            if (inf) status = inf;
        }
        __syncthreads();
        // P <- diag(q_a) P diag(1/q_b); T11 = (Q + P)/2 -> Q, T12 = (Q - P)/2 -> P
        for (int e = tid; e < n * n; e += nt) {
            const int i = e / n, j = e % n;
            cplx qai, qbj;
            if (a_inc) {
                cplx ka, kb, kc, kd;
                half_space(sb, c, c.n_inc, i % N, ka, kb, kc, kd, qai);
            } else {
                qai = qa[i];
            }
            if (b_sub) {
                cplx ka, kb, kc, kd;
                half_space(sb, c, c.n_sub, j % N, ka, kb, kc, kd, qbj);
            } else {
                qbj = qb[j];
            }
            const cplx pv = cdiv(cmul(qai, P[e]), qbj), qv = Q[e];
            Q[e] = cscale(cadd(qv, pv), 0.5);
            P[e] = cscale(csub(qv, pv), 0.5);
        }
        // X = T11 - d1 S12 T12 ; Y = d1 S12 T11 - T12   (d1 = exp(i q_a h_a) on the rows)
        blk_gemm(n, n, n, C(1.0, 0.0), S12, n, P, n, C(0.0, 0.0), X, n, &gs);
        blk_gemm(n, n, n, C(1.0, 0.0), S12, n, Q, n, C(0.0, 0.0), Y, n, &gs);
        for (int e = tid; e < n * n; e += nt) {
            const int i = e / n;
            const cplx d1 = a_inc ? C(1.0, 0.0) : cexpi(cscale(qa[i], ha));
            X[e] = cfms(d1, X[e], Q[e]);
            Y[e] = csub(cmul(d1, Y[e]), P[e]);
        }
        for (int e = tid; e < 2 * n; e += nt) {
            const int i = e / 2;
            const cplx d1 = a_inc ? C(1.0, 0.0) : cexpi(cscale(qa[i], ha));
            u[e] = cmul(d1, u[e]);
        }
        const int inf = blk_lu_blocked(n, X, n, piv, &rs, stg, &gs);
        if (inf) status = inf;
        blk_lu_solve_blocked(n, X, n, piv, n, Y, n, stg, &gs);  // Y = X^-1 (d1 S12 T11 - T12)
        blk_lu_solve_blocked(n, X, n, piv, 2, u, 2, stg, &gs);  // u = S11' a0 = X^-1 d1 S11 a0
        // S12' = Y diag(d2)
        for (int e = tid; e < n * n; e += nt) {
            const int j = e % n;
            const cplx d2 = b_sub ? C(1.0, 0.0) : cexpi(cscale(qb[j], hb));
            S12[e] = cmul(Y[e], d2);
        }
        // S21' a0 = S21 a0 + S22 T12 u'
        for (int e = tid; e < 2 * n; e += nt) stg[e] = u[e];
        __syncthreads();
        blk_matvec2(n, n, P, n, stg, w, 2, 1, false);  // w = T12 u'
        __syncthreads();
        for (int e = tid; e < 2 * n; e += nt) stg[e] = w[e];
        __syncthreads();
        blk_matvec2(n, n, S22, n, stg, vec + 2 * sb.s_n, 1, sb.s_n, true);
        // S22' = S22 (T12 S12' + T11 diag(d2))
        blk_gemm(n, n, n, C(1.0, 0.0), P, n, S12, n, C(0.0, 0.0), Z1, n, &gs);
        for (int e = tid; e < n * n; e += nt) {
            const int j = e % n;
            const cplx d2 = b_sub ? C(1.0, 0.0) : cexpi(cscale(qb[j], hb));
            Z1[e] = cfma(Q[e], d2, Z1[e]);
        }
        blk_gemm(n, n, n, C(1.0, 0.0), S22, n, Z1, n, C(0.0, 0.0), X, n, &gs);  // X is free after the solves
        for (int e = tid; e < n * n; e += nt) S22[e] = X[e];
        __syncthreads();
    }
    // exterior amplitudes for the epilogue: aN = S11 a0 (2 columns)
    for (int e = tid; e < 2 * n; e += nt) {
        const int i = e / 2, r = e % 2;
        vec[(size_t)r * sb.s_n + i] = u[e];
    }
    if (tid == 0 && status != 0) sb.info[st] = -status;
}

// ---- standalone eigensolve (eig.hpp:25) ------------------------------------------------------
// The RCWA eigen-stages on caller matrices: eig_load transposes a column-major
// (Eigen / LAPACK) matrix into the row-major H of its cell; eig_store writes the
// eigenvalues (diagonal of the Schur form) and the eigenvectors W = Z X in
// column-major order, each scaled to unit 2-norm with its largest-magnitude
// component real and positive (zgeev's normalisation).
__global__ void __launch_bounds__(kRT) eig_load(const cplx* __restrict__ A, Bucket b) {
    const int cell = blockIdx.x, n = b.n;
    const cplx* src = A + b.s_nn * cell;
    cplx* H = at(b.H, b.s_nn, cell);
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
        const int i = e / n, j = e % n;
        H[e] = src[(size_t)j * n + i];
    }
}

__global__ void __launch_bounds__(kRT) eig_store(Bucket b, cplx* __restrict__ evals, cplx* __restrict__ evecs) {
    __shared__ RedScratch rs;
    const int cell = blockIdx.x, n = b.n;
    const int tid = threadIdx.x, nt = blockDim.x;
    const cplx* H = at(b.H, b.s_nn, cell);
    const cplx* W = at(b.W, b.s_nn, cell);
    cplx* out = evecs + b.s_nn * cell;
    for (int i = tid; i < n; i += nt) evals[(size_t)cell * n + i] = H[(size_t)i * n + i];
    for (int j = 0; j < n; ++j) {
        double s2 = 0.0, big = -1.0;
        int arg = 0;
        for (int i = tid; i < n; i += nt) {
            const double m2 = cnorm2(W[(size_t)i * n + j]);
            s2 += m2;
            if (m2 > big) {
                big = m2;
                arg = i;
            }
        }
        const double tot = blk_sum(s2, &rs);
        const int imax = blk_argmax(big, arg, &rs);
        const cplx wm = W[(size_t)imax * n + j];
        const double am = cabs(wm);
        // conj(phase of the largest component) / norm
        const cplx sc = am > 0.0 && tot > 0.0 ? cscale(cconj(wm), 1.0 / (am * sqrt(tot))) : C(1.0, 0.0);
        for (int i = tid; i < n; i += nt) out[(size_t)j * n + i] = cmul(W[(size_t)i * n + j], sc);
        __syncthreads();
    }
}

// ---- flux and order-0 field (rcwa2d.cpp:416-463) ---------------------------------------------
__global__ void __launch_bounds__(kRT) rcwa_epilogue(Bucket b) {
    __shared__ RedScratch rs;
    __shared__ double sums[4];
    const int cell = blockIdx.x;
    const CellDev c = b.cells[cell];
    const int N = b.N;
    const int tid = threadIdx.x, nt = blockDim.x;
    const cplx* vec = at(b.vec, 10 * b.s_n, cell);
    const int i0 = b.Mx * (2 * b.My + 1) + b.My;
    const cplx er_i = cmul(c.n_inc, c.n_inc), ier_i = cinv(er_i);
    const cplx er_s = cmul(c.n_sub, c.n_sub), ier_s = cinv(er_s);
    const double norm = c.n_inc.x / cos(c.theta);  // rcwa2d.cpp:437
    for (int ex = 0; ex < c.nexc; ++ex) {
        // excitation coefficients: slot 0 = (ex0, ey0), slot 1 = Y (0, 1)
        const cplx fx = ex == 0 ? c.ex0 : C(0.0, 0.0);
        const cplx fy = ex == 0 ? c.ey0 : C(1.0, 0.0);
        double sR = 0.0, sT = 0.0;
        for (int i = tid; i < N; i += nt) {
            const cplx kx = kx_of(b, c, i), ky = ky_of(b, c, i);
            // incident region: a0 = -Ey0 e_i0 + Ex0 e_{N+i0}; b0 = fx b0_X + fy b0_Y
            const cplx a0s = i == i0 ? cneg(fy) : C(0.0, 0.0);
            const cplx a0p = i == i0 ? fx : C(0.0, 0.0);
            const cplx b0s = cfma(fx, vec[2 * b.s_n + i], cmul(fy, vec[3 * b.s_n + i]));
            const cplx b0p = cfma(fx, vec[2 * b.s_n + N + i], cmul(fy, vec[3 * b.s_n + N + i]));
            const cplx aNs = cfma(fx, vec[i], cmul(fy, vec[b.s_n + i]));
            const cplx aNp = cfma(fx, vec[N + i], cmul(fy, vec[b.s_n + N + i]));
            cplx ka, kb, kc, kd;
            // incident: A = kp diag(1/(omega q)), phi = I
            kp_uniform(ier_i, c.omega, kx, ky, ka, kb, kc, kd);
            const cplx iwq_i = cinv(cscale(kz_uniform(er_i, c.omega, kx, ky), c.omega));
            const cplx Aa0 = cmul(cfma(ka, a0s, cmul(kb, a0p)), iwq_i), Aa1 = cmul(cfma(kc, a0s, cmul(kd, a0p)), iwq_i);
            const cplx Ab0 = cmul(cfma(ka, b0s, cmul(kb, b0p)), iwq_i), Ab1 = cmul(cfma(kc, b0s, cmul(kd, b0p)), iwq_i);
            // bwd flux of the incident region: bxy = -Re(conj(Ab) pb) + conj(diff)
            const cplx d0 = cscale(csub(cmulc(b0s, Aa0), cmulc(Ab0, a0s)), 0.5);
            const cplx d1 = cscale(csub(cmulc(b0p, Aa1), cmulc(Ab1, a0p)), 0.5);
            const double bw = -cmulc(Ab0, b0s).x + d0.x - cmulc(Ab1, b0p).x + d1.x;  // Re(bxy_i + bxy_{N+i})
            // substrate: forward flux fxy = Re(conj(Aa) pa) + diff, b = 0
            kp_uniform(ier_s, c.omega, kx, ky, ka, kb, kc, kd);
            const cplx iwq_s = cinv(cscale(kz_uniform(er_s, c.omega, kx, ky), c.omega));
            const cplx Sa0 = cmul(cfma(ka, aNs, cmul(kb, aNp)), iwq_s), Sa1 = cmul(cfma(kc, aNs, cmul(kd, aNp)), iwq_s);
            const double fw = cmulc(Sa0, aNs).x + cmulc(Sa1, aNp).x;
            sR += -bw * norm;
            sT += fw * norm;
            if (b.ord) {  // rcwa2d.cpp:479-480
                double* o = b.ord + 2 * ((size_t)(cell * c.nexc + ex) * N + i);
                o[0] = fw * norm;
                o[1] = -bw * norm;
            }
            if (i == i0) {
                sums[0] = -bw * norm;   // de_r0
                sums[1] = fw * norm;    // de_t0
                // order-0 fields: Esub = A_sub aN, Einc = A_inc a0
                const cplx ex_inc = Aa1;
                const cplx den = cabs(ex_inc) > 1e-30 ? ex_inc : C(1.0, 0.0);
                const cplx tx = cdiv(Sa1, den), ty = cneg(cdiv(Sa0, den));
                celeris_rcwa_result* r = &b.res[(size_t)cell * c.nexc + ex];
                r->tx0[0] = tx.x;
                r->tx0[1] = tx.y;
                r->ty0[0] = ty.x;
                r->ty0[1] = ty.y;
            }
        }
        const double R = blk_sum(sR, &rs);
        const double T = blk_sum(sT, &rs);
        if (tid == 0) {
            celeris_rcwa_result* r = &b.res[(size_t)cell * c.nexc + ex];
            r->R = R;
            r->T = T;
            r->sum_de = R + T;
            r->de_r0 = sums[0];
            r->de_t0 = sums[1];
            if (b.info[cell] != 0) {
                const double nan = __longlong_as_double(0x7ff8000000000000LL);
                r->R = r->T = r->sum_de = r->de_t0 = r->de_r0 = nan;
                r->tx0[0] = r->tx0[1] = r->ty0[0] = r->ty0[1] = nan;
            }
        }
        __syncthreads();
    }
}

// ---- mirror-symmetric cells: the layer problem in its parity classes -------------------------
// A cell whose pattern is symmetric under x -> -x and under y -> -y (every
// unrotated shape of rcwa2d.cpp:37-72) at normal incidence (kx0 = ky0 = 0) has
// Kx odd and Ky even under the order map p -> -p (Px), and Einv, Exx, Eyy
// invariant under it; so M = ep2 kp - kkT commutes with Sx = diag(Px, -Px)
// (the two field blocks of rcwa2d.cpp:346-364) and likewise with Sy = diag(Py,
// -Py). Their joint eigenspaces - parity classes (a, b), a, b = +-1 - split M
// into four blocks of about n/4: the block-1 part of class (a, b) has parity
// (a, b) under (Px, Py), the block-2 part parity (-a, -b). Each class has an
// orthonormal basis of orbit vectors (the orders (+-p, +-q) of one orbit
// combined with signs a, b and weight 1/sqrt(count)). With P_c that basis,
//   M = sum_c P_c M_c P_c^T,  M_c = P_c^T M P_c,
// so the layer problem splits into one of order ~n/4 per class, each excitation lies
// in one class, and the amplitudes of the excited classes are those of the full problem
// up to rounding. M_c is built straight from the scalar parity blocks of Exx, Eyy
// and Einv (rcwa_sym_ops), never forming M. A cell whose eps operators are not mirror
// symmetric to rounding (a raster sample falling exactly on a shape boundary
// one way and not the other) is flagged kInfoAsym and solved again at full order.
// When the cell is
// also symmetric under the 90 degree rotation R (square period, Mx = My,
// fill_x = fill_y), R commutes with every operator and maps the X excitation
// onto the Y excitation, so only the X class is solved and the Y solution is R
// applied to the X one (a cell that fails that check to rounding is flagged too).
__host__ __device__ __forceinline__ int sym_class_size(int Mx, int My, int c) {
    const int a = sym_class_a(c), b = sym_class_b(c);
    return sym_count(Mx, a) * sym_count(My, b) + sym_count(Mx, -a) * sym_count(My, -b);
}

// Basis vector i of class c: its entries (2N-space indices and coefficients),
// returns their count (1, 2 or 4).
__device__ int sym_vector(int Mx, int My, int c, int i, int* idx, double* coef) {
    const int N = (2 * Mx + 1) * (2 * My + 1);
    const int a = sym_class_a(c), b = sym_class_b(c);
    const int nu = sym_count(Mx, a) * sym_count(My, b);
    int blk, pa, pb;  // field block, parities under Px, Py
    if (i < nu) {
        blk = 0, pa = a, pb = b;
    } else {
        i -= nu;
        blk = 1, pa = -a, pb = -b;
    }
    const int nq = sym_count(My, pb);
    const int p = i / nq + (pa > 0 ? 0 : 1), q = i % nq + (pb > 0 ? 0 : 1);
    const int cnt = (p > 0 ? 2 : 1) * (q > 0 ? 2 : 1);
    const double w = cnt == 4 ? 0.5 : (cnt == 2 ? 0.70710678118654752440 : 1.0);
    int k = 0;
    for (int sp = 0; sp < (p > 0 ? 2 : 1); ++sp)
        for (int sq = 0; sq < (q > 0 ? 2 : 1); ++sq) {
            const int pp = sp ? -p : p, qq = sq ? -q : q;
            idx[k] = blk * N + (pp + Mx) * (2 * My + 1) + (qq + My);
            coef[k] = w * (sp ? pa : 1) * (sq ? pb : 1);
            ++k;
        }
    return k;
}

// Orbit (p, q) >= 0 of index i in scalar parity class (a, bb).
__device__ __forceinline__ void scalar_orbit(int My, int a, int bb, int i, int& p, int& q) {
    const int nb = sym_count(My, bb);
    p = i / nb + (a > 0 ? 0 : 1);
    q = i % nb + (bb > 0 ? 0 : 1);
}
// Index of orbit (p, q) >= 0 in scalar parity class (a, bb), -1 if it has none there.
__device__ __forceinline__ int scalar_orbit_index(int My, int a, int bb, int p, int q) {
    if ((p == 0 && a < 0) || (q == 0 && bb < 0)) return -1;
    return (p - (a > 0 ? 0 : 1)) * sym_count(My, bb) + (q - (bb > 0 ? 0 : 1));
}
// ---- class operators of mirror-symmetric cells ------------------------------------------------
// Vector class c = (a, b) has its u field block in scalar class (a, b) and its v block in
// (-a, -b). Every operator of M maps parity classes onto parity classes: with kx0 =
// ky0 = 0, Kx takes the unit orbit vector of (|p|, |q|) in class (a, b) to kx = -2 pi |p| / px
// times the orbit vector of the same orbit in (-a, b), and Ky likewise in q. So with
// Eu = Eyy^(a,b), Ev = Exx^(-a,-b) and G = Einv^(a,-b), the one block of Einv that the class
// meets, and s(j) the index in (a, -b) of the orbit of j (its k is 0 where it has none):
//   Yt = Lt G, Lt[i][t] = Eu[i][t] (-ky(t));   Yb = Lb G, Lb[l][t] = Ev[l][t] kx(t)
//   M(u,u) = Yt[i][s(j)] ky(j) + w^2 Eu[i][j] - [i = j] kx^2
//   M(u,v) = -Yt[i][s(j)] kx(j) - [same orbit] kx ky
//   M(v,u) = Yb[l][s(j)] ky(j) - [same orbit] ky kx
//   M(v,v) = w^2 Ev[l][m] - Yb[l][s(m)] kx(m) - [l = m] ky^2
// (the order-space M of rcwa_build_M), the layer kp = w^2 - J Einv J^T
// (rcwa2d.cpp:346-352) as kp(u,u) = w^2 [i = j] - ky G ky, kp(u,v) = ky G kx,
// kp(v,u) = kx G ky, kp(v,v) = w^2 [i = j] - kx G kx.
//
// The scalar blocks come straight from the 1D tables (analytic rectangle) or from the
// Laurent coefficients Ge; no N x N operator is formed:
//   a Toeplitz or parity-even operator T[p][p'] between the unit orbit vectors of parity
//   a is f (T[p][p'] + a T[p][-p']), f = 1, 1/sqrt2, 1/2 by how many of p, p' are 0, times 2;
//   Laurent: B^(a,b) is the sum of the four Ge[p -+ p'][q -+ q'] with those signs, and
//   G its inverse (Gauss-Jordan of slab.cuh): one block per solved class, order ~N/4.

// factor of (T[p][p'] + a T[p][-p']) between unit orbit vectors (p, p' >= 0; p' = 0 has
// one term only, so both terms are equal there and half the sum counts)
__device__ __forceinline__ double orbit_factor(int p, int pp) {
    return p == 0 ? (pp == 0 ? 0.5 : 0.70710678118654752440) : (pp == 0 ? 0.70710678118654752440 : 1.0);
}

// ---- rasterised shapes: Fourier coefficients from sample intervals
// The samples of a raster row (one of four per pixel row, rcwa2d.cpp:74-95) that lie inside
// an unrotated shape form an interval, less an inner one for a ring: the tests compare a
// function of |x| that does not decrease away from x = 0 (with the reference's own
// roundings) with a bound. So a row is two binary searches, and its sum over the samples is a
// difference of prefix sums of the phase factors: nothing is summed over the pixels. 512
// cells on 256^2 rasters, M = 3..7, 11.9 -> 6.9 ms a call when doublings stopped at a growth of 1000
// (30 today) and buckets ran one after another; the operators of 102 M = 7 cells
// 2.1 -> 0.2 ms, of one M = 5 rectangle 0.30 -> 0.08 ms.
//
// Tables of a bucket, m = 0 .. 2 M: ph[m][i] = exp(-2 pi i m xf_i) / ng of pixel i, and
// pc[m][i] = sum of ph[m][0 .. i), the geometric series in closed form.
__global__ void rcwa_prefix_table(int ng, int mmax, cplx* ph, cplx* pc) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (mmax + 1) * (ng + 1)) return;
    const int m = e / (ng + 1), i = e - m * (ng + 1);
    double s, c;
    if (i < ng) {
        sincospi(-2.0 * m * ((i + 0.5) / ng - 0.5), &s, &c);
        ph[(size_t)m * ng + i] = C(c / ng, s / ng);
    }
    if (m % ng == 0) {  // every pixel has the same phase
        sincospi(-2.0 * m * (0.5 / ng - 0.5), &s, &c);
        pc[e] = C(c * i / ng, s * i / ng);
        return;
    }
    // e^{i pi m} e^{-i pi m i / ng} sin(pi m i / ng) / (ng sin(pi m / ng))
    const double r = sinpi((double)m * i / ng) / (ng * sinpi((double)m / ng));
    sincospi(m - (double)m * i / ng, &s, &c);
    pc[e] = C(r * c, r * s);
}

// First index in [0, cnt) at which pred holds (cnt if none); pred is monotone.
template <class Pred>
__device__ __forceinline__ int first_true(int cnt, const Pred& pred) {
    int lo = 0, hi = cnt;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (pred(mid)) hi = mid;
        else lo = mid + 1;
    }
    return lo;
}
// The samples t in [0, 2 half) with pred(t), pred true on an interval around the middle
// (monotone on either half): [lo, hi).
template <class Pred>
__device__ __forceinline__ void centred_interval(int half, const Pred& pred, int& lo, int& hi) {
    lo = first_true(half, pred);
    hi = half + first_true(half, [&](int t) { return !pred(half + t); });
}

// Shared memory of rcwa_sym_ops: a region for the raster tables (or the 1D rectangle
// tables), later the Gauss-Jordan routine's, then the coefficients.
__host__ __device__ inline size_t sym_ops_tables(int ng) { return (size_t)4 * ng * (2 * 8 + 4 * 2); }
__host__ __device__ inline size_t sym_ops_smem(int Mx, int My, int ng) {
    const int big = (Mx + 1) * (My + 1) > 2 * (Mx > My ? Mx : My) + 1 ? (Mx + 1) * (My + 1) : 2 * (Mx > My ? Mx : My) + 1;
    const size_t a = slab::shared_bytes(big), t = ng > 0 ? sym_ops_tables(ng) : 0;
    const size_t coef = ng > 0 ? (size_t)(2 * Mx + 1) * (4 * My + 1) * 16
                               : ((size_t)(4 * Mx + 1) + (4 * My + 1)) * 8 + 16;
    return ((a > t ? a : t) + 15) / 16 * 16 + coef;
}

struct RasterCoef {  // Ge from the count transform F (dp >= 0; F[-d] = conj F[d])
    const cplx* F;
    cplx eb, dE;
    int My;
    __device__ cplx operator()(int dp, int dq) const {
        const cplx f = dp >= 0 ? F[dp * (4 * My + 1) + dq + 2 * My] : cconj(F[-dp * (4 * My + 1) - dq + 2 * My]);
        const cplx v = cmul(dE, f);
        return dp == 0 && dq == 0 ? cadd(v, eb) : v;
    }
};

// F[dp][dq], dp = 0 .. 2 Mx, of the cell's inside fractions into smem (F); G1 (global):
// (2 Mx + 1) x ng. tabs: the shared tables.
__device__ void raster_transform(const Bucket& b, const CellDev& c, cplx* G1, unsigned char* tabs, cplx* F) {
    const int ng = b.ng, Mx = b.Mx, My = b.My, tid = threadIdx.x, nt = blockDim.x;
    double* tx = reinterpret_cast<double*>(tabs);
    double* ty = tx + 4 * ng;
    short* iv = reinterpret_cast<short*>(ty + 4 * ng);  // per sample row: lo, hi, inner lo, inner hi
    const double ax = c.fill_x * 0.5, ay = c.fill_y * 0.5;
    const bool round_shape = c.shape == CELERIS_SHAPE_ELLIPSE || c.shape == CELERIS_SHAPE_RING;
    const bool empty = round_shape && (ax <= 0.0 || ay <= 0.0);
    for (int t = tid; t < 4 * ng; t += nt) {
        const double xf = raster_coord(t >> 2, t & 3, ng);
        if (round_shape) {
            const double u = xf / ax, v = xf / ay;
            tx[t] = __dmul_rn(u, u);
            ty[t] = __dmul_rn(v, v);
        } else {
            tx[t] = ty[t] = fabs(xf);
        }
    }
    __syncthreads();
    const double hx = ax * c.shape_param, hy = ay * c.shape_param, ri2 = __dmul_rn(c.shape_param, c.shape_param);
    const int half = 2 * ng;
    for (int t = tid; t < 4 * ng; t += nt) {
        int lo = 0, hi = 0, ilo = 0, ihi = 0;
        const double y = ty[t];
        if (empty) {
        } else if (round_shape) {
            centred_interval(half, [&](int i) { return __dadd_rn(tx[i], y) <= 1.0; }, lo, hi);
            if (c.shape == CELERIS_SHAPE_RING)
                centred_interval(half, [&](int i) { return !(__dadd_rn(tx[i], y) >= ri2); }, ilo, ihi);
        } else {
            double bound = -1.0;
            if (y <= ay) bound = c.shape == CELERIS_SHAPE_RECT ? ax : hx;
            if (c.shape == CELERIS_SHAPE_CROSS && y <= hy) bound = fmax(bound, ax);
            if (bound >= 0.0) centred_interval(half, [&](int i) { return tx[i] <= bound; }, lo, hi);
        }
        ilo = max(ilo, lo);
        ihi = max(min(ihi, hi), ilo);
        if (ilo >= hi) ilo = ihi = hi;
        iv[4 * t] = (short)lo;
        iv[4 * t + 1] = (short)hi;
        iv[4 * t + 2] = (short)ilo;
        iv[4 * t + 3] = (short)ihi;
    }
    __syncthreads();
    // G1[dp][iy] = sum over the row's samples of ph[dp][pixel] (a sixteenth each)
    for (int e = tid; e < (2 * Mx + 1) * ng; e += nt) {
        const int dp = e / ng, iy = e - dp * ng;
        const cplx* ph = b.phx + (size_t)dp * ng;
        const cplx* pc = b.pcx + (size_t)dp * (ng + 1);
        cplx s = C(0.0, 0.0);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const short4 v = reinterpret_cast<const short4*>(iv)[4 * iy + k];
            const int end[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {  // + hi - lo, - (inner hi - inner lo)
                const double sg = (j == 1 || j == 2) ? 1.0 : -1.0;
                const int px = end[j] >> 2, rest = end[j] & 3;
                s = cadd(s, cscale(pc[px], sg * 4.0));  // four samples a pixel
                if (rest) s = cadd(s, cscale(ph[px], sg * rest));
            }
        }
        G1[e] = cscale(s, 0.0625);
    }
    __syncthreads();
    // F[dp][dq] = sum_iy G1[dp][iy] ph[dq][iy]
    const int nq = 4 * My + 1;
    for (int e = tid; e < (2 * Mx + 1) * nq; e += nt) {
        const int dp = e / nq, dq = e - dp * nq - 2 * My;
        const cplx* g = G1 + (size_t)dp * ng;
        const cplx* ph = b.phy + (size_t)abs(dq) * ng;
        const double sg = dq < 0 ? -1.0 : 1.0;
        cplx s[4] = {C(0.0, 0.0), C(0.0, 0.0), C(0.0, 0.0), C(0.0, 0.0)};
        int i = 0;
        for (; i + 4 <= ng; i += 4)
#pragma unroll
            for (int u = 0; u < 4; ++u) s[u] = cfma(g[i + u], C(ph[i + u].x, sg * ph[i + u].y), s[u]);
        for (; i < ng; ++i) s[0] = cfma(g[i], C(ph[i].x, sg * ph[i].y), s[0]);
        F[e] = cadd(cadd(s[0], s[1]), cadd(s[2], s[3]));
    }
    __syncthreads();
}

// The operators M and kp of a cell's solved classes. Flags kInfoAsym when the Laurent
// coefficients are not even in dp and in dq to the tolerance (or, for a C4 bucket, Ge(dp, dq)
// != Ge(-dq, dp)); those symmetries make M commute with the mirrors (and with the rotation).
// The analytic rectangle has them exactly. Scratch: the cell's Z and X.
template <int NT>
__global__ void __launch_bounds__(NT, NT >= 512 ? 1 : 2) rcwa_sym_ops(Bucket b) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ double red[32];
    const int cell = blockIdx.x;
    const CellDev cd = b.cells[cell];
    const int Mx = b.Mx, My = b.My, tid = threadIdx.x, nt = NT, m = b.m;
    const int nx = 2 * Mx + 1, ny = 2 * My + 1;
    const int big = max((Mx + 1) * (My + 1), max(nx, ny));
    unsigned char* coef = smem + sym_ops_smem(Mx, My, b.ng) -
                          (b.ng > 0 ? (size_t)nx * (4 * My + 1) * 16 : ((size_t)(4 * Mx + 1) + (4 * My + 1)) * 8 + 16);
    cplx* Zs = at(b.Z, b.s_nn, cell);
    cplx* Xs = at(b.X, b.s_nn, cell);
    const double w2 = cd.omega * cd.omega;
    const cplx ep = cd.eps_p, eb = cd.eps_b, ibe = cinv(eb), dI = csub(cinv(ep), ibe);
    cplx* F = reinterpret_cast<cplx*>(coef);
    double* sx = reinterpret_cast<double*>(coef);  // rect1d(d, fill_x), d = 0 .. 4 Mx
    double* sy = sx + 4 * Mx + 1;
    cplx* ax = b.G1 + b.s_g1 * cell;  // rectangle: the inverses of the 1D reciprocal Toeplitz matrices
    cplx* ay = ax + nx * nx;
    const RasterCoef Ge{F, eb, csub(ep, eb), My};
    bool asym;
    if (b.ng > 0) {
        raster_transform(b, cd, ax, smem, F);
        double dev = 0.0, mag = 0.0;
        for (int e = tid; e < (4 * Mx + 1) * (4 * My + 1); e += nt) {
            const int dp = e / (4 * My + 1) - 2 * Mx, dq = e % (4 * My + 1) - 2 * My;
            const cplx v = Ge(dp, dq);
            dev = slab::nan_max(slab::nan_max(dev, cabs(csub(v, Ge(-dp, dq)))), cabs(csub(v, Ge(dp, -dq))));
            if (b.ncls == 1) dev = slab::nan_max(dev, cabs(csub(v, Ge(-dq, dp))));
            mag = slab::nan_max(mag, cabs(v));
        }
        dev = slab::block_max(dev, red);
        mag = slab::block_max(mag, red);
        asym = !(dev < b.sym_tol * mag);  // strict: tolerance 0 flags every cell
    } else {
        for (int d = tid; d <= 4 * Mx; d += nt) sx[d] = rect1d(d, cd.fill_x);
        for (int d = tid; d <= 4 * My; d += nt) sy[d] = rect1d(d, cd.fill_y);
        __syncthreads();
        asym = !(0.0 < b.sym_tol);
        // Hx, Hy (rcwa2d.cpp:299-303, 317-321), inverted
        const slab::Shared s = slab::carve(smem, big);
        for (int axis = 0; axis < 2; ++axis) {
            const int n1 = axis ? ny : nx;
            const double* t1 = axis ? sy : sx;
            cplx* W = Zs;
            for (int e = tid; e < n1 * n1; e += nt) {
                const int i = e / n1, j = e - i * n1;
                const cplx v = cscale(dI, t1[abs(i - j)]);
                W[e] = i == j ? cadd(v, ibe) : v;
            }
            if (!slab::gauss_jordan(n1, n1, W, n1, true, s)) {
                if (tid == 0) b.info[cell] = -(axis + 1);
                return;
            }
            for (int e = tid; e < n1 * n1; e += nt) {
                const int k = e / n1, c = e - k * n1;
                (axis ? ay : ax)[(size_t)k * n1 + s.perm[c]] = W[(size_t)s.perm[k] * n1 + c];
            }
            __syncthreads();
        }
    }
    if (asym) {
        if (tid == 0) b.info[cell] = kInfoAsym;
        return;
    }
    // entry (i, j) of an operator's block in scalar class (a, bb): which = 0 Exx, 1 Eyy,
    // 2 Einv (rectangle only)
    auto entry = [&](int which, int a, int bb, int i, int j) -> cplx {
        int p, q, pp, qq;
        scalar_orbit(My, a, bb, i, p, q);
        scalar_orbit(My, a, bb, j, pp, qq);
        const double f = orbit_factor(p, pp) * orbit_factor(q, qq);
        if (b.ng > 0) {
            const cplx u = cadd(Ge(p - pp, q - qq), cscale(Ge(p + pp, q - qq), (double)a));
            const cplx v = cadd(Ge(p - pp, q + qq), cscale(Ge(p + pp, q + qq), (double)a));
            return cscale(cadd(u, cscale(v, (double)bb)), f);
        }
        const double tx = sx[abs(p - pp)] + a * sx[p + pp], ty = sy[abs(q - qq)] + bb * sy[q + qq];
        const double dx = p == pp ? 1.0 : 0.0, dy = q == qq ? 1.0 : 0.0;
        if (which == 2) {
            cplx v = cscale(dI, tx * ty * f);
            return i == j ? cadd(v, ibe) : v;
        }
        if (which == 0) {  // Ax (x) Sy + eb I (x) (I - Sy)
            const cplx A = cadd(ax[(p + Mx) * nx + pp + Mx], cscale(ax[(p + Mx) * nx - pp + Mx], (double)a));
            return cadd(cscale(A, ty * f), cscale(eb, dx * (dy - ty * orbit_factor(q, qq))));
        }
        const cplx A = cadd(ay[(q + My) * ny + qq + My], cscale(ay[(q + My) * ny - qq + My], (double)bb));
        return cadd(cscale(A, tx * f), cscale(eb, dy * (dx - tx * orbit_factor(p, pp))));
    };
    for (int cc = 0; cc < b.ncls; ++cc) {
        const int c = b.cls0 + cc;
        const int a = sym_class_a(c), bb = sym_class_b(c);
        const int su = sym_count(Mx, a) * sym_count(My, bb);    // u block: (a, b)
        const int sv = sym_count(Mx, -a) * sym_count(My, -bb);  // v block: (-a, -b)
        const int st = sym_count(Mx, a) * sym_count(My, -bb);   // Einv block: (a, -b)
        cplx* Eu = Zs;
        cplx* Ev = Eu + (size_t)su * su;
        cplx* G = Ev + (size_t)sv * sv;
        cplx* Lt = G + (size_t)st * st;
        cplx* Lb = Xs;
        cplx* Yt = Lb + (size_t)sv * st;
        cplx* Yb = Yt + (size_t)su * st;
        __syncthreads();  // the previous class's readers of the scratch are done
        for (int e = tid; e < su * su; e += nt) Eu[e] = entry(1, a, bb, e / su, e % su);
        for (int e = tid; e < sv * sv; e += nt) Ev[e] = entry(0, -a, -bb, e / sv, e % sv);
        cplx* Gb = b.ng > 0 ? Xs : G;  // the Laurent block is inverted on the way
        for (int e = tid; e < st * st; e += nt) Gb[e] = entry(2, a, -bb, e / st, e % st);
        __syncthreads();
        if (b.ng > 0 && st > 0) {
            const slab::Shared s = slab::carve(smem, big);  // the raster tables are dead
            if (!slab::gauss_jordan(st, st, Gb, st, true, s)) {
                if (tid == 0 && b.info[cell] == 0) b.info[cell] = -1;
                return;
            }
            for (int e = tid; e < st * st; e += nt) {
                const int k = e / st, l = e - k * st;
                G[(size_t)k * st + s.perm[l]] = Gb[(size_t)s.perm[k] * st + l];
            }
            __syncthreads();
        }
        // Lt[i][t] = Eu[i][orbit t in (a, b)] (-ky(t)), Lb[l][t] = Ev[l][orbit t in (-a, -b)] kx(t)
        for (int e = tid; e < (su + sv) * st; e += nt) {
            const int r = e / st, t = e % st;
            int pt, qt;
            scalar_orbit(My, a, -bb, t, pt, qt);
            if (r < su) {
                const int j = scalar_orbit_index(My, a, bb, pt, qt);
                const double ky = -(2.0 * PI * (double)qt / cd.py);
                Lt[(size_t)r * st + t] = j < 0 ? C(0.0, 0.0) : cscale(Eu[(size_t)r * su + j], -ky);
            } else {
                const int l = r - su;
                const int j = scalar_orbit_index(My, -a, -bb, pt, qt);
                const double kx = -(2.0 * PI * (double)pt / cd.px);
                Lb[(size_t)l * st + t] = j < 0 ? C(0.0, 0.0) : cscale(Ev[(size_t)l * sv + j], kx);
            }
        }
        __syncthreads();
        if (su > 0 && st > 0)
            slab::gemm(su, st, st, (const cplx*)Lt, st, (const cplx*)G, st, nullptr,
                       [=](int r, int j, cplx v) { Yt[(size_t)r * st + j] = v; });
        if (sv > 0 && st > 0)
            slab::gemm(sv, st, st, (const cplx*)Lb, st, (const cplx*)G, st, nullptr,
                       [=](int r, int j, cplx v) { Yb[(size_t)r * st + j] = v; });
        __syncthreads();
        const size_t mi = (size_t)(b.ncls * cell + cc) * m * m;
        cplx* Mc = b.cM + mi;
        cplx* Kp = b.cKp + mi;
        for (int e = tid; e < m * m; e += nt) {
            const int i = e / m, j = e % m;
            const bool ui = i < su, uj = j < su;
            const int li = ui ? i : i - su, lj = uj ? j : j - su;
            int pi, qi, pj, qj;
            scalar_orbit(My, ui ? a : -a, ui ? bb : -bb, li, pi, qi);
            scalar_orbit(My, uj ? a : -a, uj ? bb : -bb, lj, pj, qj);
            const int si = scalar_orbit_index(My, a, -bb, pi, qi), sj = scalar_orbit_index(My, a, -bb, pj, qj);
            const double kxi = -(2.0 * PI * (double)pi / cd.px), kyi = -(2.0 * PI * (double)qi / cd.py);
            const double kxj = -(2.0 * PI * (double)pj / cd.px), kyj = -(2.0 * PI * (double)qj / cd.py);
            const bool same = pi == pj && qi == qj;
            const cplx g = (si >= 0 && sj >= 0) ? G[(size_t)si * st + sj] : C(0.0, 0.0);
            cplx mv, kv;
            if (ui && uj) {
                mv = cscale(Eu[(size_t)li * su + lj], w2);
                if (sj >= 0) mv = cadd(mv, cscale(Yt[(size_t)li * st + sj], kyj));
                if (i == j) mv.x -= kxi * kxi;
                kv = cscale(g, -kyi * kyj);
                if (i == j) kv.x += w2;
            } else if (ui) {
                mv = sj >= 0 ? cscale(Yt[(size_t)li * st + sj], -kxj) : C(0.0, 0.0);
                if (same) mv.x -= kxi * kyi;
                kv = cscale(g, kyi * kxj);
            } else if (uj) {
                mv = sj >= 0 ? cscale(Yb[(size_t)li * st + sj], kyj) : C(0.0, 0.0);
                if (same) mv.x -= kyi * kxi;
                kv = cscale(g, kxi * kyj);
            } else {
                mv = cscale(Ev[(size_t)li * sv + lj], w2);
                if (sj >= 0) mv = csub(mv, cscale(Yb[(size_t)li * st + sj], kxj));
                if (i == j) mv.x -= kyi * kyi;
                kv = cscale(g, -kxi * kxj);
                if (i == j) kv.x += w2;
            }
            Mc[e] = mv;
            Kp[e] = kv;
        }
    }
}

// ---- single layers through their two-port (slab.cuh) ----------------------------------------
// A half-space's relation h = Y e of an outgoing field (h = a, e = kp q^-1 a, phi = I):
// Y = diag(kz) kp^-1 couples only the two field components of one order (of one orbit in
// a parity class): row i of Y holds d at i and o at `pair` (-1: none).
struct HalfEntry {
    cplx d, o;
    int pair;
};
// c: parity class, or -1 for the order basis.
__device__ HalfEntry half_entry(int Mx, int My, const CellDev& cd, cplx nreg, int c, int i) {
    const int N = (2 * Mx + 1) * (2 * My + 1);
    HalfEntry h;
    int p, q;
    bool u;
    if (c < 0) {
        u = i < N;
        const int o = u ? i : i - N;
        p = o / (2 * My + 1) - Mx;
        q = o % (2 * My + 1) - My;
        h.pair = u ? N + o : o;
    } else {
        const int a = sym_class_a(c), b = sym_class_b(c);
        const int su = sym_count(Mx, a) * sym_count(My, b);
        u = i < su;
        // the representative order (|p|, |q|) of the orbit
        scalar_orbit(My, u ? a : -a, u ? b : -b, u ? i : i - su, p, q);
        const int j = u ? scalar_orbit_index(My, -a, -b, p, q) : scalar_orbit_index(My, a, b, p, q);
        h.pair = j < 0 ? -1 : (u ? su + j : j);
    }
    const cplx er = cmul(nreg, nreg);
    const cplx kx = csub(cd.kx0, C(2.0 * PI * (double)p / cd.px, 0.0));
    const cplx ky = csub(cd.ky0, C(2.0 * PI * (double)q / cd.py, 0.0));
    cplx ka, kb, kc, kd;
    kp_uniform(cinv(er), cd.omega, kx, ky, ka, kb, kc, kd);
    const cplx f = cmul(kz_uniform(er, cd.omega, kx, ky), cinv(csub(cmul(ka, kd), cmul(kb, kc))));
    h.d = cmul(f, u ? kd : ka);
    h.o = cneg(cmul(f, u ? kb : kc));
    return h;
}
// The table of a half-space in shared memory (over the panel's region, free outside
// gauss_jordan); starts and ends on a barrier.
struct HalfTable {
    cplx *d, *o;
    int* pair;
    __device__ cplx times(const cplx* K, int ld, int r, int c) const {  // (Y K)[r][c]
        const cplx v = cmul(d[r], K[(size_t)r * ld + c]);
        return pair[r] < 0 ? v : cfma(o[r], K[(size_t)pair[r] * ld + c], v);
    }
};
__device__ HalfTable half_table(int Mx, int My, const CellDev& cd, cplx nreg, int c, int n, const slab::Shared& s) {
    HalfTable t;
    t.d = s.pan;
    t.o = t.d + n;
    t.pair = reinterpret_cast<int*>(t.o + n);
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const HalfEntry h = half_entry(Mx, My, cd, nreg, c, i);
        t.d[i] = h.d;
        t.o[i] = h.o;
        t.pair[i] = h.pair;
    }
    __syncthreads();
    return t;
}

// out[r][k] = sum_c A[row(r)][c] v[c][k], k < nr <= 2 (v, out: [n][2]); one warp per row.
template <class Row>
__device__ void matvec_rows2(int n, int nr, const cplx* A, int ld, const Row& row, const cplx* v, cplx* out) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarp = blockDim.x >> 5;
    for (int r = warp; r < n; r += nwarp) {
        const cplx* a = A + (size_t)row(r) * ld;
        cplx s0 = C(0.0, 0.0), s1 = s0;
        for (int c = lane; c < n; c += 32) {
            s0 = cfma(a[c], v[2 * c], s0);
            if (nr > 1) s1 = cfma(a[c], v[2 * c + 1], s1);
        }
        for (int o = 16; o > 0; o >>= 1) {
            s0.x += __shfl_down_sync(0xffffffffu, s0.x, o);
            s0.y += __shfl_down_sync(0xffffffffu, s0.y, o);
            s1.x += __shfl_down_sync(0xffffffffu, s1.x, o);
            s1.y += __shfl_down_sync(0xffffffffu, s1.y, o);
        }
        if (lane == 0) {
            out[2 * r] = s0;
            out[2 * r + 1] = s1;
        }
    }
}

// The excitation a0 of column k at index i: order basis (c < 0) X: e_{N+i0}, Y: -e_{i0}
// (rcwa2d.cpp:403-411); a class has one column (class 0: Y, class 1: X).
__device__ double excitation(int Mx, int My, int c, int i, int k) {
    const int N = (2 * Mx + 1) * (2 * My + 1), i0 = Mx * (2 * My + 1) + My;
    if (c < 0) return k == 0 ? (i == N + i0 ? 1.0 : 0.0) : (i == i0 ? -1.0 : 0.0);
    int idx[4];
    double coef[4];
    const int cnt = sym_vector(Mx, My, c, i, idx, coef), want = c == 1 ? N + i0 : i0;
    double v = 0.0;
    for (int u = 0; u < cnt; ++u)
        if (idx[u] == want) v += (c == 1 ? 1.0 : -1.0) * coef[u];
    return v;
}

// The layer, `slabs` equal slabs (A, B), between its half-spaces. With e = kp g on both
// sides of an interface,
//   substrate:  i h = i Ys kp g            ->  load L = -i Ys kp of the last slab,
//   each slab:  X = (A + L)^-1 B (g at its far side from its near side), Yin = A - B X,
//               the load of the slab before it,
//   incident:   i h(0) = -Yin g_0;  2 a0 = (i Yin + Yi kp) g_0,
//   b0 = a0 - Yi kp g_0,  aN = Ys kp X .. X g_0,
// Gauss-Jordan solves and products, for the excitation columns only. aN, b0: column k
// at + k * stride. Returns false at a zero or non-finite pivot.
template <class T>
__device__ __noinline__ bool slab_port(int Mx, int My, const CellDev& cd, int c, int n, int slabs, const T* A,
                                       const T* B, const cplx* Kp, const slab::Work& w, const slab::Shared& s,
                                       cplx* aN, cplx* b0, size_t stride) {
    const int tid = threadIdx.x, nt = blockDim.x, nr = c < 0 ? 2 : 1, n2 = 2 * n, ldg = n + 2,
              ln = slab::ld_of(n);
    cplx *Q = w.q, *G = w.e[0], *L = w.e[0], *P = w.e[1], *Pn = w.e[2];
    HalfTable ys = half_table(Mx, My, cd, cd.n_sub, c, n, s);
    HalfTable yi;
    for (int k = slabs; k >= 1; --k) {
        for (int e = tid; e < n * n; e += nt) {
            const int r = e / n, j = e - r * n;
            cplx a = slab::as_cplx(A[(size_t)r * ln + j]);
            if (k == slabs) {
                const cplx y = ys.times(Kp, n, r, j);
                a = C(a.x + y.y, a.y - y.x);
            } else {
                a = cadd(a, L[e]);
            }
            Q[(size_t)r * n2 + j] = a;
            Q[(size_t)r * n2 + n + j] = slab::as_cplx(B[(size_t)r * ln + j]);
        }
        if (!slab::gauss_jordan(n, n2, Q, n2, false, s)) return false;
        for (int i = tid; i < n; i += nt) s.perm2[i] = s.perm[i];
        yi = half_table(Mx, My, cd, cd.n_inc, c, n, s);
        if (k > 1) {
            slab::gemm(n, n, n, B, ln, (const cplx*)(Q + n), n2, s.perm2, [=](int r, int j, cplx v) {
                const size_t e = (size_t)r * n + j;
                L[e] = csub(slab::as_cplx(A[(size_t)r * ln + j]), v);
            });
            // product of the X of the slabs below the first
            if (k == slabs) {
                for (int e = tid; e < n * n; e += nt) P[e] = Q[(size_t)s.perm2[e / n] * n2 + n + e % n];
            } else {
                slab::gemm(n, n, n, (const cplx*)P, n, (const cplx*)(Q + n), n2, s.perm2,
                           [=](int r, int j, cplx v) { Pn[(size_t)r * n + j] = v; });
                cplx* t = P;
                P = Pn;
                Pn = t;
            }
            __syncthreads();
        }
    }
    slab::gemm(n, n, n, B, ln, (const cplx*)(Q + n), n2, s.perm2, [=](int r, int j, cplx v) {
        const cplx yin = csub(slab::as_cplx(A[(size_t)r * ln + j]), v), y = yi.times(Kp, n, r, j);
        G[(size_t)r * ldg + j] = C(y.x - yin.y, y.y + yin.x);
    });
    for (int e = tid; e < n * nr; e += nt) {
        const int r = e / nr, k = e - r * nr;
        G[(size_t)r * ldg + n + k] = C(2.0 * excitation(Mx, My, c, r, k), 0.0);
    }
    if (!slab::gauss_jordan(n, n + nr, G, ldg, false, s)) return false;
    cplx *g0 = w.v, *gh = g0 + n2, *kg = gh + n2, *kh = kg + n2;
    for (int e = tid; e < 2 * n; e += nt) {
        const int r = e >> 1, k = e & 1;
        g0[e] = k < nr ? G[(size_t)s.perm[r] * ldg + n + k] : C(0.0, 0.0);
    }
    __syncthreads();
    auto same = [](int r) { return r; };
    const int* xp = s.perm2;
    matvec_rows2(n, nr, Kp, n, same, g0, kg);
    matvec_rows2(n, nr, Q + n, n2, [=](int r) { return xp[r]; }, g0, gh);
    yi = half_table(Mx, My, cd, cd.n_inc, c, n, s);
    for (int e = tid; e < n * nr; e += nt) {
        const int r = e / nr, k = e - r * nr;
        const cplx y = yi.times(kg, 2, r, k);
        b0[(size_t)k * stride + r] = C(excitation(Mx, My, c, r, k) - y.x, -y.y);
    }
    if (slabs > 1) {
        matvec_rows2(n, nr, P, n, same, gh, g0);
        gh = g0;
        __syncthreads();
    }
    matvec_rows2(n, nr, Kp, n, same, gh, kh);
    ys = half_table(Mx, My, cd, cd.n_sub, c, n, s);
    for (int e = tid; e < n * nr; e += nt) {
        const int r = e / nr, k = e - r * nr;
        aN[(size_t)k * stride + r] = ys.times(kh, 2, r, k);
    }
    __syncthreads();
    return true;
}

// M = ep2 kp - kk^T and kp of a layer in the order basis (rcwa2d.cpp:346-352), from
// Einv, Exx, Eyy: one 2N x N x N product (the layer's Y of rcwa_build_M) whose epilogue
// writes M. tmp: 2 N^2 complex.
__device__ void slab_build_full(const Bucket& b, const CellDev& c, int cell, cplx* M, cplx* Kp, cplx* tmp) {
    const int N = b.N, n = b.n, tid = threadIdx.x, nt = blockDim.x;
    const cplx* Einv = at(b.Einv, b.s_NN, cell);
    const cplx* Exx = at(b.Exx, b.s_NN, cell);
    const cplx* Eyy = b.ng > 0 ? Exx : at(b.Eyy, b.s_NN, cell);
    const double w2 = c.omega * c.omega;
    for (int e = tid; e < N * N; e += nt) {
        const int i = e / N, j = e - i * N;
        const cplx kxi = kx_of(b, c, i), kyi = ky_of(b, c, i), kxj = kx_of(b, c, j), kyj = ky_of(b, c, j);
        tmp[e] = cneg(cmul(Eyy[e], kyj));
        tmp[(size_t)N * N + e] = cmul(Exx[e], kxj);
        // kp = w^2 - J Einv J^T, J = [-Ky; Kx]
        const cplx ey = cmul(Einv[e], kyj), ex = cmul(Einv[e], kxj);
        const cplx d = C(i == j ? w2 : 0.0, 0.0);
        Kp[(size_t)i * n + j] = csub(d, cmul(kyi, ey));
        Kp[(size_t)i * n + N + j] = cmul(kyi, ex);
        Kp[(size_t)(N + i) * n + j] = cmul(kxi, ey);
        Kp[(size_t)(N + i) * n + N + j] = csub(d, cmul(kxi, ex));
    }
    __syncthreads();
    slab::gemm(2 * N, N, N, (const cplx*)tmp, N, Einv, N, nullptr, [=](int r, int j, cplx y) {
        const int i = r < N ? r : r - N;
        const cplx kxj = kx_of(b, c, j), kyj = ky_of(b, c, j);
        cplx mu = cmul(y, kyj), mv = cneg(cmul(y, kxj));
        const cplx e = r < N ? Eyy[(size_t)i * N + j] : Exx[(size_t)i * N + j];
        if (r < N) mu = C(fma(w2, e.x, mu.x), fma(w2, e.y, mu.y));
        else mv = C(fma(w2, e.x, mv.x), fma(w2, e.y, mv.y));
        if (i == j) {
            const cplx ki = r < N ? kxj : kyj;
            mu = csub(mu, cmul(ki, kxj));
            mv = csub(mv, cmul(ki, kyj));
        }
        M[(size_t)r * n + j] = mu;
        M[(size_t)r * n + N + j] = mv;
    });
    __syncthreads();
}

// Orders whose whole work area fits in shared memory beside the routines' own: every
// product and copy there waits on a load or two, ~30 cycles instead of ~300 from L2
// (64 cells M = 3: 0.40 -> 0.36 ms a call when doublings stopped at a growth of 1000, 30 today).
constexpr int kSmemWork = 31;
size_t slab_smem(int n, int threads) {
    return slab::shared_bytes(n) + (threads >= 512 && n <= kSmemWork ? slab::work_size(n) * sizeof(cplx) : 0);
}

// One block per cell (order basis) or per solved parity class: the layer's two-port
// and, unless the cell is a layer of a stack (b.lA), its amplitudes between the
// half-spaces. 512 threads where a launch has no more matrices than SMs or the order
// exceeds 128 (the panel's columns then take all sixteen warps), else 256 threads with
// two blocks per SM.
template <int NT>
__global__ void __launch_bounds__(NT, NT >= 512 ? 1 : 2) rcwa_slab(Bucket b) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int skip;
    const int mi = blockIdx.x;
    const int cell = b.sym ? mi / b.ncls : mi, cc = b.sym ? mi - cell * b.ncls : 0;
    const int c = b.sym ? b.cls0 + cc : -1, n = b.sym ? b.m : b.n;
    const CellDev cd = b.cells[cell];
    if (threadIdx.x == 0) skip = b.info[cell] != 0;  // flagged by an earlier stage
    __syncthreads();
    if (skip) return;
    cplx *M, *Kp, *base;
    if (b.sym) {
        M = b.cM + (size_t)mi * n * n;
        Kp = b.cKp + (size_t)mi * n * n;
        base = at(cc ? b.X : b.Z, b.s_nn, cell);  // the class build's scratch, free now
    } else {
        base = b.slab + b.s_w * cell;
        M = base + slab::work_q(n);
        Kp = b.lA ? b.lK + b.s_nn * b.lslot[cell] : at(b.Kp, b.s_nn, cell);
    }
    slab::Shared s = slab::carve(smem, n);
    if (b.dbg) s.prof = b.dbg + kDbgSlots * (size_t)mi;
    const long long t0 = clock64();
    // small orders keep the work area in shared memory (slab_smem)
    if (NT >= 512 && n <= kSmemWork) base = reinterpret_cast<cplx*>(smem + slab::shared_bytes(n));
    const slab::Work w = slab::carve_work(base, n);
    if (!b.sym) slab_build_full(b, cd, cell, M, Kp, w.p);
    // real arithmetic where M is real up to rounding: rounding leaves imaginary parts up to 7e-16 of
    // the largest entry (400 random rasters), a raster that is not inversion symmetric ~1e-8
    bool real = cd.real_mat != 0;
    if (real) {
        double re = 0.0, im = 0.0;
        for (int e = threadIdx.x; e < n * n; e += NT) {
            re = slab::nan_max(re, fabs(M[e].x));
            im = slab::nan_max(im, fabs(M[e].y));
        }
        re = slab::block_max(re, s.red);
        im = slab::block_max(im, s.red);
        real = im <= 1e-14 * re;
    }
    cplx *aN, *b0;
    size_t stride;
    if (b.sym) {
        aN = b.cvec + (size_t)mi * 2 * n;
        b0 = aN + n;
        stride = 0;
    } else {
        aN = at(b.vec, 10 * b.s_n, cell);
        b0 = aN + 2 * b.s_n;
        stride = b.s_n;
    }
    // with permittivities of positive real part (needs_qr) no propagating mode's q exceeds the
    // bulk's, of which a complex in-plane wavevector (an absorbing incident medium) takes its
    // Im^2 from q^2 = eps w^2 - kx^2 - ky^2
    const double qmax = sqrt(cd.omega * cd.omega * fmax(cabs(cd.eps_p), cabs(cd.eps_b)) + cd.kx0.y * cd.kx0.y +
                             cd.ky0.y * cd.ky0.y);
    bool ok;
    int rest = 0;
    long long t1 = 0;
    auto finish = [&](auto* A, auto* B) {
        t1 = clock64();
        if (!b.lA) return slab_port(b.Mx, b.My, cd, c, n, 1 << rest, A, B, Kp, w, s, aN, b0, stride);
        if (threadIdx.x == 0) b.lrest[b.lslot[cell]] = rest;
        const size_t o = b.s_nn * b.lslot[cell];
        for (int e = threadIdx.x; e < n * n; e += NT) {
            const size_t p = (size_t)(e / n) * slab::ld_of(n) + e % n;
            b.lA[o + e] = slab::as_cplx(A[p]);
            b.lB[o + e] = slab::as_cplx(B[p]);
        }
        return true;
    };
    if (real) {
        double *A = nullptr, *B = nullptr;
        ok = slab::two_port<double>(n, M, cd.h, qmax, w, s, &A, &B, &rest);
        if (ok) ok = finish(A, B);
    } else {
        cplx *A = nullptr, *B = nullptr;
        ok = slab::two_port<cplx>(n, M, cd.h, qmax, w, s, &A, &B, &rest);
        if (ok) ok = finish(A, B);
    }
    if (!ok && threadIdx.x == 0) atomicCAS(&b.info[cell], 0, kInfoRedo);
    if (s.prof && threadIdx.x == 0) {
        s.prof[2] += clock64() - t0;
        s.prof[3] += clock64() - t1;
        s.prof[4] += rest;
    }
}

// A stack from the two-ports of its layers, from the substrate up: layer l's load L
// (i h = -L g at its far side) gives X_l = (A + L)^-1 B and the input relation
// Yin_l = A - B X_l; with e = kp g continuous, g_l(0) = Z_l g_{l-1}(h), Z_l = kp_l^-1 kp_{l-1},
// the next load is Yin_l Z_l. Then the fields go down: g_l(h) = X_l g_l(0). One block per
// stack; X_l and Z_l replace A_l and B_l in the layer store. work: slab::work_size(n)
// complex per stack.
struct StackPort {
    int Mx, My, n, nstack;
    const CellDev* cells;  // shared parameters of each stack (its first layer's descriptor)
    const int2* stacks;    // (layers, first slot)
    cplx *lA, *lB, *lK, *work, *vec;
    const int* lrest;
    int* info;
    size_t s_nn, s_w, s_n;
};
__global__ void __launch_bounds__(512, 1) rcwa_stack_port(StackPort sp) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int skip;
    const int st = blockIdx.x, n = sp.n, n2 = 2 * n, ldg = n + 2;
    const int tid = threadIdx.x, nt = blockDim.x;
    if (tid == 0) skip = sp.info[st] != 0;
    __syncthreads();
    if (skip) return;
    const CellDev cd = sp.cells[st];
    const int nl = sp.stacks[st].x, slot0 = sp.stacks[st].y;
    const slab::Shared s = slab::carve(smem, n);
    const slab::Work w = slab::carve_work(sp.work + sp.s_w * st, n);
    cplx *Q = w.q, *G = w.e[0], *Yin = w.p, *L = w.w1;
    bool ok = true;
    for (int l = nl - 1; l >= 0; --l) {
        cplx *A = sp.lA + sp.s_nn * (slot0 + l), *B = sp.lB + sp.s_nn * (slot0 + l);
        const cplx* K = sp.lK + sp.s_nn * (slot0 + l);
        if (l == nl - 1) {
            const HalfTable ys = half_table(sp.Mx, sp.My, cd, cd.n_sub, -1, n, s);
            for (int e = tid; e < n * n; e += nt) {
                const cplx y = ys.times(K, n, e / n, e % n);
                L[e] = C(y.y, -y.x);
            }
            __syncthreads();
        }
        const int slabs = 1 << sp.lrest[slot0 + l];
        cplx *P = w.e[1], *Pn = w.e[2];
        for (int k = slabs; k >= 1; --k) {
            const cplx* load = k == slabs ? L : Yin;
            for (int e = tid; e < n * n; e += nt) {
                const int r = e / n, j = e - r * n;
                Q[(size_t)r * n2 + j] = cadd(A[e], load[e]);
                Q[(size_t)r * n2 + n + j] = B[e];
            }
            ok = slab::gauss_jordan(n, n2, Q, n2, false, s);
            if (!ok) break;
            slab::gemm(n, n, n, (const cplx*)B, n, (const cplx*)(Q + n), n2, s.perm,
                       [=](int r, int j, cplx v) { Yin[(size_t)r * n + j] = csub(A[(size_t)r * n + j], v); });
            // product of the slabs' X
            if (k == slabs) {
                for (int e = tid; e < n * n; e += nt) P[e] = Q[(size_t)s.perm[e / n] * n2 + n + e % n];
            } else {
                slab::gemm(n, n, n, (const cplx*)P, n, (const cplx*)(Q + n), n2, s.perm,
                           [=](int r, int j, cplx v) { Pn[(size_t)r * n + j] = v; });
                cplx* t = P;
                P = Pn;
                Pn = t;
            }
            __syncthreads();
        }
        if (!ok) break;
        for (int e = tid; e < n * n; e += nt) A[e] = P[e];  // X_l
        __syncthreads();
        if (l > 0) {
            const cplx* Ku = sp.lK + sp.s_nn * (slot0 + l - 1);
            for (int e = tid; e < n * n; e += nt) {
                const int r = e / n, j = e - r * n;
                Q[(size_t)r * n2 + j] = K[e];
                Q[(size_t)r * n2 + n + j] = Ku[e];
            }
            ok = slab::gauss_jordan(n, n2, Q, n2, false, s);
            if (!ok) break;
            for (int e = tid; e < n * n; e += nt) B[e] = Q[(size_t)s.perm[e / n] * n2 + n + e % n];  // Z_l
            slab::gemm(n, n, n, (const cplx*)Yin, n, (const cplx*)(Q + n), n2, s.perm,
                       [=](int r, int j, cplx v) { L[(size_t)r * n + j] = v; });
            __syncthreads();
        }
    }
    if (ok) {
        const cplx* K0 = sp.lK + sp.s_nn * slot0;
        HalfTable yi = half_table(sp.Mx, sp.My, cd, cd.n_inc, -1, n, s);
        for (int e = tid; e < n * n; e += nt) {
            const int r = e / n, j = e - r * n;
            const cplx y = yi.times(K0, n, r, j);
            G[(size_t)r * ldg + j] = C(y.x - Yin[e].y, y.y + Yin[e].x);
        }
        for (int e = tid; e < n2; e += nt)
            G[(size_t)(e >> 1) * ldg + n + (e & 1)] = C(2.0 * excitation(sp.Mx, sp.My, -1, e >> 1, e & 1), 0.0);
        ok = slab::gauss_jordan(n, n + 2, G, ldg, false, s);
        if (ok) {
            cplx *g = w.v, *gn = g + n2, *kg = gn + n2;
            cplx* aN = sp.vec + 10 * sp.s_n * st;
            cplx* b0 = aN + 2 * sp.s_n;
            auto same = [](int r) { return r; };
            for (int e = tid; e < n2; e += nt) g[e] = G[(size_t)s.perm[e >> 1] * ldg + n + (e & 1)];
            __syncthreads();
            matvec_rows2(n, 2, K0, n, same, g, kg);
            yi = half_table(sp.Mx, sp.My, cd, cd.n_inc, -1, n, s);
            for (int e = tid; e < n2; e += nt) {
                const int r = e >> 1, k = e & 1;
                const cplx y = yi.times(kg, 2, r, k);
                b0[(size_t)k * sp.s_n + r] = C(excitation(sp.Mx, sp.My, -1, r, k) - y.x, -y.y);
            }
            for (int l = 0; l < nl; ++l) {
                __syncthreads();
                matvec_rows2(n, 2, sp.lA + sp.s_nn * (slot0 + l), n, same, g, gn);
                __syncthreads();
                const bool last = l + 1 == nl;
                matvec_rows2(n, 2, last ? sp.lK + sp.s_nn * (slot0 + l) : sp.lB + sp.s_nn * (slot0 + l + 1), n, same, gn, g);
            }
            const HalfTable ys = half_table(sp.Mx, sp.My, cd, cd.n_sub, -1, n, s);
            for (int e = tid; e < n2; e += nt) {
                const int r = e >> 1, k = e & 1;
                aN[(size_t)k * sp.s_n + r] = ys.times(g, 2, r, k);
            }
        }
    }
    if (!ok && tid == 0) sp.info[st] = kInfoRedo;
}

// QR path of one excited class: the reference's two-interface recursion restricted to the
// class (rcwa2d.cpp:376-411), from the eigenvectors W and q of its M. With Y of the incident
// and substrate half-spaces (half_entry) and D = diag(exp(i q h)):
//   A = kp W,  P = Yi A diag(1/q),  T11 = (W + P)/2,  T12 = (W - P)/2,
//   [S12 | u] = T11^-1 [-T12 D | a0],  R = diag(q) (Ys A)^-1 W,
//   (I + R - D S12 + D S12 R) y = 2 D u,  aN = W y,
//   y2 = (y - R y)/2,  b0 = T12 (u + S12 y2) + T11 D y2.
// A class matrix costs 1/64 of the order basis, which is what a thick or thin layer that
// the two-port does not take would otherwise pay (64 cells, thin or beyond 100 rad: M = 3 9.4 -> 0.75 ms,
// M = 5 48 -> 4.8 ms a call). A zero pivot sends the cell to
// the order basis (kInfoAsym).
__global__ void __launch_bounds__(512, 1) rcwa_sym_smat(Bucket b) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int skip;
    const int mi = blockIdx.x, cell = mi / b.ncls, cc = mi - cell * b.ncls, c = b.cls0 + cc, n = b.m;
    const int tid = threadIdx.x, nt = blockDim.x, Mx = b.Mx, My = b.My;
    if (tid == 0) skip = b.info[cell] != 0 || b.sinfo[mi] != 0;
    __syncthreads();
    if (skip) return;
    const CellDev cd = b.cells[cell];
    const size_t nn = (size_t)n * n;
    const cplx *W = b.sW + nn * mi, *Kp = b.cKp + nn * mi, *q = b.sq + (size_t)mi * n;
    const slab::Shared s = slab::carve(smem, n);
    const slab::Work w = slab::carve_work(at(cc ? b.X : b.Z, b.s_nn, cell), n);
    const int n2 = 2 * n, lq = n2 + 1, lc = n + 1;
    cplx *A = w.e[0], *T12 = w.w1, *G = w.p;
    cplx* S = w.q;  // [T11 | -T12 D | a0], n x lq
    cplx *T11 = w.e[1], *S12 = w.e[2];
    cplx *R = A, *Cm = S;  // where A and S are no longer needed
    slab::gemm(n, n, n, Kp, n, W, n, nullptr, [=](int r, int j, cplx v) { A[(size_t)r * n + j] = v; });
    HalfTable t = half_table(Mx, My, cd, cd.n_inc, c, n, s);
    for (int e = tid; e < n * n; e += nt) {
        const int r = e / n, j = e - r * n;
        const cplx pv = cmul(t.times(A, n, r, j), cinv(q[j])), wv = W[e];
        const cplx t11 = cscale(cadd(wv, pv), 0.5), t12 = cscale(csub(wv, pv), 0.5);
        T11[e] = t11;
        T12[e] = t12;
        S[(size_t)r * lq + j] = t11;
        S[(size_t)r * lq + n + j] = cneg(cmul(t12, cexpi(cscale(q[j], cd.h))));
    }
    for (int r = tid; r < n; r += nt) S[(size_t)r * lq + n2] = C(excitation(Mx, My, c, r, 0), 0.0);
    t = half_table(Mx, My, cd, cd.n_sub, c, n, s);
    for (int e = tid; e < n * n; e += nt) {
        const int r = e / n, j = e - r * n;
        G[(size_t)r * n2 + j] = t.times(A, n, r, j);
        G[(size_t)r * n2 + n + j] = W[e];
    }
    bool ok = slab::gauss_jordan(n, lq, S, lq, false, s);
    cplx *y = w.v, *v1 = y + n2, *v2 = v1 + n2, *v3 = v2 + n2;
    if (ok) {
        for (int e = tid; e < n * n; e += nt) S12[e] = S[(size_t)s.perm[e / n] * lq + n + e % n];
        for (int r = tid; r < n; r += nt) v3[2 * r] = S[(size_t)s.perm[r] * lq + n2];  // u
        ok = slab::gauss_jordan(n, n2, G, n2, false, s);
    }
    if (ok) {
        for (int e = tid; e < n * n; e += nt) R[e] = cmul(q[e / n], G[(size_t)s.perm[e / n] * n2 + n + e % n]);
        __syncthreads();
        slab::gemm(n, n, n, (const cplx*)S12, n, (const cplx*)R, n, nullptr, [=](int r, int j, cplx v) {
            const size_t e = (size_t)r * n + j;
            const cplx x = cadd(R[e], cmul(cexpi(cscale(q[r], cd.h)), csub(v, S12[e])));
            Cm[(size_t)r * lc + j] = r == j ? C(x.x + 1.0, x.y) : x;
        });
        for (int r = tid; r < n; r += nt)
            Cm[(size_t)r * lc + n] = cscale(cmul(cexpi(cscale(q[r], cd.h)), v3[2 * r]), 2.0);
        ok = slab::gauss_jordan(n, lc, Cm, lc, false, s);
    }
    if (!ok) {
        if (tid == 0) atomicCAS(&b.info[cell], 0, kInfoAsym);
        return;
    }
    for (int r = tid; r < n; r += nt) y[2 * r] = Cm[(size_t)s.perm[r] * lc + n];
    __syncthreads();
    cplx *aN = b.cvec + (size_t)mi * 2 * n, *b0 = aN + n;
    auto same = [](int r) { return r; };
    matvec_rows2(n, 1, W, n, same, y, v1);
    matvec_rows2(n, 1, R, n, same, y, v2);
    __syncthreads();
    for (int r = tid; r < n; r += nt) {
        aN[r] = v1[2 * r];
        v2[2 * r] = cscale(csub(y[2 * r], v2[2 * r]), 0.5);  // y2
    }
    __syncthreads();
    matvec_rows2(n, 1, S12, n, same, v2, v1);
    __syncthreads();
    for (int r = tid; r < n; r += nt) {
        y[2 * r] = cadd(v3[2 * r], v1[2 * r]);                              // u + S12 y2
        v2[2 * r] = cmul(cexpi(cscale(q[r], cd.h)), v2[2 * r]);             // D y2
    }
    __syncthreads();
    matvec_rows2(n, 1, T12, n, same, y, v1);
    matvec_rows2(n, 1, T11, n, same, v2, v3);
    __syncthreads();
    for (int r = tid; r < n; r += nt) b0[r] = cadd(v1[2 * r], v3[2 * r]);
}

// aN and b0 of both excitations into the full basis (the vector area the
// epilogue reads: aN_X, aN_Y, b0_X, b0_Y). QR path: a class eigensolve's failure becomes
// the cell's info.
__global__ void __launch_bounds__(kRT) rcwa_sym_expand(Bucket b) {
    const int cell = blockIdx.x;
    const int N = b.N, n = b.n, Mx = b.Mx, My = b.My, m = b.m, ny = 2 * My + 1;
    const int tid = threadIdx.x, nt = blockDim.x;
    cplx* vec = at(b.vec, 10 * b.s_n, cell);
    for (int e = tid; e < 4 * (int)b.s_n; e += nt) vec[e] = C(0.0, 0.0);
    __syncthreads();
    for (int cc = 0; cc < b.ncls; ++cc) {
        const int c = b.cls0 + cc, mi = b.ncls * cell + cc;
        const cplx* cv = b.cvec + (size_t)mi * 2 * m;
        cplx* dst_a = vec + (c == 1 ? 0 : b.s_n);       // aN_X : aN_Y
        cplx* dst_b = vec + (c == 1 ? 2 : 3) * b.s_n;   // b0_X : b0_Y
        for (int i = tid; i < m; i += nt) {
            int ii[4];
            double ci[4];
            const int ni = sym_vector(Mx, My, c, i, ii, ci);
            for (int u = 0; u < ni; ++u) {
                dst_a[ii[u]] = cscale(cv[i], ci[u]);
                dst_b[ii[u]] = cscale(cv[m + i], ci[u]);
            }
        }
    }
    if (b.ncls == 1) {
        // C4-symmetric cell: the Y solution is the X solution rotated by 90
        // degrees, R e_k = sigma(k) e_{rho k}: rho(u at (p, q)) = v at (-q, p)
        // with sigma = +1, rho(v at (p, q)) = u at (-q, p) with sigma = -1
        __syncthreads();
        for (int k = tid; k < n; k += nt) {
            const int bk = k / N, ok = k % N;
            const int pk = ok / ny - Mx, qk = ok % ny - My;
            const int rk = (1 - bk) * N + (-qk + Mx) * ny + (pk + My);
            const double sg = bk == 1 ? -1.0 : 1.0;
            vec[b.s_n + rk] = cscale(vec[k], sg);
            vec[3 * b.s_n + rk] = cscale(vec[2 * b.s_n + k], sg);
        }
    }
    if (b.sinfo && tid == 0 && b.info[cell] != kInfoAsym)
        for (int cc = 0; cc < b.ncls && b.info[cell] == 0; ++cc) b.info[cell] = b.sinfo[b.ncls * cell + cc];
}

// The eigen stages' bucket of a mirror-symmetric bucket's class matrices.
Bucket sym_eig_bucket(const Bucket& b) {
    Bucket e;
    std::memset(&e, 0, sizeof(e));
    e.Mx = b.Mx;
    e.My = b.My;
    e.n = b.m;
    e.N = b.m / 2;
    e.ncell = b.ncls * b.ncell;
    e.cells = b.cells;
    e.H = b.cM;
    e.Z = b.sZ;
    e.X = b.sX;
    e.W = b.sW;
    e.A = b.sA;
    e.q1 = b.sq;
    e.info = b.sinfo;
    e.dbg = b.dbg;
    e.s_nn = (size_t)e.n * e.n;
    e.s_n = (size_t)e.n;
    return e;
}

// ---- host side ------------------------------------------------------------------------------------
struct HostCell {
    CellDev d;
    int Mx, My, ng;  // ng = 0: analytic rect path
    int index;       // position in the caller's array
    int sym;         // 1: mirror-symmetric cell at normal incidence (solved in its parity classes); 2: and C4
    int qr;          // 1: through the eigendecomposition (QR) instead of the layer two-port
};

// The parity classes apply to unrotated shapes (all mirror
// symmetric, rcwa2d.cpp:37-72) at normal incidence with at least one order on
// each side of 0 in x and y; CELERIS_RCWA_SYMMETRY=0 turns it off.
bool symmetry_enabled() {
    const char* e = std::getenv("CELERIS_RCWA_SYMMETRY");
    return !(e && e[0] == '0');
}
// Mirror-asymmetry tolerance of the class split, relative to the largest Laurent
// coefficient of a rasterised cell (an analytic rectangle is symmetric exactly): rounding
// leaves ~1e-15; one raster sample on the other side of a shape boundary
// ~1e-6. CELERIS_RCWA_SYM_TOL overrides it (the test is strict, so 0 sends
// every cell to the full order through the fallback, for tests of that path).
double symmetry_tolerance() {
    const char* e = std::getenv("CELERIS_RCWA_SYM_TOL");
    return e ? std::atof(e) : 1e-9;
}
// Every bit of v (std::to_string keeps six decimals).
std::string exact_text(double v) {
    char t[40];
    std::snprintf(t, sizeof(t), "%a", v);
    return t;
}
bool sym_eligible(const celeris_rcwa_cell& c) {
    return c.theta_rad == 0.0 && c.rotation_rad == 0.0 && c.Mx >= 1 && c.My >= 1 && symmetry_enabled();
}

// Largest optical phase k0 h sqrt(max |eps|) of a layer of this order that goes through the
// two-port. A pole leaves the last doublings out, at most r of them below a phase of 2^(r+1) pi / 2
// (a growth of 30 is met within 1/47 of the pole), and each makes the complex recursion twice as long; the
// batch waits for its slowest cell. Whole calls, the eigendecomposition's time over the two-port's, at
// r <= 4 and 5: mirror-symmetric M = 2, 3, 4, 7, 64 cells, 1.13, 1.33, 1.56, 1.82 and 0.74, 0.81, 0.90, 1.02;
// oblique M = 1 .. 4 1.36, 1.73, 1.79, 1.28 and 0.86, 0.98, 0.98, 0.68. Above order 256 (12 cells) at r <= 3 and 4:
// oblique M = 6 1.29 and 0.73, classes of M = 15 1.22 and 0.71; with complex doublings at
// r <= 2, 3 and 4: oblique M = 6 1.70, 0.97 and 0.61.
double phase_limit(int order, bool real) {
    if (order <= 200) return 48.0;
    if (order <= 256) return real ? 48.0 : 24.0;
    return real ? 24.0 : 12.0;
}

// Cells of `order` (of their parity class, or of the order basis) the two-port does not take: orders
// above its limit; layers thinner than k0 h =
// 0.4 (40 nm at 633 nm; A and B are ~1 / h and only their difference counts, so
// digits go as 1 / (k0 h): against 50 digits, 48 cells of M = 1, 2 per range of k0 h, median error
// here and by the eigendecomposition 7.1e-15, 2.8e-16 in 0.01 .. 0.02, 1.1e-15, 4.4e-16 in 0.1 .. 0.2,
// 5.7e-16, 4.0e-16 in 0.2 .. 0.4, 4.7e-16, 6.1e-16 in 0.4 .. 1), zero and negative thicknesses with them; layers
// of more optical phase than phase_limit; layers with a
// permittivity of negative real part, whose plasmon modes pass the bulk's q (up to 355 times over
// 4400 random metal cells M = 1..3, so the series' slab may be at sin(q x) = 0) and whose two-port is
// less exact even where it is regular (against 50 digits, 90 % of 110 cells below 1.6e-13, the
// eigendecomposition's below 7e-14); and every
// cell while the QR iteration cap of the failure-path tests is set (the cap is about
// the eigendecomposition).
std::atomic<int> g_qr_cap_set{0};
bool needs_qr(const celeris_rcwa_cell& c, int order) {
    const double kh = 2.0 * PI / c.wavelength_um * c.thickness_um;
    const double eps = std::max(std::hypot(c.eps_pillar[0], c.eps_pillar[1]), std::hypot(c.eps_bg[0], c.eps_bg[1]));
    const bool metal = !(c.eps_pillar[0] > 0.0 && c.eps_bg[0] > 0.0);
    const bool real = c.eps_pillar[1] == 0.0 && c.eps_bg[1] == 0.0 && (c.n_inc[1] == 0.0 || c.theta_rad == 0.0);
    return metal || order > slab::kMaxOrder || !(kh >= 0.4) || !(kh * std::sqrt(eps) <= phase_limit(order, real)) ||
           g_qr_cap_set.load() != 0;
}
int full_order(int Mx, int My) { return 2 * (2 * Mx + 1) * (2 * My + 1); }
bool needs_qr(const celeris_rcwa_cell& c) {
    return needs_qr(c, sym_eligible(c) ? sym_class_size(c.Mx, c.My, 0) : full_order(c.Mx, c.My));
}

int validate(const celeris_rcwa_cell& c) {
    // every real input must be finite: a NaN or Inf would run through the
    // eigensolve and come out as a silent non-finite t, R, T
    const double v[] = {c.period_x_um, c.period_y_um, c.wavelength_um, c.theta_rad, c.phi_rad,
                        c.n_inc[0], c.n_inc[1], c.n_sub[0], c.n_sub[1], c.eps_pillar[0], c.eps_pillar[1],
                        c.eps_bg[0], c.eps_bg[1], c.fill_x, c.fill_y, c.thickness_um, c.shape_param,
                        c.rotation_rad};
    for (double x : v)
        if (!std::isfinite(x)) return set_error(CELERIS_ERR_INVALID_ARG, "cell parameter is NaN or Inf");
    if (c.Mx < 0 || c.My < 0) return set_error(CELERIS_ERR_INVALID_ARG, "M must be >= 0");
    if (c.Mx > 15 || c.My > 15) return set_error(CELERIS_ERR_TOO_LARGE, "Mx, My <= 15 supported");
    if (!(c.wavelength_um > 0) || !(c.period_x_um > 0) || !(c.period_y_um > 0))
        return set_error(CELERIS_ERR_INVALID_ARG, "wavelength and periods must be > 0");
    if (c.shape < 0 || c.shape > 3) return set_error(CELERIS_ERR_INVALID_ARG, "unknown shape %d", c.shape);
    const int n = 2 * (2 * c.Mx + 1) * (2 * c.My + 1);
    if (n > kMaxN) return set_error(CELERIS_ERR_TOO_LARGE, "2N = %d > %d", n, kMaxN);
    if (c.grid > 1024) return set_error(CELERIS_ERR_TOO_LARGE, "grid %d > 1024", c.grid);
    return CELERIS_OK;
}

HostCell make_cell(const celeris_rcwa_cell& c, int index, double ex_re, double ex_im, double ey_re, double ey_im,
                   int nexc) {
    HostCell h;
    std::memset(&h, 0, sizeof(h));
    CellDev& d = h.d;
    d.omega = 2.0 * PI / c.wavelength_um;
    d.px = c.period_x_um;
    d.py = c.period_y_um;
    d.h = c.thickness_um;
    d.theta = c.theta_rad;
    d.fill_x = c.fill_x;
    d.fill_y = c.fill_y;
    d.shape_param = c.shape_param;
    d.rot = c.rotation_rad;
    const double ni_r = c.n_inc[0], ni_i = c.n_inc[1];
    const double st = std::sin(c.theta_rad);
    // kx0 = n_inc sin(theta) cos(phi) omega (rcwa2d.cpp:234-235)
    const double fx = st * std::cos(c.phi_rad) * d.omega, fy = st * std::sin(c.phi_rad) * d.omega;
    d.kx0 = make_double2(ni_r * fx, ni_i * fx);
    d.ky0 = make_double2(ni_r * fy, ni_i * fy);
    d.eps_p = make_double2(c.eps_pillar[0], c.eps_pillar[1]);
    d.eps_b = make_double2(c.eps_bg[0], c.eps_bg[1]);
    d.n_inc = make_double2(c.n_inc[0], c.n_inc[1]);
    d.n_sub = make_double2(c.n_sub[0], c.n_sub[1]);
    d.ex0 = make_double2(ex_re, ex_im);
    d.ey0 = make_double2(ey_re, ey_im);
    d.shape = c.shape;
    d.nexc = nexc;
    d.real_mat = c.eps_pillar[1] == 0.0 && c.eps_bg[1] == 0.0 && d.kx0.y == 0.0 && d.ky0.y == 0.0;
    h.Mx = c.Mx;
    h.My = c.My;
    const bool plain_rect = c.shape == CELERIS_SHAPE_RECT && c.rotation_rad == 0.0 && !c.force_laurent;
    // reference raster size max(128, 8(2 max(Mx, My) + 1)) (rcwa2d.cpp:337)
    h.ng = plain_rect ? 0 : (c.grid > 0 ? c.grid : std::max(128, 8 * (2 * std::max(c.Mx, c.My) + 1)));
    h.index = index;
    // 2: also symmetric under the 90 degree rotation (square period, Mx = My,
    // fill_x = fill_y; every shape of rcwa2d.cpp:37-72 is then C4 symmetric):
    // the Y solution is the rotated X solution and one class is solved
    h.sym = !sym_eligible(c) ? 0
            : (c.period_x_um == c.period_y_um && c.Mx == c.My && c.fill_x == c.fill_y) ? 2 : 1;
    h.qr = needs_qr(c) ? 1 : 0;
    return h;
}

// Shared memory of the Schur kernel: two CTAs fit per SM with sizeof(AedShared);
// a launch with no more cells than SMs asks for more than half an SM's shared
// memory so that the cells spread one per SM instead of pairing up.
constexpr size_t kSchurSmemOneCta = 120 * 1024;
static_assert(sizeof(AedShared) <= kSchurSmemOneCta, "Schur shared block");
size_t schur_smem(int ncell) {
    static int sms = 0;
    if (sms == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (sms <= 0) sms = 1;
    }
    return ncell <= sms ? kSchurSmemOneCta : sizeof(AedShared);
}

// staging of blk_hessenberg_blocked
// Threads of the shared-memory Hessenberg kernel: 512 once H no longer lets
// two CTAs share an SM (order > 80), else the tuned size.
int hess_smem_threads(int n, int tuned) {
    return (size_t)n * n * sizeof(cplx) > 100 * 1024 ? kHessBigThreads : tuned;
}
size_t hess_stage_bytes(int n) { return (size_t)(n + LNB * LNB + 2 * LNB) * sizeof(cplx); }

// staging of blk_lu_blocked and the matvecs of the S-matrix kernels
size_t lu_stage_bytes(int n) { return (size_t)(2 * n + LNB * LNB) * sizeof(cplx); }

// Threads of rcwa_slab for `count` matrices of order n.
int slab_threads(int n, int count) {
    static int sms = 0;
    if (sms == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (sms <= 0) sms = 1;
    }
    return n > 128 || count <= sms ? 512 : 256;
}

size_t laurent_smem(int Mx, int My, int ng) {
    const size_t mx4 = 4 * Mx + 1, my4 = 4 * My + 1;
    const int N = (2 * Mx + 1) * (2 * My + 1);
    const size_t raster = ((size_t)laurent_g1_rows(Mx) * ng + mx4 * my4) * sizeof(cplx) + (size_t)ng * ng;
    return std::max(raster, lu_stage_bytes(N) + sizeof(GemmSmem));
}

// ---- stage configuration and autotuning -------------------------------------------------
// Every stage kernel runs with blockDim in {128, 256} (they are written for any
// multiple of 32 >= 128). For each bucket shape (Mx, My, raster) the first batch
// that meets it times every stage at both sizes on the bucket's own cells and
// keeps the faster size per stage; the table lives for the process and can be
// read with celeris_rcwa_tuning_report. CELERIS_RCWA_AUTOTUNE=0 disables it
// (all stages at 256 threads).
enum Stage { ST_FOURIER, ST_BUILD, ST_HESS, ST_SCHUR, ST_VEC, ST_SMAT1, ST_SMAT2, ST_EPI, ST_COUNT };
const char* const kStageNames[ST_COUNT] = {"fourier", "build_M", "hessenberg", "schur", "eigvec",
                                           "smat1", "smat2", "epilogue"};
constexpr int kCand[2] = {128, 256};
struct StageCfg {
    int threads[ST_COUNT];
};
StageCfg uniform_cfg(int t) {
    StageCfg c;
    for (int i = 0; i < ST_COUNT; ++i) c.threads[i] = t;
    return c;
}

std::mutex g_tune_mu;
std::map<std::tuple<int, int, int>, StageCfg>& tune_table() {
    static auto* m = new std::map<std::tuple<int, int, int>, StageCfg>();
    return *m;
}
bool tuning_enabled() {
    const char* e = std::getenv("CELERIS_RCWA_AUTOTUNE");
    return !(e && e[0] == '0');
}

struct BucketPlan {
    int Mx, My, ng, N, n, sym, qr;
    std::vector<int> ids;  // indices into the cell list
    size_t per_cell = 0, bytes = 0;
    Bucket b;
};

size_t per_cell_bytes(int n, int nexc) {
    const int N = n / 2;
    const size_t s_nn = (size_t)n * n, s_ns = (size_t)n * (n + 2), s_NN = (size_t)N * N, s_n = (size_t)n;
    return celeris_rt::align256((8 * s_nn + s_ns + 3 * s_NN + 11 * s_n) * sizeof(cplx)) +
           celeris_rt::align256(s_n * sizeof(int)) + 256 + celeris_rt::align256(sizeof(celeris_rcwa_result) * nexc) +
           celeris_rt::align256(sizeof(CellDev)) + 14 * 256;
}

// Device memory of one order-basis cell solved through its two-port: kp, the two-port's
// work area (M, the Fourier operators and their LU scratch in it), the vector area and pivots.
size_t slab_per_cell_bytes(int n, int nexc) {
    return ((size_t)n * n + slab::work_size(n) + 10 * (size_t)n) * sizeof(cplx) + (size_t)n * sizeof(int) +
           sizeof(int) + sizeof(celeris_rcwa_result) * nexc + sizeof(CellDev) + 16 * 256;
}

// Row transform of a raster (or the two 1D inverses) of one mirror-symmetric cell.
size_t sym_g1_size(int Mx, int My, int ng) {
    const size_t nx = 2 * Mx + 1, ny = 2 * My + 1;
    return std::max(nx * (size_t)ng, nx * nx + ny * ny);
}
// Z and X of one mirror-symmetric cell: the class build's scratch (full order), then a
// class's work area each, which is the larger one at Mx = My = 1.
size_t sym_scratch(int Mx, int My) {
    const size_t n = 2 * (size_t)(2 * Mx + 1) * (2 * My + 1);
    return std::max(n * n, slab::work_size(sym_class_size(Mx, My, 0)));
}
// Device memory of one mirror-symmetric cell: Z and X, the raster's row transform, the
// vector area; per solved class M, kp and 2 m amplitudes; QR path: the eigen stages'
// four matrices and q per class.
size_t sym_per_cell_bytes(int Mx, int My, int ng, int nexc, int ncls, int qr) {
    const size_t n = 2 * (size_t)(2 * Mx + 1) * (2 * My + 1);
    const size_t m = (size_t)sym_class_size(Mx, My, 0);
    return (2 * sym_scratch(Mx, My) + sym_g1_size(Mx, My, ng) + 10 * n +
            ncls * (2 * m * m + 2 * m + (qr ? 4 * m * m + m : 0))) * sizeof(cplx) + (1 + ncls) * sizeof(int) +
           sizeof(celeris_rcwa_result) * nexc + sizeof(CellDev) + 24 * 256;
}

// The largest dynamic shared memory each stage kernel needs over a wave's
// buckets; raised once per wave, outside any capture.
struct SmemNeeds {
    size_t laurent = 0, rect = 0, hess_s = 0, hess_g = 0, smat = 0, slab = 0, ops = 0, sym_smat = 0;
    bool aed = false;
    void add_eig(int n) {
        if (n <= kSmemEigMaxN) hess_s = std::max(hess_s, ((size_t)n * n + 2 * n) * sizeof(cplx));
        else hess_g = std::max(hess_g, hess_stage_bytes(n));
        aed = true;
    }
    void add(int Mx, int My, int ng, int n, int sym = 0, int qr = 1) {
        if (sym) {
            ops = std::max(ops, sym_ops_smem(Mx, My, ng));
            if (qr) sym_smat = std::max(sym_smat, slab::shared_bytes(sym_class_size(Mx, My, 0)));
        } else if (ng > 0) {
            laurent = std::max(laurent, laurent_smem(Mx, My, ng));
        } else {
            const int nx = 2 * Mx + 1, ny = 2 * My + 1;
            rect = std::max(rect, ((size_t)2 * (nx * nx + ny * ny) + 2 * std::max(nx, ny)) * sizeof(cplx));
        }
        if (!qr) {
            slab = std::max(slab, slab_smem(sym ? sym_class_size(Mx, My, 0) : n, 512));
        } else {
            add_eig(sym ? sym_class_size(Mx, My, 0) : n);
            if (!sym) smat = std::max(smat, lu_stage_bytes(n));
        }
    }
};

// Dynamic shared-memory limits are per kernel function and process-wide, so
// they only ever grow: a call that needs less never lowers the limit another
// thread's launch relies on (a larger limit does not change a launch that asks
// for less).
int raise_dyn_smem(const void* fn, size_t bytes) {
    static std::mutex mu;
    static std::map<std::pair<int, const void*>, size_t> cur;
    int dev = 0;
    CEL_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lk(mu);
    size_t& c = cur[{dev, fn}];
    if (bytes <= c) return CELERIS_OK;
    CEL_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    c = bytes;
    return CELERIS_OK;
}

int set_smem_limits(const SmemNeeds& s) {
    if (s.laurent)
        CEL_TRY(raise_dyn_smem(reinterpret_cast<const void*>(rcwa_fourier_laurent), s.laurent));
    if (s.rect)
        CEL_TRY(raise_dyn_smem(reinterpret_cast<const void*>(rcwa_fourier_rect), s.rect));
    if (s.aed)
        CEL_TRY(raise_dyn_smem(reinterpret_cast<const void*>(rcwa_schur), kSchurSmemOneCta));
    if (s.hess_g)
        CEL_TRY(raise_dyn_smem(reinterpret_cast<const void*>(rcwa_hess<false>), s.hess_g));
    if (s.hess_s) {
        CEL_TRY(raise_dyn_smem(reinterpret_cast<const void*>(rcwa_hess<true>), s.hess_s));
    }
    if (s.smat) {
        CEL_TRY(raise_dyn_smem(reinterpret_cast<const void*>(rcwa_smat1), s.smat));
        CEL_TRY(raise_dyn_smem(reinterpret_cast<const void*>(rcwa_smat2), s.smat));
    }
    if (s.sym_smat) CEL_TRY(raise_dyn_smem(reinterpret_cast<const void*>(rcwa_sym_smat), s.sym_smat));
    if (s.ops) {
        CEL_TRY(raise_dyn_smem(reinterpret_cast<const void*>(rcwa_sym_ops<256>), s.ops));
        CEL_TRY(raise_dyn_smem(reinterpret_cast<const void*>(rcwa_sym_ops<512>), s.ops));
    }
    if (s.slab) {
        CEL_TRY(raise_dyn_smem(reinterpret_cast<const void*>(rcwa_slab<256>), s.slab));
        CEL_TRY(raise_dyn_smem(reinterpret_cast<const void*>(rcwa_slab<512>), s.slab));
    }
    return CELERIS_OK;
}

// Kernels that launch_bucket launches (layer: of a stack, through the two-port).
int bucket_kernels(bool sym, int ng, bool qr, bool eig_only = false, bool layer = false) {
    const int operators = sym ? (ng > 0 ? 2 : 1) : (ng > 0 ? 3 : 1);
    if (!qr) return operators + 1 + (sym ? 1 : 0) + (layer ? 0 : 1);  // slab, expand, epilogue
    // build (order basis), hess, schur, vec; smat1 and smat2, or the classes' smat and expand; epilogue
    return operators + (sym ? 6 : eig_only ? 4 : 7);
}

// The Fourier operators of a two-port bucket into e[0] of the work areas, their LU scratch into q.
void place_operators(Bucket& b) {
    const size_t NN = (size_t)b.N * b.N;
    b.Einv = b.slab + slab::work_e(b.n);
    b.Exx = b.Einv + NN;
    b.Eyy = b.Exx + NN;
    b.s_NN = b.s_w;
    b.lu = b.slab + slab::work_q(b.n);
}

// Launch the stage sequence of one bucket on `st`. ev (ST_COUNT + 1 events) is
// optional: stage boundaries are recorded into it.
// eig_only: stop after the eigenvectors (the layers of a multi-layer stack).
// qr: through the eigendecomposition, else through the layer two-port.
void launch_bucket(const Bucket& b, const StageCfg& cfg, cudaStream_t st, cudaEvent_t* ev, bool qr,
                   bool eig_only = false) {
    const int nc = b.ncell, n = b.n;
    const int* T = cfg.threads;
    if (ev) cudaEventRecord(ev[0], st);
    count_launch(bucket_kernels(b.sym != 0, b.ng, qr, eig_only, b.lA != nullptr));
    cudaMemsetAsync(b.info, 0, sizeof(int) * nc, st);
    if (b.sym) {
        if (b.ng > 0) {
            const int mmax = 2 * std::max(b.Mx, b.My);
            rcwa_prefix_table<<<((mmax + 1) * (b.ng + 1) + 255) / 256, 256, 0, st>>>(
                b.ng, mmax, const_cast<cplx*>(b.phx), const_cast<cplx*>(b.pcx));
        }
    } else if (b.ng > 0) {
        const int Mx = b.Mx, My = b.My, ng = b.ng;
        rcwa_phase_table<<<((4 * Mx + 1) * ng + 255) / 256, 256, 0, st>>>(ng, 2 * Mx, const_cast<cplx*>(b.phx));
        rcwa_phase_table<<<((4 * My + 1) * ng + 255) / 256, 256, 0, st>>>(ng, 2 * My, const_cast<cplx*>(b.phy));
        rcwa_fourier_laurent<<<nc, T[ST_FOURIER], laurent_smem(Mx, My, ng), st>>>(b);
    } else {
        const int nx = 2 * b.Mx + 1, ny = 2 * b.My + 1;
        const size_t sm = ((size_t)2 * (nx * nx + ny * ny) + 2 * std::max(nx, ny)) * sizeof(cplx);
        rcwa_fourier_rect<<<nc, T[ST_FOURIER], sm, st>>>(b);
    }
    if (ev) cudaEventRecord(ev[1], st);
    if (b.sym) {  // class operators
        const size_t sm = sym_ops_smem(b.Mx, b.My, b.ng);
        if (slab_threads(1, nc) == 512) rcwa_sym_ops<512><<<nc, 512, sm, st>>>(b);
        else rcwa_sym_ops<256><<<nc, 256, sm, st>>>(b);
    }
    if (!qr) {
        // the layer two-port: one kernel (timed as smat1), the amplitudes of
        // mirror-symmetric cells into the order basis, the outputs
        if (ev)
            for (int i = 2; i <= 5; ++i) cudaEventRecord(ev[i], st);
        const int m = b.sym ? b.m : n, count = b.sym ? b.ncls * nc : nc;
        if (slab_threads(m, count) == 512)
            rcwa_slab<512><<<count, 512, slab_smem(m, 512), st>>>(b);
        else
            rcwa_slab<256><<<count, 256, slab_smem(m, 256), st>>>(b);
        if (ev) cudaEventRecord(ev[6], st);
        if (b.sym) rcwa_sym_expand<<<nc, T[ST_SMAT2], 0, st>>>(b);
        if (ev) cudaEventRecord(ev[7], st);
        if (!b.lA) rcwa_epilogue<<<nc, T[ST_EPI], 0, st>>>(b);
        if (ev) cudaEventRecord(ev[8], st);
        return;
    }
    const Bucket e = b.sym ? sym_eig_bucket(b) : b;
    if (b.sym) cudaMemsetAsync(e.info, 0, sizeof(int) * e.ncell, st);
    else rcwa_build_M<<<nc, T[ST_BUILD], 0, st>>>(b, b.ng > 0 ? 1 : 0);
    if (ev) cudaEventRecord(ev[2], st);
    if (e.n <= kSmemEigMaxN) {
        const size_t sm = ((size_t)e.n * e.n + 2 * e.n) * sizeof(cplx);
        rcwa_hess<true><<<e.ncell, hess_smem_threads(e.n, T[ST_HESS]), sm, st>>>(e);
    } else {
        rcwa_hess<false><<<e.ncell, T[ST_HESS], hess_stage_bytes(e.n), st>>>(e);
    }
    if (ev) cudaEventRecord(ev[3], st);
    rcwa_schur<<<e.ncell, kSchurThreads, schur_smem(e.ncell), st>>>(e);
    if (ev) cudaEventRecord(ev[4], st);
    rcwa_vec<<<e.ncell, T[ST_VEC], 0, st>>>(e);
    if (ev) cudaEventRecord(ev[5], st);
    if (b.sym) {
        rcwa_sym_smat<<<e.ncell, 512, slab::shared_bytes(e.n), st>>>(b);
        if (ev) cudaEventRecord(ev[6], st);
        rcwa_sym_expand<<<nc, T[ST_SMAT2], 0, st>>>(b);
        if (ev) cudaEventRecord(ev[7], st);
        rcwa_epilogue<<<nc, T[ST_EPI], 0, st>>>(b);
        if (ev) cudaEventRecord(ev[8], st);
        return;
    }
    if (eig_only) return;
    const size_t sm_stage = lu_stage_bytes(n);
    rcwa_smat1<<<nc, T[ST_SMAT1], sm_stage, st>>>(b);
    if (ev) cudaEventRecord(ev[6], st);
    rcwa_smat2<<<nc, T[ST_SMAT2], sm_stage, st>>>(b);
    if (ev) cudaEventRecord(ev[7], st);
    rcwa_epilogue<<<nc, T[ST_EPI], 0, st>>>(b);
    if (ev) cudaEventRecord(ev[8], st);
}

// Time each stage at every candidate size on (up to) the first 2 x SMs cells
// of the bucket; keep the faster size per stage.
int autotune(const BucketPlan& p, cudaStream_t st, StageCfg* out) {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    Bucket t = p.b;
    t.ncell = std::min(t.ncell, 2 * sms);
    cudaEvent_t ev[ST_COUNT + 1];
    for (auto& e : ev) CEL_CUDA(cudaEventCreate(&e));
    float best[ST_COUNT];
    StageCfg cfg = uniform_cfg(256);
    for (int c = 0; c < 2; ++c) {
        launch_bucket(t, uniform_cfg(kCand[c]), st, ev, p.qr != 0);
        CEL_CUDA(cudaStreamSynchronize(st));
        for (int s = 0; s < ST_COUNT; ++s) {
            float ms = 0.f;
            cudaEventElapsedTime(&ms, ev[s], ev[s + 1]);
            if (c == 0 || ms < best[s]) {
                best[s] = ms;
                cfg.threads[s] = kCand[c];
            }
        }
    }
    for (auto& e : ev) cudaEventDestroy(e);
    CEL_CUDA(cudaGetLastError());
    *out = cfg;
    return CELERIS_OK;
}

// Per-thread execution context: streams, pinned staging and the cached graph.
// The device objects follow the thread's current device (rebuilt when it
// changes) and are released, with the main stream's workspace arena, when the
// thread exits.
struct BatchCtx {
    int dev = -1;
    cudaStream_t main = nullptr;
    std::vector<cudaStream_t> side;
    cudaEvent_t fork = nullptr;
    std::vector<cudaEvent_t> join;
    void* pinned = nullptr;
    size_t pinned_cap = 0;
    cudaGraphExec_t exec = nullptr;
    std::string sig;
    uint64_t nkern = 0;  // kernels per graph launch

    void drop_device_objects() {
        if (!main) return;
        int cur = 0;
        cudaGetDevice(&cur);
        cudaSetDevice(dev);
        cudaStreamSynchronize(main);
        for (cudaStream_t s : side) cudaStreamSynchronize(s);
        if (exec) cudaGraphExecDestroy(exec);
        exec = nullptr;
        sig.clear();
        Workspace::release_stream(main);
        for (cudaStream_t s : side) {
            Workspace::release_stream(s);
            cudaStreamDestroy(s);
        }
        if (fork) cudaEventDestroy(fork);
        fork = nullptr;
        for (cudaEvent_t e : join) cudaEventDestroy(e);
        cudaStreamDestroy(main);
        side.clear();
        join.clear();
        main = nullptr;
        dev = -1;
        cudaSetDevice(cur);
        cudaGetLastError();  // a failure here (e.g. the runtime shutting down) is nobody's call's error
    }
    ~BatchCtx() {
        drop_device_objects();
        if (pinned) cudaFreeHost(pinned);
        cudaGetLastError();
    }
};
thread_local BatchCtx t_ctx;

int ensure_streams(int nb) {
    BatchCtx& c = t_ctx;
    int cur = 0;
    CEL_CUDA(cudaGetDevice(&cur));
    if (c.main && c.dev != cur) c.drop_device_objects();
    if (!c.main) {
        CEL_CUDA(cudaEventCreateWithFlags(&c.fork, cudaEventDisableTiming));
        const cudaError_t e = cudaStreamCreateWithFlags(&c.main, cudaStreamNonBlocking);
        if (e != cudaSuccess) {
            cudaEventDestroy(c.fork);
            c.fork = nullptr;
            c.main = nullptr;
            return celeris_rt::cuda_error(e, "stream of the RCWA batch");
        }
        c.dev = cur;
    }
    while ((int)c.side.size() < nb) {
        cudaStream_t s;
        cudaEvent_t j;
        CEL_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
        CEL_CUDA(cudaEventCreateWithFlags(&j, cudaEventDisableTiming));
        c.side.push_back(s);
        c.join.push_back(j);
    }
    return CELERIS_OK;
}

// Free device memory, cached per device for the batch planner.
struct FreeMemCache {
    std::mutex mu;
    std::map<int, std::pair<size_t, std::chrono::steady_clock::time_point>> by_dev;
};
FreeMemCache& free_mem_cache() {
    static FreeMemCache c;
    return c;
}
int query_free_memory(int dev, size_t* free_b) {
    size_t total_b = 0;
    CEL_CUDA(cudaMemGetInfo(free_b, &total_b));
    FreeMemCache& c = free_mem_cache();
    std::lock_guard<std::mutex> lk(c.mu);
    c.by_dev[dev] = {*free_b, std::chrono::steady_clock::now()};
    return CELERIS_OK;
}
// The cached figure if it is under 2 s old, else 0.
size_t cached_free_memory(int dev) {
    FreeMemCache& c = free_mem_cache();
    std::lock_guard<std::mutex> lk(c.mu);
    const auto it = c.by_dev.find(dev);
    if (it == c.by_dev.end()) return 0;
    const double age = std::chrono::duration<double>(std::chrono::steady_clock::now() - it->second.second).count();
    return age < 2.0 ? it->second.first : 0;
}

int run_cells(std::vector<HostCell>& cells, celeris_rcwa_result* out, int* info_out, int nexc) {
    CEL_TRY(celeris_rt::require_device());
    // ---- plan: buckets by (Mx, My, raster), largest first so they start first
    std::map<std::tuple<int, int, int, int, int>, std::vector<int>> by;
    for (int i = 0; i < (int)cells.size(); ++i)
        by[std::make_tuple(cells[i].Mx, cells[i].My, cells[i].ng, cells[i].sym, cells[i].qr)].push_back(i);
    std::vector<BucketPlan> plans;
    std::vector<std::vector<int>> waves;
    CEL_TRY(ensure_streams(1));
    int dev = 0, smem_optin = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    Workspace& ws0 = Workspace::for_stream(t_ctx.main);
    // the memory budget: a free-memory figure up to 2 s old is used only when
    // the resulting plan needs no larger arena (no allocation can then fail);
    // the query itself is a driver call that costs ~0.1-1 ms, a sizeable part
    // of a small batch
    bool fresh = false;
    size_t free_b = cached_free_memory(dev);
    if (free_b == 0) {
        CEL_TRY(query_free_memory(dev, &free_b));
        fresh = true;
    }
    auto make_plan = [&](size_t free_now) -> int {
        plans.clear();
        waves.clear();
        const size_t budget = (size_t)(0.6 * (double)(free_now + ws0.capacity()));
        for (auto& kv : by) {
            BucketPlan p;
            p.Mx = std::get<0>(kv.first);
            p.My = std::get<1>(kv.first);
            p.ng = std::get<2>(kv.first);
            p.sym = std::get<3>(kv.first);
            p.qr = std::get<4>(kv.first);
            p.N = (2 * p.Mx + 1) * (2 * p.My + 1);
            p.n = 2 * p.N;
            if (p.ng > 0 && laurent_smem(p.Mx, p.My, p.ng) + 1024 > (size_t)smem_optin)
                return set_error(CELERIS_ERR_TOO_LARGE, "raster %d with M=(%d,%d) exceeds shared memory", p.ng, p.Mx, p.My);
            p.per_cell = p.sym  ? sym_per_cell_bytes(p.Mx, p.My, p.ng, nexc, p.sym == 2 ? 1 : 2, p.qr)
                         : p.qr ? per_cell_bytes(p.n, nexc)
                                : slab_per_cell_bytes(p.n, nexc);
            // split buckets that alone exceed the budget
            const size_t max_cells = std::max<size_t>(1, budget / std::max<size_t>(1, p.per_cell));
            for (size_t c0 = 0; c0 < kv.second.size(); c0 += max_cells) {
                BucketPlan q = p;
                const size_t c1 = std::min(kv.second.size(), c0 + max_cells);
                q.ids.assign(kv.second.begin() + c0, kv.second.begin() + c1);
                q.bytes = q.per_cell * q.ids.size() +
                          (q.ng > 0 ? celeris_rt::align256(((size_t)(4 * q.Mx + 1) + (4 * q.My + 1)) * q.ng *
                                                           sizeof(cplx)) + 512
                                    : 0);
                plans.push_back(q);
            }
        }
        std::sort(plans.begin(), plans.end(), [](const BucketPlan& a, const BucketPlan& b) { return a.n > b.n; });
        // ---- waves of buckets that fit the memory budget together
        size_t acc = 0;
        for (int i = 0; i < (int)plans.size(); ++i) {
            if (waves.empty() || acc + plans[i].bytes > budget) {
                waves.emplace_back();
                acc = 0;
            }
            waves.back().push_back(i);
            acc += plans[i].bytes;
        }
        return CELERIS_OK;
    };
    CEL_TRY(make_plan(free_b));
    if (!fresh) {
        size_t max_need = 0;
        for (const auto& wave : waves) {
            size_t need = 0;
            for (int i : wave) need += plans[i].bytes + 4096;
            max_need = std::max(max_need, need);
        }
        if (max_need > ws0.capacity()) {  // the arena must grow: plan on a fresh figure
            CEL_TRY(query_free_memory(dev, &free_b));
            CEL_TRY(make_plan(free_b));
        }
    }
    std::vector<celeris_rcwa_result> hres(cells.size() * nexc);
    std::vector<int> hinfo(cells.size(), 0);
    const bool prof = std::getenv("CELERIS_RCWA_STAGE_CLOCKS") != nullptr;
    for (const auto& wave : waves) {
        CEL_TRY(ensure_streams((int)wave.size()));
        BatchCtx& ctx = t_ctx;
        cudaStream_t st = ctx.main;
        Workspace& ws = Workspace::for_stream(st);
        size_t need = 0, pin_need = 0;
        for (int i : wave) {
            need += plans[i].bytes + 4096;
            pin_need += celeris_rt::align256(sizeof(CellDev) * plans[i].ids.size()) +
                        celeris_rt::align256(sizeof(celeris_rcwa_result) * nexc * plans[i].ids.size()) +
                        celeris_rt::align256(sizeof(int) * plans[i].ids.size());
        }
        void* old_base = ws.base();
        CEL_TRY(ws.reserve(st, need));
        if (ws.base() != old_base && ctx.exec) {  // the cached graph points at the old arena
            cudaGraphExecDestroy(ctx.exec);
            ctx.exec = nullptr;
            ctx.sig.clear();
        }
        if (ctx.pinned_cap < pin_need) {
            if (ctx.exec) {
                cudaGraphExecDestroy(ctx.exec);
                ctx.exec = nullptr;
                ctx.sig.clear();
            }
            if (ctx.pinned) cudaFreeHost(ctx.pinned);
            ctx.pinned = nullptr;
            ctx.pinned_cap = 0;
            CEL_CUDA(cudaHostAlloc(&ctx.pinned, pin_need, cudaHostAllocDefault));
            ctx.pinned_cap = pin_need;
        }
        // ---- carve the arena and the pinned staging, fill the descriptors
        char* pin = static_cast<char*>(ctx.pinned);
        std::string sig = "n" + std::to_string(nexc);
        std::vector<CellDev*> hdesc(wave.size());
        std::vector<celeris_rcwa_result*> hres_pin(wave.size());
        std::vector<int*> hinfo_pin(wave.size());
        SmemNeeds needs;
        for (size_t w = 0; w < wave.size(); ++w) {
            BucketPlan& p = plans[wave[w]];
            const int nc = (int)p.ids.size();
            Bucket& b = p.b;
            std::memset(&b, 0, sizeof(b));
            b.Mx = p.Mx;
            b.My = p.My;
            b.N = p.N;
            b.n = p.n;
            b.ng = p.ng;
            b.ncell = nc;
            b.s_nn = (size_t)p.n * p.n;
            b.s_ns = (size_t)p.n * (p.n + 2);
            b.s_NN = (size_t)p.N * p.N;
            b.s_n = (size_t)p.n;
            CellDev* dcells = static_cast<CellDev*>(ws.take(sizeof(CellDev) * nc));
            b.cells = dcells;
            auto take = [&](size_t count) { return static_cast<cplx*>(ws.take(sizeof(cplx) * count)); };
            if (p.sym) b.s_nn = sym_scratch(p.Mx, p.My);  // Z and X are its only square buffers
            if (p.qr && !p.sym) {
                cplx** mats[] = {&b.H, &b.Z, &b.X, &b.W, &b.A, &b.T11, &b.T11lu, &b.T12};
                for (cplx** m : mats) *m = take(b.s_nn * nc);
                b.S12 = take(b.s_ns * nc);
                b.q1 = take(b.s_n * nc);
            } else if (p.sym) {
                for (cplx** m : {&b.Z, &b.X}) *m = take(b.s_nn * nc);
                b.s_g1 = sym_g1_size(p.Mx, p.My, p.ng);
                b.G1 = take(b.s_g1 * nc);
            } else {
                b.Kp = take(b.s_nn * nc);
                b.s_w = slab::work_size(p.n);
                b.slab = take(b.s_w * nc);
                place_operators(b);
            }
            if (!p.sym) {
                if (p.qr)
                    for (cplx** m : {&b.Einv, &b.Exx, &b.Eyy}) *m = take(b.s_NN * nc);
                b.piv = static_cast<int*>(ws.take(sizeof(int) * b.s_n * nc));
            }
            b.vec = take(10 * b.s_n * nc);
            b.info = static_cast<int*>(ws.take(sizeof(int) * nc));
            b.res = static_cast<celeris_rcwa_result*>(ws.take(sizeof(celeris_rcwa_result) * nexc * nc));
            if (p.ng > 0 && p.sym) {  // one table for both axes
                const size_t mt = 2 * std::max(p.Mx, p.My) + 1;
                b.phx = b.phy = take(mt * p.ng);
                b.pcx = take(mt * (p.ng + 1));
            } else if (p.ng > 0) {
                b.phx = take((size_t)(4 * p.Mx + 1) * p.ng);
                b.phy = take((size_t)(4 * p.My + 1) * p.ng);
            }
            b.sym = p.sym;
            b.sym_tol = symmetry_tolerance();
            if (p.sym) {
                // the excited classes of order m
                b.ncls = p.sym == 2 ? 1 : 2;
                b.cls0 = p.sym == 2 ? 1 : 0;
                b.m = sym_class_size(p.Mx, p.My, 0);
                const size_t nm = (size_t)b.ncls * nc, m = (size_t)b.m;  // class matrices in the bucket
                b.cM = take(m * m * nm);
                b.cKp = take(m * m * nm);
                b.cvec = take(2 * m * nm);
                if (p.qr) {
                    for (cplx** x : {&b.sZ, &b.sX, &b.sW, &b.sA}) *x = take(m * m * nm);
                    b.sq = take(m * nm);
                    b.sinfo = static_cast<int*>(ws.take(sizeof(int) * nm));
                }
            }
            hdesc[w] = reinterpret_cast<CellDev*>(pin);
            pin += celeris_rt::align256(sizeof(CellDev) * nc);
            hres_pin[w] = reinterpret_cast<celeris_rcwa_result*>(pin);
            pin += celeris_rt::align256(sizeof(celeris_rcwa_result) * nexc * nc);
            hinfo_pin[w] = reinterpret_cast<int*>(pin);
            pin += celeris_rt::align256(sizeof(int) * nc);
            for (int i = 0; i < nc; ++i) hdesc[w][i] = cells[p.ids[i]].d;
            needs.add(p.Mx, p.My, p.ng, p.n, p.sym, p.qr);
            sig += "|" + std::to_string(p.Mx) + "," + std::to_string(p.My) + "," + std::to_string(p.ng) + "," +
                   std::to_string(p.sym) + "," + std::to_string(p.qr) + "," + std::to_string(nc) + "," +
                   exact_text(b.sym_tol);  // the tolerance is an argument of the captured kernels
        }
        CEL_TRY(set_smem_limits(needs));
        // ---- tune unseen bucket shapes (descriptors must be on the device)
        std::vector<StageCfg> cfgs(wave.size(), uniform_cfg(256));
        for (size_t w = 0; w < wave.size(); ++w) {
            const BucketPlan& p = plans[wave[w]];
            // key: shape and batch class (fewer than, or at least, one cell per SM)
            int sms = 148;
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
            const auto key = std::make_tuple(p.Mx, p.My, 8 * p.ng + (p.qr ? 0 : 4) + 2 * (p.sym != 0) + ((int)p.ids.size() >= sms ? 1 : 0));
            bool have = false;
            {
                std::lock_guard<std::mutex> lk(g_tune_mu);
                auto it = tune_table().find(key);
                if (it != tune_table().end()) {
                    cfgs[w] = it->second;
                    have = true;
                }
            }
            if (!have && tuning_enabled() && !prof) {
                CEL_CUDA(cudaMemcpyAsync(const_cast<CellDev*>(p.b.cells), hdesc[w], sizeof(CellDev) * p.ids.size(),
                                         cudaMemcpyHostToDevice, st));
                CEL_TRY(autotune(p, st, &cfgs[w]));
                std::lock_guard<std::mutex> lk(g_tune_mu);
                tune_table()[key] = cfgs[w];
            }
            for (int s = 0; s < ST_COUNT; ++s) sig += (cfgs[w].threads[s] == 128 ? "a" : "b");
        }
        if (prof) {
            // diagnostics: one bucket after the other, events per stage
            for (size_t w = 0; w < wave.size(); ++w) {
                BucketPlan& p = plans[wave[w]];
                const int nc = (int)p.ids.size();
                CEL_CUDA(cudaMemcpyAsync(const_cast<CellDev*>(p.b.cells), hdesc[w], sizeof(CellDev) * nc,
                                         cudaMemcpyHostToDevice, st));
                long long* dbg = nullptr;  // 2 nc slots: a class bucket has up to two matrices per cell
                CEL_CUDA(cudaMalloc(&dbg, sizeof(long long) * kDbgSlots * 2 * nc));
                CEL_CUDA(cudaMemsetAsync(dbg, 0, sizeof(long long) * kDbgSlots * 2 * nc, st));
                p.b.dbg = dbg;
                cudaEvent_t ev[ST_COUNT + 1];
                for (auto& e : ev) cudaEventCreate(&e);
                launch_bucket(p.b, cfgs[w], st, ev, p.qr != 0);
                CEL_CUDA(cudaMemcpyAsync(hres_pin[w], p.b.res, sizeof(celeris_rcwa_result) * nexc * nc,
                                         cudaMemcpyDeviceToHost, st));
                CEL_CUDA(cudaMemcpyAsync(hinfo_pin[w], p.b.info, sizeof(int) * nc, cudaMemcpyDeviceToHost, st));
                CEL_CUDA(cudaStreamSynchronize(st));
                std::vector<long long> h(kDbgSlots * 2 * nc);
                cudaMemcpy(h.data(), dbg, sizeof(long long) * kDbgSlots * 2 * nc, cudaMemcpyDeviceToHost);
                double sw = 0, ph[kDbgSlots] = {};
                for (int i = 0; i < 2 * nc; ++i) {
                    sw += (double)h[kDbgSlots * i + 6];
                    for (int q = 0; q < kDbgSlots; ++q) ph[q] += (double)h[kDbgSlots * i + q];
                }
                std::string line = "[rcwa stages] n=" + std::to_string(p.n) + " cells=" + std::to_string(nc) + " ms:";
                for (int s = 0; s < ST_COUNT; ++s) {
                    float ms = 0.f;
                    cudaEventElapsedTime(&ms, ev[s], ev[s + 1]);
                    char buf[64];
                    std::snprintf(buf, sizeof(buf), " %s %.2f", kStageNames[s], ms);
                    line += buf;
                }
                if (!p.qr) {
                    char b3[256];
                    std::snprintf(b3, sizeof(b3), " | two-port Mcycles/cell: %.3f (between the half-spaces %.3f); panels %.3f, their updates %.3f; "
                                  "left-out doublings %.3f\n",
                                  ph[2] / nc * 1e-6, ph[3] / nc * 1e-6, ph[0] / nc * 1e-6, ph[1] / nc * 1e-6, ph[4] / nc);
                    std::fprintf(stderr, "%s%s", line.c_str(), b3);
                    for (auto& e : ev) cudaEventDestroy(e);
                    cudaFree(dbg);
                    p.b.dbg = nullptr;
                    continue;
                }
                char buf[64];
                std::snprintf(buf, sizeof(buf), " | sweeps/cell %.1f", sw / nc);
                char buf2[512];
                std::snprintf(buf2, sizeof(buf2), " | schur Mcycles/cell: aed %.2f (qr %.2f, %.0f rot) aed_far %.2f sweep %.2f (%.0f steps) sweep_far %.2f small %.2f"
                              " | hess Mcycles/cell: columns %.2f (matvec %.2f) updates %.2f"
                              " | small QR Mcycles/cell: aed chase %.2f deferred %.2f, block chase %.2f deferred %.2f\n",
                              ph[0] / nc * 1e-6, ph[5] / nc * 1e-6, ph[8] / nc, ph[1] / nc * 1e-6, ph[2] / nc * 1e-6,
                              ph[7] / nc, ph[3] / nc * 1e-6, ph[4] / nc * 1e-6, ph[9] / nc * 1e-6, ph[10] / nc * 1e-6,
                              ph[11] / nc * 1e-6, ph[12] / nc * 1e-6, ph[13] / nc * 1e-6, ph[14] / nc * 1e-6,
                              ph[15] / nc * 1e-6);
                std::fprintf(stderr, "%s%s%s", line.c_str(), buf, buf2);
                for (auto& e : ev) cudaEventDestroy(e);
                cudaFree(dbg);
                p.b.dbg = nullptr;
            }
        } else {
            // ---- the whole wave as one CUDA graph: descriptors in, every bucket
            // on its own stream (fork/join), results out; cached per shape.
            if (!ctx.exec || ctx.sig != sig) {
                if (ctx.exec) {
                    cudaGraphExecDestroy(ctx.exec);
                    ctx.exec = nullptr;
                }
                cudaGraph_t graph = nullptr;
                CEL_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
                celeris_rt::set_launch_counting(false);
                uint64_t nk = 0;
                // one fork before the first bucket and the joins behind the last: a join in
                // between would hold the next bucket's fork back until the buckets before it are done
                cudaEventRecord(ctx.fork, st);
                for (size_t w = 0; w < wave.size(); ++w) {
                    const BucketPlan& p = plans[wave[w]];
                    const int nc = (int)p.ids.size();
                    cudaStream_t bs = ctx.side[w];
                    cudaStreamWaitEvent(bs, ctx.fork, 0);
                    cudaMemcpyAsync(const_cast<CellDev*>(p.b.cells), hdesc[w], sizeof(CellDev) * nc,
                                    cudaMemcpyHostToDevice, bs);
                    launch_bucket(p.b, cfgs[w], bs, nullptr, p.qr != 0);
                    nk += bucket_kernels(p.sym != 0, p.ng, p.qr != 0);
                    cudaMemcpyAsync(hres_pin[w], p.b.res, sizeof(celeris_rcwa_result) * nexc * nc,
                                    cudaMemcpyDeviceToHost, bs);
                    cudaMemcpyAsync(hinfo_pin[w], p.b.info, sizeof(int) * nc, cudaMemcpyDeviceToHost, bs);
                    cudaEventRecord(ctx.join[w], bs);
                }
                for (size_t w = 0; w < wave.size(); ++w) cudaStreamWaitEvent(st, ctx.join[w], 0);
                const cudaError_t ce = cudaStreamEndCapture(st, &graph);
                celeris_rt::set_launch_counting(true);
                if (ce != cudaSuccess) return celeris_rt::cuda_error(ce, "capture of the RCWA batch");
                const cudaError_t ie = cudaGraphInstantiate(&ctx.exec, graph, 0);
                cudaGraphDestroy(graph);
                if (ie != cudaSuccess) {
                    ctx.exec = nullptr;
                    return celeris_rt::cuda_error(ie, "instantiate the RCWA batch graph");
                }
                ctx.sig = sig;
                ctx.nkern = nk;
            }
            CEL_CUDA(cudaGraphLaunch(ctx.exec, st));
            count_launch(ctx.nkern);
            CEL_CUDA(cudaStreamSynchronize(st));
        }
        CEL_CUDA(cudaGetLastError());
        for (size_t w = 0; w < wave.size(); ++w) {
            const BucketPlan& p = plans[wave[w]];
            for (int i = 0; i < (int)p.ids.size(); ++i) {
                const int idx = cells[p.ids[i]].index;
                for (int e = 0; e < nexc; ++e) hres[(size_t)idx * nexc + e] = hres_pin[w][(size_t)i * nexc + e];
                hinfo[idx] = hinfo_pin[w][i];
            }
        }
    }
    // cells flagged as not mirror symmetric to rounding are solved again at full order,
    // cells whose two-port was ill conditioned through the eigendecomposition
    std::vector<int> redo;
    for (size_t i = 0; i < hinfo.size(); ++i)
        if (hinfo[i] == kInfoAsym || hinfo[i] == kInfoRedo) redo.push_back((int)i);
    if (!redo.empty()) {
        std::vector<int> pos(cells.size(), -1);
        for (int i = 0; i < (int)cells.size(); ++i) pos[cells[i].index] = i;
        std::vector<HostCell> sub;
        for (size_t j = 0; j < redo.size(); ++j) {
            HostCell h = cells[pos[redo[j]]];
            if (hinfo[redo[j]] == kInfoAsym) h.sym = 0;
            h.qr = h.qr || hinfo[redo[j]] == kInfoRedo || (!h.sym && 2 * (2 * h.Mx + 1) * (2 * h.My + 1) > slab::kMaxOrder);
            h.index = (int)j;
            sub.push_back(h);
        }
        std::vector<celeris_rcwa_result> sub_out(sub.size() * nexc);
        std::vector<int> sub_info(sub.size(), 0);
        CEL_TRY(run_cells(sub, sub_out.data(), sub_info.data(), nexc));
        for (size_t j = 0; j < redo.size(); ++j) {
            for (int e = 0; e < nexc; ++e) hres[(size_t)redo[j] * nexc + e] = sub_out[j * nexc + e];
            hinfo[redo[j]] = sub_info[j];
        }
    }
    std::memcpy(out, hres.data(), sizeof(celeris_rcwa_result) * hres.size());
    int first_bad = -1;
    for (size_t i = 0; i < hinfo.size(); ++i) {
        if (info_out) info_out[i] = hinfo[i];
        if (hinfo[i] != 0 && first_bad < 0) first_bad = (int)i;
    }
    // with an info array the per-cell codes are the report (LAPACK style)
    if (first_bad >= 0 && !info_out) {
        const int v = hinfo[first_bad];
        return set_error(v > 0 ? CELERIS_ERR_EIG_NOCONV : CELERIS_ERR_SINGULAR,
                         "cell %d: %s (info %d)", first_bad,
                         v > 0 ? "QR eigensolve did not converge" : "singular pivot in an LU factorization", v);
    }
    return CELERIS_OK;
}

// ---- multi-layer stacks ----------------------------------------------------------------------
// Sub-allocation from one reserved region (the stack path's per-stream
// workspace arena): no cudaMalloc / cudaFree per call.
struct Bump {
    char* p = nullptr;
    size_t left = 0;
    template <typename T>
    int get(T** out, size_t count) {
        const size_t b = celeris_rt::align256(std::max<size_t>(count, 1) * sizeof(T));
        if (b > left) return set_error(CELERIS_ERR_OOM, "stack workspace: carve of %zu bytes over its plan", b);
        *out = reinterpret_cast<T*>(p);
        p += b;
        left -= b;
        return CELERIS_OK;
    }
};
size_t a256(size_t b) { return celeris_rt::align256(std::max<size_t>(b, 1)); }

// stacks[s] = (first layer index, layer count) into `layers`; exc holds 4 doubles
// (Ex0 re, im, Ey0 re, im) per stack; results nexc per stack.
// ord_out (may be NULL): per stack and excitation N x (de_t, de_r).
// Through the eigendecompositions of the layers (rcwa_stack_smat).
int run_stacks_qr(const celeris_rcwa_cell* layers, const std::vector<std::pair<int, int>>& stacks,
                  const double* exc, celeris_rcwa_result* out, int* info_out, int nexc, double* ord_out) {
    CEL_TRY(celeris_rt::require_device());
    int dev = 0, smem_optin = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    // one stream (and so one workspace arena) per calling thread for the stack path
    static thread_local celeris_rt::ThreadStream t_stack_st;
    cudaStream_t st = nullptr;
    CEL_TRY(t_stack_st.get(&st));
    Workspace& ws = Workspace::for_stream(st);
    // stacks grouped by (Mx, My): one layer store and one recursion launch per group
    std::map<std::pair<int, int>, std::vector<int>> groups;
    for (int s = 0; s < (int)stacks.size(); ++s) {
        const celeris_rcwa_cell& f = layers[stacks[s].first];
        groups[{f.Mx, f.My}].push_back(s);
    }
    size_t free_b = 0, total_b = 0;
    CEL_CUDA(cudaMemGetInfo(&free_b, &total_b));
    const size_t budget = free_b / 2;
    for (auto& g : groups) {
        const int Mx = g.first.first, My = g.first.second;
        const int N = (2 * Mx + 1) * (2 * My + 1), n = 2 * N;
        const size_t s_nn = (size_t)n * n, s_n = (size_t)n, s_NN = (size_t)N * N;
        // stacks in chunks whose layer store, eigen buffers and recursion buffers fit the budget
        const size_t per_layer = (7 * s_nn + 3 * s_NN + 4 * s_n) * sizeof(cplx) + 4096;
        const size_t per_stack = (7 * s_nn + 11 * s_n) * sizeof(cplx) + 4096;
        size_t c0 = 0;
        while (c0 < g.second.size()) {
            std::vector<int> ids;
            size_t bytes = 0;
            while (c0 < g.second.size()) {
                const size_t need = per_stack + per_layer * stacks[g.second[c0]].second;
                if (!ids.empty() && bytes + need > budget) break;
                ids.push_back(g.second[c0++]);
                bytes += need;
            }
            const int ns = (int)ids.size();
            // layer store slots, in stack order
            std::vector<HostCell> sub;
            std::vector<int> first_slot(ns);
            for (int k = 0; k < ns; ++k) {
                first_slot[k] = (int)sub.size();
                const auto& sp = stacks[ids[k]];
                for (int l = 0; l < sp.second; ++l)
                    sub.push_back(make_cell(layers[sp.first + l], (int)sub.size(), 1.0, 0.0, 0.0, 0.0, 2));
            }
            const int nslot = (int)sub.size();
            std::map<int, std::vector<int>> by_ng;
            for (int i = 0; i < nslot; ++i) by_ng[sub[i].ng].push_back(i);
            // region plan: layer store + recursion, then one raster class's bucket at a time
            const size_t c16 = sizeof(cplx);
            size_t fixed = 2 * a256(s_nn * nslot * c16) + a256(s_n * nslot * c16) + a256(nslot * sizeof(double)) +
                           7 * a256(s_nn * ns * c16) + a256(10 * s_n * ns * c16) + a256(s_n * ns * sizeof(int)) +
                           a256(ns * sizeof(int)) + a256(ns * sizeof(CellDev)) + a256(ns * sizeof(StackDev)) +
                           a256(ns * nexc * sizeof(celeris_rcwa_result));
            if (ord_out) fixed += a256((size_t)ns * nexc * N * 2 * sizeof(double));
            size_t class_max = 0;
            for (auto& kv : by_ng) {
                const size_t nc = kv.second.size(), ng = (size_t)std::max(kv.first, 0);
                size_t b = a256(nc * sizeof(CellDev)) + 5 * a256(s_nn * nc * c16) + 3 * a256(s_NN * nc * c16) +
                           a256(s_n * nc * c16) + a256(s_n * nc * sizeof(int)) + 2 * a256(nc * sizeof(int));
                if (ng > 0) b += a256((4 * Mx + 1) * ng * c16) + a256((4 * My + 1) * ng * c16);
                class_max = std::max(class_max, b);
            }
            CEL_TRY(ws.reserve(st, fixed + class_max));
            char* region = static_cast<char*>(ws.take(fixed + class_max));
            Bump mem{region, fixed};
            cplx *LW, *LA, *Lq;
            double* Lh;
            CEL_TRY(mem.get(&LW, s_nn * nslot));
            CEL_TRY(mem.get(&LA, s_nn * nslot));
            CEL_TRY(mem.get(&Lq, s_n * nslot));
            CEL_TRY(mem.get(&Lh, (size_t)nslot));
            std::vector<int> sub_info(nslot, 0);
            // eigen-solutions of every layer, one bucket per raster class
            for (auto& kv : by_ng) {
                const int ng = kv.first;
                const std::vector<int>& si = kv.second;
                const int nc = (int)si.size();
                if (ng > 0 && laurent_smem(Mx, My, ng) + 1024 > (size_t)smem_optin)
                    return set_error(CELERIS_ERR_TOO_LARGE, "raster %d with M=(%d,%d) exceeds shared memory", ng,
                                     Mx, My);
                Bump bm{region + fixed, class_max};  // reused by each class in turn (the stream is synchronised)
                Bucket b;
                std::memset(&b, 0, sizeof(b));
                b.Mx = Mx;
                b.My = My;
                b.N = N;
                b.n = n;
                b.ng = ng;
                b.ncell = nc;
                b.s_nn = s_nn;
                b.s_ns = (size_t)n * (n + 2);
                b.s_NN = s_NN;
                b.s_n = s_n;
                CellDev* dcells;
                CEL_TRY(bm.get(&dcells, (size_t)nc));
                b.cells = dcells;
                cplx** mats[] = {&b.H, &b.Z, &b.X, &b.W, &b.A};
                for (cplx** m : mats) CEL_TRY(bm.get(m, s_nn * nc));
                CEL_TRY(bm.get(&b.Einv, s_NN * nc));
                CEL_TRY(bm.get(&b.Exx, s_NN * nc));
                CEL_TRY(bm.get(&b.Eyy, s_NN * nc));
                CEL_TRY(bm.get(&b.q1, s_n * nc));
                CEL_TRY(bm.get(&b.piv, s_n * nc));
                CEL_TRY(bm.get(&b.info, (size_t)nc));
                if (ng > 0) {
                    cplx *phx, *phy;
                    CEL_TRY(bm.get(&phx, (size_t)(4 * Mx + 1) * ng));
                    CEL_TRY(bm.get(&phy, (size_t)(4 * My + 1) * ng));
                    b.phx = phx;
                    b.phy = phy;
                }
                std::vector<CellDev> hd(nc);
                std::vector<int> hslot(nc);
                for (int i = 0; i < nc; ++i) {
                    hd[i] = sub[si[i]].d;
                    hslot[i] = si[i];
                }
                int* dslot;
                CEL_TRY(bm.get(&dslot, (size_t)nc));
                CEL_CUDA(cudaMemcpyAsync(dcells, hd.data(), sizeof(CellDev) * nc, cudaMemcpyHostToDevice, st));
                CEL_CUDA(cudaMemcpyAsync(dslot, hslot.data(), sizeof(int) * nc, cudaMemcpyHostToDevice, st));
                SmemNeeds needs;
                needs.add(Mx, My, ng, n);
                CEL_TRY(set_smem_limits(needs));
                launch_bucket(b, uniform_cfg(256), st, nullptr, true, true);
                rcwa_layer_out<<<nc, kRT, 0, st>>>(b, LW, LA, Lq, Lh, dslot);
                count_launch(1);
                CEL_CUDA(cudaGetLastError());
                std::vector<int> hinfo(nc);
                CEL_CUDA(cudaMemcpyAsync(hinfo.data(), b.info, sizeof(int) * nc, cudaMemcpyDeviceToHost, st));
                CEL_CUDA(cudaStreamSynchronize(st));
                for (int i = 0; i < nc; ++i) sub_info[si[i]] = hinfo[i];
            }
            // S-matrix recursion and outputs, one CTA per stack
            StackBucket sb;
            std::memset(&sb, 0, sizeof(sb));
            sb.Mx = Mx;
            sb.My = My;
            sb.N = N;
            sb.n = n;
            sb.nstack = ns;
            sb.LW = LW;
            sb.LA = LA;
            sb.Lq = Lq;
            sb.Lh = Lh;
            sb.s_nn = s_nn;
            sb.s_n = s_n;
            cplx** smats[] = {&sb.S12, &sb.S22, &sb.Q, &sb.P, &sb.X, &sb.Y, &sb.Z1};
            for (cplx** m : smats) CEL_TRY(mem.get(m, s_nn * ns));
            CEL_TRY(mem.get(&sb.vec, 10 * s_n * ns));
            CEL_TRY(mem.get(&sb.piv, s_n * ns));
            CEL_TRY(mem.get(&sb.info, (size_t)ns));
            CellDev* scells;
            StackDev* sdev;
            celeris_rcwa_result* dres;
            CEL_TRY(mem.get(&scells, (size_t)ns));
            CEL_TRY(mem.get(&sdev, (size_t)ns));
            CEL_TRY(mem.get(&dres, (size_t)ns * nexc));
            std::vector<CellDev> hc(ns);
            std::vector<StackDev> hs(ns);
            std::vector<int> hinfo(ns, 0);
            for (int k = 0; k < ns; ++k) {
                const auto& sp = stacks[ids[k]];
                const double* e = exc + 4 * (size_t)ids[k];
                hc[k] = make_cell(layers[sp.first], ids[k], e[0], e[1], e[2], e[3], nexc).d;
                hs[k].nl = sp.second;
                hs[k].slot0 = first_slot[k];
                for (int l = 0; l < sp.second; ++l)
                    if (sub_info[first_slot[k] + l] != 0 && hinfo[k] == 0) hinfo[k] = sub_info[first_slot[k] + l];
            }
            CEL_CUDA(cudaMemcpyAsync(scells, hc.data(), sizeof(CellDev) * ns, cudaMemcpyHostToDevice, st));
            CEL_CUDA(cudaMemcpyAsync(sdev, hs.data(), sizeof(StackDev) * ns, cudaMemcpyHostToDevice, st));
            CEL_CUDA(cudaMemcpyAsync(sb.info, hinfo.data(), sizeof(int) * ns, cudaMemcpyHostToDevice, st));
            sb.cells = scells;
            sb.stacks = sdev;
            const size_t sm_stage = lu_stage_bytes(n);
            CEL_TRY(raise_dyn_smem(reinterpret_cast<const void*>(rcwa_stack_smat), sm_stage));
            rcwa_stack_smat<<<ns, kRT, sm_stage, st>>>(sb);
            Bucket eb;
            std::memset(&eb, 0, sizeof(eb));
            eb.Mx = Mx;
            eb.My = My;
            eb.N = N;
            eb.n = n;
            eb.ncell = ns;
            eb.cells = scells;
            eb.vec = sb.vec;
            eb.info = sb.info;
            eb.res = dres;
            eb.s_n = s_n;
            eb.s_nn = s_nn;
            if (ord_out) CEL_TRY(mem.get(&eb.ord, (size_t)ns * nexc * N * 2));
            rcwa_epilogue<<<ns, kRT, 0, st>>>(eb);
            count_launch(2);
            CEL_CUDA(cudaGetLastError());
            std::vector<celeris_rcwa_result> hres((size_t)ns * nexc);
            CEL_CUDA(cudaMemcpyAsync(hres.data(), dres, sizeof(celeris_rcwa_result) * ns * nexc,
                                     cudaMemcpyDeviceToHost, st));
            CEL_CUDA(cudaMemcpyAsync(hinfo.data(), sb.info, sizeof(int) * ns, cudaMemcpyDeviceToHost, st));
            std::vector<double> hord;
            if (ord_out) {
                hord.resize((size_t)ns * nexc * N * 2);
                CEL_CUDA(cudaMemcpyAsync(hord.data(), eb.ord, sizeof(double) * hord.size(), cudaMemcpyDeviceToHost,
                                         st));
            }
            CEL_CUDA(cudaStreamSynchronize(st));
            if (ord_out)
                for (int k = 0; k < ns; ++k)
                    std::memcpy(ord_out + (size_t)ids[k] * nexc * N * 2, hord.data() + (size_t)k * nexc * N * 2,
                                sizeof(double) * nexc * N * 2);
            for (int k = 0; k < ns; ++k) {
                for (int e = 0; e < nexc; ++e) out[(size_t)ids[k] * nexc + e] = hres[(size_t)k * nexc + e];
                if (info_out) info_out[ids[k]] = hinfo[k];
            }
            if (!info_out)
                for (int k = 0; k < ns; ++k) {
                    if (hinfo[k] > 0)
                        return set_error(CELERIS_ERR_EIG_NOCONV, "eigensolve did not converge (a layer of stack %d)",
                                         ids[k]);
                    if (hinfo[k] < 0)
                        return set_error(CELERIS_ERR_SINGULAR, "singular interface system (stack %d)", ids[k]);
                }
        }
    }
    return CELERIS_OK;
}

// Device memory of `ns` stacks of `nslot` layers in all, of order n, on the two-port path: three
// matrices a layer, and work areas for the layers or the stacks that run at a time. Up to eight layers
// per SM run in one launch: at one or two blocks per SM, more of them would save little.
size_t work_areas(size_t ns, size_t nslot, int sms) { return std::min(nslot, std::max(ns, (size_t)8 * sms)); }
size_t stacks_bytes(size_t ns, size_t nslot, int n, int nexc, int sms) {
    return (3 * (size_t)n * n * nslot + slab::work_size(n) * work_areas(ns, nslot, sms) + 10 * (size_t)n * ns) * sizeof(cplx) +
           (size_t)nexc * n * sizeof(double) * ns + 4096 * (ns + nslot);
}

// The same through the layers' two-ports (rcwa_slab, rcwa_stack_port). info_out (required):
// 0 or kInfoRedo per stack; results of flagged stacks are not written.
int run_stacks_slab(const celeris_rcwa_cell* layers, const std::vector<std::pair<int, int>>& stacks, const double* exc,
                    celeris_rcwa_result* out, int* info_out, int nexc, double* ord_out) {
    CEL_TRY(celeris_rt::require_device());
    int dev = 0, smem_optin = 0, sms = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    static thread_local celeris_rt::ThreadStream t_slab_st;
    cudaStream_t st = nullptr;
    CEL_TRY(t_slab_st.get(&st));
    Workspace& ws = Workspace::for_stream(st);
    // stacks grouped by (Mx, My): one layer store and one recursion launch per group
    std::map<std::pair<int, int>, std::vector<int>> groups;
    for (int s = 0; s < (int)stacks.size(); ++s) {
        const celeris_rcwa_cell& f = layers[stacks[s].first];
        groups[{f.Mx, f.My}].push_back(s);
    }
    const size_t c16 = sizeof(cplx);
    // the budget matters only when the arena must grow: the driver's query (a call that
    // can take milliseconds) is left out while every group fits the arena that is there
    size_t most = 0;
    for (auto& g : groups) {
        const int N = (2 * g.first.first + 1) * (2 * g.first.second + 1), n = 2 * N;
        size_t nslot = 0;
        for (int k : g.second) nslot += stacks[k].second;
        most = std::max(most, stacks_bytes(g.second.size(), nslot, n, nexc, sms) + ((size_t)1 << 22));
    }
    size_t budget = ws.capacity();
    if (most > budget) {
        size_t free_b = 0;
        CEL_TRY(query_free_memory(dev, &free_b));
        budget = (free_b + ws.capacity()) / 2;
    }
    for (auto& g : groups) {
        const int Mx = g.first.first, My = g.first.second;
        const int N = (2 * Mx + 1) * (2 * My + 1), n = 2 * N;
        const size_t s_nn = (size_t)n * n, s_n = (size_t)n, s_w = slab::work_size(n);
        size_t c0 = 0;
        while (c0 < g.second.size()) {
            std::vector<int> ids;
            size_t slots = 0;
            while (c0 < g.second.size()) {
                const size_t more = slots + stacks[g.second[c0]].second;
                if (!ids.empty() && stacks_bytes(ids.size() + 1, more, n, nexc, sms) > budget) break;
                ids.push_back(g.second[c0++]);
                slots = more;
            }
            const int ns = (int)ids.size();
            std::vector<HostCell> sub;
            std::vector<CellDev> head;
            std::vector<int2> hs(ns);
            for (int k = 0; k < ns; ++k) {
                const auto& sp = stacks[ids[k]];
                const double* e = exc + 4 * (size_t)ids[k];
                hs[k] = make_int2(sp.second, (int)sub.size());
                head.push_back(make_cell(layers[sp.first], ids[k], e[0], e[1], e[2], e[3], nexc).d);
                for (int l = 0; l < sp.second; ++l)
                    sub.push_back(make_cell(layers[sp.first + l], (int)sub.size(), 1.0, 0.0, 0.0, 0.0, 2));
            }
            const int nslot = (int)sub.size();
            // buckets by raster: (ng, cells)
            std::map<int, std::vector<int>> by_ng;
            for (int i = 0; i < nslot; ++i) by_ng[sub[i].ng].push_back(i);
            // one block up (descriptors), one block down (results, status words), the rest
            size_t up_bytes = a256(ns * sizeof(CellDev)) + a256(ns * sizeof(int2));
            size_t down_bytes = a256(ns * nexc * sizeof(celeris_rcwa_result)) + a256(ns * sizeof(int));
            if (ord_out) down_bytes += a256((size_t)ns * nexc * N * 2 * sizeof(double));
            const size_t areas = work_areas(ns, nslot, sms);
            size_t fixed = 3 * a256(s_nn * nslot * c16) + a256(s_w * areas * c16) + a256(10 * s_n * ns * c16) +
                           a256(nslot * sizeof(int)) + a256(s_n * areas * sizeof(int));
            for (auto& kv : by_ng) {
                const size_t nc = kv.second.size(), ng = (size_t)std::max(kv.first, 0);
                up_bytes += a256(nc * sizeof(CellDev)) + a256(nc * sizeof(int));
                down_bytes += a256(nc * sizeof(int));
                if (ng > 0) fixed += a256((4 * Mx + 1) * ng * c16) + a256((4 * My + 1) * ng * c16);
            }
            CEL_TRY(ws.reserve(st, up_bytes + down_bytes + fixed));
            char* region = static_cast<char*>(ws.take(up_bytes + down_bytes + fixed));
            char* pin = static_cast<char*>(celeris_rt::pinned_staging(up_bytes + down_bytes));
            if (!pin) return set_error(CELERIS_ERR_OOM, "pinned staging of %zu bytes failed", up_bytes + down_bytes);
            Bump up{region, up_bytes}, down{region + up_bytes, down_bytes};
            Bump mem{region + up_bytes + down_bytes, fixed};
            // the host copy of a pointer into the up or down block
            auto host = [&](const void* d) { return pin + (static_cast<const char*>(d) - region); };
            StackPort sp;
            std::memset(&sp, 0, sizeof(sp));
            sp.Mx = Mx;
            sp.My = My;
            sp.n = n;
            sp.nstack = ns;
            sp.s_nn = s_nn;
            sp.s_w = s_w;
            sp.s_n = s_n;
            CEL_TRY(mem.get(&sp.lA, s_nn * nslot));
            CEL_TRY(mem.get(&sp.lB, s_nn * nslot));
            CEL_TRY(mem.get(&sp.lK, s_nn * nslot));
            CEL_TRY(mem.get(&sp.work, s_w * areas));  // the layers', then the stacks'
            int* piv;
            CEL_TRY(mem.get(&piv, s_n * areas));
            CEL_TRY(mem.get(&sp.vec, 10 * s_n * ns));
            CEL_TRY(down.get(&sp.info, (size_t)ns));
            int* lrest;
            CEL_TRY(mem.get(&lrest, (size_t)nslot));
            sp.lrest = lrest;
            CellDev* scells;
            int2* sstacks;
            celeris_rcwa_result* dres;
            CEL_TRY(up.get(&scells, (size_t)ns));
            CEL_TRY(up.get(&sstacks, (size_t)ns));
            CEL_TRY(down.get(&dres, (size_t)ns * nexc));
            sp.cells = scells;
            sp.stacks = sstacks;
            std::memcpy(host(scells), head.data(), sizeof(CellDev) * ns);
            std::memcpy(host(sstacks), hs.data(), sizeof(int2) * ns);
            // the layers' buckets, one per raster class
            std::vector<Bucket> buckets;
            for (auto& kv : by_ng) {
                const int ng = kv.first, nc = (int)kv.second.size();
                if (ng > 0 && laurent_smem(Mx, My, ng) + 1024 > (size_t)smem_optin)
                    return set_error(CELERIS_ERR_TOO_LARGE, "raster %d with M=(%d,%d) exceeds shared memory", ng,
                                     Mx, My);
                Bucket b;
                std::memset(&b, 0, sizeof(b));
                b.Mx = Mx;
                b.My = My;
                b.N = N;
                b.n = n;
                b.ng = ng;
                b.ncell = nc;
                b.s_nn = s_nn;
                b.s_n = s_n;
                b.s_w = s_w;
                b.slab = sp.work;
                place_operators(b);
                b.piv = piv;
                b.lA = sp.lA;
                b.lB = sp.lB;
                b.lK = sp.lK;
                b.lrest = lrest;
                CellDev* dcells;
                int* dslot;
                CEL_TRY(up.get(&dcells, (size_t)nc));
                CEL_TRY(down.get(&b.info, (size_t)nc));
                CEL_TRY(up.get(&dslot, (size_t)nc));
                if (ng > 0) {
                    cplx *phx, *phy;
                    CEL_TRY(mem.get(&phx, (size_t)(4 * Mx + 1) * ng));
                    CEL_TRY(mem.get(&phy, (size_t)(4 * My + 1) * ng));
                    b.phx = phx;
                    b.phy = phy;
                }
                b.cells = dcells;
                b.lslot = dslot;
                CellDev* hd = reinterpret_cast<CellDev*>(host(dcells));
                for (int i = 0; i < nc; ++i) hd[i] = sub[kv.second[i]].d;
                std::memcpy(host(dslot), kv.second.data(), sizeof(int) * nc);
                SmemNeeds needs;
                needs.add(Mx, My, ng, n, 0, 0);
                CEL_TRY(set_smem_limits(needs));
                buckets.push_back(b);
            }
            CEL_CUDA(cudaMemcpyAsync(region, pin, up_bytes, cudaMemcpyHostToDevice, st));
            CEL_CUDA(cudaMemsetAsync(region + up_bytes, 0, down_bytes, st));  // status words, results
            CEL_CUDA(cudaMemsetAsync(lrest, 0, sizeof(int) * nslot, st));
            for (const Bucket& b : buckets)
                for (int i = 0; i < b.ncell; i += (int)areas) {
                    Bucket part = b;
                    part.ncell = std::min(b.ncell - i, (int)areas);
                    part.cells += i;
                    part.lslot += i;
                    part.info += i;
                    launch_bucket(part, uniform_cfg(256), st, nullptr, false);
                }
            CEL_CUDA(cudaGetLastError());
            CEL_TRY(raise_dyn_smem(reinterpret_cast<const void*>(rcwa_stack_port), slab::shared_bytes(n)));
            rcwa_stack_port<<<ns, 512, slab::shared_bytes(n), st>>>(sp);
            Bucket eb;
            std::memset(&eb, 0, sizeof(eb));
            eb.Mx = Mx;
            eb.My = My;
            eb.N = N;
            eb.n = n;
            eb.ncell = ns;
            eb.cells = scells;
            eb.vec = sp.vec;
            eb.info = sp.info;
            eb.res = dres;
            eb.s_n = s_n;
            eb.s_nn = s_nn;
            if (ord_out) CEL_TRY(down.get(&eb.ord, (size_t)ns * nexc * N * 2));
            rcwa_epilogue<<<ns, kRT, 0, st>>>(eb);
            count_launch(2);
            CEL_CUDA(cudaGetLastError());
            CEL_CUDA(cudaMemcpyAsync(pin + up_bytes, region + up_bytes, down_bytes, cudaMemcpyDeviceToHost, st));
            CEL_CUDA(cudaStreamSynchronize(st));
            const auto* hres = reinterpret_cast<const celeris_rcwa_result*>(host(dres));
            const int* hinfo = reinterpret_cast<const int*>(host(sp.info));
            const double* hord = ord_out ? reinterpret_cast<const double*>(host(eb.ord)) : nullptr;
            // a flagged layer flags its stack (its part of the layer store was not written)
            std::vector<char> bad(nslot, 0);
            size_t k = 0;
            for (auto& kv : by_ng) {
                const int* li = reinterpret_cast<const int*>(host(buckets[k].info));
                for (size_t i = 0; i < kv.second.size(); ++i) bad[kv.second[i]] = li[i] != 0;
                ++k;
            }
            for (int i = 0; i < ns; ++i) {
                int f = hinfo[i];
                for (int l = 0; l < hs[i].x; ++l)
                    if (bad[hs[i].y + l]) f = kInfoRedo;
                info_out[ids[i]] = f;
                if (f != 0) continue;
                for (int e = 0; e < nexc; ++e) out[(size_t)ids[i] * nexc + e] = hres[(size_t)i * nexc + e];
                if (ord_out)
                    std::memcpy(ord_out + (size_t)ids[i] * nexc * N * 2, hord + (size_t)i * nexc * N * 2,
                                sizeof(double) * nexc * N * 2);
            }
        }
    }
    return CELERIS_OK;
}

// Stacks through the two-ports; those it does not take (needs_qr of a layer) and those
// it flags through the eigendecompositions.
int run_stacks(const celeris_rcwa_cell* layers, const std::vector<std::pair<int, int>>& stacks, const double* exc,
               celeris_rcwa_result* out, int* info_out, int nexc, double* ord_out = nullptr) {
    const int ns = (int)stacks.size();
    std::vector<int> info(ns, 0), direct, rest;
    for (int s = 0; s < ns; ++s) {
        bool qr = false;
        for (int l = 0; l < stacks[s].second; ++l) {
            const celeris_rcwa_cell& c = layers[stacks[s].first + l];
            qr = qr || needs_qr(c, full_order(c.Mx, c.My));  // stacks are solved in the order basis
        }
        (qr ? rest : direct).push_back(s);
    }
    // a subset of the stacks through one of the two, results back at their places
    auto run = [&](const std::vector<int>& sel, bool qr) -> int {
        if (sel.empty()) return CELERIS_OK;
        const int k = (int)sel.size();
        std::vector<std::pair<int, int>> st(k);
        std::vector<double> ex(4 * (size_t)k);
        std::vector<celeris_rcwa_result> res((size_t)k * nexc);
        std::vector<int> inf(k, 0);
        size_t per = 0;  // order records per stack: one stack at a time is asked for them
        if (ord_out) {
            const celeris_rcwa_cell& f = layers[stacks[0].first];
            per = (size_t)nexc * (2 * f.Mx + 1) * (2 * f.My + 1) * 2;
        }
        std::vector<double> ord(per * k);
        for (int i = 0; i < k; ++i) {
            st[i] = stacks[sel[i]];
            std::memcpy(&ex[4 * (size_t)i], exc + 4 * (size_t)sel[i], 4 * sizeof(double));
        }
        double* o = ord_out ? ord.data() : nullptr;
        CEL_TRY(qr ? run_stacks_qr(layers, st, ex.data(), res.data(), inf.data(), nexc, o)
                   : run_stacks_slab(layers, st, ex.data(), res.data(), inf.data(), nexc, o));
        for (int i = 0; i < k; ++i) {
            info[sel[i]] = inf[i];
            if (!qr && inf[i] != 0) continue;
            for (int e = 0; e < nexc; ++e) out[(size_t)sel[i] * nexc + e] = res[(size_t)i * nexc + e];
            if (o) std::memcpy(ord_out + per * sel[i], o + per * i, per * sizeof(double));
        }
        return CELERIS_OK;
    };
    CEL_TRY(run(direct, false));
    for (int s : direct)
        if (info[s] != 0) rest.push_back(s);
    CEL_TRY(run(rest, true));
    for (int s = 0; s < ns; ++s) {
        if (info_out) info_out[s] = info[s];
        else if (info[s] > 0)
            return set_error(CELERIS_ERR_EIG_NOCONV, "eigensolve did not converge (a layer of stack %d)", s);
        else if (info[s] < 0)
            return set_error(CELERIS_ERR_SINGULAR, "singular interface system (stack %d)", s);
    }
    return CELERIS_OK;
}

// Layers of one stack must share everything but the pattern, materials and thickness.
int validate_stack(const celeris_rcwa_cell* l, int nl) {
    if (nl < 1) return set_error(CELERIS_ERR_INVALID_ARG, "a stack needs at least one layer");
    for (int i = 0; i < nl; ++i) CEL_TRY(validate(l[i]));
    const celeris_rcwa_cell& f = l[0];
    for (int i = 1; i < nl; ++i) {
        const celeris_rcwa_cell& c = l[i];
        if (c.Mx != f.Mx || c.My != f.My || c.period_x_um != f.period_x_um || c.period_y_um != f.period_y_um ||
            c.wavelength_um != f.wavelength_um || c.theta_rad != f.theta_rad || c.phi_rad != f.phi_rad ||
            c.n_inc[0] != f.n_inc[0] || c.n_inc[1] != f.n_inc[1] || c.n_sub[0] != f.n_sub[0] ||
            c.n_sub[1] != f.n_sub[1])
            return set_error(CELERIS_ERR_INVALID_ARG,
                             "layer %d of a stack differs from layer 0 in orders, periods, wavelength, angles or "
                             "half-spaces",
                             i);
    }
    return CELERIS_OK;
}

// ---- standalone eigensolve: batches of n x n matrices through the eigen-stages ------------
int run_eig(const double* A, int n, int count, double* evals, double* evecs, int* info_out) {
    CEL_TRY(celeris_rt::require_device());
    const size_t s_nn = (size_t)n * n, s_n = (size_t)n;
    int dev = 0;
    CEL_CUDA(cudaGetDevice(&dev));
    static thread_local celeris_rt::ThreadStream t_eig_st;  // one stream and arena per calling thread
    cudaStream_t st = nullptr;
    CEL_TRY(t_eig_st.get(&st));
    Workspace& ws = Workspace::for_stream(st);
    if (n <= kSmemEigMaxN)
        CEL_TRY(raise_dyn_smem(reinterpret_cast<const void*>(rcwa_hess<true>), (s_nn + 2 * s_n) * sizeof(cplx)));
    else
        CEL_TRY(raise_dyn_smem(reinterpret_cast<const void*>(rcwa_hess<false>), hess_stage_bytes(n)));
    CEL_TRY(raise_dyn_smem(reinterpret_cast<const void*>(rcwa_schur), kSchurSmemOneCta));
    size_t free_b = 0, total_b = 0;
    CEL_CUDA(cudaMemGetInfo(&free_b, &total_b));
    const size_t per = (7 * s_nn + 2 * s_n) * sizeof(cplx) + 4096;
    const int chunk = (int)std::max<size_t>(1, std::min<size_t>((size_t)count, (free_b / 2) / per));
    for (int c0 = 0; c0 < count; c0 += chunk) {
        const int nc = std::min(chunk, count - c0);
        const size_t c16 = sizeof(cplx);
        const size_t plan = 6 * a256(s_nn * nc * c16) + 2 * a256(s_n * nc * c16) + a256(nc * sizeof(int));
        CEL_TRY(ws.reserve(st, plan));
        Bump mem{static_cast<char*>(ws.take(plan)), plan};
        Bucket b;
        std::memset(&b, 0, sizeof(b));
        b.n = n;
        b.N = n / 2;
        b.ncell = nc;
        b.s_nn = s_nn;
        b.s_n = s_n;
        cplx *dA, *dval, *dvec;
        CEL_TRY(mem.get(&dA, s_nn * nc));
        cplx** mats[] = {&b.H, &b.Z, &b.X, &b.W, &b.A};
        for (cplx** m : mats) CEL_TRY(mem.get(m, s_nn * nc));
        CEL_TRY(mem.get(&b.q1, s_n * nc));
        CEL_TRY(mem.get(&b.info, (size_t)nc));
        CEL_TRY(mem.get(&dval, s_n * nc));
        dvec = b.A;  // free after the eigenvectors
        CEL_CUDA(cudaMemcpyAsync(dA, A + 2 * s_nn * c0, sizeof(cplx) * s_nn * nc, cudaMemcpyHostToDevice, st));
        CEL_CUDA(cudaMemsetAsync(b.info, 0, sizeof(int) * nc, st));
        eig_load<<<nc, kRT, 0, st>>>(dA, b);
        if (n <= kSmemEigMaxN)
            rcwa_hess<true><<<nc, kRT, (s_nn + 2 * s_n) * sizeof(cplx), st>>>(b);
        else
            rcwa_hess<false><<<nc, kRT, hess_stage_bytes(n), st>>>(b);
        rcwa_schur<<<nc, kSchurThreads, schur_smem(nc), st>>>(b);
        rcwa_vec<<<nc, kRT, 0, st>>>(b);
        eig_store<<<nc, kRT, 0, st>>>(b, dval, dvec);
        count_launch(6);
        CEL_CUDA(cudaGetLastError());
        std::vector<int> hinfo(nc);
        CEL_CUDA(cudaMemcpyAsync(evals + 2 * s_n * c0, dval, sizeof(cplx) * s_n * nc, cudaMemcpyDeviceToHost, st));
        CEL_CUDA(cudaMemcpyAsync(evecs + 2 * s_nn * c0, dvec, sizeof(cplx) * s_nn * nc, cudaMemcpyDeviceToHost, st));
        CEL_CUDA(cudaMemcpyAsync(hinfo.data(), b.info, sizeof(int) * nc, cudaMemcpyDeviceToHost, st));
        CEL_CUDA(cudaStreamSynchronize(st));
        for (int i = 0; i < nc; ++i) {
            if (info_out) info_out[c0 + i] = hinfo[i];
            else if (hinfo[i] != 0)
                return set_error(CELERIS_ERR_EIG_NOCONV, "QR did not converge (info %d)", hinfo[i]);
        }
    }
    return CELERIS_OK;
}

}  // namespace

extern "C" {

int celeris_solve_rcwa_2d(const celeris_rcwa_cell* cell, const double* Ex0, const double* Ey0,
                          celeris_rcwa_result* out) {
    if (!cell || !Ex0 || !Ey0 || !out) return set_error(CELERIS_ERR_INVALID_ARG, "NULL argument");
    CEL_TRY(validate(*cell));
    std::vector<HostCell> cells{make_cell(*cell, 0, Ex0[0], Ex0[1], Ey0[0], Ey0[1], 1)};
    return run_cells(cells, out, nullptr, 1);
}

int celeris_rcwa_tuning_report(char* buf, int len) {
    if (!buf || len <= 0) return set_error(CELERIS_ERR_INVALID_ARG, "bad buffer");
    std::string s;
    std::lock_guard<std::mutex> lk(g_tune_mu);
    for (const auto& kv : tune_table()) {
        s += "Mx=" + std::to_string(std::get<0>(kv.first)) + " My=" + std::to_string(std::get<1>(kv.first)) +
             " grid=" + std::to_string(std::get<2>(kv.first) / 8) +
             ((std::get<2>(kv.first) & 4) ? "" : " eigensolve") +
             ((std::get<2>(kv.first) & 2) ? " parity-classes" : "") +
             ((std::get<2>(kv.first) & 1) ? " batch>=SMs:" : " batch<SMs:");
        for (int st = 0; st < ST_COUNT; ++st)
            s += std::string(" ") + kStageNames[st] + "=" + std::to_string(kv.second.threads[st]);
        s += "\n";
    }
    std::snprintf(buf, (size_t)len, "%s", s.c_str());
    return CELERIS_OK;
}

int celeris_solve_rcwa_2d_stack(const celeris_rcwa_cell* layers, int nlayers, const double* Ex0, const double* Ey0,
                                celeris_rcwa_result* out) {
    if (!layers || !Ex0 || !Ey0 || !out) return set_error(CELERIS_ERR_INVALID_ARG, "NULL argument");
    CEL_TRY(validate_stack(layers, nlayers));
    const double exc[4] = {Ex0[0], Ex0[1], Ey0[0], Ey0[1]};
    return run_stacks(layers, {{0, nlayers}}, exc, out, nullptr, 1);
}

int celeris_eig_general_batch(const double* A, int n, int count, double* evals, double* evecs, int* info) {
    if (n < 1 || count < 0) return set_error(CELERIS_ERR_INVALID_ARG, "n must be >= 1 and count >= 0");
    if (n > kMaxN) return set_error(CELERIS_ERR_TOO_LARGE, "n = %d > %d", n, kMaxN);
    if (count == 0) return CELERIS_OK;
    if (!A || !evals || !evecs) return set_error(CELERIS_ERR_INVALID_ARG, "NULL argument");
    {   // x * 0 is NaN exactly when x is NaN or Inf: one branch-free pass
        const size_t per = 2 * (size_t)n * n;
        for (int c = 0; c < count; ++c) {
            double z = 0.0;
            for (size_t i = 0; i < per; ++i) z += A[c * per + i] * 0.0;
            if (z != 0.0) return set_error(CELERIS_ERR_INVALID_ARG, "matrix %d holds NaN or Inf", c);
        }
    }
    if (n == 1) {  // nothing to reduce
        for (int c = 0; c < count; ++c) {
            evals[2 * c] = A[2 * c];
            evals[2 * c + 1] = A[2 * c + 1];
            evecs[2 * c] = 1.0;
            evecs[2 * c + 1] = 0.0;
            if (info) info[c] = 0;
        }
        return CELERIS_OK;
    }
    return run_eig(A, n, count, evals, evecs, info);
}

int celeris_eig_general(const double* A, int n, double* evals, double* evecs) {
    return celeris_eig_general_batch(A, n, 1, evals, evecs, nullptr);
}

int celeris_solve_rcwa_2d_orders(const celeris_rcwa_cell* layers, int nlayers, const double* Ex0, const double* Ey0,
                                 celeris_rcwa_result* out, celeris_rcwa_order* orders, int max_orders) {
    if (!layers || !Ex0 || !Ey0 || !out || !orders) return set_error(CELERIS_ERR_INVALID_ARG, "NULL argument");
    CEL_TRY(validate_stack(layers, nlayers));
    const celeris_rcwa_cell& f = layers[0];
    const int N = (2 * f.Mx + 1) * (2 * f.My + 1);
    if (max_orders < N) return set_error(CELERIS_ERR_INVALID_ARG, "orders holds %d records, %d needed", max_orders, N);
    const double exc[4] = {Ex0[0], Ex0[1], Ey0[0], Ey0[1]};
    std::vector<double> ord((size_t)N * 2);
    CEL_TRY(run_stacks(layers, {{0, nlayers}}, exc, out, nullptr, 1, ord.data()));
    // order labels and the propagation test of rcwa2d.cpp:469-484 (same arithmetic)
    typedef std::complex<double> cd;
    const double k0 = 2.0 * PI / f.wavelength_um;
    const cd n_inc(f.n_inc[0], f.n_inc[1]);
    const cd kx0 = n_inc * std::sin(f.theta_rad) * std::cos(f.phi_rad) * k0;
    const cd ky0 = n_inc * std::sin(f.theta_rad) * std::sin(f.phi_rad) * k0;
    const double k0sub = (f.n_sub[0] * k0) * (f.n_sub[0] * k0);
    const double k0inc = (f.n_inc[0] * k0) * (f.n_inc[0] * k0);
    for (int p = -f.Mx; p <= f.Mx; ++p)
        for (int q = -f.My; q <= f.My; ++q) {
            const int i = (p + f.Mx) * (2 * f.My + 1) + (q + f.My);
            const cd kx = kx0 - 2.0 * PI * (double)p / f.period_x_um;
            const cd ky = ky0 - 2.0 * PI * (double)q / f.period_y_um;
            const double kt2 = (kx * kx + ky * ky).real();
            celeris_rcwa_order& o = orders[i];
            o.p = p;
            o.q = q;
            o.de_t = ord[2 * (size_t)i];
            o.de_r = ord[2 * (size_t)i + 1];
            o.prop_t = k0sub - kt2 > 0.0;
            o.prop_r = k0inc - kt2 > 0.0;
        }
    return CELERIS_OK;
}

int celeris_rcwa_stack_batch(const celeris_rcwa_cell* layers, const int* layer_start, int nstack,
                             celeris_rcwa_result* out, int* info) {
    if (nstack < 0) return set_error(CELERIS_ERR_INVALID_ARG, "nstack < 0");
    if (nstack == 0) return CELERIS_OK;
    if (!layers || !layer_start || !out) return set_error(CELERIS_ERR_INVALID_ARG, "NULL argument");
    std::vector<std::pair<int, int>> stacks;
    std::vector<double> exc(4 * (size_t)nstack, 0.0);
    for (int s = 0; s < nstack; ++s) {
        const int a = layer_start[s], nl = layer_start[s + 1] - layer_start[s];
        if (a < 0 || nl < 1) return set_error(CELERIS_ERR_INVALID_ARG, "stack %d: bad layer range", s);
        CEL_TRY(validate_stack(layers + a, nl));
        stacks.push_back({a, nl});
        exc[4 * (size_t)s] = 1.0;  // slot 0 = X polarization (Ex0 = 1), slot 1 = Y
    }
    return run_stacks(layers, stacks, exc.data(), out, info, 2);
}

int celeris_rcwa_batch(const celeris_rcwa_cell* cells, int ncell, celeris_rcwa_result* out, int* info) {
    if (ncell < 0) return set_error(CELERIS_ERR_INVALID_ARG, "ncell < 0");
    if (ncell == 0) return CELERIS_OK;
    if (!cells || !out) return set_error(CELERIS_ERR_INVALID_ARG, "NULL argument");
    std::vector<HostCell> hc;
    hc.reserve(ncell);
    for (int i = 0; i < ncell; ++i) {
        const int v = validate(cells[i]);
        if (v != CELERIS_OK) {
            const std::string msg = celeris_last_error();
            return set_error(v, "cell %d: %s", i, msg.c_str());
        }
        hc.push_back(make_cell(cells[i], i, 1.0, 0.0, 0.0, 0.0, 2));
    }
    return run_cells(hc, out, info, 2);
}

int celeris_debug_qr_iteration_cap(int cap) {
    if (cap < 0) return set_error(CELERIS_ERR_INVALID_ARG, "cap < 0");
    CEL_TRY(celeris_rt::require_device());
    CEL_CUDA(cudaMemcpyToSymbol(g_qr_iter_cap, &cap, sizeof(int)));
    g_qr_cap_set.store(cap);
    return CELERIS_OK;
}

}  // extern "C"
