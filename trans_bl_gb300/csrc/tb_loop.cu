// tb_loop.cu -- the stage driver (drv_fi/drv_les, RK4 update, wall forcing)
// and the velocity recovery of loop() except the v-Poisson solve.
#include "tb_internal.h"
#include "tb_warp.cuh"
#include <cmath>
#include <cstring>

namespace {

__device__ __forceinline__ cplx cm(double s, cplx a) { return make_double2(s * a.x, s * a.y); }
__device__ __forceinline__ cplx ca(cplx a, cplx b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ cplx cs_(cplx a, cplx b) { return make_double2(a.x - b.x, a.y - b.y); }
// v_kb(k) * a with v_kb = -i (k-1) beta  (main_par.f:1888)
__device__ __forceinline__ cplx ikb(double kb, cplx a) { return make_double2(kb * a.y, -kb * a.x); }

// ---------------------------------------------------------------------------
// drv_fi / drv_les combine (main_par.f:1312-1333, 1550-1571), rows j >= 2.
struct CombArgs {
    const cplx *dady, *b, *xx0, *yy0, *wx;
    const cplx *c, *dadx, *xx1, *yy1, *wy;
    const cplx *dbdx, *dcdy, *xx2, *yy2, *wz;
    const cplx *fx, *fy, *dfzdy, *dfzdx, *dfxdy, *dfydx;  // force terms, null if none
    const cplx *gd, *gdddx;                               // drv_gv's d and dd/dx, null if none
    cplx *dvx, *dvy, *dvz;
    const double* k2b2;
    int nx, ny, K;
    double beta, invRe, fac_y, varg;
};
__global__ void k_combine(CombArgs A) {
    size_t n = (size_t)A.nx * A.ny * A.K;
    size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (q >= n) return;
    int j = (int)((q / A.nx) % A.ny);
    if (j < 1) return;
    int k = (int)(q / ((size_t)A.nx * A.ny));
    double kb = (double)k * A.beta, k2 = A.k2b2[k], fy = A.fac_y;
    cplx vx = ca(cs_(ikb(kb, A.b[q]), A.dady[q]), cm(A.invRe, ca(ca(A.xx0[q], cm(fy, A.yy0[q])), cm(k2, A.wx[q]))));
    cplx vy = ca(cs_(A.dadx[q], ikb(kb, A.c[q])), cm(A.invRe, ca(ca(A.xx1[q], cm(fy, A.yy1[q])), cm(k2, A.wy[q]))));
    cplx vz = ca(cs_(A.dcdy[q], A.dbdx[q]), cm(A.invRe, ca(ca(A.xx2[q], cm(fy, A.yy2[q])), cm(k2, A.wz[q]))));
    if (A.fx) {
        vx = cs_(ca(vx, cm(1.0 / fy, ikb(kb, A.fy[q]))), A.dfzdy[q]);
        vy = cs_(ca(vy, A.dfzdx[q]), ikb(kb, A.fx[q]));
        vz = cs_(ca(vz, A.dfxdy[q]), cm(1.0 / fy, A.dfydx[q]));
    }
    if (A.gd) {   // drv_gv (main_par.f:1382-1396): - v_kb d varg, + varg dd/dx
        vx = cs_(vx, cm(A.varg, ikb(kb, A.gd[q])));
        vz = ca(vz, cm(A.varg, A.gdddx[q]));
    }
    A.dvx[q] = vx; A.dvy[q] = vy; A.dvz[q] = vz;
}

// RK4 update (main_par.f:170-246): j = 2..jmax-1, i = 3..ptsx.
struct RkArgs {
    cplx *wx, *wy, *wz, *wx1, *wy1, *wz1, *d1x, *d1y, *d1z;
    const cplx *d2x, *d2y, *d2z;
    int nx, ny, K, stage;
    double dt, dt2, dt6;
};
__global__ void k_rk(RkArgs A) {
    size_t n = (size_t)A.nx * A.ny * A.K;
    size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (q >= n) return;
    int i = (int)(q % A.nx), j = (int)((q / A.nx) % A.ny);
    if (j < 1 || j > A.ny - 2 || i < 2) return;
    if (A.stage == 1) {
        cplx x = A.wx[q], y = A.wy[q], z = A.wz[q];
        A.wx1[q] = x; A.wy1[q] = y; A.wz1[q] = z;
        A.wx[q] = ca(x, cm(A.dt2, A.d1x[q]));
        A.wy[q] = ca(y, cm(A.dt2, A.d1y[q]));
        A.wz[q] = ca(z, cm(A.dt2, A.d1z[q]));
    } else if (A.stage == 2 || A.stage == 3) {
        double h = (A.stage == 2) ? A.dt2 : A.dt;
        cplx ex = A.d2x[q], ey = A.d2y[q], ez = A.d2z[q];
        A.wx[q] = ca(A.wx1[q], cm(h, ex));
        A.wy[q] = ca(A.wy1[q], cm(h, ey));
        A.wz[q] = ca(A.wz1[q], cm(h, ez));
        A.d1x[q] = ca(A.d1x[q], cm(2.0, ex));
        A.d1y[q] = ca(A.d1y[q], cm(2.0, ey));
        A.d1z[q] = ca(A.d1z[q], cm(2.0, ez));
    } else {
        A.wx[q] = ca(A.wx1[q], cm(A.dt6, ca(A.d1x[q], A.d2x[q])));
        A.wy[q] = ca(A.wy1[q], cm(A.dt6, ca(A.d1y[q], A.d2y[q])));
        A.wz[q] = ca(A.wz1[q], cm(A.dt6, ca(A.d1z[q], A.d2z[q])));
    }
}

// bzone (loop_par.f:6-45) for j >= 2 and bzonew (691-725) for j = 1; bdfc
// holds the two ramp rows bdfc(1,:), bdfc(2,:) one after the other.
__global__ void k_bzone(cplx* wx, cplx* wy, cplx* wz, const double* bdfc, const double* wzb, int nx, int ny, int K,
                        int wall, int form) {
    size_t n = (size_t)nx * (wall ? 1 : ny) * K;
    size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (t >= n) return;
    int i, j, k;
    if (wall) { i = (int)(t % nx); k = (int)(t / nx); j = 0; }
    else { i = (int)(t % nx); j = (int)((t / nx) % ny); k = (int)(t / ((size_t)nx * ny)); if (j < 1) return; }
    size_t q = (size_t)i + (size_t)nx * (j + (size_t)ny * k);
    double bd = bdfc[(k == 2 ? (size_t)nx : 0) + i];   // bdt = 2 for the third mode (loop_par.f:19-20)
    wx[q] = cm(bd, wx[q]);
    wy[q] = cm(bd, wy[q]);
    if ((form == 0 || form == 4) && k == 0) {
        double b = wzb[i + (size_t)nx * j];
        cplx v = wz[q];
        wz[q] = make_double2((v.x - b) * bd + b, v.y * bd);
    } else {
        wz[q] = cm(bd, wz[q]);
    }
}

// outuy tail (loop_par.f:96-114): Dirichlet uy at the outflow column, j >= 2.
__global__ void k_outuy_bc(cplx* uy, const double* uyb, int nx, int ny, int K, int form) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= ny * K) return;
    int j = t % ny, k = t / ny;
    if (j < 1) return;
    size_t q = (size_t)(nx - 1) + (size_t)nx * (j + (size_t)ny * k);
    uy[q] = ((form == 0 || form == 4) && k == 0) ? make_double2(uyb[(nx - 1) + (size_t)nx * j], 0.0) : make_double2(0.0, 0.0);
}

// ---------------------------------------------------------------------------
// x-direction recurrences, one warp per line (tb_warp.cuh).  Shared memory
// per warp: two line buffers of 32 x Sp complex (inputs E, rows V).

// The 4th-order implicit x integration of poi_ux mode 0 (loop_par.f:452-499)
// and of wz_wall (loop_par.f:361-425): w_0 given,
//   w_1     = (sg dx (251 r0 + 646 r1 - 264 r2 + 106 r3 - 19 r4) + 720 w_0) / 720
//   w_i     = (sg dx (281 r_{i-2} + 2056 r_{i-1} + 1176 r_i - 104 r_{i+1} + 11 r_{i+2}) / 90
//              + 11 w_{i-2} + 16 w_{i-1}) / 27                       2 <= i <= n-3
//   w_{n-2} = (sg dx (10 r_{n-4} + 57 r_{n-3} + 24 r_{n-2} - r_{n-1}) + 33 w_{n-4} + 24 w_{n-3}) / 57
//   w_{n-1} = (sg dx (251 r_{n-1} + 646 r_{n-2} - 264 r_{n-3} + 106 r_{n-4} - 19 r_{n-5}) + 720 w_{n-2}) / 720
// with r in E (lane chunks), w_0 = w0; the result (rows 1..n-1) goes to out.
__device__ void xint_line(const cplx* E, cplx* V, const WarpLine& L, int lane, cplx w0, double sgdx, cplx* out) {
    const int n = L.n, r0 = lane * L.S, r1 = min(n, r0 + L.S);
    const double i720 = 1.0 / 720.0, i27 = 1.0 / 27.0, i90 = 1.0 / 90.0, i57 = 1.0 / 57.0;
    auto e = [&](int i) { return E[L.slot(i)]; };
    cplx* Vl = V + lane * L.Sp;
    for (int i = r0; i < r1; i++) {
        cplx v;
        if (i == 0) v = w0;
        else if (i == 1) {
            cplx a = e(0), b = e(1), c = e(2), d = e(3), f = e(4);
            v = make_double2(sgdx * (251.0 * a.x + 646.0 * b.x - 264.0 * c.x + 106.0 * d.x - 19.0 * f.x) * i720,
                             sgdx * (251.0 * a.y + 646.0 * b.y - 264.0 * c.y + 106.0 * d.y - 19.0 * f.y) * i720);
        } else if (i <= n - 3) {
            cplx a = e(i - 2), b = e(i - 1), c = e(i), d = e(i + 1), f = e(i + 2);
            v = make_double2(sgdx * (281.0 * a.x + 2056.0 * b.x + 1176.0 * c.x - 104.0 * d.x + 11.0 * f.x) * i90 * i27,
                             sgdx * (281.0 * a.y + 2056.0 * b.y + 1176.0 * c.y - 104.0 * d.y + 11.0 * f.y) * i90 * i27);
        } else if (i == n - 2) {
            cplx a = e(i - 2), b = e(i - 1), c = e(i), d = e(i + 1);
            v = make_double2(sgdx * (10.0 * a.x + 57.0 * b.x + 24.0 * c.x - d.x) * i57,
                             sgdx * (10.0 * a.y + 57.0 * b.y + 24.0 * c.y - d.y) * i57);
        } else {
            cplx a = e(i), b = e(i - 1), c = e(i - 2), d = e(i - 3), f = e(i - 4);
            v = make_double2(sgdx * (251.0 * a.x + 646.0 * b.x - 264.0 * c.x + 106.0 * d.x - 19.0 * f.x) * i720,
                             sgdx * (251.0 * a.y + 646.0 * b.y - 264.0 * c.y + 106.0 * d.y - 19.0 * f.y) * i720);
        }
        Vl[i - r0] = v;
    }
    auto ca_ = [=](int i) -> double {
        if (i == 0) return 0.0;
        if (i == 1 || i == n - 1) return -720.0 * i720;
        if (i == n - 2) return -24.0 * i57;
        return -16.0 * i27;
    };
    auto cb_ = [=](int i) -> double {
        if (i <= 1 || i == n - 1) return 0.0;
        if (i == n - 2) return -33.0 * i57;
        return -11.0 * i27;
    };
    warp_rec2_fwd(Vl, r0, r1, lane, ca_, cb_);
    __syncwarp();
    for (int i = lane; i < n; i += 32)
        if (i >= 1) out[i] = V[L.slot(i)];
}

// poi_ux mode 0: ux(:, j, 0) from duydy by x integration, one warp per row j = 1..ny-2.
__global__ void __launch_bounds__(64) k_ux_mode0(cplx* ux, const cplx* duydy, int nx, int ny, double dx) {
    extern __shared__ cplx wsm[];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int j = 1 + blockIdx.x * (blockDim.x >> 5) + wib;
    if (j > ny - 2) return;
    const WarpLine L{nx, WarpLine::chunk(nx), WarpLine::padded(nx)};
    cplx* E = wsm + (size_t)wib * 64 * L.Sp;
    cplx* V = E + 32 * L.Sp;
    const cplx* D = duydy + (size_t)nx * j;
    for (int i = lane; i < nx; i += 32) E[L.slot(i)] = D[i];
    __syncwarp();
    cplx* U = ux + (size_t)nx * j;
    xint_line(E, V, L, lane, U[0], -dx, U);
}

// wz_wall: wall wz of mode k from r = v_kb wx - lapv by x integration, one warp per mode.
__global__ void __launch_bounds__(64) k_wz_wall(cplx* wz, const cplx* wx, const cplx* lapv, int nx, int ny, int K, double dx,
                                                double beta) {
    extern __shared__ cplx wsm[];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int k = blockIdx.x * (blockDim.x >> 5) + wib;
    if (k >= K) return;
    const WarpLine L{nx, WarpLine::chunk(nx), WarpLine::padded(nx)};
    cplx* E = wsm + (size_t)wib * 64 * L.Sp;
    cplx* V = E + 32 * L.Sp;
    const double kb = (double)k * beta;
    const cplx* WX = wx + (size_t)nx * ny * k;
    const cplx* LV = lapv + (size_t)nx * k;
    for (int i = lane; i < nx; i += 32) { cplx v = ikb(kb, WX[i]); cplx l = LV[i]; E[L.slot(i)] = make_double2(v.x - l.x, v.y - l.y); }
    __syncwarp();
    cplx* W = wz + (size_t)nx * ny * k;
    xint_line(E, V, L, lane, W[0], dx, W);
}

// Pentadiagonal x solve with the LU of lhs5 (lusolver / lusolver_1,
// penta_par.f:53-208) of one mode, by one warp for the real or the imaginary part
// of a line.  The plane L (lane t's rows [tS, tS + S) at t (S | 1)) holds e and takes
// the solution; in units of 8 dx^2 the rhs rows are
//   r_0 = boundary value, r_1 = (e_0 + 10 e_1 + e_2) / 96, r_i = e_{i-1} + 5.5 e_i + e_{i+1},
//   r_{n-2} = (e_{n-1} + 10 e_{n-2} + e_{n-3}) / 96, r_{n-1} = rn,
// r0v and rn given unscaled.  T: the mode's row tables (penta_table_size), entries of
// row tS + q at q * 32 + t: L1 L2 of the forward sweep, SI = 8 dx^2 / u3, C D of
// the backward sweep, the responses H1 H2 (with SI) and K1 K2 of the rows to the states
// entering the chunk, then the Kogge-Stone matrices of both sweeps.
__device__ __forceinline__ void penta_sweeps(const double* __restrict__ T, int S, int n, double* L, double* E, int lane, double r0v,
                                             double rn, double unit) {
    const int Sp = S | 1, r0 = min(n, lane * S), r1 = min(n, r0 + S);
    double* Ul = L + lane * Sp;
    const double* Tr = T + lane;
    const int N = 32 * S;   // doubles of one row table
    auto e = [&](int i) { return L[(i / S) * Sp + i % S]; };
    if (lane < 4) {   // r_0, r_1, r_{n-2}, r_{n-1}
        const int i = lane == 1 ? 1 : n - 2;
        const bool mid = lane == 1 || lane == 2;
        E[lane] = (mid ? fma(10.0, e(i), e(i - 1) + e(i + 1)) : lane ? rn : r0v) * (mid ? 1.0 / 96.0 : unit);
    }
    double ep = (r0 >= 1 && r0 < r1) ? e(r0 - 1) : 0.0;
    const double en = r1 < n ? e(r1) : 0.0;
    __syncwarp();
    double y1 = 0.0, y2 = 0.0;
    for (int q = 0; q < r1 - r0; q++) {
        const int i = r0 + q;
        const double b = Ul[q], c = (i + 1 < r1) ? Ul[q + 1] : en;
        double t = fma(5.5, b, ep + c);
        if (i < 2 || i >= n - 2) t = E[i < 2 ? i : i - n + 4];
        ep = b;
        const double y = fma(-Tr[N + 32 * q], y1, fma(-Tr[32 * q], y2, t));
        Ul[q] = y;
        y2 = y1; y1 = y;
    }
    const double* Pf = Tr + 9 * N;
#pragma unroll
    for (int d = 0, off = 1; d < 5; d++, off <<= 1) {
        const double o1 = __shfl_up_sync(0xffffffffu, y1, off), o2 = __shfl_up_sync(0xffffffffu, y2, off);
        if (lane >= off) {
            y1 = fma(Pf[128 * d], o1, fma(Pf[128 * d + 32], o2, y1));
            y2 = fma(Pf[128 * d + 64], o1, fma(Pf[128 * d + 96], o2, y2));
        }
    }
    double Y1 = __shfl_up_sync(0xffffffffu, y1, 1), Y2 = __shfl_up_sync(0xffffffffu, y2, 1);
    if (lane == 0) { Y1 = 0.0; Y2 = 0.0; }
    double x1 = 0.0, x2 = 0.0;
#pragma unroll 2
    for (int q = r1 - r0 - 1; q >= 0; q--) {
        const double* t = Tr + 32 * q;
        const double r = fma(t[5 * N], Y1, fma(t[6 * N], Y2, t[2 * N] * Ul[q]));
        const double x = fma(-t[3 * N], x1, fma(-t[4 * N], x2, r));
        Ul[q] = x;
        x2 = x1; x1 = x;
    }
    const double* Pb = Pf + 640;
#pragma unroll
    for (int d = 0, off = 1; d < 5; d++, off <<= 1) {
        const double o1 = __shfl_down_sync(0xffffffffu, x1, off), o2 = __shfl_down_sync(0xffffffffu, x2, off);
        if (lane + off < 32) {
            x1 = fma(Pb[128 * d], o1, fma(Pb[128 * d + 32], o2, x1));
            x2 = fma(Pb[128 * d + 64], o1, fma(Pb[128 * d + 96], o2, x2));
        }
    }
    double X1 = __shfl_down_sync(0xffffffffu, x1, 1), X2 = __shfl_down_sync(0xffffffffu, x2, 1);
    if (lane == 31) { X1 = 0.0; X2 = 0.0; }
#pragma unroll 2
    for (int q = 0; q < r1 - r0; q++) Ul[q] = fma(Tr[7 * N + 32 * q], X1, fma(Tr[8 * N + 32 * q], X2, Ul[q]));
}

// Points t64, t64 + 64, ... of a line shared by a pair of warps: fn(i, slot).
template <class Fn>
__device__ __forceinline__ void pair_points(int t64, int S, int n, Fn fn) {
    const int dc = 64 / S, dr = 64 % S, Sp = S | 1;
    int c = t64 / S, r = t64 % S;
#pragma unroll 4
    for (int i = t64; i < n; i += 64) {
        fn(i, c * Sp + r);
        c += dc; r += dr;
        if (r >= S) { r -= S; c++; }
    }
}
__device__ __forceinline__ void pair_barrier(int id) { asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory"); }
__host__ __device__ inline int penta_line_size(int S) { return 64 * (S | 1) + 8; }   // two planes and the end rows

// x-penta Poisson of poi_ux / poi_uz (loop_par.f:519-563, 641-685), a pair of
// warps per line (j >= 1, k >= 1), one for its real and one for its imaginary part:
// with g = -1 (ux) or 1 (uz), e = g D - v_kb W, and the last row is
// (v_kb W - g D) / (k beta)^2.
//
// Bound by the FP64 pipe: 12 instructions a real value (22 with the chunk's
// responses followed in the sweeps) and the scans.  A block takes a run of lines in the
// order of the modes and keeps the row tables of the mode it is at in shared
// memory: 598 us before, 367 us at 1025 x 193 x 32.
struct PentaArgs {
    const cplx* D;   // d2uydxdy or dwydx
    const cplx* W;   // wy or duydy
    cplx* out;       // ux or uz
    const double* tab;
    int nx, ny, K, S, staged;
    double g, beta, unit;
};
constexpr int PENTA_MAX = 8;   // lines per block at most
__global__ void __launch_bounds__(64 * PENTA_MAX) k_penta_x(PentaArgs A) {
    extern __shared__ double ps[];
    const int pair = threadIdx.x >> 6, part = (threadIdx.x >> 5) & 1, lane = threadIdx.x & 31, t64 = threadIdx.x & 63;
    const int W = blockDim.x >> 6, n = A.nx, S = A.S, rows = A.ny - 1, plane = 32 * (S | 1), tsz = penta_table_size(S);
    double* F = ps + (A.staged ? tsz : 0) + (size_t)pair * penta_line_size(S);
    double* L = F + part * plane;
    const long total = (long)rows * (A.K - 1);
    const int end = (int)(total * (blockIdx.x + 1) / gridDim.x);
    for (int first = (int)(total * blockIdx.x / gridDim.x); first < end;) {
        const int k = 1 + first / rows, last = min(end, k * rows);   // the run's lines of mode k
        const double* T = A.tab + (size_t)k * tsz;
        if (A.staged) {
            __syncthreads();
            for (int q = threadIdx.x; q < tsz; q += blockDim.x) ps[q] = T[q];
            __syncthreads();
            T = ps;
        }
        const double kb = (double)k * A.beta, den = 1.0 / ((double)k * (double)k * A.beta * A.beta);
        for (int t = first + pair; t < last; t += W) {
            const int j = 1 + t - (k - 1) * rows;
            const size_t base = (size_t)n * (j + (size_t)A.ny * k);
            const cplx *D = A.D + base, *Wv = A.W + base;
            cplx* O = A.out + base;
            pair_points(t64, S, n, [&](int i, int slot) {
                const cplx d = D[i], w = Wv[i];
                F[slot] = fma(-kb, w.y, A.g * d.x);
                F[plane + slot] = fma(kb, w.x, A.g * d.y);
            });
            pair_barrier(1 + pair);
            const double r0v = reinterpret_cast<const double*>(O)[part];
            const double rn = -den * L[((n - 1) / S) * (S | 1) + (n - 1) % S];
            __syncwarp();
            penta_sweeps(T, S, n, L, F + 2 * plane + 4 * part, lane, r0v, rn, A.unit);
            pair_barrier(1 + pair);
            pair_points(t64, S, n, [&](int i, int slot) {
                if (i >= 1) O[i] = make_double2(F[slot], F[plane + slot]);
            });
            pair_barrier(1 + pair);
        }
        first = last;
    }
}

// lapv (loop_par.f:194-205) for every (i, k).
__global__ void k_lapv(cplx* lapv, const cplx* uy, const cplx* d2uydx2, const double* k2b2, const double* w, int nx, int ny,
                       int K, double inv_dyyw1) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nx * K) return;
    int i = t % nx, k = t / nx;
    const cplx* U = uy + (size_t)i + (size_t)nx * ny * k;
    size_t s = nx;
    cplx acc = make_double2(0, 0);
#pragma unroll
    for (int m = 0; m < 7; m++) { cplx v = U[m * s]; acc.x += w[2 + m] * v.x; acc.y += w[2 + m] * v.y; }
    cplx d = d2uydx2[t];
    cplx u1 = U[0];
    lapv[t] = make_double2(d.x + acc.x * inv_dyyw1 + k2b2[k] * u1.x, d.y + acc.y * inv_dyyw1 + k2b2[k] * u1.y);
}

// wall dwy/dy (der2wydxdy first loop, loop_par.f:313-321) per (i, k).
__global__ void k_dwydy_wall(cplx* out, const cplx* wy, const double* w, int nx, int ny, int K, double invdy) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nx * K) return;
    int i = t % nx, k = t / nx;
    const cplx* W = wy + (size_t)i + (size_t)nx * ny * k;
    size_t s = nx;
    cplx acc = make_double2(0, 0);
#pragma unroll
    for (int m = 0; m < 7; m++) { cplx v = W[m * s]; acc.x += w[1 + m] * v.x; acc.y += w[1 + m] * v.y; }
    out[t] = make_double2(invdy * acc.x, invdy * acc.y);
}

// wx_wall (loop_par.f:174-255): per mode k >= 1, d2wy/dxdy by explicit
// stencils, then the x-penta solve with the LU of lhs5 (lusolver_1,
// penta_par.f:53-127); a pair of warps per mode.
__global__ void __launch_bounds__(64) k_wx_wall(cplx* wx, const cplx* dwdy, const cplx* lapv, const double* tab, int nx,
                                                int ny, int S, double dx, double unit, double beta) {
    extern __shared__ double ws[];
    const int part = threadIdx.x >> 5, lane = threadIdx.x & 31, plane = 32 * (S | 1);
    const int k = 1 + blockIdx.x, n = nx;
    double* L = ws + part * plane;
    const cplx* dw = dwdy + (size_t)nx * k;
    const cplx* LV = lapv + (size_t)nx * k;
    cplx* WX = wx + (size_t)nx * ny * k;  // row j = 1
    const double kb = (double)k * beta;
    const double idx6 = 1.0 / 6.0 / dx, idx60 = 1.0 / 60.0 / dx, idx12 = 1.0 / 12.0 / dx, idx2 = 1.0 / 2.0 / dx;
    auto d2 = [&](int i) -> cplx {  // d2wydxdy(i), 0-based i
        if (i >= 3 && i <= n - 4) {
            cplx a = dw[i + 1], b = dw[i - 1], c = dw[i - 2], d = dw[i + 2], e = dw[i + 3], f = dw[i - 3];
            return make_double2((45.0 * (a.x - b.x) + 9.0 * (c.x - d.x) + e.x - f.x) * idx60,
                                (45.0 * (a.y - b.y) + 9.0 * (c.y - d.y) + e.y - f.y) * idx60);
        }
        if (i == n - 3) {
            cplx a = dw[n - 5], b = dw[n - 4], c = dw[n - 2], d = dw[n - 1];
            return make_double2((a.x - 8.0 * b.x + 8.0 * c.x - d.x) * idx12, (a.y - 8.0 * b.y + 8.0 * c.y - d.y) * idx12);
        }
        if (i == n - 2) {
            cplx a = dw[n - 1], b = dw[n - 2], c = dw[n - 3], d = dw[n - 4];
            return make_double2((2.0 * a.x + 3.0 * b.x - 6.0 * c.x + d.x) * idx6, (2.0 * a.y + 3.0 * b.y - 6.0 * c.y + d.y) * idx6);
        }
        if (i == n - 1) {
            cplx a = dw[n - 1], b = dw[n - 2], c = dw[n - 3];
            return make_double2((3.0 * a.x - 4.0 * b.x + c.x) * idx2, (3.0 * a.y - 4.0 * b.y + c.y) * idx2);
        }
        const double W0[7] = {-14.7, 36.0, -45.0, 40.0, -22.5, 7.2, -1.0};
        const double W1[7] = {-1.0, -7.7, 15.0, -10.0, 5.0, -1.5, 0.2};
        const double W2[7] = {0.2, -2.4, -3.5, 8.0, -3.0, 0.8, -0.1};
        const double* cw = (i == 0) ? W0 : (i == 1) ? W1 : W2;
        cplx acc = make_double2(0, 0);
        for (int m = 0; m < 7; m++) { acc.x += cw[m] * dw[m].x; acc.y += cw[m] * dw[m].y; }
        return make_double2(acc.x * idx6, acc.y * idx6);
    };
    pair_points(threadIdx.x, S, n, [&](int i, int slot) {
        const cplx a = d2(i), v = ikb(kb, LV[i]);
        ws[slot] = v.x - a.x;
        ws[plane + slot] = v.y - a.y;
    });
    __syncthreads();
    const double den = 1.0 / ((double)k * (double)k * beta * beta);
    const double r0v = reinterpret_cast<const double*>(WX)[part], rn = -den * L[((n - 1) / S) * (S | 1) + (n - 1) % S];
    __syncwarp();
    penta_sweeps(tab + (size_t)k * penta_table_size(S), S, n, L, ws + 2 * plane + 4 * part, lane, r0v, rn, unit);
    __syncthreads();
    pair_points(threadIdx.x, S, n, [&](int i, int slot) {
        if (i >= 1) WX[i] = make_double2(ws[slot], ws[plane + slot]);
    });
}

// Shared memory of the warp-per-line x kernels (two line buffers per warp).
constexpr int XW_WARPS = 2;
size_t xw_smem(int nx) { return (size_t)XW_WARPS * 64 * WarpLine::padded(nx) * sizeof(cplx); }

// A run of lines per block (k_penta_x), as many blocks as the SMs hold, with up to
// 8 lines at a time.  Blocks of two lines that read the tables from global memory
// where an SM has fewer than 8 lines, which the copy to shared memory would hold up,
// and where the tables leave no room for two.  With and without the copy, us:
// 4.4 lines an SM 31 and 24 (257 points), 78 and 59 (1025 points); 6.9 lines 47 and 45
// (513), 83 and 82 (1025); 9.3 lines 57 and 46 (257), 64 and 69 (513), 112 and 145
// (1025); 39 lines 143 and 140 (257), 213 and 233 (513), 366 and 461 (1025).
int launch_penta(tb_ctx* c, const cplx* D, const cplx* W, cplx* out, double g) {
    PentaArgs A{D, W, out, c->px.tab, c->g.nx, c->g.ny, c->g.K, c->px.S, 0, g, c->cfg.beta, c->px.unit};
    const size_t tab = (size_t)penta_table_size(A.S) * sizeof(double), line = (size_t)penta_line_size(A.S) * sizeof(double);
    const size_t room = (size_t)226 * 1024, sms = c->sm_count > 0 ? c->sm_count : 148;
    const size_t lines = (size_t)(A.ny - 1) * (A.K - 1);
    if (line > room) { tb_set_error("x-line of %d points exceeds shared memory", A.nx); return TB_ERR_ARG; }
    A.staged = tab + 2 * line <= room && lines >= 8 * sms;
    const size_t t0 = A.staged ? tab : 0;
    size_t w = std::min<size_t>(A.staged ? PENTA_MAX : 2, (room - t0) / line);
    if (w >= 4) w &= ~(size_t)3;   // the SM's four sub-partitions
    const size_t per = std::max<size_t>(1, std::min<size_t>(A.staged ? 3 : 16, room / (t0 + w * line + 1024)));
    const size_t nb = std::min((lines + w - 1) / w, per * sms);
    cudaEvent_t ps = nullptr;
    int r;
    if ((r = tb_prof_begin(c, PROF_PENTA, &ps))) return r;
    TB_CUDA(cudaFuncSetAttribute(k_penta_x, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    k_penta_x<<<(unsigned)nb, (unsigned)(64 * w), t0 + w * line, c->stream>>>(A);
    TB_CHECK_LAUNCH(c);
    return tb_prof_end(c, PROF_PENTA, ps);
}

// ts2d_pert / ts3d_pert (main_par.f:1613-1685) for each forced mode.
struct PertArgs {
    cplx *uy, *d2uydx2;
    const double *fcx, *fcllx;
    int nx, ny, i1, i2, nf;
    int mode[4];
    double fct[4];
    const double* fct_dev;   // when set, the amplitudes are read here (a recorded step graph)
};
__global__ void k_ts_pert(PertArgs A) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;  // 0-based
    if (i < A.i1 || i > A.i2 - 2) return;          // 1-based i1+1 .. i2-1
    for (int m = 0; m < A.nf; m++) {
        int k = A.mode[m];
        double f = A.fct_dev ? A.fct_dev[m] : A.fct[m];
        A.uy[(size_t)i + (size_t)A.nx * A.ny * k] = make_double2(A.fcx[i] * f, 0.0);
        A.d2uydx2[(size_t)i + (size_t)A.nx * k] = make_double2(A.fcllx[i] * f, 0.0);
    }
}

// lterms_gv (nlterms_par.f:89-112): the disturbance times the 2D base flow,
// pointwise in every mode.
__global__ void k_lterms_gv(const cplx* ux, const cplx* uy, const cplx* wx, const cplx* wy, const cplx* wz,
                            const double* uxb, const double* uyb, const double* wzb, cplx* a, cplx* b, cplx* c,
                            cplx* d, int nx, int ny, int K) {
    const size_t n2 = (size_t)nx * ny;
    const size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (q >= n2 * K) return;
    const size_t p = q % n2;
    const double U = uxb[p], V = uyb[p], W = wzb[p];
    const cplx ex = wx[q], ey = wy[q], ez = wz[q], u = ux[q], v = uy[q];
    a[q] = cs_(cm(V, ex), cm(U, ey));
    b[q] = ca(cm(U, ez), cm(W, u));
    c[q] = cs_(cm(-V, ez), cm(W, v));
    d[q] = cm(2.0 * U, u);
}

// gv_pert (main_par.f:1577-1610): the steady Goertler strip in every mode
// k >= 1 (0-based), wall row, 1-based i1+1 .. i2-1; amplitude a (or *a_dev
// in a recorded step).
__global__ void k_gv_pert(cplx* uy, cplx* d2uydx2, const double* fcx2, const double* fcllx2, int nx, int ny, int K,
                          int i1, int i2, double a, const double* a_dev) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = t % nx, k = 1 + t / nx;
    if (k >= K || i < i1 || i > i2 - 2) return;
    const double A = a_dev ? *a_dev : a;
    uy[(size_t)i + (size_t)nx * ny * k] = make_double2(A * fcx2[i], 0.0);
    d2uydx2[(size_t)i + (size_t)nx * k] = make_double2(A * fcllx2[i], 0.0);
}

}  // namespace

// drv_gv (main_par.f:1338-1401): linear terms about the base flow, their
// derivatives, the viscous terms and the curvature terms with varg =
// Go^2 / sqrt(Re) at every point (init_gv, main_par.f:944-970); dvargdx, the
// compact x-derivative of the constant varg, is zero and left out.
int tb_drv_gv(tb_ctx* c, cplx* dvx, cplx* dvy, cplx* dvz) {
    cplx** t = c->tmp;
    int r;
    k_lterms_gv<<<tb_blocks(tb_n3(c), 256), 256, 0, c->stream>>>(c->ux, c->uy, c->wx, c->wy, c->wz, c->uxb, c->uyb,
                                                                  c->wzb, t[0], t[1], t[2], t[13], c->g.nx, c->g.ny,
                                                                  c->g.K);
    TB_CHECK_LAUNCH(c);
    XJob xj[6] = {{t[0], t[3], XOP_D1}, {t[1], t[4], XOP_D1}, {t[13], t[14], XOP_D1},
                  {c->wx, t[5], XOP_D2}, {c->wy, t[6], XOP_D2}, {c->wz, t[7], XOP_D2}};
    YJob yj[5] = {{t[0], t[8], YOP_D1}, {t[2], t[9], YOP_D1},
                  {c->wx, t[10], YOP_D2}, {c->wy, t[11], YOP_D2}, {c->wz, t[12], YOP_D2}};
    if ((r = tb_launch_xlines(c, xj, 6))) return r;
    if ((r = tb_launch_ylines(c, yj, 5))) return r;
    return tb_combine_gv(c, t[3], t[8], t[1], t[5], t[10], t[2], t[6], t[11], t[4], t[9], t[7], t[12], t[13], t[14],
                         c->cfg.go_number * c->cfg.go_number / std::sqrt(c->cfg.Re), dvx, dvy, dvz);
}

// The momentum part of drv_gv / drv_gvth from its derivative fields.
int tb_combine_gv(tb_ctx* c, const cplx* dadx, const cplx* dady, const cplx* b, const cplx* xx0, const cplx* yy0,
                  const cplx* cc, const cplx* xx1, const cplx* yy1, const cplx* dbdx, const cplx* dcdy,
                  const cplx* xx2, const cplx* yy2, const cplx* d, const cplx* dddx, double varg, cplx* dvx, cplx* dvy,
                  cplx* dvz) {
    CombArgs A;
    std::memset(&A, 0, sizeof A);
    A.dady = dady; A.b = b; A.xx0 = xx0; A.yy0 = yy0; A.wx = c->wx;
    A.c = cc; A.dadx = dadx; A.xx1 = xx1; A.yy1 = yy1; A.wy = c->wy;
    A.dbdx = dbdx; A.dcdy = dcdy; A.xx2 = xx2; A.yy2 = yy2; A.wz = c->wz;
    A.gd = d; A.gdddx = dddx; A.varg = varg;
    A.dvx = dvx; A.dvy = dvy; A.dvz = dvz; A.k2b2 = c->k2b2;
    A.nx = c->g.nx; A.ny = c->g.ny; A.K = c->g.K; A.beta = c->cfg.beta; A.invRe = 1.0 / c->cfg.Re; A.fac_y = c->cfg.fac_y;
    k_combine<<<tb_blocks(tb_n3(c), 256), 256, 0, c->stream>>>(A);
    TB_CHECK_LAUNCH(c);
    return TB_OK;
}

// ===========================================================================
int tb_drv_k(tb_ctx* c, cplx* dvx, cplx* dvy, cplx* dvz) {
    cplx** t = c->tmp;
    int r;
    if (c->cfg.my_form == 1) return tb_drv_gv(c, dvx, dvy, dvz);
    if (c->cfg.my_form == 2) return tb_drv_gvth(c, dvx, dvy, dvz, dvx == c->dv1x ? c->dv1t : c->dv2t);
    if (c->cfg.my_form == 4 || c->cfg.ibm) {
        cplx* f[3] = {t[16], t[17], t[18]};
        cplx* df[4] = {t[19], t[20], t[21], t[22]};
        return tb_drv_forced(c, dvx, dvy, dvz, f, df);
    }
    // nonlinear terms a, b, c -> t[0..2]
    if ((r = tb_launch_nlterms(c, t[0], t[1], t[2]))) return r;
    XJob xj[5] = {{t[0], t[3], XOP_D1}, {t[1], t[4], XOP_D1},
                  {c->wx, t[5], XOP_D2}, {c->wy, t[6], XOP_D2}, {c->wz, t[7], XOP_D2}};
    YJob yj[5] = {{t[0], t[8], YOP_D1}, {t[2], t[9], YOP_D1},
                  {c->wx, t[10], YOP_D2}, {c->wy, t[11], YOP_D2}, {c->wz, t[12], YOP_D2}};
    if ((r = tb_launch_xlines(c, xj, 5))) return r;
    if ((r = tb_launch_ylines(c, yj, 5))) return r;
    CombArgs A;
    std::memset(&A, 0, sizeof A);
    A.dady = t[8]; A.b = t[1]; A.xx0 = t[5]; A.yy0 = t[10]; A.wx = c->wx;
    A.c = t[2]; A.dadx = t[3]; A.xx1 = t[6]; A.yy1 = t[11]; A.wy = c->wy;
    A.dbdx = t[4]; A.dcdy = t[9]; A.xx2 = t[7]; A.yy2 = t[12]; A.wz = c->wz;
    A.dvx = dvx; A.dvy = dvy; A.dvz = dvz; A.k2b2 = c->k2b2;
    A.nx = c->g.nx; A.ny = c->g.ny; A.K = c->g.K; A.beta = c->cfg.beta; A.invRe = 1.0 / c->cfg.Re; A.fac_y = c->cfg.fac_y;
    k_combine<<<tb_blocks(tb_n3(c), 256), 256, 0, c->stream>>>(A);
    TB_CHECK_LAUNCH(c);
    return TB_OK;
}

// drv with LES and/or IBM forcing: forces first (they use tmp[0..11] as
// scratch), the force curl terms, then the standard terms.
int tb_drv_forced(tb_ctx* c, cplx* dvx, cplx* dvy, cplx* dvz, cplx* f[3], cplx* df[4]) {
    int r;
    bool les = c->cfg.my_form == 4, ibm = c->cfg.ibm != 0;
    if (les) { if ((r = tb_launch_les(c, f[0], f[1], f[2]))) return r; }
    if (ibm) { if ((r = tb_launch_cvirt(c, f[0], f[1], f[2], les))) return r; }
    XJob fx[2] = {{f[1], df[0], XOP_D1}, {f[2], df[1], XOP_D1}};   // dfydx, dfzdx
    YJob fy[2] = {{f[0], df[2], YOP_D1}, {f[2], df[3], YOP_D1}};   // dfxdy, dfzdy
    if ((r = tb_launch_xlines(c, fx, 2))) return r;
    if ((r = tb_launch_ylines(c, fy, 2))) return r;
    cplx** t = c->tmp;
    if ((r = tb_launch_nlterms(c, t[0], t[1], t[2]))) return r;
    XJob xj[5] = {{t[0], t[3], XOP_D1}, {t[1], t[4], XOP_D1},
                  {c->wx, t[5], XOP_D2}, {c->wy, t[6], XOP_D2}, {c->wz, t[7], XOP_D2}};
    YJob yj[5] = {{t[0], t[8], YOP_D1}, {t[2], t[9], YOP_D1},
                  {c->wx, t[10], YOP_D2}, {c->wy, t[11], YOP_D2}, {c->wz, t[12], YOP_D2}};
    if ((r = tb_launch_xlines(c, xj, 5))) return r;
    if ((r = tb_launch_ylines(c, yj, 5))) return r;
    CombArgs A;
    std::memset(&A, 0, sizeof A);
    A.dady = t[8]; A.b = t[1]; A.xx0 = t[5]; A.yy0 = t[10]; A.wx = c->wx;
    A.c = t[2]; A.dadx = t[3]; A.xx1 = t[6]; A.yy1 = t[11]; A.wy = c->wy;
    A.dbdx = t[4]; A.dcdy = t[9]; A.xx2 = t[7]; A.yy2 = t[12]; A.wz = c->wz;
    A.fx = f[0]; A.fy = f[1]; A.dfydx = df[0]; A.dfzdx = df[1]; A.dfxdy = df[2]; A.dfzdy = df[3];
    A.dvx = dvx; A.dvy = dvy; A.dvz = dvz; A.k2b2 = c->k2b2;
    A.nx = c->g.nx; A.ny = c->g.ny; A.K = c->g.K; A.beta = c->cfg.beta; A.invRe = 1.0 / c->cfg.Re; A.fac_y = c->cfg.fac_y;
    k_combine<<<tb_blocks(tb_n3(c), 256), 256, 0, c->stream>>>(A);
    TB_CHECK_LAUNCH(c);
    return TB_OK;
}

int tb_rk_update(tb_ctx* c, int stage) {
    RkArgs A{c->wx, c->wy, c->wz, c->wx1, c->wy1, c->wz1, c->dv1x, c->dv1y, c->dv1z, c->dv2x, c->dv2y, c->dv2z,
             c->g.nx, c->g.ny, c->g.K, stage, c->dt, c->dt2, c->dt6};
    k_rk<<<tb_blocks(tb_n3(c), 256), 256, 0, c->stream>>>(A);
    TB_CHECK_LAUNCH(c);
    return c->cfg.my_form == 2 ? tb_rk_update_th(c, stage) : TB_OK;
}

// filter_trid (filter_par.f:144-177), in place on rows i >= 2, j >= 2 (1-based)
int tb_filter(tb_ctx* c) {
    XJob xj[3] = {{c->wx, c->wx, XOP_FILTER}, {c->wy, c->wy, XOP_FILTER}, {c->wz, c->wz, XOP_FILTER}};
    return tb_launch_xlines(c, xj, 3);
}

int tb_bzone_k(tb_ctx* c) {
    k_bzone<<<tb_blocks(tb_n3(c), 256), 256, 0, c->stream>>>(c->wx, c->wy, c->wz, c->bdfc, c->wzb, c->g.nx, c->g.ny, c->g.K, 0,
                                                              c->cfg.my_form);
    TB_CHECK_LAUNCH(c);
    return c->cfg.my_form == 2 ? tb_bzone_th(c) : TB_OK;
}
int tb_bzonew_k(tb_ctx* c) {
    k_bzone<<<tb_blocks((size_t)c->g.nx * c->g.K, 256), 256, 0, c->stream>>>(c->wx, c->wy, c->wz, c->bdfc, c->wzb, c->g.nx,
                                                                              c->g.ny, c->g.K, 1, c->cfg.my_form);
    TB_CHECK_LAUNCH(c);
    return TB_OK;
}
int tb_outuy_k(tb_ctx* c, cplx* dwzdx) {
    XJob xj[1] = {{c->wz, dwzdx, XOP_D1}};
    int r;
    if ((r = tb_launch_xlines(c, xj, 1))) return r;
    k_outuy_bc<<<tb_blocks((size_t)c->g.ny * c->g.K, 128), 128, 0, c->stream>>>(c->uy, c->uyb, c->g.nx, c->g.ny, c->g.K,
                                                                                 c->cfg.my_form);
    TB_CHECK_LAUNCH(c);
    return TB_OK;
}
int tb_poi_ux_k(tb_ctx* c, cplx* duydy) {
    int r;
    YJob yj[1] = {{c->uy, duydy, YOP_D1FV}};
    if ((r = tb_launch_ylines(c, yj, 1))) return r;
    size_t sm = xw_smem(c->g.nx);
    TB_CUDA(cudaFuncSetAttribute(k_ux_mode0, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    k_ux_mode0<<<tb_blocks(c->g.ny - 2, XW_WARPS), 32 * XW_WARPS, sm, c->stream>>>(c->ux, duydy, c->g.nx, c->g.ny, c->cfg.dx);
    TB_CHECK_LAUNCH(c);
    if (c->g.K < 2) return TB_OK;
    cplx* d2 = c->tmp[13];
    XJob xj[1] = {{duydy, d2, XOP_D1}};
    if ((r = tb_launch_xlines(c, xj, 1))) return r;
    return launch_penta(c, d2, c->wy, c->ux, -1.0);
}
int tb_poi_uz_k(tb_ctx* c, const cplx* duydy) {
    if (c->g.K < 2) return TB_OK;
    int r;
    cplx* dwydx = c->tmp[14];
    XJob xj[1] = {{c->wy, dwydx, XOP_D1}};
    if ((r = tb_launch_xlines(c, xj, 1))) return r;
    return launch_penta(c, dwydx, duydy, c->uz, 1.0);
}
int tb_wx_wall_k(tb_ctx* c, cplx* lapv) {
    const double* wat = c->coefs.data() + 100 + 24 * c->g.msh - 17;  // w_at_w_coef(9) on the host
    const double* dcoef = c->wcoef;   // device copy of w_at_w_coef(9), dwydy_coef(8)
    double dyy = c->cfg.dy * c->cfg.dy;
    unsigned nb = tb_blocks((size_t)c->g.nx * c->g.K, 128);
    k_lapv<<<nb, 128, 0, c->stream>>>(lapv, c->uy, c->d2uydx2, c->k2b2, dcoef, c->g.nx, c->g.ny, c->g.K,
                                       1.0 / (dyy * wat[0]));
    TB_CHECK_LAUNCH(c);
    if (c->g.K < 2) return TB_OK;
    cplx* dw = c->tmp[15];
    k_dwydy_wall<<<nb, 128, 0, c->stream>>>(dw, c->wy, dcoef + 9, c->g.nx, c->g.ny, c->g.K, 1.0 / c->cfg.dy);
    TB_CHECK_LAUNCH(c);
    const size_t sm = (size_t)penta_line_size(c->px.S) * sizeof(double);
    TB_CUDA(cudaFuncSetAttribute(k_wx_wall, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    k_wx_wall<<<c->g.K - 1, 64, sm, c->stream>>>(c->wx, dw, lapv, c->px.tab, c->g.nx, c->g.ny, c->px.S, c->cfg.dx, c->px.unit,
                                                 c->cfg.beta);
    TB_CHECK_LAUNCH(c);
    return TB_OK;
}
int tb_wz_wall_k(tb_ctx* c, const cplx* lapv) {
    size_t sm = xw_smem(c->g.nx);
    TB_CUDA(cudaFuncSetAttribute(k_wz_wall, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    k_wz_wall<<<tb_blocks(c->g.K, XW_WARPS), 32 * XW_WARPS, sm, c->stream>>>(c->wz, c->wx, lapv, c->g.nx, c->g.ny, c->g.K,
                                                                             c->cfg.dx, c->cfg.beta);
    TB_CHECK_LAUNCH(c);
    return TB_OK;
}
// Wall-forcing amplitude of each forced mode at step t + tempt, in the order
// of the forced modes that exist on this grid; returns their number.
int tb_ts_pert_fct(tb_ctx* c, int t, double tempt, double* out) {
    const tb_config& cf = c->cfg;
    if (cf.my_form == 1) {   // gv_pert (main_par.f:1577-1600): steady after the ramp
        double A = 1e-6 * std::sqrt(cf.fac_y);
        if (t < cf.stpp) {
            double ep = (double)t / (double)cf.stpp;
            A = A * ((6.0 * ep - 15.0) * ep + 10.0) * tb_powi(ep, 3);
        }
        out[0] = A;
        return 1;
    }
    int nf = 0;
    for (int m = 0; m < cf.n_forced && m < 4; m++) {
        int k = cf.forced_mode[m];
        if (k < 0 || k >= c->g.K) continue;
        double Aamp = cf.forced_amp[m] * std::sqrt(cf.fac_y);
        double H = 1.0;
        double arg = H * ((double)t + tempt) * cf.omega * c->dt;
        if (cf.forced_phase[m] != 0.0) arg = arg + cf.forced_phase[m];
        double fct = Aamp * std::sin(arg);
        if (t < cf.stpp) {
            double ept = (double)t / (double)cf.stpp;
            fct = fct * ((6.0 * ept - 15.0) * ept + 10.0) * tb_powi(ept, 3);
        }
        out[nf++] = fct;
    }
    return nf;
}

int tb_ts_pert_k(tb_ctx* c, int t, double tempt) {
    const tb_config& cf = c->cfg;
    if (cf.my_form == 1) {
        double a = 0.0;
        tb_ts_pert_fct(c, t, tempt, &a);
        const double* a_dev = c->capturing ? c->d_fct + (tempt < 0.75 ? 0 : 4) : nullptr;
        if (c->g.K < 2) return TB_OK;
        k_gv_pert<<<tb_blocks((size_t)c->g.nx * (c->g.K - 1), 128), 128, 0, c->stream>>>(
            c->uy, c->d2uydx2, c->fcx2, c->fcllx2, c->g.nx, c->g.ny, c->g.K, cf.i1, cf.i2, a, a_dev);
        TB_CHECK_LAUNCH(c);
        return TB_OK;
    }
    PertArgs A;
    std::memset(&A, 0, sizeof A);
    A.uy = c->uy; A.d2uydx2 = c->d2uydx2; A.fcx = c->fcx; A.fcllx = c->fcllx;
    A.nx = c->g.nx; A.ny = c->g.ny; A.i1 = cf.i1; A.i2 = cf.i2;
    for (int m = 0; m < cf.n_forced && m < 4; m++) {
        int k = cf.forced_mode[m];
        if (k < 0 || k >= c->g.K) continue;
        A.mode[A.nf++] = k;
    }
    tb_ts_pert_fct(c, t, tempt, A.fct);
    // in a recorded step the amplitudes of stage 1 (tempt 0.5) and stage 3
    // (tempt 1) are uploaded before each replay
    if (c->capturing) A.fct_dev = c->d_fct + (tempt < 0.75 ? 0 : 4);
    if (A.nf == 0) return TB_OK;
    k_ts_pert<<<tb_blocks(c->g.nx, 128), 128, 0, c->stream>>>(A);
    TB_CHECK_LAUNCH(c);
    return TB_OK;
}

// loop(erro) (main_par.f:1762-1785)
int tb_loop_impl(tb_ctx* c, double erro, bool filter) {
    int r;
    if (filter && (r = tb_filter(c))) return r;
    if ((r = tb_bzone_k(c))) return r;
    cplx* dwzdx = c->tmp[0];
    cplx* duydy = c->tmp[1];
    if ((r = tb_outuy_k(c, dwzdx))) return r;
    if (c->cfg.precision == TB_FORM_MIXED) r = tb_poi_uy_mixed(c, dwzdx, erro);
    else r = tb_poi_uy_k(c, dwzdx, erro);
    if (r) return r;
    if ((r = tb_poi_ux_k(c, duydy))) return r;
    if ((r = tb_poi_uz_k(c, duydy))) return r;
    if ((r = tb_wx_wall_k(c, c->lapv))) return r;
    if ((r = tb_wz_wall_k(c, c->lapv))) return r;
    return tb_bzonew_k(c);
}
