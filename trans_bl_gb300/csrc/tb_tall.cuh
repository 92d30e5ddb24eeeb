// tb_tall.cuh -- the FP32 V-cycle's levels of more than 272 rows (included by
// tb_mixed.cu).
//
// The strips of tb_cycle.cuh hold 96 lines in the registers of one CTA, and above
// 272 rows they do not fit: with 33 rows a chunk they spilled 6 KB a thread.  So the
// levels that keep all rows of such a grid (the finest and those coarsened in x
// only) relax a line on a warp, one launch per colour, e in global memory
// (k_relax).  The levels below have half the rows and stay in strips.  The
// V-cycles of two corrections at 1025 points and 32 modes, ms:
//   rows                                         273   321   385   505
//   strips on all levels, 33 rows a chunk        12.6  12.8  13.0  13.9
//   this                                          5.9   7.3   8.3  12.1
// and a solve with them against every level a line on a warp:
//   this                                          8.2   9.9  11.4  16.2
//   every level so                               10.5  12.7  19.9  24.3
//
// Layout: lines contiguous, element (i, j) of level l at off[l] + n i + j.  The
// finest level's right-hand side comes from the colour planes and its e
// goes back to them (k_in, k_out), and the restriction to the first strip
// level and the interpolation from it cross over too.
#pragma once
#include "tb_cycle.cuh"

namespace tall {

constexpr int STRIP_ROWS = 272;   // rows that the strips take
constexpr int THREADS = 128;      // 4 warps, a line each

struct Levels {
    float2 *e, *r, *rr;    // per mode blocks of `elems`; rr (nx[0] * n) holds one level's residual
    const float* tab;      // (2, NL, K) blocks of tab_size: line tables per type
    const float *coef, *qdy2;   // of the finest level: sp(7) cp(8) pp(4) lp(5), 1/dy^2
    const double* k2b2;
    const int* state;      // per mode: [2k] active
    int K, NL, n;
    int nx[mg::MAX_LEVELS];
    size_t off[mg::MAX_LEVELS], elems;
    float qx[mg::MAX_LEVELS];   // 1 / (12 dx_l^2 fac_y)
    float ify, alpha2;          // 1 / fac_y, alpha^2
};
// L1 L2 U1 U2 ID h1 h2 k1 k2 (n each), Kogge-Stone matrices Pf Pb (5, 32, 4)
__host__ __device__ inline size_t tab_size(int n) { return 9 * (size_t)n + 1280; }
// Rows per lane: the smallest odd S from 9 with 32 S >= n (an even one has the lanes
// meet in the banks of the line staged in shared memory: 505 rows took 17.1 ms with
// 16 rows a lane, 12.1 with 17).
inline int pick_rows(int n) { return n <= 288 ? 9 : n <= 352 ? 11 : n <= 416 ? 13 : n <= 480 ? 15 : 17; }

__device__ __forceinline__ float2 f2(float a, float b) { return make_float2(a, b); }

// The FP32 operator of a level at a point.
struct PointOp {
    int nx, n;
    const float *cf, *Q2;
    float k2b2, den, ify, alpha2;
};
// s - L e at the interior point (i, j), the operator of defect
// (poisson_par.f:543-793) term by term; f(i, j) reads e.
template <class F>
__device__ __forceinline__ float2 point_resid(const PointOp& O, int i, int j, float2 s, const F& f) {
    const int nxl = O.nx, n = O.n;
    const float *SP = O.cf, *CP = SP + 7, *PP = SP + 15, *LP = SP + 19, *Q2 = O.Q2;
    const float k2b2 = O.k2b2;
    auto bx = [&](int jj) -> float2 {
        if (i == 1 || i == nxl - 2) {
            int e = (i == 1) ? 1 : -1;
            float2 a = f(i - e, jj), c0 = f(i, jj), b = f(i + e, jj), c = f(i + 2 * e, jj), d = f(i + 3 * e, jj), g = f(i + 4 * e, jj);
            return f2(10.f * a.x - 15.f * c0.x - 4.f * b.x + 14.f * c.x - 6.f * d.x + g.x,
                      10.f * a.y - 15.f * c0.y - 4.f * b.y + 14.f * c.y - 6.f * d.y + g.y);
        }
        float2 a = f(i - 2, jj), b = f(i - 1, jj), c0 = f(i, jj), c = f(i + 1, jj), d = f(i + 2, jj);
        return f2(-a.x + 16.f * b.x - 30.f * c0.x + 16.f * c.x - d.x, -a.y + 16.f * b.y - 30.f * c0.y + 16.f * c.y - d.y);
    };
    float2 b, cc, d;
    float q2, top = 0.f;
    if (j == 1) {
        float2 b1 = bx(1), b2 = bx(2);
        b = f2(SP[2] * b2.x + SP[1] * b1.x, SP[2] * b2.y + SP[1] * b1.y);
        float2 g0 = f(i, 0), g1 = f(i, 1), g2 = f(i, 2), g3 = f(i, 3);
        cc = f2(SP[3] * g0.x + SP[4] * g1.x + SP[5] * g2.x + SP[6] * g3.x, SP[3] * g0.y + SP[4] * g1.y + SP[5] * g2.y + SP[6] * g3.y);
        d = f2(k2b2 * (SP[1] * g1.x + SP[2] * g2.x), k2b2 * (SP[1] * g1.y + SP[2] * g2.y));
        q2 = Q2[0];
    } else if (j <= n - 3) {
        float2 ba = bx(j - 1), bb = bx(j), bc = bx(j + 1);
        b = f2(CP[0] * ba.x + CP[1] * bb.x + CP[2] * bc.x, CP[0] * ba.y + CP[1] * bb.y + CP[2] * bc.y);
        float2 fm2 = f(i, j - 2), fm1 = f(i, j - 1), g0 = f(i, j), fp1 = f(i, j + 1), fp2 = f(i, j + 2);
        cc = f2(CP[3] * fm2.x + CP[4] * fm1.x + CP[5] * g0.x + CP[6] * fp1.x + CP[7] * fp2.x,
                CP[3] * fm2.y + CP[4] * fm1.y + CP[5] * g0.y + CP[6] * fp1.y + CP[7] * fp2.y);
        d = f2(k2b2 * (CP[0] * fm1.x + CP[1] * g0.x + CP[2] * fp1.x), k2b2 * (CP[0] * fm1.y + CP[1] * g0.y + CP[2] * fp1.y));
        q2 = Q2[j - 2];
    } else if (j == n - 2) {
        b = bx(j);
        float2 fm1 = f(i, j - 1), g0 = f(i, j), fp1 = f(i, j + 1);
        cc = f2(PP[3] * fp1.x + PP[2] * g0.x + PP[1] * fm1.x, PP[3] * fp1.y + PP[2] * g0.y + PP[1] * fm1.y);
        d = f2(k2b2 * g0.x, k2b2 * g0.y);
        q2 = Q2[j - 1];
    } else {
        b = bx(j);
        float2 fm2 = f(i, j - 2), fm1 = f(i, j - 1), g0 = f(i, j);
        cc = f2(LP[2] * g0.x + LP[3] * fm1.x + LP[4] * fm2.x, LP[2] * g0.y + LP[3] * fm1.y + LP[4] * fm2.y);
        d = f2(k2b2 * g0.x, k2b2 * g0.y);
        q2 = Q2[j - 2];
        top = LP[1] * sqrtf((O.alpha2 - k2b2) * O.ify) * sqrtf(q2);
    }
    float2 fij = f(i, j);
    return f2(s.x - (b.x * O.den + cc.x * q2 + d.x * O.ify - top * fij.x),
              s.y - (b.y * O.den + cc.y * q2 + d.y * O.ify - top * fij.y));
}

// Relax one group of lines at level l: lines i = first + step*t, t < nlines,
// in every active mode; e(i, :) <- line solve of L e = r with the other lines
// frozen.  One warp per (line, mode); the pentadiagonal solve is split into
// 32 row chunks (local recurrences, warp scan of precomputed 2x2 chunk
// propagators, fix-up with precomputed homogeneous responses).
template <int S>
__global__ void __launch_bounds__(THREADS, 6) k_relax(const __grid_constant__ Levels M, int l, int first, int step, int nlines) {
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int gw = blockIdx.x * (THREADS / 32) + wib;
    const int k = gw / nlines;
    if (k >= M.K || !M.state[2 * k]) return;   // uniform over the warp
    const int i = first + step * (gw - k * nlines);
    const int nxl = M.nx[l], n = M.n;
    const bool border = i == 1 || i == nxl - 2;
    const int dir = (i == 1) ? 1 : -1;
    extern __shared__ float2 smf[];
    float2* g = smf + (size_t)wib * 2 * n;
    float2* rs = g + n;
    float2* E = M.e + (size_t)k * M.elems + M.off[l];
    const float2* R = M.r + (size_t)k * M.elems + M.off[l] + (size_t)n * i;
    // x-stencil sums without the diagonal (rhs_center / rhs_border,
    // poisson_par.f:229-540), rows j = lane + 32 q, q < S (32 S >= n): all loads
    // of the line issue at once
    auto xsum = [&](int j) -> float2 {
        auto at = [&](int ii) { return E[(size_t)n * ii + j]; };
        if (!border) {
            float2 a = at(i - 2), b = at(i - 1), c = at(i + 1), d = at(i + 2);
            return f2(16.f * (b.x + c.x) - (a.x + d.x), 16.f * (b.y + c.y) - (a.y + d.y));
        }
        float2 a = at(i - dir), b = at(i + dir), c = at(i + 2 * dir), d = at(i + 3 * dir), f = at(i + 4 * dir);
        return f2(10.f * a.x - 4.f * b.x + 14.f * c.x - 6.f * d.x + f.x, 10.f * a.y - 4.f * b.y + 14.f * c.y - 6.f * d.y + f.y);
    };
    float2 rv[S];
#pragma unroll
    for (int q = 0; q < S; q++) {
        int j = lane + 32 * q;
        if (j < n) { g[j] = xsum(j); rv[q] = R[j]; }
    }
    __syncwarp();
    const float* cf = M.coef;
    const float sp2 = cf[1], sp3 = cf[2], cp1 = cf[7], cp2 = cf[8], cp3 = cf[9];
    const float qx = M.qx[l];
#pragma unroll
    for (int q = 0; q < S; q++) {
        int j = lane + 32 * q;
        if (j >= n) break;
        float2 v = f2(0.f, 0.f);
        if (j >= 1) {
            float2 t;
            if (j == 1) t = f2(sp3 * g[2].x + sp2 * g[1].x, sp3 * g[2].y + sp2 * g[1].y);
            else if (j <= n - 3)
                t = f2(cp1 * g[j - 1].x + cp2 * g[j].x + cp3 * g[j + 1].x, cp1 * g[j - 1].y + cp2 * g[j].y + cp3 * g[j + 1].y);
            else t = g[j];
            float2 s = rv[q];
            v = f2(s.x - qx * t.x, s.y - qx * t.y);
        }
        rs[j] = v;
    }
    __syncwarp();
    const float* T = M.tab + (((size_t)(border ? 1 : 0) * M.NL + l) * M.K + k) * tab_size(n);
    const float *L1 = T, *L2 = T + n, *U1 = T + 2 * n, *U2 = T + 3 * n, *ID = T + 4 * n;
    const float *h1 = T + 5 * n, *h2 = T + 6 * n, *k1 = T + 7 * n, *k2 = T + 8 * n;
    const float* Pf = T + 9 * n;
    const float* Pb = Pf + 640;
    const int r0 = lane * S, r1 = min(n, r0 + S);
    float2 y[S];
    float2 ym1 = f2(0.f, 0.f), ym2 = f2(0.f, 0.f);
#pragma unroll
    for (int s = 0; s < S; s++) {
        int j = r0 + s;
        if (j < r1) {
            float2 v = rs[j];
            float a1 = L1[j], a2 = L2[j];
            float2 yy = f2(v.x - a2 * ym2.x - a1 * ym1.x, v.y - a2 * ym2.y - a1 * ym1.y);
            y[s] = yy; ym2 = ym1; ym1 = yy;
        }
    }
    float2 b0 = ym1, b1 = ym2;
#pragma unroll
    for (int d = 0, off = 1; d < 5; d++, off <<= 1) {
        float2 o0, o1;
        o0.x = __shfl_up_sync(0xffffffffu, b0.x, off); o0.y = __shfl_up_sync(0xffffffffu, b0.y, off);
        o1.x = __shfl_up_sync(0xffffffffu, b1.x, off); o1.y = __shfl_up_sync(0xffffffffu, b1.y, off);
        if (lane >= off) {
            const float* P = Pf + (d * 32 + lane) * 4;
            b0 = f2(b0.x + P[0] * o0.x + P[1] * o1.x, b0.y + P[0] * o0.y + P[1] * o1.y);
            b1 = f2(b1.x + P[2] * o0.x + P[3] * o1.x, b1.y + P[2] * o0.y + P[3] * o1.y);
        }
    }
    float2 Y1, Y2;
    Y1.x = __shfl_up_sync(0xffffffffu, b0.x, 1); Y1.y = __shfl_up_sync(0xffffffffu, b0.y, 1);
    Y2.x = __shfl_up_sync(0xffffffffu, b1.x, 1); Y2.y = __shfl_up_sync(0xffffffffu, b1.y, 1);
    if (lane == 0) { Y1 = f2(0.f, 0.f); Y2 = f2(0.f, 0.f); }
#pragma unroll
    for (int s = 0; s < S; s++) {
        int j = r0 + s;
        if (j < r1) y[s] = f2(y[s].x + h1[j] * Y1.x + h2[j] * Y2.x, y[s].y + h1[j] * Y1.y + h2[j] * Y2.y);
    }
    float2 xp1 = f2(0.f, 0.f), xp2 = f2(0.f, 0.f);
#pragma unroll
    for (int s = S - 1; s >= 0; s--) {
        int j = r0 + s;
        if (j < r1) {
            float u1 = U1[j], u2 = U2[j], id = ID[j];
            float2 xx = f2((y[s].x - u1 * xp1.x - u2 * xp2.x) * id, (y[s].y - u1 * xp1.y - u2 * xp2.y) * id);
            y[s] = xx; xp2 = xp1; xp1 = xx;
        }
    }
    b0 = xp1; b1 = xp2;
#pragma unroll
    for (int d = 0, off = 1; d < 5; d++, off <<= 1) {
        float2 o0, o1;
        o0.x = __shfl_down_sync(0xffffffffu, b0.x, off); o0.y = __shfl_down_sync(0xffffffffu, b0.y, off);
        o1.x = __shfl_down_sync(0xffffffffu, b1.x, off); o1.y = __shfl_down_sync(0xffffffffu, b1.y, off);
        if (lane + off < 32) {
            const float* P = Pb + (d * 32 + lane) * 4;
            b0 = f2(b0.x + P[0] * o0.x + P[1] * o1.x, b0.y + P[0] * o0.y + P[1] * o1.y);
            b1 = f2(b1.x + P[2] * o0.x + P[3] * o1.x, b1.y + P[2] * o0.y + P[3] * o1.y);
        }
    }
    float2 X1, X2;
    X1.x = __shfl_down_sync(0xffffffffu, b0.x, 1); X1.y = __shfl_down_sync(0xffffffffu, b0.y, 1);
    X2.x = __shfl_down_sync(0xffffffffu, b1.x, 1); X2.y = __shfl_down_sync(0xffffffffu, b1.y, 1);
    if (lane == 31) { X1 = f2(0.f, 0.f); X2 = f2(0.f, 0.f); }
    __syncwarp();
#pragma unroll
    for (int s = 0; s < S; s++) {
        int j = r0 + s;
        if (j < r1) rs[j] = f2(y[s].x + k1[j] * X1.x + k2[j] * X2.x, y[s].y + k1[j] * X1.y + k2[j] * X2.y);
    }
    __syncwarp();
    float2* Ei = E + (size_t)n * i;
#pragma unroll
    for (int q = 0; q < S; q++) {
        int j = lane + 32 * q;
        if (j >= 1 && j < n) Ei[j] = rs[j];
    }
}

// A thread's point (mode k, line i, row j) of `lines` x n points per mode; false
// beyond them or in a mode that is done.
__device__ __forceinline__ bool point(const Levels& M, int lines, int& k, int& i, int& j) {
    const size_t per = (size_t)lines * M.n, q = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (q >= per * M.K) return false;
    k = (int)(q / per);
    const size_t rq = q % per;
    i = (int)(rq / M.n);
    j = (int)(rq % M.n);
    return M.state[2 * k] != 0;
}

// rr = r - L e at level l.
__global__ void k_resid(const __grid_constant__ Levels M, int l) {
    int k, i, j;
    if (!point(M, M.nx[l], k, i, j) || i < 1 || i > M.nx[l] - 2 || j < 1) return;
    const float2* E = M.e + (size_t)k * M.elems + M.off[l];
    const size_t o = (size_t)M.n * i + j;
    const PointOp O{M.nx[l], M.n, M.coef, M.qdy2, (float)M.k2b2[k], M.qx[l], M.ify, M.alpha2};
    M.rr[(size_t)k * M.nx[0] * M.n + o] =
        point_resid(O, i, j, M.r[(size_t)k * M.elems + M.off[l] + o], [&](int ii, int jj) { return E[(size_t)M.n * ii + jj]; });
}

// rr of level l into r(l+1), weights (1/4, 1/2, 1/4) in x; e(l+1) starts at 0.
__global__ void k_restrict_x(const __grid_constant__ Levels M, int l) {
    int k, i, j;
    if (!point(M, M.nx[l + 1], k, i, j)) return;
    const size_t n = M.n, oc = (size_t)k * M.elems + M.off[l + 1] + n * i + j;
    M.e[oc] = f2(0.f, 0.f);
    float2 v = f2(0.f, 0.f);
    if (i >= 1 && i <= M.nx[l + 1] - 2 && j >= 1) {
        const float2* D = M.rr + (size_t)k * M.nx[0] * n + j;
        float2 a = D[n * (2 * i - 1)], b = D[n * (2 * i)], c = D[n * (2 * i + 1)];
        v = f2(0.25f * (a.x + 2.f * b.x + c.x), 0.25f * (a.y + 2.f * b.y + c.y));
    }
    M.r[oc] = v;
}

// e(l) of an x-only coarsened level, interpolated, added to e(l-1).
__global__ void k_prolong_x(const __grid_constant__ Levels M, int l) {
    int k, i, j;
    if (!point(M, M.nx[l - 1], k, i, j) || i < 1 || i > M.nx[l - 1] - 2 || j < 1) return;
    const size_t n = M.n;
    const float2* C = M.e + (size_t)k * M.elems + M.off[l] + j;
    float2 t = C[n * (i / 2)];
    if (i & 1) {
        float2 b = C[n * (i / 2 + 1)];
        t = f2(0.5f * (t.x + b.x), 0.5f * (t.y + b.y));
    }
    float2& fe = M.e[(size_t)k * M.elems + M.off[l - 1] + n * i + j];
    fe = f2(fe.x + t.x, fe.y + t.y);
}

// rr of the last of these levels into r of the first strip level, weights of
// restrict (poisson_par.f:796-874); interior points only, the others hold zeros.
__global__ void k_restrict_out(const __grid_constant__ Levels M, const __grid_constant__ mg::Cycle S) {
    const mg::Level& N = S.lv[M.NL];
    const int k = blockIdx.z, j = 1 + blockIdx.y, i = 1 + blockIdx.x * blockDim.x + threadIdx.x, n = M.n;
    if (!M.state[2 * k] || i > N.nx - 2) return;
    const float2* D = M.rr + (size_t)k * M.nx[0] * n;
    auto df = [&](int ii, int jj) { return D[(size_t)n * ii + jj]; };
    const int fi = 2 * i, fj = j <= N.n - 2 ? 2 * j : n - 1;
    float2 v;
    if (j <= N.n - 2) {
        float2 a = df(fi - 1, fj), b = df(fi + 1, fj), c = df(fi, fj - 1), d = df(fi, fj + 1), e = df(fi, fj);
        float2 g1 = df(fi + 1, fj + 1), g2 = df(fi + 1, fj - 1), g3 = df(fi - 1, fj + 1), g4 = df(fi - 1, fj - 1);
        v.x = 0.0625f * (2.f * (a.x + b.x + c.x + d.x) + 4.f * e.x + g1.x + g2.x + g3.x + g4.x);
        v.y = 0.0625f * (2.f * (a.y + b.y + c.y + d.y) + 4.f * e.y + g1.y + g2.y + g3.y + g4.y);
    } else {
        float2 a = df(fi - 1, fj), e = df(fi, fj), b = df(fi + 1, fj);
        v = f2(0.25f * (a.x + 2.f * e.x + b.x), 0.25f * (a.y + 2.f * e.y + b.y));
    }
    S.r[(size_t)k * S.elems + mg::el(N, i, j)] = v;
}

// eb of the first strip level, interpolated bilinearly (intpol,
// poisson_par.f:877-920), added to e of the last of these levels.
__global__ void k_prolong_in(const __grid_constant__ Levels M, const __grid_constant__ mg::Cycle S) {
    const int l = M.NL - 1;
    int k, i, j;
    if (!point(M, M.nx[l], k, i, j) || i < 1 || i > M.nx[l] - 2 || j < 1) return;
    const mg::Level& N = S.lv[M.NL];
    const float2* C = S.eb + (size_t)k * S.elems;
    auto row = [&](int cj) -> float2 {
        float2 a = C[mg::el(N, i / 2, cj)];
        if ((i & 1) == 0) return a;
        float2 b = C[mg::el(N, i / 2 + 1, cj)];
        return f2(0.5f * (a.x + b.x), 0.5f * (a.y + b.y));
    };
    float2 t = row(j / 2);
    if (j & 1) {
        float2 b = row(j / 2 + 1);
        t = f2(0.5f * (t.x + b.x), 0.5f * (t.y + b.y));
    }
    float2& fe = M.e[(size_t)k * M.elems + M.off[l] + (size_t)M.n * i + j];
    fe = f2(fe.x + t.x, fe.y + t.y);
}

// The finest level's r out of the colour planes, e = 0 (OUT false), or its e into
// them (OUT true), in 32 x 32 tiles through shared memory.
template <bool OUT>
__global__ void __launch_bounds__(256) k_cross(const __grid_constant__ Levels M, const __grid_constant__ mg::Cycle S) {
    __shared__ float2 tile[32][33];
    const int k = blockIdx.z, i0 = blockIdx.x * 32, j0 = blockIdx.y * 32, nx = M.nx[0], n = M.n;
    if (!M.state[2 * k]) return;   // uniform over the block
    const size_t line = (size_t)k * M.elems, plane = (size_t)k * S.elems;
    for (int q = threadIdx.y; q < 32; q += 8) {
        const int i = i0 + (OUT ? q : threadIdx.x), j = j0 + (OUT ? threadIdx.x : q);
        if (i < nx && j < n) tile[q][threadIdx.x] = OUT ? M.e[line + (size_t)n * i + j] : S.r[plane + mg::el(S.lv[0], i, j)];
    }
    __syncthreads();
    for (int q = threadIdx.y; q < 32; q += 8) {
        const int i = i0 + (OUT ? threadIdx.x : q), j = j0 + (OUT ? q : threadIdx.x);
        if (i >= nx || j >= n) continue;
        const float2 v = tile[threadIdx.x][q];
        if (OUT) S.eb[plane + mg::el(S.lv[0], i, j)] = v;
        else {
            M.r[line + (size_t)n * i + j] = v;
            M.e[line + (size_t)n * i + j] = f2(0.f, 0.f);
        }
    }
}

}  // namespace tall
