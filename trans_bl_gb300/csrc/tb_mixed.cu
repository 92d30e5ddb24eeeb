// tb_mixed.cu -- mixed-precision form of the v-Poisson solve (poi_uy).
//
// The reference solves each mode's v-Poisson problem with an FP64 FAS
// multigrid whose smoother relaxes the y-lines in lexicographic x order
// (poisson_par.f:6-963): every line waits for the one before it.  This form
// keeps the reference's discrete problem and its stopping rule and changes
// how the answer is reached:
//
//   outer loop, FP64 (defect correction on the reference's fine operator):
//     d = sc - L u        -- same kernel as the plain form (poisson_par.f:543-793)
//     stop a mode once max|d| < tol  (verifica_poi, poisson_par.f:945-963)
//     solve L e = d       -- FP32 correction-scheme multigrid, e = 0 at start
//     u += e
//
// The FP32 multigrid uses the reference's level operators (compact y-weights
// and 4th-order x-stencils of coef_center/coef_border), full-weighting
// restriction and bilinear prolongation on the reference's msh levels.  Below
// them it keeps coarsening in x only (same y-level operators, dx doubled,
// (1/4, 1/2, 1/4) restriction, linear prolongation) until a level has at most
// DIRECT_MAX unknowns, which is solved exactly: its operator is inverted per
// mode at set-up (FP64 Gauss-Jordan, stored in FP32) and applied as one
// matrix-vector product.  The smoother relaxes y-lines in four
// groups: the two border lines, then the centre lines by colour i mod 3.  The
// centre stencil reaches i+-2 and the border stencil reaches 4 lines inwards,
// so the lines of one group never read each other and a whole group is solved
// at once (tb_cycle.cuh: the V-cycle's kernels and the layout of its levels;
// tb_tall.cuh: levels of more than 272 rows).
#include "tb_internal.h"
#include "tb_cycle.cuh"
#include "tb_tall.cuh"
#include <algorithm>
#include <array>
#include <cmath>
#include <cstring>
#include <thread>

namespace {

// Relaxation sweeps before / after the coarse correction, V-cycles per FP64
// correction, and whether the hierarchy starts with x-only coarsening
// (until dx >= the largest y-spacing, so that y-coupling dominates at every
// point of the coarser levels and y-line relaxation smooths everywhere).
#ifndef TB_MG_NU_PRE
#define TB_MG_NU_PRE 1
#endif
#ifndef TB_MG_NU_POST
#define TB_MG_NU_POST 2
#endif
#ifndef TB_MG_INNER
#define TB_MG_INNER 2
#endif
#ifndef TB_MG_SEMI_FIRST
#define TB_MG_SEMI_FIRST 1
#endif
constexpr int NU_PRE = TB_MG_NU_PRE, NU_POST = TB_MG_NU_POST, INNER_VCYCLES = TB_MG_INNER;
constexpr int MG_MAX = mg::MAX_LEVELS;   // levels of the FP32 hierarchy
constexpr int DIRECT_MAX = 400;      // unknowns per mode below which coarsening stops

struct Mixed {
    float2 *ea = nullptr, *eb = nullptr, *r = nullptr;   // per mode blocks of `elems` (layout: tb_cycle.cuh)
    float4* tab = nullptr;    // per mode: line-solve and residual rows of every level (mg::Cycle::tab)
    double* drow = nullptr;   // rows and modes of the FP64 defect (DefectRows)
    float* coef = nullptr;    // sp(7) cp(8) pp(4) lp(5) per reference level
    float* qdy2 = nullptr;    // (ny, msh)
    float* ainv = nullptr;    // (K, N, N) inverse of the coarsest operator per mode
    unsigned long long* maxsq = nullptr;   // (K) max |defect|^2 as double bits
    // warm start: per RK stage the v of the last two steps' solves (h0 the
    // newer), how many of them are usable (device, per stage) and the step
    // of the last solve (host)
    cplx* hist[4][2] = {{nullptr, nullptr}, {nullptr, nullptr}, {nullptr, nullptr}, {nullptr, nullptr}};
    int* hvalid = nullptr;
    int last_t[4] = {-9, -9, -9, -9};
    int hv_host[4] = {0, 0, 0, 0};   // host copy of hvalid for host-launched solves
    int* lkeep = nullptr;            // (K, 2) learned correction kept per mode, in the layout of pstate
    int* iter = nullptr;      // corrections tested so far in a recorded solve loop
    int NL = 0, N = 0;
    int ptsx[MG_MAX], ptsy[MG_MAX], ylvl[MG_MAX], semi[MG_MAX];
    double dx2[MG_MAX];
    size_t elems = 0;
    mg::Cycle cyc;            // launch arguments of the V-cycle kernels
    tall::Levels tl;          // the levels above the strips (NL of them: 0 on most grids)
};

// The finest FP32 level for the kernels outside the V-cycle.
struct FineDev {
    float2 *e, *r;
    const float* coef;
    const float* qdy2;
    const double* k2b2;
    const int* state;
    mg::Level L;
    int nx, ny, K;
    size_t elems;
    float den;              // 1 / (12 dx^2 fac_y)
    float ify, alpha2;      // 1 / fac_y, alpha^2
};

__device__ __forceinline__ float2 f2(float a, float b) { return make_float2(a, b); }

// FP32 residual r - L e at the interior point (i, j) of the finest level, point
// by point (the learned correction's judge and its tests; the V-cycle's strips have
// their own fused form).
__device__ __forceinline__ float2 fine_resid(const FineDev& M, int k, int i, int j) {
    const float2* E = M.e + (size_t)k * M.elems;
    const tall::PointOp O{M.nx, M.ny, M.coef, M.qdy2, (float)M.k2b2[k], M.den, M.ify, M.alpha2};
    return tall::point_resid(O, i, j, M.r[(size_t)k * M.elems + mg::el(M.L, i, j)],
                             [&](int ii, int jj) { return E[mg::el(M.L, ii, jj)]; });
}

// The residual of one mode into out, line-contiguous (nx, ny).
__global__ void k_fine_resid(FineDev M, int k, float2* out) {
    const size_t per = (size_t)(M.nx - 2) * (M.ny - 1);
    const size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (q >= per) return;
    const int j = 1 + (int)(q % (M.ny - 1)), i = 1 + (int)(q / (M.ny - 1));
    out[(size_t)M.ny * i + j] = fine_resid(M, k, i, j);
}

// Warm start of one stage's solve from its history h0 (previous step), h1
// (the step before), of which *valid are usable: with both, fc = 2 h0 - h1
// on the interior of the FP64 fine level (the boundary rows and columns keep
// this stage's Dirichlet data).  h1 <- h0 then makes room for this solve,
// which the caller copies into h0.
__global__ void k_extrap(cplx* fc, size_t elems64, cplx* h0, cplx* h1, const int* valid, int nx, int ny, int K,
                         int shift) {
    const int nv = *valid;
    if (nv == 0) return;
    size_t per = (size_t)nx * ny;
    size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (q >= per * K) return;
    int k = (int)(q / per);
    int i = (int)((q % per) % nx), j = (int)((q % per) / nx);
    cplx a = h0[q];
    if (nv >= 2 && i >= 1 && i <= nx - 2 && j >= 1) {
        cplx b = h1[q];
        fc[(size_t)k * elems64 + (q % per)] = make_double2(2.0 * a.x - b.x, 2.0 * a.y - b.y);
    }
    if (shift) h1[q] = a;
}

// warm_start = 2: the previous solve's solution fc (stage p = s - 1 of this
// step, or stage 4 of the last step for s = 1) plus the increment between
// the same two solves one step earlier, fc + v_s(n-1) - v_p(n-1), from this
// stage's newest history entry h0 and stage p's older one hp1.  Stages 2 and 4
// solve at the same time as the stage before them, so the increment is the
// difference of two RK stage estimates and changes by O(dt^3) per step;
// stages 1 and 3 carry half a step of time change, O(dt^2) with half the
// constant of the linear extrapolation.  Needs one entry of this stage's
// history and two of stage p's; shifts this stage's history as k_extrap.
__global__ void k_extrap_inc(cplx* fc, size_t elems64, cplx* h0, cplx* h1, const cplx* hp1, const int* valid,
                             const int* valid_p, int nx, int ny, int K, int shift) {
    const int nv = *valid, np = *valid_p;
    if (nv == 0) return;
    const size_t per = (size_t)nx * ny;
    const size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (q >= per * K) return;
    const int k = (int)(q / per);
    const int i = (int)((q % per) % nx), j = (int)((q % per) / nx);
    const cplx a = h0[q];
    if (np >= 2 && i >= 1 && i <= nx - 2 && j >= 1) {
        cplx& f = fc[(size_t)k * elems64 + (q % per)];
        const cplx b = hp1[q];
        f = make_double2(f.x + (a.x - b.x), f.y + (a.y - b.y));
    }
    if (shift) h1[q] = a;
}

// ---- learned first correction (network and training in tb_learn.cu) -------
// Per mode maxima over both parts of |v1| and |v1 - v2| (history,
// x-contiguous) and of |D^-1 d0| (d0: the FP32 copy r of the FP64 defect of
// the guess), as float bits in scl (K, 3).
__global__ void k_learn_scale(FineDev M, const cplx* h0, const cplx* h1, const int* valid, unsigned* scl, const float* invD,
                              int nx) {
    if (*valid < 2) return;
    const int k = blockIdx.y, ny = M.ny;
    const size_t per = (size_t)nx * ny;
    float a = 0.f, b = 0.f, d = 0.f;
    for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < per; q += (size_t)gridDim.x * blockDim.x) {
        const cplx u = h0[(size_t)k * per + q], w = h1[(size_t)k * per + q];
        a = fmaxf(a, fmaxf(fabsf((float)u.x), fabsf((float)u.y)));
        b = fmaxf(b, fmaxf(fabsf((float)(u.x - w.x)), fabsf((float)(u.y - w.y))));
        const int i = (int)(q % nx), j = (int)(q / nx);
        const float2 r = M.r[(size_t)k * M.elems + mg::el(M.L, i, j)];
        d = fmaxf(d, invD[(size_t)k * ny + j] * fmaxf(fabsf(r.x), fabsf(r.y)));
    }
    for (int o = 16; o > 0; o >>= 1) {
        a = fmaxf(a, __shfl_xor_sync(0xffffffffu, a, o));
        b = fmaxf(b, __shfl_xor_sync(0xffffffffu, b, o));
        d = fmaxf(d, __shfl_xor_sync(0xffffffffu, d, o));
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMax(&scl[3 * k], __float_as_uint(a));
        atomicMax(&scl[3 * k + 1], __float_as_uint(b));
        atomicMax(&scl[3 * k + 2], __float_as_uint(d));
    }
}

// The network's input planes X (2K, 4, nx, ny) and the history shift
// h1 <- h0 that k_extrap leaves to this kernel when the network runs.
__global__ void k_learn_prep(FineDev M, const cplx* h0, cplx* h1, const int* valid, const float* scl, const float* invD,
                             const float* mfeat, float* X, int nx) {
    const int nv = *valid;
    if (nv == 0) return;
    __shared__ float2 t0[32][33], t1[32][33];   // [j][i]: v1, v1 - v2
    const int k = blockIdx.z, ny = M.ny, i0 = blockIdx.x * 32, j0 = blockIdx.y * 32;
    const size_t per = (size_t)nx * ny;
    for (int r = threadIdx.y; r < 32; r += 8) {
        const int i = i0 + threadIdx.x, j = j0 + r;
        float2 a = f2(0.f, 0.f), b = f2(0.f, 0.f);
        if (i < nx && j < ny) {
            const size_t o = (size_t)k * per + (size_t)j * nx + i;
            const cplx u = h0[o], w = h1[o];
            a = f2((float)u.x, (float)u.y);
            b = f2((float)(u.x - w.x), (float)(u.y - w.y));
            h1[o] = u;
        }
        t0[r][threadIdx.x] = a;
        t1[r][threadIdx.x] = b;
    }
    if (nv < 2) return;   // uniform over the block
    __syncthreads();
    // one scale for the three field planes: s = max|v1 - v2|
    const float si = scl[3 * k + 1];
    const float ii = si > 0.f ? 1.f / si : 0.f, iv = ii, id = ii;
    float* Xr = X + (size_t)(2 * k) * 4 * per;   // planes of the real part, then of the imaginary part
    float* Xi = Xr + 4 * per;
    for (int r = threadIdx.y; r < 32; r += 8) {
        const int i = i0 + r, j = j0 + threadIdx.x;
        if (i >= nx || j >= ny) continue;
        const float2 a = t0[threadIdx.x][r], b = t1[threadIdx.x][r];
        const float2 d = M.r[(size_t)k * M.elems + mg::el(M.L, i, j)];
        const float sj = invD[(size_t)k * ny + j] * id, mf = mfeat[(size_t)k * ny + j];
        const size_t o = (size_t)ny * i + j;
        Xr[o] = a.x * iv; Xr[per + o] = b.x * ii; Xr[2 * per + o] = d.x * sj; Xr[3 * per + o] = mf;
        Xi[o] = a.y * iv; Xi[per + o] = b.y * ii; Xi[2 * per + o] = d.y * sj; Xi[3 * per + o] = mf;
    }
}

// Candidate correction e = max|v1 - v2| * network output on the fine interior.
__global__ void k_learn_emit(FineDev M, const float* out, const float* scl, const int* valid, int nx) {
    if (*valid < 2) return;
    const int ny = M.ny;
    const size_t per = (size_t)(nx - 2) * (ny - 1), img = (size_t)nx * ny;
    const size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (q >= per * M.K) return;
    const int k = (int)(q / per);
    const size_t rq = q % per;
    const int j = 1 + (int)(rq % (ny - 1)), i = 1 + (int)(rq / (ny - 1));
    const float s = scl[3 * k + 1];
    const size_t o = (size_t)ny * i + j;
    M.e[(size_t)k * M.elems + mg::el(M.L, i, j)] = f2(s * out[(size_t)(2 * k) * img + o], s * out[(size_t)(2 * k + 1) * img + o]);
}

// max |r - L e|^2 per mode (blockIdx.y) over the fine interior, float bits.
__global__ void k_learn_judge(FineDev M, unsigned* jmax, const int* valid, int nx) {
    if (*valid < 2) return;
    const int k = blockIdx.y, ny = M.ny;
    const size_t per = (size_t)(nx - 2) * (ny - 1);
    float m = 0.f;
    for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < per; q += (size_t)gridDim.x * blockDim.x) {
        const int j = 1 + (int)(q % (ny - 1)), i = 1 + (int)(q / (ny - 1));
        const float2 v = fine_resid(M, k, i, j);
        m = fmaxf(m, v.x * v.x + v.y * v.y);
    }
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(&jmax[k], __float_as_uint(m));
}

// Gated evaluation of the network for one stage's solve.  It runs the first
// time, once every `probe` solves, and in the solve after one where it ran
// and the solve needed fewer corrections than the stage's last solve
// without it: the network is kept on only while it saves multigrid work;
// otherwise the solve falls back to the warm-start guess without running it.
// g (per stage): [solves since it last ran, ran in the last solve,
// evaluations, solves, corrections of the last solve without it, of the
// last solve with it].  The decision goes to a conditional graph node (h)
// or, for host-launched solves, to *flag.
__global__ void k_learn_gate(int* g, int probe, cudaGraphConditionalHandle h, int use_handle, int* flag) {
    const int saved = g[1] && g[5] < g[4];
    const int run = (g[2] == 0 || saved || g[0] >= probe - 1) ? 1 : 0;
    if (run) { g[0] = 0; g[2] += 1; }
    else g[0] += 1;
    g[1] = run;
    g[3] += 1;
    if (use_handle) cudaGraphSetConditional(h, (unsigned)run);
    else *flag = run;
}

// After a gated solve: its corrections (the largest count over the modes)
// into the stage's slot for solves with or without the network.
__global__ void k_learn_after(const int* state, int K, int* g) {
    int c = 0;
    for (int k = 0; k < K; k++) {
        int v = state[2 * k + 1];
        if (v < 0) v = -v - 1;
        c = max(c, v);
    }
    if (g[1]) g[5] = c;
    else g[4] = c;
}

// Keep the candidate for a mode when it lowers the max defect by 5% or more
// (max|d0 - L e|^2 < 0.9 max|d0|^2: a zero correction, whose FP32 defect
// differs from the FP64 one by rounding only, is never kept); count the
// solves tried and the corrections kept; clear the maxima for the loop.
__global__ void k_learn_keep(unsigned long long* maxsq, unsigned* jmax, int* keep, long long* tally, const int* valid,
                             int K, int* gate_kept) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= K) return;
    int ok = 0;
    if (*valid >= 2) {
        const double d0 = __longlong_as_double((long long)maxsq[k]);
        const double d1 = (double)__uint_as_float(jmax[k]);
        ok = d1 < 0.9 * d0;
        tally[2 * k] += 1;
        tally[2 * k + 1] += ok;
        if (ok && gate_kept) atomicAdd(gate_kept, 1);
    }
    keep[2 * k] = ok;
    keep[2 * k + 1] = 0;
    maxsq[k] = 0ull;
    jmax[k] = 0u;
}

__global__ void k_hist_count(int* valid) { *valid = min(*valid + 1, 2); }

// u += e on the interior of the FP64 fine level (fc layout: x-contiguous).
__global__ void k_apply(FineDev M, cplx* fc, size_t elems64) {
    const int k = blockIdx.z;
    if (!M.state[2 * k]) return;
    const int i = 1 + blockIdx.x * 128 + threadIdx.x, j = 1 + blockIdx.y;
    if (i > M.nx - 2) return;
    const float2 e = M.e[(size_t)k * M.elems + mg::el(M.L, i, j)];
    cplx& u = fc[(size_t)k * elems64 + (size_t)i + (size_t)M.nx * j];
    u = make_double2(u.x + (double)e.x, u.y + (double)e.y);
}

// Per-mode test of the FP64 defect (max |d| over the interior, as
// get_max_value/verifica_poi, from the max |d|^2 the defect kernel folded
// into maxsq): converged modes leave the active set with the number of
// corrections applied; a non-finite defect stops the mode with
// -1 - corrections.  maxsq is cleared for the next defect.
__device__ __forceinline__ int check_mode(unsigned long long* maxsq, int* state, double* err, int k, double tol, int it,
                                          int last) {
    if (!state[2 * k]) return 0;
    double m2 = __longlong_as_double((long long)maxsq[k]);
    maxsq[k] = 0ull;
    double e = sqrt(m2);
    if (!(e <= 1.7e308)) { err[k] = __longlong_as_double(0x7ff8000000000000LL); state[2 * k] = 0; state[2 * k + 1] = -1 - it; }
    else {
        err[k] = e;
        if (e < tol) { state[2 * k] = 0; state[2 * k + 1] = it; }
        else if (last) state[2 * k + 1] = it;   // stays active: not converged
    }
    return state[2 * k];
}
__global__ void k_check_sq(unsigned long long* maxsq, int* state, double* err, int K, double tol, int it, int last) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < K) check_mode(maxsq, state, err, k, tol, it, last);
}
// The same test inside a recorded solve (one block): the correction count
// lives in *iter, and the loop's WHILE condition becomes "some mode is still
// active and fewer than max_outer corrections were applied".
constexpr int CHECK_THREADS = 256;
__global__ void __launch_bounds__(CHECK_THREADS) k_check_loop(unsigned long long* maxsq, int* state, double* err, int K,
                                                              double tol, int* iter, int first, int max_outer,
                                                              cudaGraphConditionalHandle h) {
    const int it = first ? 0 : *iter;
    int act = 0;
    for (int k = threadIdx.x; k < K; k += blockDim.x) act |= check_mode(maxsq, state, err, k, tol, it, it == max_outer);
    act = __syncthreads_or(act);
    if (threadIdx.x == 0) {
        *iter = it + 1;
        cudaGraphSetConditional(h, (act && it < max_outer) ? 1u : 0u);
    }
}

Mixed* get(tb_ctx* c) { return static_cast<Mixed*>(c->mixed); }

FineDev make(tb_ctx* c) {
    Mixed* m = get(c);
    FineDev M;
    std::memset(&M, 0, sizeof M);
    M.e = m->eb; M.r = m->r;
    M.coef = m->coef + 24 * m->ylvl[0];
    M.qdy2 = m->qdy2 + (size_t)c->g.ny * m->ylvl[0];
    M.k2b2 = c->k2b2; M.state = c->pstate;
    M.L = m->cyc.lv[0];
    M.elems = m->elems;
    M.nx = c->g.nx; M.ny = c->g.ny; M.K = c->g.K;
    M.den = (float)(1.0 / (12.0 * m->dx2[0] * c->cfg.fac_y));
    M.ify = (float)(1.0 / c->cfg.fac_y);
    M.alpha2 = (float)(c->cfg.alpha * c->cfg.alpha);
    return M;
}

template <class T>
int upl(T** d, const std::vector<T>& h) {
    if (*d) cudaFree(*d);
    *d = nullptr;
    TB_CUDA(cudaMalloc((void**)d, h.size() * sizeof(T)));
    TB_CUDA(cudaMemcpy(*d, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice));
    return TB_OK;
}

// The level operator L (defect, poisson_par.f:543-793) at interior point
// (i, j) of a level with nxl x n points, applied to u (line-contiguous), FP64.
struct HostOp {
    const double *SP, *CP, *PP, *LP, *Q2;
    double den, ify, k2b2, topc;
    int nxl, n;
    double apply(const std::vector<double>& u, int i, int j) const {
        auto f = [&](int ii, int jj) { return u[(size_t)n * ii + jj]; };
        auto bx = [&](int jj) {
            if (i == 1 || i == nxl - 2) {
                int e = (i == 1) ? 1 : -1;
                return 10.0 * f(i - e, jj) - 15.0 * f(i, jj) - 4.0 * f(i + e, jj) + 14.0 * f(i + 2 * e, jj) -
                       6.0 * f(i + 3 * e, jj) + f(i + 4 * e, jj);
            }
            return -f(i - 2, jj) + 16.0 * f(i - 1, jj) - 30.0 * f(i, jj) + 16.0 * f(i + 1, jj) - f(i + 2, jj);
        };
        double b, cc, d, q2, top = 0.0;
        if (j == 1) {
            b = SP[2] * bx(2) + SP[1] * bx(1);
            cc = SP[3] * f(i, 0) + SP[4] * f(i, 1) + SP[5] * f(i, 2) + SP[6] * f(i, 3);
            d = k2b2 * (SP[1] * f(i, 1) + SP[2] * f(i, 2));
            q2 = Q2[0];
        } else if (j <= n - 3) {
            b = CP[0] * bx(j - 1) + CP[1] * bx(j) + CP[2] * bx(j + 1);
            cc = CP[3] * f(i, j - 2) + CP[4] * f(i, j - 1) + CP[5] * f(i, j) + CP[6] * f(i, j + 1) + CP[7] * f(i, j + 2);
            d = k2b2 * (CP[0] * f(i, j - 1) + CP[1] * f(i, j) + CP[2] * f(i, j + 1));
            q2 = Q2[j - 2];
        } else if (j == n - 2) {
            b = bx(j);
            cc = PP[3] * f(i, j + 1) + PP[2] * f(i, j) + PP[1] * f(i, j - 1);
            d = k2b2 * f(i, j);
            q2 = Q2[j - 1];
        } else {
            b = bx(j);
            cc = LP[2] * f(i, j) + LP[3] * f(i, j - 1) + LP[4] * f(i, j - 2);
            d = k2b2 * f(i, j);
            q2 = Q2[j - 2];
            top = LP[1] * topc * std::sqrt(q2);
        }
        return b * den + cc * q2 + d * ify - top * f(i, j);
    }
};

// Inverse of the coarsest-level operator of one mode (N x N, row-major),
// by Gauss-Jordan elimination with partial pivoting in FP64.
bool coarse_inverse(const HostOp& op, int N, float* out) {
    const int nxl = op.nxl, n = op.n, m = n - 1;
    std::vector<double> A((size_t)N * N, 0.0), X((size_t)N * N, 0.0), u((size_t)nxl * n, 0.0);
    for (int q = 0; q < N; q++) {
        int iq = 1 + q / m, jq = 1 + q % m;
        u[(size_t)n * iq + jq] = 1.0;
        for (int i = std::max(1, iq - 4); i <= std::min(nxl - 2, iq + 4); i++)
            for (int j = std::max(1, jq - 3); j <= std::min(n - 1, jq + 3); j++)
                A[(size_t)((i - 1) * m + (j - 1)) * N + q] = op.apply(u, i, j);
        u[(size_t)n * iq + jq] = 0.0;
    }
    for (int p = 0; p < N; p++) X[(size_t)p * N + p] = 1.0;
    for (int c = 0; c < N; c++) {
        int piv = c;
        for (int p = c + 1; p < N; p++)
            if (std::fabs(A[(size_t)p * N + c]) > std::fabs(A[(size_t)piv * N + c])) piv = p;
        if (A[(size_t)piv * N + c] == 0.0) return false;
        if (piv != c)
            for (int q = 0; q < N; q++) {
                std::swap(A[(size_t)piv * N + q], A[(size_t)c * N + q]);
                std::swap(X[(size_t)piv * N + q], X[(size_t)c * N + q]);
            }
        double inv = 1.0 / A[(size_t)c * N + c];
        for (int q = 0; q < N; q++) { A[(size_t)c * N + q] *= inv; X[(size_t)c * N + q] *= inv; }
        for (int p = 0; p < N; p++) {
            if (p == c) continue;
            double f = A[(size_t)p * N + c];
            if (f == 0.0) continue;
            for (int q = 0; q < N; q++) {
                A[(size_t)p * N + q] -= f * A[(size_t)c * N + q];
                X[(size_t)p * N + q] -= f * X[(size_t)c * N + q];
            }
        }
    }
    for (size_t q = 0; q < X.size(); q++) out[q] = (float)X[q];
    return true;
}

int apply(tb_ctx* c, const FineDev& M) {
    k_apply<<<dim3(tb_blocks(c->g.nx - 2, 128), c->g.ny - 1, c->g.K), 128, 0, c->stream>>>(M, c->pfc, c->g.lvl_elems);
    TB_CHECK_LAUNCH(c);
    return TB_OK;
}

int defect(tb_ctx* c) {
    Mixed* m = get(c);
    return tb_poisson_defect_f32(c, DefectRows{m->drow, m->drow + (size_t)DEFECT_ROW * c->g.ny}, m->r, m->elems, m->cyc.lv[0].T, m->cyc.lv[0].np, m->maxsq);
}

template <int S>
int launch_strip(tb_ctx* c, const mg::Cycle& M, int l, int up, int from) {
    const mg::Level& L = M.lv[l];
    const size_t smem = mg::strip_bytes(L);
    const dim3 grid((unsigned)(up ? L.up : L.down), (unsigned)M.K);
    if (up) mg::k_up<S><<<grid, mg::NT, smem, c->stream>>>(M, l);
    else mg::k_down<S><<<grid, mg::NT, smem, c->stream>>>(M, l, from);
    TB_CHECK_LAUNCH(c);
    return TB_OK;
}
int strip(tb_ctx* c, const mg::Cycle& M, int l, int up, int from) {
    cudaEvent_t p0 = nullptr;
    int r;
    if (l == 0 && up && (r = tb_prof_begin(c, PROF_RELAX0, &p0))) return r;
    switch (M.lv[l].S) {
        case 2: r = launch_strip<2>(c, M, l, up, from); break;
        case 4: r = launch_strip<4>(c, M, l, up, from); break;
        case 5: r = launch_strip<5>(c, M, l, up, from); break;
        case 7: r = launch_strip<7>(c, M, l, up, from); break;
        case 9: r = launch_strip<9>(c, M, l, up, from); break;
        case 13: r = launch_strip<13>(c, M, l, up, from); break;
        default: r = launch_strip<17>(c, M, l, up, from); break;
    }
    if (r) return r;
    return l == 0 && up ? tb_prof_end(c, PROF_RELAX0, p0) : TB_OK;
}
// the largest dynamic shared memory any context may ask of the cycle's kernels
template <int S>
int strip_attr() {
    TB_CUDA(cudaFuncSetAttribute(mg::k_down<S>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    TB_CUDA(cudaFuncSetAttribute(mg::k_up<S>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    return TB_OK;
}
int cycle_attrs() {
    int r;
    if ((r = strip_attr<2>()) || (r = strip_attr<4>()) || (r = strip_attr<5>()) || (r = strip_attr<7>()) || (r = strip_attr<9>()) ||
        (r = strip_attr<13>()) || (r = strip_attr<17>()))
        return r;
    return TB_OK;
}

// One relaxation sweep of a tall level: border lines, then centre colours 0, 1, 2.
int tall_sweep(tb_ctx* c, const tall::Levels& T, int l) {
    const size_t smem = (size_t)(tall::THREADS / 32) * 2 * T.n * sizeof(float2);
    auto relax = [&](int first, int step, int nlines) -> int {
        const unsigned nb = tb_blocks((size_t)nlines * T.K, tall::THREADS / 32);
        switch (tall::pick_rows(T.n)) {
            case 9: tall::k_relax<9><<<nb, tall::THREADS, smem, c->stream>>>(T, l, first, step, nlines); break;
            case 11: tall::k_relax<11><<<nb, tall::THREADS, smem, c->stream>>>(T, l, first, step, nlines); break;
            case 13: tall::k_relax<13><<<nb, tall::THREADS, smem, c->stream>>>(T, l, first, step, nlines); break;
            case 15: tall::k_relax<15><<<nb, tall::THREADS, smem, c->stream>>>(T, l, first, step, nlines); break;
            default: tall::k_relax<17><<<nb, tall::THREADS, smem, c->stream>>>(T, l, first, step, nlines); break;
        }
        TB_CHECK_LAUNCH(c);
        return TB_OK;
    };
    const int nxl = T.nx[l];
    int r = relax(1, nxl - 3, 2);
    for (int first = 2; !r && first < 5 && first <= nxl - 3; first++) r = relax(first, 3, (nxl - 3 - first) / 3 + 1);
    return r;
}
// The tall levels on the way down, from e of the finest one, and on the way up.
int tall_down(tb_ctx* c, const tall::Levels& T, const mg::Cycle& M) {
    int r;
    for (int l = 0; l < T.NL; l++) {
        for (int s = 0; s < NU_PRE; s++)
            if ((r = tall_sweep(c, T, l))) return r;
        tall::k_resid<<<tb_blocks((size_t)T.nx[l] * T.n * T.K, 256), 256, 0, c->stream>>>(T, l);
        TB_CHECK_LAUNCH(c);
        if (l + 1 < T.NL) tall::k_restrict_x<<<tb_blocks((size_t)T.nx[l + 1] * T.n * T.K, 256), 256, 0, c->stream>>>(T, l);
        else {
            const mg::Level& N = M.lv[T.NL];
            tall::k_restrict_out<<<dim3(tb_blocks(N.nx - 2, 128), N.n - 1, T.K), 128, 0, c->stream>>>(T, M);
        }
        TB_CHECK_LAUNCH(c);
    }
    return TB_OK;
}
int tall_up(tb_ctx* c, const tall::Levels& T, const mg::Cycle& M) {
    cudaEvent_t p0 = nullptr;
    int r;
    for (int l = T.NL - 1; l >= 0; l--) {
        if (l == 0 && (r = tb_prof_begin(c, PROF_RELAX0, &p0))) return r;
        const unsigned nb = tb_blocks((size_t)T.nx[l] * T.n * T.K, 256);
        if (l + 1 < T.NL) tall::k_prolong_x<<<nb, 256, 0, c->stream>>>(T, l + 1);
        else tall::k_prolong_in<<<nb, 256, 0, c->stream>>>(T, M);
        TB_CHECK_LAUNCH(c);
        for (int s = 0; s < NU_POST; s++)
            if ((r = tall_sweep(c, T, l))) return r;
    }
    return tb_prof_end(c, PROF_RELAX0, p0);
}

// The V-cycles of one correction.
int vcycles(tb_ctx* c) {
    Mixed* m = get(c);
    cudaEvent_t ps = nullptr;
    int r;
    if ((r = tb_prof_begin(c, PROF_SOR, &ps))) return r;
    mg::Cycle M = m->cyc;
    M.state = c->pstate;
    tall::Levels T = m->tl;
    T.state = c->pstate;
    T.k2b2 = c->k2b2;
    const int bot = M.NL - 1;
    const dim3 tiles(tb_blocks(c->g.nx, 32), tb_blocks(c->g.ny, 32), M.K), tile(32, 8);
    if (T.NL) { tall::k_cross<false><<<tiles, tile, 0, c->stream>>>(T, M); TB_CHECK_LAUNCH(c); }
    for (int v = 0; v < INNER_VCYCLES; v++) {
        if (T.NL && (r = tall_down(c, T, M))) return r;
        for (int l = T.NL; l < bot; l++)
            if ((r = strip(c, M, l, 0, v > 0 && l == 0))) return r;
        mg::k_direct<<<dim3(tb_blocks(M.N, 4 * mg::NW), M.K), mg::NT, 0, c->stream>>>(M);
        TB_CHECK_LAUNCH(c);
        for (int l = bot - 1; l >= T.NL; l--)
            if ((r = strip(c, M, l, 1, 0))) return r;
        if (T.NL && (r = tall_up(c, T, M))) return r;
    }
    if (T.NL) { tall::k_cross<true><<<tiles, tile, 0, c->stream>>>(T, M); TB_CHECK_LAUNCH(c); }
    return tb_prof_end(c, PROF_SOR, ps);
}

// A float4 table of doubled coefficients: pair q of the row at out.
void put_pairs(float4* out, const double* v, int n) {
    for (int q = 0; q < n; q += 2) out[q / 2] = make_float4((float)v[q], (float)v[q], (float)v[q + 1], (float)v[q + 1]);
}

// Line-solve rows of one level, line type and mode (mg::Cycle::tab): per row
// the weights of the right-hand side's x-stencil sums (-qx and the sums' unit
// folded in), the forward recurrence, the chunk responses and the backward
// recurrence (1/D folded in), then the 2x2 propagators (mg::MATS per direction).
// Row 0 (Dirichlet) and the pad rows hold zeros.
void line_tables(int n, int S, double unit, double qx, const double* cf, const double* L1, const double* L2, const double* U1,
                 const double* U2, const double* ID, float4* out) {
    std::vector<double> h1(n), h2(n), k1(n), k2(n);
    double Mf[mg::NW][4], Mb[mg::NW][4];
    for (int t = 0; t < mg::NW; t++) {
        const int r0 = std::min(n, t * S), r1 = std::min(n, r0 + S);
        for (int u = 0; u < 2; u++) {
            double ym1 = (u == 0) ? 1.0 : 0.0, ym2 = (u == 0) ? 0.0 : 1.0;
            for (int j = r0; j < r1; j++) {
                const double y = j == 0 ? 0.0 : -L2[j] * ym2 - L1[j] * ym1;
                (u == 0 ? h1 : h2)[j] = y;
                ym2 = ym1; ym1 = y;
            }
            Mf[t][u] = ym1; Mf[t][2 + u] = ym2;
        }
        for (int u = 0; u < 2; u++) {
            double xp1 = (u == 0) ? 1.0 : 0.0, xp2 = (u == 0) ? 0.0 : 1.0;
            for (int j = r1 - 1; j >= r0; j--) {
                const double x = j == 0 ? 0.0 : (-U1[j] * xp1 - U2[j] * xp2) * ID[j];
                (u == 0 ? k1 : k2)[j] = x;
                xp2 = xp1; xp1 = x;
            }
            Mb[t][u] = xp1; Mb[t][2 + u] = xp2;
        }
    }
    // per direction, in the order the carry takes: the chunks' propagators, the
    // products of the chunks before each one in its group of four, the groups' products
    for (int dir = 0; dir < 2; dir++) {
        float4* prop = out + (size_t)mg::ROW4 * mg::NW * S + dir * 2 * mg::MATS;
        double acc[4] = {1, 0, 0, 1};
        for (int v = 0; v < mg::NW; v++) {
            const double* m = dir ? Mb[mg::NW - 1 - v] : Mf[v];
            if (v % 4 == 0) { acc[0] = acc[3] = 1.0; acc[1] = acc[2] = 0.0; }
            put_pairs(prop + 2 * v, m, 4);
            put_pairs(prop + 2 * (mg::NW + v), acc, 4);
            const double a0 = m[0] * acc[0] + m[1] * acc[2], a1 = m[0] * acc[1] + m[1] * acc[3];
            const double a2 = m[2] * acc[0] + m[3] * acc[2], a3 = m[2] * acc[1] + m[3] * acc[3];
            acc[0] = a0; acc[1] = a1; acc[2] = a2; acc[3] = a3;
            if (v % 4 == 3) put_pairs(prop + 2 * (2 * mg::NW + v / 4), acc, 4);
        }
    }
    for (int j = 1; j < n; j++) {
        double w[3] = {0.0, 0.0, 0.0};
        if (j == 1) { w[1] = -qx * cf[1]; w[2] = -qx * cf[2]; }
        else if (j <= n - 3) for (int q = 0; q < 3; q++) w[q] = -qx * cf[7 + q];
        else w[1] = -qx;
        const double row[12] = {unit * w[0], unit * w[1], unit * w[2], -L1[j], -L2[j], ID[j] * h1[j], ID[j] * h2[j],
                                -U1[j] * ID[j], -U2[j] * ID[j], ID[j], k1[j], k2[j]};
        put_pairs(out + (size_t)mg::ROW4 * j, row, 12);
    }
}

// Line tables of a tall level, type and mode (tall::tab_size): the band LU rows,
// the responses h1 h2 (k1 k2) of a lane's S rows to the states entering them
// forward (backward), and the Kogge-Stone matrices of the lanes' propagators.
void tall_tables(int n, int S, const double* L1, const double* L2, const double* U1, const double* U2, const double* ID, float* out) {
    using M2 = std::array<double, 4>;
    auto mul = [](const M2& A, const M2& B) {
        return M2{A[0] * B[0] + A[1] * B[2], A[0] * B[1] + A[1] * B[3], A[2] * B[0] + A[3] * B[2], A[2] * B[1] + A[3] * B[3]};
    };
    const double* lu[5] = {L1, L2, U1, U2, ID};
    for (int q = 0; q < 5; q++)
        for (int j = 0; j < n; j++) out[(size_t)q * n + j] = (float)lu[q][j];
    float *h = out + 5 * (size_t)n, *kk = h + 2 * (size_t)n, *Pf = kk + 2 * (size_t)n, *Pb = Pf + 640;
    M2 Mf[32], Mb[32];
    for (int t = 0; t < 32; t++) {
        const int r0 = std::min(n, t * S), r1 = std::min(n, r0 + S);
        for (int u = 0; u < 2; u++) {
            double p1 = u == 0, p2 = u == 1;
            for (int j = r0; j < r1; j++) {
                const double y = -L2[j] * p2 - L1[j] * p1;
                h[(size_t)u * n + j] = (float)y;
                p2 = p1; p1 = y;
            }
            Mf[t][u] = p1; Mf[t][2 + u] = p2;
            p1 = u == 0; p2 = u == 1;
            for (int j = r1 - 1; j >= r0; j--) {
                const double x = (-U1[j] * p1 - U2[j] * p2) * ID[j];
                kk[(size_t)u * n + j] = (float)x;
                p2 = p1; p1 = x;
            }
            Mb[t][u] = p1; Mb[t][2 + u] = p2;
        }
    }
    for (int d = 0, off = 1; d < 5; d++, off <<= 1) {
        M2 nf[32], nb[32];
        for (int t = 0; t < 32; t++) {
            for (int q = 0; q < 4; q++) { Pf[(d * 32 + t) * 4 + q] = (float)Mf[t][q]; Pb[(d * 32 + t) * 4 + q] = (float)Mb[t][q]; }
            nf[t] = t >= off ? mul(Mf[t], Mf[t - off]) : Mf[t];
            nb[t] = t + off < 32 ? mul(Mb[t], Mb[t + off]) : Mb[t];
        }
        std::copy(nf, nf + 32, Mf);
        std::copy(nb, nb + 32, Mb);
    }
}

// The operator's row j (1 <= j < n) of one level: weights w1 of the x-stencil sums
// (and of the k^2 term) of rows j-1 .. j+1, w2 of the values of rows j-2 .. j+2
// in the y-derivative, whose factor q2 is returned (defect, poisson_par.f:543-793).
double operator_row(int j, int n, const double* cf, const double* Q2, double* w1, double* w2) {
    const double *SP = cf, *CP = cf + 7, *PP = cf + 15, *LP = cf + 19;
    std::fill(w1, w1 + 3, 0.0);
    std::fill(w2, w2 + 5, 0.0);
    if (j == 1) {
        w1[1] = SP[1]; w1[2] = SP[2];
        for (int q = 0; q < 4; q++) w2[1 + q] = SP[3 + q];
        return Q2[0];
    }
    if (j <= n - 3) {
        for (int q = 0; q < 3; q++) w1[q] = CP[q];
        for (int q = 0; q < 5; q++) w2[q] = CP[3 + q];
        return Q2[j - 2];
    }
    w1[1] = 1.0;
    if (j == n - 2) {
        w2[3] = PP[3]; w2[2] = PP[2]; w2[1] = PP[1];
        return Q2[j - 1];
    }
    w2[2] = LP[2]; w2[1] = LP[3]; w2[0] = LP[4];
    return Q2[j - 2];
}
// The boundary term of the top row: its multiple of the value there is subtracted.
double top_term(int n, double ify, double k2b2, double alpha2, const double* cf, const double* Q2) {
    return cf[20] * std::sqrt((alpha2 - k2b2) * ify) * std::sqrt(Q2[n - 3]);
}

// The row as weights of the x-stencil sums of rows j-1 .. j+1 (w[0..2]) and of
// the values of rows j-2 .. j+2 (w[3..7]), the centre stencil's diagonal (-30)
// folded into the latter: L u = sum_q w1[q] X(j+q) + sum_q w2[q] u(j+q).
void residual_row(int j, int n, double den, double ify, double k2b2, double alpha2, const double* cf, const double* Q2,
                  double* w) {
    double *w1 = w, *w2 = w + 3;
    const double q2 = operator_row(j, n, cf, Q2, w1, w2), kk = k2b2 * ify;
    for (int q = 0; q < 5; q++) w2[q] *= q2;
    for (int q = 0; q < 3; q++) w2[1 + q] += kk * w1[q];
    if (j == n - 1) w2[2] -= top_term(n, ify, k2b2, alpha2, cf, Q2);
    for (int q = 0; q < 3; q++) {
        w1[q] *= den;
        w2[1 + q] -= 30.0 * w1[q];
    }
}

// FP32 residual rows of one level and mode, negated, the sums in units of 16.
void residual_rows(int n, double den, double ify, double k2b2, double alpha2, const double* cf, const double* Q2,
                   float4* out) {
    for (int j = 1; j < n; j++) {
        double w[8];
        residual_row(j, n, den, ify, k2b2, alpha2, cf, Q2, w);
        for (int q = 0; q < 8; q++) w[q] *= q < 3 ? -16.0 : -1.0;
        put_pairs(out + (size_t)mg::RES4 * j, w, 8);
    }
}

}  // namespace

int tb_mixed_setup(tb_ctx* c) {
    tb_mixed_free(c);
    const int K = c->g.K, ny = c->g.ny, msh = c->g.msh;
    Mixed* m = new Mixed();
    c->mixed = m;
    // hierarchy: x-only coarsening while dx < max dy (if enabled), the
    // reference's y-levels with x and y halved together, then x-only
    // coarsening down to a level small enough for the direct solve
    double dy_max = 0.0;
    for (int j = 0; j + 1 < ny; j++) dy_max = std::max(dy_max, 1.0 / c->h_qdy[j]);
    auto push = [&](int px, int py, int yl, double dx2) {
        int l = m->NL++;
        m->ptsx[l] = px; m->ptsy[l] = py; m->ylvl[l] = yl; m->dx2[l] = dx2; m->semi[l] = 0;
    };
    m->NL = 0;
    push(c->g.nx, ny, 0, c->h_dx2[0]);
    const int full_steps = msh - 1, fdiv = 1 << full_steps;
    while (TB_MG_SEMI_FIRST && m->NL < MG_MAX - msh) {
        int l = m->NL - 1, px = m->ptsx[l];
        int pxn = (px + 1) / 2;
        if (std::sqrt(m->dx2[l]) >= dy_max || (px - 1) % 2 || (pxn - 1) % fdiv || (pxn - 1) / fdiv + 1 < 10) break;
        m->semi[l] = 1;
        push(pxn, m->ptsy[l], 0, 4.0 * m->dx2[l]);
    }
    for (int yl = 1; yl <= full_steps; yl++) {
        int l = m->NL - 1;
        push((m->ptsx[l] + 1) / 2, c->g.ptsy[yl], yl, 4.0 * m->dx2[l]);
    }
    while (m->NL < MG_MAX) {
        int l = m->NL - 1, px = m->ptsx[l], py = m->ptsy[l];
        if ((long)(px - 2) * (py - 1) <= DIRECT_MAX || (px - 1) % 2 || (px + 1) / 2 < 10) break;
        m->semi[l] = 1;
        push((px + 1) / 2, py, m->ylvl[l], 4.0 * m->dx2[l]);
    }
    const int NL = m->NL, lc = NL - 1;
    if (m->ptsx[lc] < 10) {
        tb_set_error("mixed form needs at least 10 points in x on the coarsest level (got %d)", m->ptsx[lc]);
        return TB_ERR_ARG;
    }
    m->N = (m->ptsx[lc] - 2) * (m->ptsy[lc] - 1);
    if (m->N > mg::DIRECT_LIMIT) {
        tb_set_error("mixed form: coarsest level has %d unknowns per mode (limit %d); raise msh", m->N, mg::DIRECT_LIMIT);
        return TB_ERR_ARG;
    }
    mg::Cycle& cy = m->cyc;
    tall::Levels& tl = m->tl;
    std::memset(&cy, 0, sizeof cy);
    std::memset(&tl, 0, sizeof tl);
    while (m->ptsy[tl.NL] > tall::STRIP_ROWS) tl.NL++;   // at least one level has half the rows
    cy.nu_pre = NU_PRE; cy.nu_post = NU_POST;
    size_t off = 0;
    int t4 = 0;   // tables per mode
    for (int l = 0; l < NL; l++) {
        mg::Level& L = cy.lv[l];
        L.nx = m->ptsx[l]; L.n = m->ptsy[l]; L.semi = m->semi[l];
        const int Tn = L.nx / 3 + 1;   // elements of a colour plane
        L.T = (Tn + 3) & ~3;
        if (l < tl.NL) {   // of these levels only the finest has colour planes
            L.np = L.n + 2;
            if (l > 0) continue;
        } else {
            L.S = mg::pick_rows(L.n);
            L.np = mg::NW * L.S + 2;
            L.down = mg::strips(Tn, NU_PRE, 1);
            L.up = mg::strips(Tn, NU_POST, 0);
            if (l < NL - 1) { L.tab = t4; t4 += mg::level4(L); }
        }
        L.off = (int)off;
        off += (size_t)3 * L.np * L.T;
        if (off > 0x7fffffffu) { tb_set_error("mixed form: grid too large for the FP32 hierarchy"); return TB_ERR_ARG; }
    }
    cy.tab4 = t4;
    cy.elems = m->elems = off;
    cy.K = K; cy.NL = NL; cy.N = m->N;
    int r;
    if ((r = cycle_attrs())) return r;
    size_t w = (size_t)K * m->elems;
    for (float2** p : {&m->ea, &m->eb, &m->r}) {
        TB_CUDA(cudaMalloc(p, w * sizeof(float2)));
        TB_CUDA(cudaMemset(*p, 0, w * sizeof(float2)));
    }
    cy.ea = m->ea; cy.eb = m->eb; cy.r = m->r;
    if (tl.NL) {
        tl.K = K; tl.n = ny;
        tl.ify = (float)(1.0 / c->cfg.fac_y);
        tl.alpha2 = (float)(c->cfg.alpha * c->cfg.alpha);
        for (int l = 0; l < tl.NL; l++) {
            tl.nx[l] = m->ptsx[l];
            tl.qx[l] = (float)(1.0 / (12.0 * m->dx2[l] * c->cfg.fac_y));
            tl.off[l] = tl.elems;
            tl.elems += (size_t)m->ptsx[l] * ny;
        }
        const size_t te = (size_t)K * tl.elems, tr = (size_t)K * c->g.nx * ny;
        for (const auto& p : {std::make_pair(&tl.e, te), std::make_pair(&tl.r, te), std::make_pair(&tl.rr, tr)}) {
            TB_CUDA(cudaMalloc(p.first, p.second * sizeof(float2)));
            TB_CUDA(cudaMemset(*p.first, 0, p.second * sizeof(float2)));
        }
    }
    TB_CUDA(cudaMalloc(&m->maxsq, K * sizeof(unsigned long long)));
    TB_CUDA(cudaMemset(m->maxsq, 0, K * sizeof(unsigned long long)));
    TB_CUDA(cudaMalloc(&m->hvalid, 4 * sizeof(int)));
    TB_CUDA(cudaMemset(m->hvalid, 0, 4 * sizeof(int)));
    TB_CUDA(cudaMalloc(&m->iter, sizeof(int)));
    TB_CUDA(cudaMemset(m->iter, 0, sizeof(int)));
    TB_CUDA(cudaMalloc(&m->lkeep, 2 * K * sizeof(int)));
    TB_CUDA(cudaMemset(m->lkeep, 0, 2 * K * sizeof(int)));
    if (c->cfg.warm_start)
        for (auto& h : m->hist)
            for (cplx*& p : h) TB_CUDA(cudaMalloc(&p, tb_n3(c) * sizeof(cplx)));
    const double* blob = c->coefs.data();
    std::vector<double> cf64((size_t)24 * msh);
    for (int l = 0; l < msh; l++) {   // sp_poi(7,msh) cp_poi(8,msh) pp_poi(4,msh) lp_poi(5,msh) from blob[83]
        for (int q = 0; q < 7; q++) cf64[24 * l + q] = blob[83 + 7 * l + q];
        for (int q = 0; q < 8; q++) cf64[24 * l + 7 + q] = blob[83 + 7 * msh + 8 * l + q];
        for (int q = 0; q < 4; q++) cf64[24 * l + 15 + q] = blob[83 + 15 * msh + 4 * l + q];
        for (int q = 0; q < 5; q++) cf64[24 * l + 19 + q] = blob[83 + 19 * msh + 5 * l + q];
    }
    // line-solve tables per mode, line type and level (band5 factors of the
    // level's y-line matrix and chunk tables) and residual rows, in FP32
    std::vector<float4> t32((size_t)K * cy.tab4, make_float4(0.f, 0.f, 0.f, 0.f));
    std::vector<double> a, L1(ny), L2(ny), U1(ny), U2(ny), ID(ny);
    std::vector<float> ttall((size_t)2 * tl.NL * K * tall::tab_size(ny), 0.f);
    for (int type = 0; type < 2; type++)
        for (int l = 0; l < tl.NL; l++)
            for (int k = 0; k < K; k++) {
                tb_poisson_band_matrix_dx(c, type, 1, k + 1, m->dx2[l], a);
                tb_band5_factor(ny, a, L1.data(), L2.data(), U1.data(), U2.data(), ID.data());
                tall_tables(ny, tall::pick_rows(ny), L1.data(), L2.data(), U1.data(), U2.data(), ID.data(),
                            &ttall[(((size_t)type * tl.NL + l) * K + k) * tall::tab_size(ny)]);
            }
    for (int k = 0; k < K; k++)
        for (int l = tl.NL; l < NL - 1; l++) {
            const mg::Level& L = cy.lv[l];
            const double* cfl = &cf64[24 * m->ylvl[l]];
            const double qx = 1.0 / (12.0 * m->dx2[l] * c->cfg.fac_y);
            float4* T = &t32[(size_t)k * cy.tab4];
            for (int type = 0; type < 2; type++) {
                tb_poisson_band_matrix_dx(c, type, m->ylvl[l] + 1, k + 1, m->dx2[l], a);
                tb_band5_factor(L.n, a, L1.data(), L2.data(), U1.data(), U2.data(), ID.data());
                line_tables(L.n, L.S, type ? 1.0 : 16.0, qx, cfl, L1.data(), L2.data(), U1.data(), U2.data(), ID.data(),
                            T + L.tab + type * mg::line4(L));
            }
            residual_rows(L.n, qx, 1.0 / c->cfg.fac_y, c->h_k2b2[k], c->cfg.alpha * c->cfg.alpha, cfl,
                          &c->h_qdy2[(size_t)ny * m->ylvl[l]], T + L.tab + 2 * mg::line4(L));
        }
    if ((r = upl(&m->tab, t32))) return r;
    cy.tab = m->tab;
    std::vector<double> drow((size_t)DEFECT_ROW * ny + 2 * K, 0.0);
    {
        const double den = 1.0 / (12.0 * c->h_dx2[0] * c->cfg.fac_y), ify = 1.0 / c->cfg.fac_y;
        for (int j = 1; j < ny; j++) {
            double* w = &drow[(size_t)DEFECT_ROW * j];
            w[8] = -operator_row(j, ny, &cf64[0], &c->h_qdy2[0], w, w + 3);
            for (int q = 0; q < 3; q++) w[q] *= -den;
        }
        for (int k = 0; k < K; k++) {
            double* md = &drow[(size_t)DEFECT_ROW * ny + 2 * k];
            md[0] = c->h_k2b2[k] * ify / den;
            md[1] = top_term(ny, ify, c->h_k2b2[k], c->cfg.alpha * c->cfg.alpha, &cf64[0], &c->h_qdy2[0]);
        }
    }
    if ((r = upl(&m->drow, drow))) return r;
    std::vector<float> cf(cf64.begin(), cf64.end());
    if ((r = upl(&m->coef, cf))) return r;
    std::vector<float> q2(c->h_qdy2.begin(), c->h_qdy2.end());
    if ((r = upl(&m->qdy2, q2))) return r;
    if (tl.NL) {
        float* t = nullptr;
        r = upl(&t, ttall);
        tl.tab = t;
        if (r) return r;
        tl.coef = m->coef;
        tl.qdy2 = m->qdy2;
    }
    // exact inverse of the coarsest operator per mode (modes in parallel)
    const int N = m->N;
    std::vector<float> ainv((size_t)K * N * N);
    std::vector<int> ok(K, 0);
    auto work = [&](int k0, int k1) {
        for (int k = k0; k < k1; k++) {
            HostOp op;
            const double* base = &cf64[24 * m->ylvl[lc]];
            op.SP = base; op.CP = base + 7; op.PP = base + 15; op.LP = base + 19;
            op.Q2 = &c->h_qdy2[(size_t)ny * m->ylvl[lc]];
            op.den = 1.0 / (12.0 * m->dx2[lc] * c->cfg.fac_y);
            op.ify = 1.0 / c->cfg.fac_y;
            op.k2b2 = c->h_k2b2[k];
            op.topc = std::sqrt((c->cfg.alpha * c->cfg.alpha - op.k2b2) / c->cfg.fac_y);
            op.nxl = m->ptsx[lc]; op.n = m->ptsy[lc];
            ok[k] = coarse_inverse(op, N, &ainv[(size_t)k * N * N]);
        }
    };
    int nt = (int)std::min<unsigned>(std::max(1u, std::thread::hardware_concurrency()), (unsigned)K);
    std::vector<std::thread> th;
    for (int t = 0; t < nt; t++) th.emplace_back(work, K * t / nt, K * (t + 1) / nt);
    for (auto& t : th) t.join();
    for (int k = 0; k < K; k++)
        if (!ok[k]) { tb_set_error("mixed form: coarsest operator of mode %d is singular", k); return TB_ERR_ARG; }
    if ((r = upl(&m->ainv, ainv))) return r;
    cy.ainv = m->ainv;
    return TB_OK;
}

void tb_mixed_invalidate(tb_ctx* c) {
    Mixed* m = get(c);
    if (!m) return;
    for (int& t : m->last_t) t = -9;
    for (int& v : m->hv_host) v = 0;
}

int tb_mixed_graph_pre(tb_ctx* c, int t, cudaStream_t s) {
    Mixed* m = get(c);
    if (!m) { tb_set_error("mixed form not set up"); return TB_ERR_STATE; }
    for (int q = 0; q < 4; q++)
        if (m->last_t[q] != t - 1) TB_CUDA(cudaMemsetAsync(m->hvalid + q, 0, sizeof(int), s));
    return TB_OK;
}

void tb_mixed_graph_post(tb_ctx* c, int t) {
    Mixed* m = get(c);
    if (!m || !c->cfg.warm_start) return;
    for (int q = 0; q < 4; q++) {
        m->hv_host[q] = m->last_t[q] == t - 1 ? std::min(m->hv_host[q] + 1, 2) : 1;
        m->last_t[q] = t;
    }
}

void tb_mixed_free(tb_ctx* c) {
    Mixed* m = get(c);
    if (!m) return;
    for (auto& h : m->hist)
        for (cplx* p : h)
            if (p) cudaFree(p);
    for (void* p : {(void*)m->ea, (void*)m->eb, (void*)m->r, (void*)m->tab, (void*)m->drow, (void*)m->coef, (void*)m->qdy2, (void*)m->ainv,
                    (void*)m->maxsq, (void*)m->hvalid, (void*)m->iter, (void*)m->lkeep, (void*)m->tl.e, (void*)m->tl.r,
                    (void*)m->tl.rr, (void*)m->tl.tab})
        if (p) cudaFree(p);
    delete m;
    c->mixed = nullptr;
}

// One FP64 correction recorded as the body of the solve's WHILE node:
// INNER_VCYCLES V-cycles of the FP32 hierarchy, u += e, the new defect and
// its test (which sets the loop condition).
static int record_body(tb_ctx* c, const FineDev& M, double erro, cudaGraphConditionalHandle h) {
    Mixed* m = get(c);
    int r;
    if ((r = vcycles(c))) return r;
    if ((r = apply(c, M))) return r;
    if ((r = defect(c))) return r;
    k_check_loop<<<1, CHECK_THREADS, 0, c->stream>>>(m->maxsq, c->pstate, c->perr, c->g.K, erro, m->iter, 0,
                                                     c->cfg.max_vcycles, h);
    TB_CHECK_LAUNCH(c);
    return TB_OK;
}

// The correction loop of a solve being recorded into a step graph: first
// defect and test, then a conditional WHILE node that repeats the body
// above until every mode has converged or max_vcycles corrections ran.
static int record_loop(tb_ctx* c, const FineDev& M, double erro) {
    Mixed* m = get(c);
    cudaStreamCaptureStatus st;
    cudaGraph_t g = nullptr;
    TB_CUDA(cudaStreamGetCaptureInfo(c->stream, &st, nullptr, &g, nullptr, nullptr, nullptr));
    if (st != cudaStreamCaptureStatusActive || !g) { tb_set_error("step graph: stream is not recording"); return TB_ERR_STATE; }
    cudaGraphConditionalHandle h;
    TB_CUDA(cudaGraphConditionalHandleCreate(&h, g, 0, 0));
    int r;
    if ((r = defect(c))) return r;
    k_check_loop<<<1, CHECK_THREADS, 0, c->stream>>>(m->maxsq, c->pstate, c->perr, c->g.K, erro, m->iter, 1,
                                                     c->cfg.max_vcycles, h);
    TB_CHECK_LAUNCH(c);
    const cudaGraphNode_t* deps = nullptr;
    size_t nd = 0;
    TB_CUDA(cudaStreamGetCaptureInfo(c->stream, &st, nullptr, &g, &deps, nullptr, &nd));
    cudaGraphNodeParams p = {};
    std::memset(&p, 0, sizeof p);
    p.type = cudaGraphNodeTypeConditional;
    p.conditional.handle = h;
    p.conditional.type = cudaGraphCondTypeWhile;
    p.conditional.size = 1;
    cudaGraphNode_t node;
    TB_CUDA(cudaGraphAddNode(&node, g, deps, nullptr, nd, &p));
    TB_CUDA(cudaStreamUpdateCaptureDependencies(c->stream, &node, nullptr, 1, cudaStreamSetCaptureDependencies));
    cudaGraph_t body = p.conditional.phGraph_out[0];
    cudaStream_t outer = c->stream;
    c->stream = c->body_stream;
    const long long l0 = c->launches;
    cudaError_t e = cudaStreamBeginCaptureToGraph(c->stream, body, nullptr, nullptr, 0, cudaStreamCaptureModeRelaxed);
    if (e != cudaSuccess) {
        c->stream = outer;
        tb_set_error("step graph: recording the solve loop: %s", cudaGetErrorString(e));
        return TB_ERR_CUDA;
    }
    r = record_body(c, M, erro, h);
    cudaGraph_t got = nullptr;
    e = cudaStreamEndCapture(c->stream, &got);
    c->stream = outer;
    if (r) return r;
    if (e != cudaSuccess) { tb_set_error("step graph: recording the solve loop: %s", cudaGetErrorString(e)); return TB_ERR_CUDA; }
    if (c->g_stage >= 1 && c->g_stage <= 4) c->g_body[c->g_stage - 1] = c->launches - l0;
    return TB_OK;
}

// 1 / |diagonal| of the fine y-line operator per mode and row, and the share
// of k^2 beta^2 in it (rows j >= 1; the wall row is Dirichlet: 0).
int tb_mixed_line_diag(tb_ctx* c, std::vector<float>& invD, std::vector<float>& mfeat) {
    const int K = c->g.K, ny = c->g.ny;
    invD.assign((size_t)K * ny, 0.f);
    mfeat.assign((size_t)K * ny, 0.f);
    std::vector<double> a, a0;
    tb_poisson_band_matrix_dx(c, 0, 1, 1, c->h_dx2[0], a0);
    for (int k = 0; k < K; k++) {
        tb_poisson_band_matrix_dx(c, 0, 1, k + 1, c->h_dx2[0], a);
        const int n = (int)(a.size() / 5);
        if (n != ny) { tb_set_error("line operator has %d rows, expected %d", n, ny); return TB_ERR_STATE; }
        for (int j = 1; j < ny; j++) {
            const double d = a[(size_t)j + (size_t)n * 2], d0 = a0[(size_t)j + (size_t)n * 2];
            if (d != 0.0) {
                invD[(size_t)k * ny + j] = (float)(1.0 / std::fabs(d));
                mfeat[(size_t)k * ny + j] = (float)(std::fabs(d - d0) / std::fabs(d));
            }
        }
    }
    return TB_OK;
}

// The learned first correction of stage ws's solve, before the loop: the
// FP64 defect d0 of the extrapolated guess, the network's inputs (which also
// shift the stage's history), then (when applying the network) its candidate
// correction, kept per mode where max|d0 - L e| < max|d0|.  While sampling,
// the guess is kept for the training targets.
static int learned_first(tb_ctx* c, const FineDev& M, int ws, LearnSolve* L) {
    Mixed* m = get(c);
    const int K = c->g.K, nx = c->g.nx, ny = c->g.ny;
    int r;
    if ((r = defect(c))) return r;
    TB_CUDA(cudaMemsetAsync(L->scl, 0, 3 * K * sizeof(float), c->stream));
    const int* valid = m->hvalid + ws;
    cplx *h0 = m->hist[ws][0], *h1 = m->hist[ws][1];
    const unsigned nb = std::min<unsigned>(tb_blocks((size_t)nx * ny, 256), 64);
    k_learn_scale<<<dim3(nb, K), 256, 0, c->stream>>>(M, h0, h1, valid, reinterpret_cast<unsigned*>(L->scl), L->invD, nx);
    TB_CHECK_LAUNCH(c);
    k_learn_prep<<<dim3(tb_blocks(nx, 32), tb_blocks(ny, 32), K), dim3(32, 8), 0, c->stream>>>(M, h0, h1, valid, L->scl,
                                                                                             L->invD, L->mfeat, L->X, nx);
    TB_CHECK_LAUNCH(c);
    if (L->sample) {
        const size_t pitch = c->g.lvl_elems * sizeof(cplx);
        TB_CUDA(cudaMemcpy2DAsync(L->g0, pitch, c->pfc, pitch, (size_t)nx * ny * sizeof(cplx), K, cudaMemcpyDeviceToDevice,
                                  c->stream));
    }
    if (!L->infer) {
        TB_CUDA(cudaMemsetAsync(m->maxsq, 0, K * sizeof(unsigned long long), c->stream));
        return TB_OK;
    }
    int* gk = nullptr;
    // the network, its judge and the kept corrections; when it does not run,
    // maxsq keeps the guess's defect, which the loop's first defect recomputes
    auto network = [&]() -> int {
        int rr;
        if ((rr = tb_learn_run_net(c))) return rr;
        const size_t per = (size_t)(nx - 2) * (ny - 1);
        k_learn_emit<<<tb_blocks(per * K, 256), 256, 0, c->stream>>>(M, L->out, L->scl, valid, nx);
        TB_CHECK_LAUNCH(c);
        const unsigned nj = std::min<unsigned>(tb_blocks(per, 256), 64);
        k_learn_judge<<<dim3(nj, K), 256, 0, c->stream>>>(M, L->jmax, valid, nx);
        TB_CHECK_LAUNCH(c);
        k_learn_keep<<<tb_blocks(K, 64), 64, 0, c->stream>>>(m->maxsq, L->jmax, m->lkeep, L->tally, valid, K, gk);
        TB_CHECK_LAUNCH(c);
        FineDev Mk = M;
        Mk.state = m->lkeep;
        return apply(c, Mk);
    };
    if (!L->gated) return network();
    if (!c->capturing) {
        k_learn_gate<<<1, 1, 0, c->stream>>>(L->gate + 8 * ws, L->probe, 0, 0, L->gate + 32);
        TB_CHECK_LAUNCH(c);
        int run = 0;
        TB_CUDA(cudaMemcpyAsync(&run, L->gate + 32, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
        TB_CUDA(cudaStreamSynchronize(c->stream));
        return run ? network() : TB_OK;
    }
    // recorded step: the network's kernels become the body of a conditional
    // IF node whose condition the gate kernel sets at every replay
    cudaStreamCaptureStatus st;
    cudaGraph_t g = nullptr;
    TB_CUDA(cudaStreamGetCaptureInfo(c->stream, &st, nullptr, &g, nullptr, nullptr, nullptr));
    if (st != cudaStreamCaptureStatusActive || !g) { tb_set_error("step graph: stream is not recording"); return TB_ERR_STATE; }
    cudaGraphConditionalHandle h;
    TB_CUDA(cudaGraphConditionalHandleCreate(&h, g, 0, 0));
    k_learn_gate<<<1, 1, 0, c->stream>>>(L->gate + 8 * ws, L->probe, h, 1, nullptr);
    TB_CHECK_LAUNCH(c);
    const cudaGraphNode_t* deps = nullptr;
    size_t nd = 0;
    TB_CUDA(cudaStreamGetCaptureInfo(c->stream, &st, nullptr, &g, &deps, nullptr, &nd));
    cudaGraphNodeParams p = {};
    std::memset(&p, 0, sizeof p);
    p.type = cudaGraphNodeTypeConditional;
    p.conditional.handle = h;
    p.conditional.type = cudaGraphCondTypeIf;
    p.conditional.size = 1;
    cudaGraphNode_t node;
    TB_CUDA(cudaGraphAddNode(&node, g, deps, nullptr, nd, &p));
    TB_CUDA(cudaStreamUpdateCaptureDependencies(c->stream, &node, nullptr, 1, cudaStreamSetCaptureDependencies));
    cudaGraph_t body = p.conditional.phGraph_out[0];
    cudaStream_t outer = c->stream;
    c->stream = c->body_stream;
    cudaError_t e = cudaStreamBeginCaptureToGraph(c->stream, body, nullptr, nullptr, 0, cudaStreamCaptureModeRelaxed);
    if (e != cudaSuccess) {
        c->stream = outer;
        tb_set_error("step graph: recording the learned correction: %s", cudaGetErrorString(e));
        return TB_ERR_CUDA;
    }
    const long long l0 = c->launches;
    r = network();
    if (c->g_stage >= 1 && c->g_stage <= 4) c->g_learn[c->g_stage - 1] = c->launches - l0;
    cudaGraph_t got = nullptr;
    e = cudaStreamEndCapture(c->stream, &got);
    c->stream = outer;
    if (r) return r;
    if (e != cudaSuccess) { tb_set_error("step graph: recording the learned correction: %s", cudaGetErrorString(e)); return TB_ERR_CUDA; }
    return TB_OK;
}

int tb_mixed_fine_op(tb_ctx* c, FineOp* op) {
    Mixed* m = get(c);
    if (!m) { tb_set_error("mixed form not set up"); return TB_ERR_STATE; }
    FineDev M = make(c);
    op->coef = M.coef;
    op->qdy2 = M.qdy2;
    op->k2b2 = M.k2b2;
    op->den = M.den;
    op->ify = M.ify;
    op->alpha2 = M.alpha2;
    op->nx = m->ptsx[0];
    op->ny = M.ny;
    op->K = M.K;
    return TB_OK;
}

// -L e on the finest level of mode k alone (r = 0), through fine_resid.
int tb_mixed_resid_mode(tb_ctx* c, int k, const float* e, float* out) {
    Mixed* m = get(c);
    if (!m) { tb_set_error("mixed form not set up"); return TB_ERR_STATE; }
    const int K = c->g.K, nx = c->g.nx, ny = c->g.ny;
    if (k < 0 || k >= K) { tb_set_error("mode out of range"); return TB_ERR_ARG; }
    FineDev M = make(c);
    const size_t img = (size_t)nx * ny, lvl = (size_t)3 * M.L.np * M.L.T;
    std::vector<float2> h(lvl, make_float2(0.f, 0.f)), o(img, make_float2(0.f, 0.f));
    for (int i = 0; i < nx; i++)
        for (int j = 0; j < ny; j++) h[mg::el(M.L, i, j)] = make_float2(e[(size_t)ny * i + j], 0.f);
    float2* d = nullptr;
    TB_CUDA(cudaStreamSynchronize(c->stream));
    TB_CUDA(cudaMalloc(&d, img * sizeof(float2)));
    auto run = [&]() -> int {
        TB_CUDA(cudaMemcpy(m->eb + (size_t)k * m->elems, h.data(), lvl * sizeof(float2), cudaMemcpyHostToDevice));
        TB_CUDA(cudaMemset(m->r + (size_t)k * m->elems, 0, lvl * sizeof(float2)));
        TB_CUDA(cudaMemset(d, 0, img * sizeof(float2)));
        const size_t per = (size_t)(nx - 2) * (ny - 1);
        k_fine_resid<<<tb_blocks(per, 256), 256, 0, c->stream>>>(M, k, d);
        TB_CHECK_LAUNCH(c);
        TB_CUDA(cudaMemcpyAsync(o.data(), d, img * sizeof(float2), cudaMemcpyDeviceToHost, c->stream));
        TB_CUDA(cudaStreamSynchronize(c->stream));
        TB_CUDA(cudaMemset(m->eb + (size_t)k * m->elems, 0, lvl * sizeof(float2)));
        return TB_OK;
    };
    const int r = run();
    cudaFree(d);
    if (r) return r;
    for (size_t q = 0; q < img; q++) out[q] = o[q].x;
    return TB_OK;
}

// One solve's per-mode state (hs: active flag and corrections, per mode)
// and final defect (he) into the statistics.
int tb_mixed_absorb_stats(tb_ctx* c, const int* hs, const double* he) {
    const int K = c->g.K;
    c->stats.noconv = 0;
    int nonfinite = 0;
    for (int k = 0; k < K && k < 256; k++) {
        int vc = hs[2 * k + 1];
        if (hs[2 * k]) c->stats.noconv++;
        if (vc < 0) { nonfinite = 1; vc = -vc - 1; }
        c->stats.vcycles[k] = vc;
        c->stats.residual[k] = he[k];
        c->stats.total_vcycles += vc;
    }
    c->stats.solves++;
    if (nonfinite) { tb_set_error("poi_uy (mixed form): non-finite defect"); return TB_ERR_NONFINITE; }
    return TB_OK;
}

// poi_uy (poisson_par.f:6-64), mixed form: at most max_vcycles FP64
// corrections per solve; stats.vcycles[k] counts the corrections applied to
// mode k.
int tb_poi_uy_mixed(tb_ctx* c, const cplx* dwzdx, double erro) {
    if (!c->mixed) { tb_set_error("mixed form not set up"); return TB_ERR_STATE; }
    const int K = c->g.K, nx = c->g.nx, ny = c->g.ny, max_outer = c->cfg.max_vcycles;
    FineDev M = make(c);
    Mixed* mx = get(c);
    int r;
    cudaEvent_t pall = nullptr;
    if ((r = tb_prof_begin(c, PROF_POISSON, &pall))) return r;
    if ((r = tb_poisson_begin(c, dwzdx))) return r;
    const int ws = (c->cfg.warm_start && c->ws_stage >= 1 && c->ws_stage <= 4) ? c->ws_stage - 1 : -1;
    LearnSolve* L = ws >= 0 ? tb_learn_solve(c) : nullptr;
    int hv = 0;   // usable history entries, known to the host in host-launched solves
    if (ws >= 0) {
        // a recorded step checks the continuity of its steps before each replay
        if (!c->capturing && mx->last_t[ws] != c->ws_t - 1) {
            TB_CUDA(cudaMemsetAsync(mx->hvalid + ws, 0, sizeof(int), c->stream));
            mx->hv_host[ws] = 0;
        }
        hv = mx->hv_host[ws];
        if (c->cfg.warm_start == 2) {
            const int p = (ws + 3) % 4;
            k_extrap_inc<<<tb_blocks(tb_n3(c), 256), 256, 0, c->stream>>>(
                c->pfc, c->g.lvl_elems, mx->hist[ws][0], mx->hist[ws][1], mx->hist[p][1], mx->hvalid + ws,
                mx->hvalid + p, nx, ny, K, L ? 0 : 1);
        } else {
            k_extrap<<<tb_blocks(tb_n3(c), 256), 256, 0, c->stream>>>(c->pfc, c->g.lvl_elems, mx->hist[ws][0],
                                                                      mx->hist[ws][1], mx->hvalid + ws, nx, ny, K,
                                                                      L ? 0 : 1);
        }
        TB_CHECK_LAUNCH(c);
        if (L && (r = learned_first(c, M, ws, L))) return r;
    }
    if (c->capturing) {
        if ((r = record_loop(c, M, erro))) return r;
    } else {
        std::vector<int> hs(2 * K);
        for (int it = 0; it <= max_outer; it++) {
            Mixed* m = get(c);
            if ((r = defect(c))) return r;
            k_check_sq<<<tb_blocks(K, 64), 64, 0, c->stream>>>(m->maxsq, c->pstate, c->perr, K, erro, it, it == max_outer);
            TB_CHECK_LAUNCH(c);
            if (it == max_outer) break;
            TB_CUDA(cudaMemcpyAsync(hs.data(), c->pstate, 2 * K * sizeof(int), cudaMemcpyDeviceToHost, c->stream));
            TB_CUDA(cudaStreamSynchronize(c->stream));
            bool any = false;
            for (int k = 0; k < K; k++) any = any || hs[2 * k];
            if (!any) break;
            if ((r = vcycles(c))) return r;
            if ((r = apply(c, M))) return r;
        }
    }
    if (L && L->infer && L->gated) {
        k_learn_after<<<1, 1, 0, c->stream>>>(c->pstate, K, L->gate + 8 * ws);
        TB_CHECK_LAUNCH(c);
    }
    if (L && L->sample && !c->capturing && hv >= 2 && (r = tb_learn_collect(c))) return r;
    if ((r = tb_poisson_end(c))) return r;
    if (ws >= 0) {   // this solve becomes the newest entry of the stage's history
        TB_CUDA(cudaMemcpyAsync(mx->hist[ws][0], c->uy, tb_n3(c) * sizeof(cplx), cudaMemcpyDeviceToDevice, c->stream));
        k_hist_count<<<1, 1, 0, c->stream>>>(mx->hvalid + ws);
        TB_CHECK_LAUNCH(c);
        if (!c->capturing) {
            mx->last_t[ws] = c->ws_t;
            mx->hv_host[ws] = std::min(hv + 1, 2);
        }
    }
    if ((r = tb_prof_end(c, PROF_POISSON, pall))) return r;
    if (c->capturing) {   // the step's statistics are read after each replay
        const int s = c->g_stage - 1;
        if (s < 0 || s > 3) { tb_set_error("step graph: solve outside a stage"); return TB_ERR_STATE; }
        TB_CUDA(cudaMemcpyAsync(c->gsnap + (size_t)2 * K * s, c->pstate, 2 * K * sizeof(int), cudaMemcpyDeviceToDevice,
                                c->stream));
        TB_CUDA(cudaMemcpyAsync(c->gerr + (size_t)K * s, c->perr, K * sizeof(double), cudaMemcpyDeviceToDevice, c->stream));
        return TB_OK;
    }
    std::vector<int> hs(2 * K);
    std::vector<double> he(K);
    TB_CUDA(cudaMemcpyAsync(hs.data(), c->pstate, 2 * K * sizeof(int), cudaMemcpyDeviceToHost, c->stream));
    TB_CUDA(cudaMemcpyAsync(he.data(), c->perr, K * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
    TB_CUDA(cudaStreamSynchronize(c->stream));
    return tb_mixed_absorb_stats(c, hs.data(), he.data());
}
