// tb_poisson.cu -- the pieces of poi_uy (poisson_par.f:6-164) that the mixed
// form shares: the source and start state (function_source) in the complex
// x-contiguous work arrays, the fine-level FP64 defect of the correction
// equation and the write-back of fc into uy.  The plain FP64 form's V-cycle is in tb_plain.cu.
#include "tb_internal.h"
#include <cmath>
#include <cstring>
#include <algorithm>



namespace {

struct PoiDev {
    cplx *fc, *sc;         // blocks of elems per mode, x-contiguous
    const double* coef;    // sp(7) cp(8) pp(4) lp(5) of the fine level
    const int* state;      // per mode: [2k] active, [2k+1] corrections done
    int nx, ny, K;
    size_t elems;
    double fac_y, alpha;
};

__device__ __forceinline__ cplx& AT(cplx* base, const PoiDev& P, int k, int i, int j) {
    return base[(size_t)k * P.elems + (size_t)i + (size_t)P.nx * j];
}

// ---------------------------------------------------------------------------
// function_source (poisson_par.f:111-164) for all modes.
__global__ void k_source(PoiDev P, const cplx* wx, const cplx* dwzdx, const cplx* uy, const double* duexmdx,
                         const double* uyb, double beta, double dy, double stf_pow, int form) {
    size_t n = (size_t)P.nx * P.ny * P.K;
    size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (q >= n) return;
    int i = (int)(q % P.nx), j = (int)((q / P.nx) % P.ny), k = (int)(q / ((size_t)P.nx * P.ny));
    const double* c0 = P.coef;  // level 1
    double kb = (double)k * beta;
    int J = P.ny;
    auto S = [&](int jj) {
        size_t o = (size_t)i + (size_t)P.nx * (jj + (size_t)J * k);
        cplx w = wx[o], d = dwzdx[o];
        return make_double2(kb * w.y - d.x, -kb * w.x - d.y);
    };
    cplx s;
    if (j == 0) s = make_double2(0, 0);
    else if (j == 1) { cplx a = S(1), b = S(2); s = make_double2(c0[1] * a.x + c0[2] * b.x, c0[1] * a.y + c0[2] * b.y); }
    else if (j <= J - 3) {
        cplx a = S(j - 1), b = S(j), d = S(j + 1);
        s = make_double2(c0[7] * a.x + c0[8] * b.x + c0[9] * d.x, c0[7] * a.y + c0[8] * b.y + c0[9] * d.y);
    } else if (j == J - 2) s = S(J - 2);
    else {
        s = make_double2(0, 0);
        if ((form == 0 || form == 4) && k == 0) {
            double dya = dy * stf_pow;
            size_t o = (size_t)i + (size_t)P.nx * (J - 1);
            double lp1 = c0[19], lp2 = c0[20];
            s = make_double2(-(lp1 * dwzdx[o].x) + lp2 * duexmdx[i] / dya - lp2 * P.alpha * uyb[o] / dya / sqrt(P.fac_y),
                             -(lp1 * dwzdx[o].y));
        }
    }
    AT(P.sc, P, k, i, j) = s;
    AT(P.fc, P, k, i, j) = uy[q];
}

// ---------------------------------------------------------------------------
// Fine-level FP64 defect d = sc - L fc for the mixed form (the operator of
// defect, poisson_par.f:543-793): stored as FP32 in the right-hand side r32 of
// the correction equation (line i = 3t + c - 1, row j of mode k at
// k*elems32 + (c*np + j + 1)*T + t, tb_cycle.cuh), and max |d|^2 of each mode
// folded into maxsq[k] (bit pattern of a non-negative double; a non-finite
// defect records +inf).
//
// An FP64 warp instruction holds its pipe for 64 cycles, so their number is
// what the kernel costs.  A thread marches down a column with the values and
// the x-stencil sums of its rows in registers, so a sum is formed once, and the k^2
// term rides on the sums as one more centre term: 28 FP64 instructions a complex
// point (46 with the operator's terms formed one by one).  This defect stops the
// solve, so its rounding must stay that of those terms: the sums cancel
// before they meet 1/(12 dx^2), the y-derivative before it meets 1/dy^2.  With all
// constants and the diagonal folded into row weights it takes 24, but leaves 2.5 to
// 5 times the error (rms against 80-bit sums, 65 to 257 rows); this order has that of the
// terms one by one.
// Rows per thread, with two more stencil sums a chunk: 16 and 24 rows leave small grids
// idle (257 x 97 x 8: 37 and 52 us, 31 with 8 rows) and gain nothing on large ones
// (1025 x 193 x 32: 425, 430 and 428 us).
constexpr int DEF_ROWS = 8;
__global__ void __launch_bounds__(128) k_defect_f32(PoiDev P, DefectRows D, float2* r32, size_t elems32, int T,
                                                    int np, unsigned long long* maxsq) {
    __shared__ unsigned long long wmax[4];
    const int k = blockIdx.z;
    if (!P.state[2 * k]) return;   // uniform over the block
    const int nx = P.nx, ny = P.ny;
    const int i = 1 + blockIdx.x * 128 + threadIdx.x;
    const int j0 = 1 + blockIdx.y * DEF_ROWS, j1 = min(ny, j0 + DEF_ROWS);
    unsigned long long m = 0;
    if (i <= nx - 2) {
        const cplx* F = P.fc + (size_t)k * P.elems + i;
        const cplx* SC = P.sc + (size_t)k * P.elems + i;
        const double kd = D.modes[2 * k], top = D.modes[2 * k + 1];
        const int iq = i + 1;
        float2* out = r32 + (size_t)k * elems32 + ((size_t)(iq % 3) * np + 1) * T + iq / 3;   // row 0 of this line
        const bool border = i == 1 || i == nx - 2;
        const int e = (i == 1) ? 1 : -1;
        const cplx z = make_double2(0.0, 0.0);
        auto val = [&](int j) -> cplx { return (j >= 0 && j < ny) ? F[(size_t)nx * j] : z; };
        // x-stencil sum of row j (rhs_center, rhs_border; one-sided on a border line) and its k^2 term
        auto sum = [&](int j, cplx f) -> cplx {
            if (j < 1 || j >= ny) return z;   // weight 0
            const cplx* R = F + (size_t)nx * j;
            cplx s;
            if (border) {
                const cplx a = R[-e], b = R[e], c = R[2 * e], d = R[3 * e], g = R[4 * e];
                s = make_double2(fma(-6.0, d.x, fma(14.0, c.x, fma(-4.0, b.x, fma(-15.0, f.x, 10.0 * a.x)))) + g.x,
                                 fma(-6.0, d.y, fma(14.0, c.y, fma(-4.0, b.y, fma(-15.0, f.y, 10.0 * a.y)))) + g.y);
            } else {
                const cplx a = R[-2], b = R[-1], c = R[1], d = R[2];
                s = make_double2(fma(16.0, c.x, fma(-30.0, f.x, fma(16.0, b.x, -a.x))) - d.x,
                                 fma(16.0, c.y, fma(-30.0, f.y, fma(16.0, b.y, -a.y))) - d.y);
            }
            return make_double2(fma(kd, f.x, s.x), fma(kd, f.y, s.y));
        };
        cplx f0 = val(j0 - 2), f1 = val(j0 - 1), f2 = val(j0), f3 = val(j0 + 1);
        cplx x0 = sum(j0 - 1, f1), x1 = sum(j0, f2);
        const unsigned long long largest = (unsigned long long)__double_as_longlong(1.7e308);
#pragma unroll 2
        for (int j = j0; j < j1; j++) {
            const cplx f4 = val(j + 2), x2 = sum(j + 1, f3);
            const double* w = D.rows + DEFECT_ROW * j;
            const cplx t[5] = {f0, f1, f2, f3, f4}, X[3] = {x0, x1, x2};
            cplx cc = make_double2(w[3] * f0.x, w[3] * f0.y);
#pragma unroll
            for (int q = 1; q < 5; q++) cc = make_double2(fma(w[3 + q], t[q].x, cc.x), fma(w[3 + q], t[q].y, cc.y));
            cplx v = SC[(size_t)nx * j];
            v = make_double2(fma(w[8], cc.x, v.x), fma(w[8], cc.y, v.y));
#pragma unroll
            for (int q = 0; q < 3; q++) v = make_double2(fma(w[q], X[q].x, v.x), fma(w[q], X[q].y, v.y));
            if (j == ny - 1) v = make_double2(fma(top, f2.x, v.x), fma(top, f2.y, v.y));
            const unsigned long long a = (unsigned long long)__double_as_longlong(fma(v.x, v.x, v.y * v.y));
            m = max(m, a > largest ? 0x7ff0000000000000ull : a);
            out[(size_t)j * T] = make_float2((float)v.x, (float)v.y);
            f0 = f1; f1 = f2; f2 = f3; f3 = f4;
            x0 = x1; x1 = x2;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) wmax[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) atomicMax(&maxsq[k], max(max(wmax[0], wmax[1]), max(wmax[2], wmax[3])));
}

// uy(i,j,k) = fc(i,j,1) for j >= 2, 2 <= i <= ptsx-1 (poisson_par.f:53-57).
__global__ void k_write_uy(PoiDev P, cplx* uy) {
    size_t n = (size_t)P.nx * P.ny * P.K;
    size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (q >= n) return;
    int i = (int)(q % P.nx), j = (int)((q / P.nx) % P.ny), k = (int)(q / ((size_t)P.nx * P.ny));
    if (j < 1 || i < 1 || i > P.nx - 2) return;
    uy[q] = AT(P.fc, P, k, i, j);
}

__global__ void k_activate(int* state, int K) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < K) { state[2 * k] = 1; state[2 * k + 1] = 0; }
}

PoiDev make_dev(tb_ctx* c) {
    PoiDev P;
    std::memset(&P, 0, sizeof P);
    P.fc = c->pfc; P.sc = c->psc; P.coef = c->pcoef; P.state = c->pstate;
    P.nx = c->g.nx; P.ny = c->g.ny; P.K = c->g.K;
    P.elems = c->g.lvl_elems;
    P.fac_y = c->cfg.fac_y; P.alpha = c->cfg.alpha;
    return P;
}

}  // namespace

int tb_poisson_setup(tb_ctx* c) {
    const int K = c->g.K;
    const size_t w = (size_t)K * c->g.lvl_elems;
    for (cplx** p : {&c->pfc, &c->psc}) {
        if (*p) cudaFree(*p);
        TB_CUDA(cudaMalloc(p, w * sizeof(cplx)));
        TB_CUDA(cudaMemset(*p, 0, w * sizeof(cplx)));
    }
    if (!c->pstate) TB_CUDA(cudaMalloc(&c->pstate, 2 * K * sizeof(int)));
    if (!c->perr) TB_CUDA(cudaMalloc(&c->perr, K * sizeof(double)));
    return TB_OK;
}

// Pieces of poi_uy shared with the mixed form: the source and the start
// state (fc = uy, every mode active) and the write-back of fc into uy.
int tb_poisson_begin(tb_ctx* c, const cplx* dwzdx) {
    PoiDev P = make_dev(c);
    double stf_pow = tb_powi(c->cfg.stf, c->g.ny - 3);
    k_source<<<tb_blocks(tb_n3(c), 256), 256, 0, c->stream>>>(P, c->wx, dwzdx, c->uy, c->duexmdx, c->uyb, c->cfg.beta,
                                                               c->cfg.dy, stf_pow, c->cfg.my_form);
    TB_CHECK_LAUNCH(c);
    k_activate<<<tb_blocks(c->g.K, 64), 64, 0, c->stream>>>(c->pstate, c->g.K);
    TB_CHECK_LAUNCH(c);
    return TB_OK;
}

int tb_poisson_end(tb_ctx* c) {
    PoiDev P = make_dev(c);
    k_write_uy<<<tb_blocks(tb_n3(c), 256), 256, 0, c->stream>>>(P, c->uy);
    TB_CHECK_LAUNCH(c);
    return TB_OK;
}

int tb_poisson_defect_f32(tb_ctx* c, const DefectRows& D, float2* r32, size_t elems32, int T, int np, unsigned long long* maxsq) {
    PoiDev P = make_dev(c);
    dim3 grid(tb_blocks(c->g.nx - 2, 128), tb_blocks(c->g.ny - 1, DEF_ROWS), c->g.K);
    cudaEvent_t ps = nullptr;
    if (tb_prof_begin(c, PROF_DEFECT, &ps)) return TB_ERR_CUDA;
    k_defect_f32<<<grid, 128, 0, c->stream>>>(P, D, r32, elems32, T, np, maxsq);
    TB_CHECK_LAUNCH(c);
    return tb_prof_end(c, PROF_DEFECT, ps);
}
