// tb_deriv.cu -- batched compact line operators of the stage.
//
// x-lines (derparx/derparxx, filter_trid; tb_xline.cuh) and y-lines (dery/
// deryfv/deryy derivs_par.f:116-177 with rhsy/rhsyfv/rhsyy 400-611 and tridy
// 947-975).  Every line is an independent tridiagonal solve with a constant
// LHS.  A y-line is strided by nx, so one thread per line already reads
// coalesced rows across a warp; an x-line is contiguous, so two warps
// share one x-line (k_xwarp).  Launches batch several fields so that each SM
// sub-partition has full warps of FP64 work (GB300 issues one FP64 warp
// instruction per 64 cycles per sub-partition whatever the active-lane count).
#include "tb_internal.h"
#include "tb_xline.cuh"
#include <algorithm>
#include <cstring>

namespace {

struct XArgs {
    XJob job[8];
    int njobs, nx, ny, K;
    int fp32_modes;   // lines of modes k >= 1 in FP32 (mixed form)
    int inner;        // in place, rows i >= 1 of the lines j >= 1 only (filter_trid's copy-back)
    int staged;       // the tables are copied to shared memory
    int S;
    const double* tab;
    const float* tabf;
    xl::Weights w;
};

// The batched jobs' x-lines of one operator, two warps per line; lines of
// modes k >= 1 run in FP32 when A.fp32_modes is set (the mixed form: they hold
// only the disturbance).  A block keeps one copy of the operator's tables in
// shared memory for all the lines its warps take in turn.  Bound by the FP64 pipe:
// a field at 1025 x 193 x 32 takes 261 (D1) and 289 us (D2); 317 and 371 us with
// the tables read from global memory by blocks of two one-warp lines, whose lines
// left no room for them in L1.
constexpr int XW_MAX = 8;   // lines per block at most
template <int OP>
__global__ void __launch_bounds__(64 * XW_MAX) k_xwarp(XArgs A) {
    extern __shared__ double xs[];
    const int pair = threadIdx.x >> 6, part = (threadIdx.x >> 5) & 1, W = blockDim.x >> 6;
    const int tsz = xl::table_size(A.S);
    const double* T = A.tab;
    double* lines = xs;
    if (A.staged) {
        for (int q = threadIdx.x; q < tsz; q += blockDim.x) xs[q] = A.tab[q];
        T = xs;
        lines = xs + tsz;
        __syncthreads();
    }
    double* F = lines + (size_t)pair * xl::line_size(A.S);
    const long nlines = (long)A.ny * A.K, total = nlines * A.njobs;
    for (long gw = (long)pair * gridDim.x + blockIdx.x; gw < total; gw += (long)gridDim.x * W) {
        const int jb = (int)(gw / nlines), line = (int)(gw - jb * nlines);
        if (A.inner && line % A.ny == 0) continue;
        const cplx* f = A.job[jb].src + (size_t)line * A.nx;
        cplx* o = A.job[jb].dst + (size_t)line * A.nx;
        if (A.fp32_modes && line >= A.ny)
            xl::xline<OP, float>(A.w, A.tabf, A.S, A.nx, f, o, A.inner, reinterpret_cast<float*>(F), part, 1 + pair);
        else xl::xline<OP, double>(A.w, T, A.S, A.nx, f, o, A.inner, F, part, 1 + pair);
    }
}

struct YArgs {
    YJob job[8];
    int nx2, ny, K;
    TriLHS t[3];
    YRhs r[3];
};

// One real line a thread: the real and the imaginary parts of a field are
// lines of their own, neighbours in memory.  The right-hand side is formed with the
// scheme's weights as they are, in units of the row's 1/dy or 1/dy^2, which together
// with 1/pivot enters the backward sweep beside its chain: an interior row takes 5
// instructions for its right-hand side and 1 and 2 for the sweeps, and its weights
// stay in registers.  (All factors folded into the weights take one less, but each weight
// is then rounded for itself and the derivative no longer cancels: 1.3 to 5 times the
// error on 33 to 257 rows.)  All jobs run in one launch, blockIdx.y the job.  Bound by
// the FP64 pipe on large grids and by the chain of rows on small ones: dery and deryfv
// of a field, a launch each, take 0.10 ms at 257 x 97 x 8 and 0.48 ms at 1025 x 193 x 32;
// a complex line a thread, which reads a row's five weights and takes one instruction
// more a row on its chain, took 0.20 and 0.61 ms.
__global__ void __launch_bounds__(128) k_ylines(YArgs A) {
    const int line = blockIdx.x * blockDim.x + threadIdx.x, ny = A.ny;
    if (line >= A.nx2 * A.K) return;
    const YJob& J = A.job[blockIdx.y];
    const int i = line % A.nx2, k = line / A.nx2;
    const size_t s = A.nx2, base = (size_t)i + s * ny * k;
    const double* __restrict__ f = reinterpret_cast<const double*>(J.src) + base;
    double* __restrict__ o = reinterpret_cast<double*>(J.dst) + base;
    const double* __restrict__ ta = A.t[J.op].a;
    const double* __restrict__ tg = A.t[J.op].g;
    const double* __restrict__ tib = A.t[J.op].ib;
    const YRhs& R = A.r[J.op];
    const double* __restrict__ wr = R.w;
    double u = 0.0;
    // one row of the forward sweep with its rhs from the tables (boundary rows)
    auto generic = [&](int j) {
        double r = 0.0;
        const int c0 = R.cnt[j], of = R.off[j];
        const double* w = wr + 7 * j;
        for (int m = 0; m < c0; m++) r = fma(w[m], f[(size_t)(j + of + m) * s], r);
        u = fma(-ta[j], u, r);
        o[(size_t)j * s] = u;
    };
    // The sweeps are sequential in j, so each row's loads are issued YPD rows
    // ahead into a register ring; the interior rows j = 2 .. ny-3 (five-point
    // rhs f[j-2 .. j+2], derivs_par.f:400-611) keep their window in registers.
    constexpr int YPD = 8;
    generic(0);
    generic(1);
    {
        const double c0 = wr[14], c1 = wr[15], c2 = wr[16], c3 = wr[17], c4 = wr[18];
        double w0 = f[0], w1 = f[s], w2 = f[2 * s], w3 = f[3 * s];
        double pre[YPD];
#pragma unroll
        for (int q = 0; q < YPD; q++) pre[q] = (4 + q < ny) ? f[(size_t)(4 + q) * s] : 0.0;
        for (int jb = 2; jb < ny - 2; jb += YPD) {
#pragma unroll
            for (int q = 0; q < YPD; q++) {
                const int j = jb + q;
                if (j < ny - 2) {
                    const double w4 = pre[q];   // row j + 2
                    const int nr = j + 2 + YPD;
                    if (nr < ny) pre[q] = f[(size_t)nr * s];
                    double r = c0 * w0;
                    r = fma(c1, w1, r);
                    r = fma(c2, w2, r);
                    r = fma(c3, w3, r);
                    r = fma(c4, w4, r);
                    u = fma(-ta[j], u, r);
                    o[(size_t)j * s] = u;
                    w0 = w1; w1 = w2; w2 = w3; w3 = w4;
                }
            }
        }
    }
    generic(ny - 2);
    generic(ny - 1);
    // backward sweep, rows ny-2 .. 0, the forward values read YPD rows ahead
    u *= tib[ny - 1];
    o[(size_t)(ny - 1) * s] = u;
    {
        double pre[YPD];
#pragma unroll
        for (int q = 0; q < YPD; q++) pre[q] = (ny - 2 - q >= 0) ? o[(size_t)(ny - 2 - q) * s] : 0.0;
        for (int jb = ny - 2; jb >= 0; jb -= YPD) {
#pragma unroll
            for (int q = 0; q < YPD; q++) {
                const int j = jb - q;
                if (j >= 0) {
                    const double v = pre[q];
                    const int nr = j - YPD;
                    if (nr >= 0) pre[q] = o[(size_t)nr * s];
                    u = fma(-tg[j + 1], u, tib[j] * v);
                    o[(size_t)j * s] = u;
                }
            }
        }
    }
}

// Launch of one operator's jobs.  A line's time is its FP64 instructions, so an SM
// takes lines in fours, dealt evenly over its sub-partitions: blocks of 8
// lines where one or more fit an SM beside the tables, else 4 or fewer; half as many
// where the tuner found that faster.  Where every pair of warps has one line at
// most, or a line is so long that the tables leave no room for two, the tables are read
// from global memory by blocks of two lines, without the copy to shared memory
// (D1 of 33 lines of 1025 points: 33 us, 49 with it; of 129 lines of 385: 20 and 28;
// near the line the two meet: of 1032 lines of 385, one a pair, 29 and 28).
template <int OP>
int launch_xop(tb_ctx* c, XArgs& A, const TriLHS& t) {
    A.S = t.S; A.tab = t.xt; A.tabf = t.xtf;
    const size_t tab = (size_t)xl::table_size(t.S) * sizeof(double), line = (size_t)xl::line_size(t.S) * sizeof(double);
    const size_t room = (size_t)226 * 1024, lines = (size_t)A.njobs * A.ny * A.K;
    const size_t sms = c->sm_count > 0 ? c->sm_count : 148;
    if (line > room) { tb_set_error("x-line of %d points exceeds shared memory", A.nx); return TB_ERR_ARG; }
    int W = 2;
    size_t per = 1;   // blocks per SM
    A.staged = tab + 2 * line <= room;
    if (A.staged) {
        W = tab + 8 * line <= room ? 8 : tab + 4 * line <= room ? 4 : 2;
        per = std::max<size_t>(1, std::min<size_t>(4, room / (tab + W * line + 1024)));
        A.staged = lines > sms * per * W;
    }
    if (!A.staged) {
        W = 2 * line <= room ? 2 : 1;
        per = std::max<size_t>(1, std::min<size_t>(16, room / (W * line + 1024)));
    }
    if (c->tune_xw == 1 && W > 1) W /= 2;
    const size_t smem = (A.staged ? tab : 0) + W * line;
    const unsigned nb = (unsigned)std::min<size_t>((lines + W - 1) / W, per * sms);
    TB_CUDA(cudaFuncSetAttribute(k_xwarp<OP>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    k_xwarp<OP><<<nb, 64 * W, smem, c->stream>>>(A);
    TB_CHECK_LAUNCH(c);
    return TB_OK;
}

}  // namespace

int tb_launch_xlines(tb_ctx* c, const XJob* jobs, int njobs) {
    if (njobs <= 0) return TB_OK;
    if (njobs > 8) {
        int r = tb_launch_xlines(c, jobs, 8);
        if (r) return r;
        return tb_launch_xlines(c, jobs + 8, njobs - 8);
    }
    cudaEvent_t ps = nullptr;
    if (tb_prof_begin(c, PROF_XLINES, &ps)) return TB_ERR_CUDA;
    for (int op = 0; op < 3; op++) {
        XArgs A;
        std::memset(&A, 0, sizeof A);
        for (int q = 0; q < njobs; q++) {
            if (jobs[q].op != op) continue;
            // the filter may overwrite its field: the lines' rows as filter_trid copies them back
            if (jobs[q].src == jobs[q].dst) {
                if (op != XOP_FILTER) { tb_set_error("x-line job %d: in-place operation", q); return TB_ERR_ARG; }
                A.inner = 1;
            }
            A.job[A.njobs++] = jobs[q];
        }
        if (!A.njobs) continue;
        A.nx = c->g.nx; A.ny = c->g.ny; A.K = c->g.K;
        A.fp32_modes = (c->cfg.precision == TB_FORM_MIXED && c->fp32_lines) ? 1 : 0;
        A.w = tb_filter_weights(c->cfg.alphaf);
        int r;
        if (op == XOP_D1) r = launch_xop<xl::D1>(c, A, c->tx1);
        else if (op == XOP_D2) r = launch_xop<xl::D2>(c, A, c->tx2);
        else r = launch_xop<xl::FILTER>(c, A, c->tfil);
        if (r) return r;
    }
    return tb_prof_end(c, PROF_XLINES, ps);
}

int tb_launch_ylines(tb_ctx* c, const YJob* jobs, int njobs) {
    if (njobs <= 0) return TB_OK;
    if (njobs > 8) {
        int r = tb_launch_ylines(c, jobs, 8);
        if (r) return r;
        return tb_launch_ylines(c, jobs + 8, njobs - 8);
    }
    YArgs A;
    std::memset(&A, 0, sizeof A);
    for (int q = 0; q < njobs; q++) {
        if (jobs[q].src == jobs[q].dst) { tb_set_error("y-line job %d: in-place operation", q); return TB_ERR_ARG; }
        A.job[q] = jobs[q];
    }
    A.nx2 = 2 * c->g.nx; A.ny = c->g.ny; A.K = c->g.K;
    A.t[0] = c->ty1; A.t[1] = c->tyfv; A.t[2] = c->ty2;
    A.r[0] = c->ry1; A.r[1] = c->ryfv; A.r[2] = c->ry2;
    const int yt = (c->tune_yt == 32 || c->tune_yt == 64) ? c->tune_yt : 128;   // threads per block (tb_autotune)
    cudaEvent_t ps = nullptr;
    if (tb_prof_begin(c, PROF_YLINES, &ps)) return TB_ERR_CUDA;
    k_ylines<<<dim3(tb_blocks((size_t)A.nx2 * A.K, yt), njobs), yt, 0, c->stream>>>(A);
    TB_CHECK_LAUNCH(c);
    return tb_prof_end(c, PROF_YLINES, ps);
}
