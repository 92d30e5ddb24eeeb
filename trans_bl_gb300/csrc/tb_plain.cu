// tb_plain.cu -- multigrid v-Poisson per spanwise mode, plain FP64 form
// (poi_uy and its helpers, poisson_par.f:6-963; band solves penta_par.f:308-404).
//
// The reference relaxes y-lines in lexicographic order: in every sweep the
// border line i=2, the border line i=ptsx-1, then the centre lines 3..ptsx-2
// (1-based), each line solve using the lines i-1, i-2 already updated in the
// same sweep and i+1, i+2 from the previous one (sor, poisson_par.f:167-226).
// This file keeps that order and its iterates, and runs it as follows:
//
//  - Real and imaginary parts are independent problems (every operator
//    coefficient is real), so each (mode, part) is one CTA with its own
//    line-contiguous copy of the multigrid arrays: element (i, j) of level l
//    at off[l] + i*ptsy[l] + j, so a y-line is one contiguous run.
//  - Successive sweeps overlap as a wavefront: sweep s relaxes the centre
//    line i at step i-1+5s, the border line 2 at step 5s and the border line
//    ptsx-1 at step ptsx-8+5s (0-based line indices 1 and ptsx-2).  Every line
//    solve then reads exactly the values the sequential order gives it, and
//    no two solves of one step touch a line that the other writes (the
//    border stencils reach 4 lines inwards, which sets the lag of 5).  The last
//    sweep of a V-cycle on the fine level runs in one wavefront with the first
//    three of the next.
//  - What a step costs is the FP64 instructions of one line solve: a warp's
//    holds its sub-partition's FP64 pipe for ~64 cycles whatever the number of
//    active lanes.  So the sweeps of a wavefront sit on different SMs, in the
//    CTAs of a cluster, and a line on all four sub-partitions of its SM, one
//    row a lane where 128 lanes suffice (k_wsor).
// Defect, restriction, correction and interpolation are grid-parallel.
#include "tb_internal.h"
#include <algorithm>
#include <array>
#include <cmath>
#include <cstring>

namespace {

constexpr int LAG = 5;      // steps between successive sweeps of the wavefront
constexpr int RING = 16;    // lines of a slot's ring: a sweep and the one behind it touch 14
constexpr int NGROUP = 3;   // line groups of 1, 2 and 4 warps
constexpr int MAX_CLUSTER = 8;

__host__ __device__ inline int group_warps(int gi) { return 1 << gi; }
// Rows per lane of a line of n points (rows 1 .. n-1) on G warps, rounded up to
// a size the kernel is built for.
__host__ __device__ inline int rows_per_lane(int n, int G) {
    const int s = (n - 1 + 32 * G - 1) / (32 * G);
    return s <= 4 ? (s < 1 ? 1 : s) : s <= 6 ? 6 : s <= 8 ? 8 : s <= 12 ? 12 : 16;
}
// Line-solve tables of one (group, type, level, mode): entry e of chunk c (lane
// c % 32 of warp c / 32, rows 1 + c S .. c S + S) at e * 32 G + c.
//   per row s, from 8 s: weights WL WC WR of the x-stencil sums of rows j-1, j,
//     j+1 in the right-hand side (negative), L1 L2, U1 U2 (times ID), ID
//   WZ  -L times the fixed value of row 0, rows 1 and 2 (entries of rows s < 2)
//   per row the responses H1 H2 (forward) and K1 K2 (backward) to the states
//     entering the chunk
//   PF, PB  5 x 4: Kogge-Stone matrices of the chunk propagators in a warp
//   CF, CB  3 x 4: response of the state entering the chunk to the state
//     leaving warp w of those before (after) it
__host__ __device__ constexpr int tab_wz(int S) { return 8 * S; }
__host__ __device__ constexpr int tab_h(int S) { return 8 * S + (S < 2 ? 1 : 2); }
__host__ __device__ constexpr int tab_pf(int S) { return tab_h(S) + 4 * S; }
__host__ __device__ constexpr int tab_pb(int S) { return tab_pf(S) + 20; }
__host__ __device__ constexpr int tab_cf(int S) { return tab_pb(S) + 20; }
__host__ __device__ constexpr int tab_cb(int S) { return tab_cf(S) + 12; }
__host__ __device__ constexpr int tab_entries(int S) { return tab_cb(S) + 12; }
__host__ __device__ inline int tab_size(int n, int G) { return tab_entries(rows_per_lane(n, G)) * 32 * G; }
__host__ __device__ inline size_t tab_block(int ny) {
    const int a = tab_size(ny, 1), b = tab_size(ny, 2), c = tab_size(ny, 4), m = a > b ? a : b;
    return (size_t)(m > c ? m : c);
}

struct PlainDev {
    double *fc, *sc, *fct, *def;   // per block b = 2k + part: pelems doubles (fc, sc, fct), dstride (def)
    const double* tab;             // line-solve tables per (group, type, level, mode), blocks of tabs
    const double* coef;            // sp(7) cp(8) pp(4) lp(5) per level
    const double* qdy2;            // (ny, msh)
    const double* k2b2;
    int* state;                    // per mode: [2k] active, [2k+1] vcycles done
    double* err;
    unsigned long long* maxsq;     // per mode: max |defect|^2 of the fine level (double bits)
    int nx, ny, K, msh;
    int ptsx[TB_MAX_MSH], ptsy[TB_MAX_MSH];
    size_t off[TB_MAX_MSH], pelems, dstride, tabs;
    double den[TB_MAX_MSH];        // 1 / (12 dx2 fac_y)
    double fac_y, alpha, ify;
};

__device__ __forceinline__ const double* tab_ptr(const PlainDev& P, int gi, int type, int l, int k) {
    return P.tab + ((((size_t)gi * 2 + type) * P.msh + l) * P.K + k) * P.tabs;
}

__device__ __forceinline__ void group_barrier(int id, int nthreads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}

__device__ __forceinline__ void push(uint32_t addr, double v) {   // into a CTA of the cluster
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}
__device__ __forceinline__ uint32_t in_cta(const double* p, int rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// ---------------------------------------------------------------------------
// One y-line solve of sor on a group of G warps: rhs_center / rhs_border1 /
// rhs_border2 (poisson_par.f:343-540), banbk5_poi (penta_par.f:367-404) and
// fc + rf (x - fc) for the rows j >= 1 (0-based), S rows a lane.  Each chunk
// runs its local recurrences with zero carry, the chunk-end 2x2 propagators
// are scanned within each warp (Kogge-Stone, `lv` levels), the states leaving the
// other warps enter through precomputed responses, and the rows follow from the
// state that enters their chunk.  Row 0 keeps its value f0, which enters rows 1
// and 2.  Rows past the line have zero tables.
//
// With one or two rows a lane the scanned states are the rows themselves, but a row
// taken from there carries the rounding of every level: the defect that three sweeps
// leave of a solved problem on 129 rows is 1.4 times that of sequential sweeps, 1.05 times
// with the rows formed from the entering state.
//
// FP64 instructions a warp, four warps of one row a lane: 3 stencil, 3 weights,
// twice 1 + 16 scan and 2 for the rows, 12 for the three other warps, 1 scaling, 2
// update: 59 of ~64 cycles.  The x-stencil lines come as pointers to the
// chunk's rows (stride NC = 32 G): for a centre line (i-2, i-1, i+1, i+2), for
// a border line the four inner lines in order of distance and the outer line.
template <int S>
__device__ __forceinline__ void line_solve(bool border, const double* T, int G, int g, int lane, int lv, const double* a0,
                                           const double* a1, const double* a2, const double* a3, const double* a4,
                                           const double* F, const double (&sc)[S], double f0, double rf, double (&out)[S],
                                           double* xch, int bar) {
    const int NC = 32 * G, c = 32 * g + lane;
    const double* t = T + c;
    auto tab = [&](int e) { return t[e * NC]; };
    // x-stencil sums of the chunk's rows, and of the row on either side
    double gs[S];
    if (!border) {
#pragma unroll
        for (int s = 0; s < S; s++) gs[s] = fma(16.0, a1[s * NC] + a2[s * NC], -(a0[s * NC] + a3[s * NC]));
    } else {
#pragma unroll
        for (int s = 0; s < S; s++)
            gs[s] = 10.0 * a4[s * NC] - 4.0 * a0[s * NC] + 14.0 * a1[s * NC] - 6.0 * a2[s * NC] + a3[s * NC];
    }
    double gm = __shfl_up_sync(0xffffffffu, gs[S - 1], 1), gp = __shfl_down_sync(0xffffffffu, gs[0], 1);
    if (G > 1) {
        if (lane == 0) xch[2 * g] = gs[0];
        if (lane == 31) xch[2 * g + 1] = gs[S - 1];
        group_barrier(bar, 32 * G);
        if (lane == 0 && g > 0) gm = xch[2 * (g - 1) + 1];
        if (lane == 31 && g + 1 < G) gp = xch[2 * (g + 1)];
    }
    double y[S];
#pragma unroll
    for (int s = 0; s < S; s++) {
        double r = fma(tab(8 * s + 1), gs[s], sc[s]);
        r = fma(tab(8 * s), s ? gs[s > 0 ? s - 1 : 0] : gm, r);
        r = fma(tab(8 * s + 2), s + 1 < S ? gs[s + 1 < S ? s + 1 : 0] : gp, r);
        if (s < 2 && g == 0) r = fma(tab(tab_wz(S) + s), f0, r);
        if (s > 0) r = fma(-tab(8 * s + 3), y[s > 0 ? s - 1 : 0], r);
        if (s > 1) r = fma(-tab(8 * s + 4), y[s > 1 ? s - 2 : 0], r);
        y[s] = r;
    }
    // forward: scan of the chunk-end states (y_e, y_{e-1}) within the warp
    double b0 = y[S - 1], b1 = S > 1 ? y[S > 1 ? S - 2 : 0] : 0.0;
#pragma unroll
    for (int d = 0, off = 1; d < 5; d++, off <<= 1) {
        if (d >= lv) break;
        const double o0 = __shfl_up_sync(0xffffffffu, b0, off), o1 = __shfl_up_sync(0xffffffffu, b1, off);
        if (lane >= off) {
            const int e = tab_pf(S) + 4 * d;
            if (S == 1 && d == 0) {   // one row: the propagator is (m0 m1; 1 0)
                b0 = fma(tab(e), o0, b0);
                b1 = o0;
            } else {
                b0 = fma(tab(e), o0, fma(tab(e + 1), o1, b0));
                b1 = fma(tab(e + 2), o0, fma(tab(e + 3), o1, b1));
            }
        }
    }
    double* xf = xch + 2 * G;
    if (G > 1) {
        if (lane == 31) { xf[2 * g] = b0; xf[2 * g + 1] = b1; }
        group_barrier(bar, 32 * G);
    }
    b0 = __shfl_up_sync(0xffffffffu, b0, 1);
    b1 = __shfl_up_sync(0xffffffffu, b1, 1);
    if (lane == 0) { b0 = 0.0; b1 = 0.0; }
#pragma unroll
    for (int w = 0; w < 3; w++)
        if (w < g) {
            const double z0 = xf[2 * w], z1 = xf[2 * w + 1];
            const int e = tab_cf(S) + 4 * w;
            b0 = fma(tab(e), z0, fma(tab(e + 1), z1, b0));
            b1 = fma(tab(e + 2), z0, fma(tab(e + 3), z1, b1));
        }
#pragma unroll
    for (int s = 0; s < S; s++) y[s] = fma(tab(tab_h(S) + 4 * s), b0, fma(tab(tab_h(S) + 4 * s + 1), b1, y[s]));
    // backward, likewise from the high lanes
#pragma unroll
    for (int s = S - 1; s >= 0; s--) {
        double x = tab(8 * s + 7) * y[s];
        if (s + 1 < S) x = fma(-tab(8 * s + 5), y[s + 1 < S ? s + 1 : 0], x);
        if (s + 2 < S) x = fma(-tab(8 * s + 6), y[s + 2 < S ? s + 2 : 0], x);
        y[s] = x;
    }
    b0 = y[0]; b1 = S > 1 ? y[S > 1 ? 1 : 0] : 0.0;
#pragma unroll
    for (int d = 0, off = 1; d < 5; d++, off <<= 1) {
        if (d >= lv) break;
        const double o0 = __shfl_down_sync(0xffffffffu, b0, off), o1 = __shfl_down_sync(0xffffffffu, b1, off);
        if (lane + off < 32) {
            const int e = tab_pb(S) + 4 * d;
            if (S == 1 && d == 0) {
                b0 = fma(tab(e), o0, b0);
                b1 = o0;
            } else {
                b0 = fma(tab(e), o0, fma(tab(e + 1), o1, b0));
                b1 = fma(tab(e + 2), o0, fma(tab(e + 3), o1, b1));
            }
        }
    }
    double* xb = xch + 4 * G;
    if (G > 1) {
        if (lane == 0) { xb[2 * g] = b0; xb[2 * g + 1] = b1; }
        group_barrier(bar, 32 * G);
    }
    b0 = __shfl_down_sync(0xffffffffu, b0, 1);
    b1 = __shfl_down_sync(0xffffffffu, b1, 1);
    if (lane == 31) { b0 = 0.0; b1 = 0.0; }
#pragma unroll
    for (int w = 0; w < 3; w++)
        if (g + 1 + w < G) {   // the warps after this one
            const double z0 = xb[2 * (g + 1 + w)], z1 = xb[2 * (g + 1 + w) + 1];
            const int e = tab_cb(S) + 4 * w;
            b0 = fma(tab(e), z0, fma(tab(e + 1), z1, b0));
            b1 = fma(tab(e + 2), z0, fma(tab(e + 3), z1, b1));
        }
#pragma unroll
    for (int s = 0; s < S; s++) y[s] = fma(tab(tab_h(S) + 4 * s + 2), b0, fma(tab(tab_h(S) + 4 * s + 3), b1, y[s]));
#pragma unroll
    for (int s = 0; s < S; s++) {
        out[s] = y[s];
        if (rf != 1.0) {
            const double fo = F[s * NC];
            out[s] = fma(rf, y[s] - fo, fo);
        }
    }
}

// Shapes of one k_wsor launch.
struct Wave {
    int l, ns, gi;      // level, sweeps, line group
    int C, W;           // CTAs of a cluster, line groups (slots) of a CTA
    int lv;             // scan levels
    int seq;            // too few lines for the wavefront: the reference's order on one group
    int parity;         // rings per slot: 2 where a slot runs several sweeps
    int staged;         // tables in shared memory: 2 both types, 1 the centre lines'
    double rf0, rf;     // relaxation factor of the first sweep and of the others
};
__host__ __device__ inline size_t wave_lines(const Wave& v, int NC, int S) {
    return ((size_t)v.W * v.parity * RING + 2) * NC * S;
}

// `ns` lexicographic sweeps at level l of one (mode, part) with an active mode
// on one cluster.  A slot is a group of G warps with a ring of lines; slot q of
// the cluster's C W runs the sweeps q, q + C W, ...  The first sweep reads its
// lines from global memory, every sweep hands each relaxed line to the ring
// of the slot behind it (in another CTA through distributed shared memory),
// and the last one writes it back; one cluster barrier a step orders this.
// A further group per CTA solves the far border line of its slots' sweeps
// beside their centre lines.  A slot that runs several sweeps alternates
// between two rings.
//
// One CTA per (mode, part), two warps a line and all sweeps of a wavefront on
// the SM's four FP64 pipes took 411 ms a step at 385 x 129 x 1 and 450 ms at
// 513 x 129 x 8; this takes 149 and 204 ms, 3.8 us a step of the wavefront of four
// sweeps on 129 rows.
// STAGED: both types' tables fit shared memory beside the rings, and every load
// of a solve is one from shared memory.
template <int S, bool STAGED>
__global__ void __launch_bounds__(256) k_wsor(PlainDev P, Wave V) {
    const int C = V.C, rank = blockIdx.x % C, b = blockIdx.x / C, k = b >> 1, l = V.l;
    if (!P.state[2 * k]) return;   // uniform over the cluster
    const int nxl = P.ptsx[l], n = P.ptsy[l], m = nxl - 2, ns = V.ns;
    const int G = 1 << V.gi, NC = 32 * G, LS = NC * S, W = V.W, NS = C * W;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int grp = warp >> V.gi, g = warp & (G - 1), c = 32 * g + lane;
    extern __shared__ double smem[];
    double* rings = smem;                                        // (W, parity, RING, S, NC)
    double* edge = rings + (size_t)W * V.parity * RING * LS;     // lines 0 and nxl - 1
    double* xch = edge + 2 * LS + 6 * G * grp;                   // group exchange
    double* ts = edge + 2 * LS + 6 * G * (W + 1);                // staged tables
    const double *tc = tab_ptr(P, V.gi, 0, l, k), *tb = tab_ptr(P, V.gi, 1, l, k);
    double* Fg = P.fc + (size_t)b * P.pelems + P.off[l];
    const double* SCg = P.sc + (size_t)b * P.pelems + P.off[l];
    {
        const int tsz = tab_entries(S) * NC;
        if (STAGED || V.staged) {
            for (int q = tid; q < tsz; q += blockDim.x) ts[q] = tc[q];
            tc = ts;
        }
        if (STAGED) {
            for (int q = tid; q < tsz; q += blockDim.x) ts[tsz + q] = tb[q];
            tb = ts + tsz;
        }
        // rows past the line stay zero in every ring
        for (int q = tid; q < W * V.parity * RING * LS; q += blockDim.x) rings[q] = 0.0;
    }
    __syncthreads();
    const int row0 = 1 + c * S;   // the chunk's first row
    auto ring = [&](int w, int s) { return rings + (size_t)(w * V.parity + (V.parity > 1 ? (s / NS) & 1 : 0)) * RING * LS; };
    // line q of a sweep as its slot sees it, at the chunk's rows
    auto at = [&](const double* R, int q) -> const double* {
        return (q == 0 ? edge : q == nxl - 1 ? edge + LS : R + (size_t)(q & (RING - 1)) * LS) + c;
    };
    auto fill = [&](double* dst, int q) {
#pragma unroll
        for (int s = 0; s < S; s++) dst[s * NC + c] = (row0 + s < n) ? Fg[(size_t)q * n + row0 + s] : 0.0;
    };
    if (grp == 0) {
        fill(edge, 0);
        fill(edge + LS, nxl - 1);
        if (rank == 0)
            for (int q = 1; q <= min(m, 7); q++) fill(rings + (size_t)(q & (RING - 1)) * LS, q);
    }
    if (C > 1) {
        cluster_arrive();
        cluster_wait();
    } else __syncthreads();
    auto load_sc = [&](int line, double (&v)[S], double& f0) {
#pragma unroll
        for (int s = 0; s < S; s++) v[s] = (row0 + s < n) ? SCg[(size_t)line * n + row0 + s] : 0.0;
        if (g == 0) f0 = Fg[(size_t)line * n];
    };
    // the last sweep's line (0: none) on its way to global memory
    int done = 0;
    double res[S];
    auto write_back = [&]() {
        if (done) {
#pragma unroll
            for (int q = 0; q < S; q++)
                if (row0 + q < n) Fg[(size_t)done * n + row0 + q] = res[q];
            done = 0;
        }
    };
    // relax line `line` of sweep s in slot w (of this CTA)
    auto relax = [&](int w, int s, int line, const double (&sc)[S], double f0) {
        double* R = ring(w, s);
        const bool lo = line == 1, hi = line == m, bd = lo || hi;
        const int e = lo ? 1 : -1;
        const double* F = at(R, line);
        double out[S];
        line_solve<S>(bd, bd ? tb : tc, G, g, lane, V.lv, at(R, bd ? line + e : line - 2), at(R, bd ? line + 2 * e : line - 1),
                      at(R, bd ? line + 3 * e : line + 1), at(R, bd ? line + 4 * e : line + 2), bd ? at(R, line - e) : nullptr, F,
                      sc, f0, s == 0 ? V.rf0 : V.rf, out, xch, 1 + grp);
        double* own = R + (size_t)(line & (RING - 1)) * LS + c;
#pragma unroll
        for (int q = 0; q < S; q++) own[q * NC] = out[q];
        if (s == ns - 1) {
            done = line;
#pragma unroll
            for (int q = 0; q < S; q++) res[q] = out[q];
        } else if (!V.seq) {
            const int slot = (s + 1) % NS, w2 = slot % W, r2 = slot / W;
            double* next = ring(w2, s + 1) + (size_t)(line & (RING - 1)) * LS + c;
            if (r2 == rank) {
#pragma unroll
                for (int q = 0; q < S; q++) next[q * NC] = out[q];
            } else {
                const uint32_t a = in_cta(next, r2);
#pragma unroll
                for (int q = 0; q < S; q++) push(a + 8u * q * NC, out[q]);
            }
        }
    };
    if (V.seq) {
        // one group in the reference's order; lines 0 .. 8 at most, all in the ring
        if (grp == 0)
            for (int q = 0; q < ns * m; q++) {
                const int s = q / m, r = q - s * m, line = r == 0 ? 1 : r == 1 ? m : r;
                double sc[S], f0 = 0.0;
                load_sc(line, sc, f0);
                relax(0, s, line, sc, f0);
                write_back();
                if (G > 1) group_barrier(1, 32 * G); else __syncwarp();
            }
        return;
    }
    // A line group runs its slot's sweep s at step u = t - 5 s: line 1, then the
    // centre lines.  The last group watches all slots of the CTA for the step
    // of the far border line.
    const bool bgrp = grp == W;
    const int turn = V.parity > 1 ? LAG * NS : 0x3fffffff;   // steps from a slot's sweep to its next
    int sw = rank * W + (bgrp ? 0 : grp);   // current sweep of the group's (first) slot
    double scn[S], f0n = 0.0, fln[S];
#pragma unroll
    for (int q = 0; q < S; q++) { scn[q] = 0.0; fln[q] = 0.0; }
    // the task of the group at step t: line (0: none) of sweep `s` in slot `w`
    auto task = [&](int t, int& w, int& s) -> int {
        if (!bgrp) {
            w = grp; s = sw;
            if (t - LAG * s >= turn) s += NS;
            const int u = t - LAG * s;
            return (u < 0 || u > m - 2 || s >= ns) ? 0 : u + 1;
        }
        for (int q = 0; q < W; q++) {
            s = sw + q;
            if (t - LAG * s >= turn) s += NS;
            if (t - LAG * s == m - 6 && s < ns) { w = q; return m; }
        }
        return 0;
    };
    int w = 0, s = 0, line = task(0, w, s);
    if (line) load_sc(line, scn, f0n);
    const int T = m - 1 + LAG * (ns - 1);
    for (int t = 0; t < T; t++) {
        double sc[S], f0 = f0n;
#pragma unroll
        for (int q = 0; q < S; q++) sc[q] = scn[q];
        int w2 = 0, s2 = 0;
        const int line2 = task(t + 1, w2, s2);
        if (line2) load_sc(line2, scn, f0n);
        const bool feed = rank == 0 && grp == 0 && t + 8 <= m;   // line t + 8 of the first sweep
        if (feed) {
#pragma unroll
            for (int q = 0; q < S; q++) fln[q] = (row0 + q < n) ? Fg[(size_t)(t + 8) * n + row0 + q] : 0.0;
        }
        if (line) relax(w, s, line, sc, f0);
        if (feed) {
            double* dst = rings + (size_t)((t + 8) & (RING - 1)) * LS + c;
#pragma unroll
            for (int q = 0; q < S; q++) dst[q * NC] = fln[q];
        }
        // written between the barrier's halves, or its release would wait for global memory
        __syncwarp();
        if (C > 1) cluster_arrive();
        write_back();
        line = line2; w = w2; s = s2;
        if (t + 1 - LAG * sw - (bgrp ? LAG * (W - 1) : 0) >= turn) sw += NS;
        __syncwarp();
        if (C > 1) cluster_wait(); else __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// The level-l operator of defect (poisson_par.f:543-793) at the interior point
// (i, j) of block b: L fc = den*Dxx + q2*Dyy + k2b2*ify*M - top (real part).
__device__ __forceinline__ double plain_bx(const double* F, int n, int nxl, int i, int jj) {
    auto f = [&](int ii) { return F[(size_t)ii * n + jj]; };
    if (i == 1 || i == nxl - 2) {
        int e = (i == 1) ? 1 : -1;
        return 10.0 * f(i - e) - 15.0 * f(i) - 4.0 * f(i + e) + 14.0 * f(i + 2 * e) - 6.0 * f(i + 3 * e) + f(i + 4 * e);
    }
    return -f(i - 2) + 16.0 * f(i - 1) - 30.0 * f(i) + 16.0 * f(i + 1) - f(i + 2);
}

__device__ __forceinline__ double plain_Lu(const PlainDev& P, int l, int k, const double* F, int i, int j) {
    const int nxl = P.ptsx[l], n = P.ptsy[l];
    const double* cf = P.coef + 24 * l;
    const double *SPc = cf, *CPc = cf + 7, *PPc = cf + 15, *LPc = cf + 19;
    const double k2b2 = P.k2b2[k], den = P.den[l], ify = P.ify;
    const double* Fi = F + (size_t)i * n;
    auto bx = [&](int jj) { return plain_bx(F, n, nxl, i, jj); };
    double b, cc, d, q2, top = 0.0;
    if (j == 1) {
        b = SPc[2] * bx(2) + SPc[1] * bx(1);
        cc = SPc[3] * Fi[0] + SPc[4] * Fi[1] + SPc[5] * Fi[2] + SPc[6] * Fi[3];
        d = k2b2 * (SPc[1] * Fi[1] + SPc[2] * Fi[2]);
        q2 = P.qdy2[(size_t)P.ny * l];
    } else if (j <= n - 3) {
        b = CPc[0] * bx(j - 1) + CPc[1] * bx(j) + CPc[2] * bx(j + 1);
        cc = CPc[3] * Fi[j - 2] + CPc[4] * Fi[j - 1] + CPc[5] * Fi[j] + CPc[6] * Fi[j + 1] + CPc[7] * Fi[j + 2];
        d = k2b2 * (CPc[0] * Fi[j - 1] + CPc[1] * Fi[j] + CPc[2] * Fi[j + 1]);
        q2 = P.qdy2[(j - 2) + (size_t)P.ny * l];
    } else if (j == n - 2) {
        b = bx(j);
        cc = PPc[3] * Fi[j + 1] + PPc[2] * Fi[j] + PPc[1] * Fi[j - 1];
        d = k2b2 * Fi[j];
        q2 = P.qdy2[(j - 1) + (size_t)P.ny * l];
    } else {
        b = bx(j);
        cc = LPc[2] * Fi[j] + LPc[3] * Fi[j - 1] + LPc[4] * Fi[j - 2];
        d = k2b2 * Fi[j];
        q2 = P.qdy2[(j - 2) + (size_t)P.ny * l];
        top = LPc[1] * sqrt((P.alpha * P.alpha - k2b2) / P.fac_y) * sqrt(q2);
    }
    return b * den + cc * q2 + d * ify - top * Fi[j];
}

// defect (poisson_par.f:543-793): def = sc + si * (L fc) at level l, points
// 1 <= i <= ptsx-2, 1 <= j <= ptsy-1, both parts of mode blockIdx.y per
// thread; si > 0 also stores it into sc(l).  On the fine level (l = 0) the
// block's max |def|^2 goes into maxsq[k] (double bits, non-negative; a
// non-finite defect records +inf) for k_pcheck.
__global__ void k_pdefect(PlainDev P, int l, double si) {
    const int k = blockIdx.y;
    if (!P.state[2 * k]) return;   // uniform over the block
    const int nxl = P.ptsx[l], n = P.ptsy[l];
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    double m = 0.0;
    bool bad = false;
    if (q < (nxl - 2) * (n - 1)) {
        const int i = 1 + q / (n - 1), j = 1 + q % (n - 1);
        const size_t o = (size_t)i * n + j;
        double v[2];
#pragma unroll
        for (int part = 0; part < 2; part++) {
            const int b = 2 * k + part;
            const double* F = P.fc + (size_t)b * P.pelems + P.off[l];
            double* SC = P.sc + (size_t)b * P.pelems + P.off[l];
            v[part] = SC[o] + si * plain_Lu(P, l, k, F, i, j);
            P.def[(size_t)b * P.dstride + o] = v[part];
            if (si > 0) SC[o] = v[part];
        }
        const double a = v[0] * v[0] + v[1] * v[1];
        if (!(a <= 1.7e308)) bad = true;
        else m = a;
    }
    if (l != 0) return;   // uniform over the block
    if (bad) m = __longlong_as_double(0x7ff0000000000000LL);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    __shared__ double wm[8];
    if ((threadIdx.x & 31) == 0) wm[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        double bm = wm[0];
        for (int w = 1; w < (int)(blockDim.x >> 5); w++) bm = fmax(bm, wm[w]);
        atomicMax(&P.maxsq[k], (unsigned long long)__double_as_longlong(bm));
    }
}

// get_max_value + verifica_poi (poisson_par.f:67-108, 945-963): max |defect|
// of each mode from the fine-level defect's maxima; converged modes stop.
__global__ void k_pcheck(PlainDev P, double tol, int vcycle) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= P.K || !P.state[2 * k]) return;
    const double a = __longlong_as_double((long long)P.maxsq[k]);
    P.maxsq[k] = 0ull;
    if (!(a <= 1.7e308)) {
        P.err[k] = __longlong_as_double(0x7ff8000000000000LL);
        P.state[2 * k] = 0;
        P.state[2 * k + 1] = -1 - vcycle;
        return;
    }
    const double e = sqrt(a);
    P.err[k] = e;
    if (e < tol) { P.state[2 * k] = 0; P.state[2 * k + 1] = vcycle - 1; }
}

// restrict (poisson_par.f:796-874): level l -> l+1 (injection of fc into fc
// and fct, full weighting of the defect into sc at interior points, the top
// row from three points).
__global__ void k_prestrict(PlainDev P, int l) {
    const int b = blockIdx.y, k = b >> 1;
    if (!P.state[2 * k]) return;
    const int nxc = P.ptsx[l + 1], nyc = P.ptsy[l + 1], nxf = P.ptsx[l], nyf = P.ptsy[l];
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= nxc * nyc) return;
    const int i = q / nyc, j = q % nyc;
    const double* Ff = P.fc + (size_t)b * P.pelems + P.off[l];
    const double* Df = P.def + (size_t)b * P.dstride;
    double* Fc = P.fc + (size_t)b * P.pelems + P.off[l + 1];
    double* Tc = P.fct + (size_t)b * P.pelems + P.off[l + 1];
    double* Sc = P.sc + (size_t)b * P.pelems + P.off[l + 1];
    auto df = [&](int ii, int jj) { return Df[(size_t)ii * nyf + jj]; };
    int fi = (i == nxc - 1) ? nxf - 1 : 2 * i, fj = (j == nyc - 1) ? nyf - 1 : 2 * j;
    const size_t o = (size_t)i * nyc + j;
    double v = Ff[(size_t)fi * nyf + fj];
    Fc[o] = v;
    Tc[o] = v;
    if (i >= 1 && i <= nxc - 2) {
        if (j >= 1 && j <= nyc - 2) {
            Sc[o] = 6.25e-2 * (2.0 * (df(fi - 1, fj) + df(fi + 1, fj) + df(fi, fj - 1) + df(fi, fj + 1)) + 4.0 * df(fi, fj) +
                               df(fi + 1, fj + 1) + df(fi + 1, fj - 1) + df(fi - 1, fj + 1) + df(fi - 1, fj - 1));
        } else if (j == nyc - 1) {
            Sc[o] = 0.25 * (df(fi - 1, fj) + 2.0 * df(fi, fj) + df(fi + 1, fj));
        }
    }
}

// correction (poisson_par.f:923-942) at the coarse level l.
__global__ void k_pcorrection(PlainDev P, int l) {
    const int b = blockIdx.y, k = b >> 1;
    if (!P.state[2 * k]) return;
    const int nxl = P.ptsx[l], n = P.ptsy[l];
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= (nxl - 2) * n) return;
    const size_t o = (size_t)n + q;   // lines 1 .. nxl-2
    double* F = P.fc + (size_t)b * P.pelems + P.off[l];
    const double* T = P.fct + (size_t)b * P.pelems + P.off[l];
    F[o] = F[o] - T[o];
}

// intpol (poisson_par.f:877-920): add the bilinear interpolant of level l to
// level l-1 at lines 1 .. ptsx(l-1)-2.
__global__ void k_pintpol(PlainDev P, int l) {
    const int b = blockIdx.y, k = b >> 1;
    if (!P.state[2 * k]) return;
    const int nyc = P.ptsy[l], nxf = P.ptsx[l - 1], nyf = P.ptsy[l - 1];
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= (nxf - 2) * nyf) return;
    const int i = 1 + q / nyf, j = q % nyf;
    const double* C = P.fc + (size_t)b * P.pelems + P.off[l];
    auto cv = [&](int ci, int cj) { return C[(size_t)ci * nyc + cj]; };
    auto row = [&](int jj) -> double {
        int cj = jj / 2;
        if ((i & 1) == 0) return cv(i / 2, cj);
        return 0.5 * (cv(i / 2, cj) + cv(i / 2 + 1, cj));
    };
    double t = ((j & 1) == 0) ? row(j) : 0.5 * (row(j + 1) + row(j - 1));
    double* F = P.fc + (size_t)b * P.pelems + P.off[l - 1];
    F[(size_t)i * nyf + j] += t;
}

// function_source (poisson_par.f:111-164) for all modes, into the
// line-contiguous real/imaginary planes of level 0: sc and fc = uy.  32 x 32
// tiles transposed through shared memory (x-rows in, y-lines out).
__global__ void k_psource(PlainDev P, const cplx* wx, const cplx* dwzdx, const cplx* uy, const double* duexmdx,
                          const double* uyb, double beta, double dy, double stf_pow, int form) {
    __shared__ cplx ts[32][33], tu[32][33];
    const int k = blockIdx.z, J = P.ny, nx = P.nx;
    const int i0 = blockIdx.x * 32, j0 = blockIdx.y * 32;
    const double* c0 = P.coef;
    const double kb = (double)k * beta;
    auto S = [&](int i, int jj) {
        size_t o = (size_t)i + (size_t)nx * (jj + (size_t)J * k);
        cplx w = wx[o], d = dwzdx[o];
        return make_double2(kb * w.y - d.x, -kb * w.x - d.y);
    };
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        int i = i0 + threadIdx.x, j = j0 + r;
        if (i < nx && j < J) {
            cplx s;
            if (j == 0) s = make_double2(0, 0);
            else if (j == 1) { cplx a = S(i, 1), b = S(i, 2); s = make_double2(c0[1] * a.x + c0[2] * b.x, c0[1] * a.y + c0[2] * b.y); }
            else if (j <= J - 3) {
                cplx a = S(i, j - 1), b = S(i, j), d = S(i, j + 1);
                s = make_double2(c0[7] * a.x + c0[8] * b.x + c0[9] * d.x, c0[7] * a.y + c0[8] * b.y + c0[9] * d.y);
            } else if (j == J - 2) s = S(i, J - 2);
            else {
                s = make_double2(0, 0);
                if ((form == 0 || form == 4) && k == 0) {
                    double dya = dy * stf_pow;
                    size_t o = (size_t)i + (size_t)nx * (J - 1);
                    double lp1 = c0[19], lp2 = c0[20];
                    s = make_double2(-(lp1 * dwzdx[o].x) + lp2 * duexmdx[i] / dya - lp2 * P.alpha * uyb[o] / dya / sqrt(P.fac_y),
                                     -(lp1 * dwzdx[o].y));
                }
            }
            ts[r][threadIdx.x] = s;
            tu[r][threadIdx.x] = uy[(size_t)i + (size_t)nx * (j + (size_t)J * k)];
        }
    }
    __syncthreads();
    double *sr = P.sc + (size_t)(2 * k) * P.pelems, *si = sr + P.pelems;
    double *fr = P.fc + (size_t)(2 * k) * P.pelems, *fi = fr + P.pelems;
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        int i = i0 + r, j = j0 + threadIdx.x;
        if (i < nx && j < J) {
            size_t o = (size_t)i * J + j;
            cplx s = ts[threadIdx.x][r], u = tu[threadIdx.x][r];
            sr[o] = s.x; si[o] = s.y; fr[o] = u.x; fi[o] = u.y;
        }
    }
}

// uy(i,j,k) = fc(i,j,1) for j >= 2, 2 <= i <= ptsx-1 (poisson_par.f:53-57).
__global__ void k_pwrite_uy(PlainDev P, cplx* uy) {
    __shared__ cplx tile[32][33];
    const int k = blockIdx.z, J = P.ny, nx = P.nx;
    const int i0 = blockIdx.x * 32, j0 = blockIdx.y * 32;
    const double *fr = P.fc + (size_t)(2 * k) * P.pelems, *fi = fr + P.pelems;
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        int i = i0 + r, j = j0 + threadIdx.x;
        if (i < nx && j < J) {
            size_t o = (size_t)i * J + j;
            tile[r][threadIdx.x] = make_double2(fr[o], fi[o]);
        }
    }
    __syncthreads();
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        int i = i0 + threadIdx.x, j = j0 + r;
        if (i >= 1 && i <= nx - 2 && j >= 1 && j < J) uy[(size_t)i + (size_t)nx * (j + (size_t)J * k)] = tile[threadIdx.x][r];
    }
}

__global__ void k_pactivate(int* state, int K) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < K) { state[2 * k] = 1; state[2 * k + 1] = 0; }
}

PlainDev make_plain(tb_ctx* c) {
    PlainDev P;
    std::memset(&P, 0, sizeof P);
    P.fc = c->pl_fc; P.sc = c->pl_sc; P.fct = c->pl_fct; P.def = c->pl_def; P.tab = c->pl_tab; P.coef = c->pcoef;
    P.qdy2 = c->pqdy2; P.k2b2 = c->k2b2; P.state = c->pstate; P.err = c->perr; P.maxsq = c->pl_maxsq;
    P.nx = c->g.nx; P.ny = c->g.ny; P.K = c->g.K; P.msh = c->g.msh;
    for (int l = 0; l < c->g.msh; l++) {
        P.ptsx[l] = c->g.ptsx[l]; P.ptsy[l] = c->g.ptsy[l]; P.off[l] = c->g.lvl_off[l];
        P.den[l] = 1.0 / (12.0 * c->h_dx2[l] * c->cfg.fac_y);
    }
    P.ify = 1.0 / c->cfg.fac_y;
    P.pelems = c->g.lvl_elems; P.dstride = (size_t)c->g.nx * c->g.ny; P.tabs = tab_block(c->g.ny);
    P.fac_y = c->cfg.fac_y; P.alpha = c->cfg.alpha;
    return P;
}

// Line-solve tables (layout above tab_wz) of one (group, type, level, mode)
// for G warps of 32 chunks of S rows, from the band LU rows L1 L2 U1 U2 ID.  The rows
// past the line are rows of zeros, so every chunk has S.
void group_tables(int n, int S, int G, const double* L1, const double* L2, const double* U1, const double* U2,
                  const double* ID, const double* cf, double qx, double* out) {
    const int NC = 32 * G;
    using M2 = std::array<double, 4>;
    auto mul = [](const M2& A, const M2& B) {   // A B
        return M2{A[0] * B[0] + A[1] * B[2], A[0] * B[1] + A[1] * B[3], A[2] * B[0] + A[3] * B[2], A[2] * B[1] + A[3] * B[3]};
    };
    std::vector<M2> Mf(NC), Mb(NC);
    for (int c = 0; c < NC; c++) {
        auto at = [&](int e) -> double& { return out[(size_t)e * NC + c]; };
        std::vector<double> l1(S), l2(S), u1(S), u2(S);
        for (int s = 0; s < S; s++) {
            const int j = 1 + c * S + s;
            const bool in = j < n;
            if (in) {
                // sc - qx (weights . x-stencil sums), rhs_center / rhs_border (poisson_par.f:343-540)
                at(8 * s) = (j > 1 && j <= n - 3) ? -qx * cf[7] : 0.0;
                at(8 * s + 1) = j == 1 ? -qx * cf[1] : j <= n - 3 ? -qx * cf[8] : -qx;
                at(8 * s + 2) = j == 1 ? -qx * cf[2] : j <= n - 3 ? -qx * cf[9] : 0.0;
            }
            l1[s] = (in && j > 1) ? L1[j] : 0.0; l2[s] = (in && j > 2) ? L2[j] : 0.0;
            u1[s] = in ? U1[j] * ID[j] : 0.0; u2[s] = in ? U2[j] * ID[j] : 0.0;
            at(8 * s + 3) = l1[s]; at(8 * s + 4) = l2[s];
            at(8 * s + 5) = u1[s]; at(8 * s + 6) = u2[s];
            at(8 * s + 7) = in ? ID[j] : 0.0;
            if (s < 2) at(tab_wz(S) + s) = in && j == 1 ? -L1[1] : in && j == 2 ? -L2[2] : 0.0;
        }
        // responses to the entering states (y_{-1}, y_{-2}) and (x_S, x_{S+1})
        for (int u = 0; u < 2; u++) {
            double p1 = u == 0, p2 = u == 1;
            for (int s = 0; s < S; s++) {
                const double y = -l1[s] * p1 - l2[s] * p2;
                at(tab_h(S) + 4 * s + u) = y;
                p2 = p1; p1 = y;
            }
            Mf[c][u] = p1; Mf[c][2 + u] = p2;
            p1 = u == 0; p2 = u == 1;
            for (int s = S - 1; s >= 0; s--) {
                const double x = -u1[s] * p1 - u2[s] * p2;
                at(tab_h(S) + 4 * s + 2 + u) = x;
                p2 = p1; p1 = x;
            }
            Mb[c][u] = p1; Mb[c][2 + u] = p2;
        }
    }
    const M2 I{1.0, 0.0, 0.0, 1.0};
    std::vector<M2> A(G, I), B(G, I);   // propagators of whole warps
    for (int g = 0; g < G; g++)
        for (int t = 0; t < 32; t++) {
            A[g] = mul(Mf[32 * g + t], A[g]);
            B[g] = mul(Mb[32 * g + 31 - t], B[g]);
        }
    for (int g = 0; g < G; g++) {
        std::vector<M2> a(Mf.begin() + 32 * g, Mf.begin() + 32 * g + 32), b(Mb.begin() + 32 * g, Mb.begin() + 32 * g + 32);
        for (int d = 0, off = 1; d < 5; d++, off <<= 1) {
            std::vector<M2> na = a, nb = b;
            for (int t = 0; t < 32; t++) {
                for (int q = 0; q < 4; q++) {
                    out[(size_t)(tab_pf(S) + 4 * d + q) * NC + 32 * g + t] = a[t][q];
                    out[(size_t)(tab_pb(S) + 4 * d + q) * NC + 32 * g + t] = b[t][q];
                }
                if (t >= off) na[t] = mul(a[t], a[t - off]);
                if (t + off < 32) nb[t] = mul(b[t], b[t + off]);
            }
            a = na; b = nb;
        }
        M2 f = I, r = I;   // from the warp's start (end) to the chunk's
        for (int t = 0; t < 32; t++) {
            const int cf_ = 32 * g + t, cb_ = 32 * g + 31 - t;
            M2 x = f;
            for (int w = g - 1; w >= 0; w--) {   // from warp w's end to this warp's start
                for (int q = 0; q < 4; q++) out[(size_t)(tab_cf(S) + 4 * w + q) * NC + cf_] = x[q];
                x = mul(x, A[w]);
            }
            x = r;
            for (int w = g + 1; w < G; w++) {
                for (int q = 0; q < 4; q++) out[(size_t)(tab_cb(S) + 4 * (w - g - 1) + q) * NC + cb_] = x[q];
                x = mul(x, B[w]);
            }
            f = mul(Mf[cf_], f);
            r = mul(Mb[cb_], r);
        }
    }
}

// Warps per line (as log2, the table group) of a launch with `slots` sweeps in
// flight on lines of n points: one row a lane as far as four warps go, for the
// shortest line solve, and fewer warps where the sub-partitions of all SMs have more
// than a warp each, for fewer instructions in all (a line takes 4 x 59 on four
// warps, 2 x 72 on two); or what the tuner chose.  Timed at 385 x 129, three sweeps,
// the fastest is four warps at 1, 8 and 16 modes, two at 32, one at 64, as here.
int plain_group(const tb_ctx* c, int n, int itera, int slots) {
    const int tuned = itera == 1 ? c->tune_pg1 : c->tune_pg3;
    int gi = tuned ? tuned - 1 : NGROUP - 1;
    while (gi > 0 && n - 1 <= 32 * group_warps(gi - 1)) gi--;
    const int sms = c->sm_count > 0 ? c->sm_count : 148;
    if (!tuned)
        while (gi > 0 && (long)2 * c->g.K * slots * group_warps(gi) > 4L * sms) gi--;
    return gi;
}

template <int S, bool STAGED>
int launch_wsor_t(tb_ctx* c, const PlainDev& P, const Wave& V, size_t smem) {
    TB_CUDA(cudaFuncSetAttribute(k_wsor<S, STAGED>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = (unsigned)V.C; at.val.clusterDim.y = 1; at.val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)(2 * c->g.K * V.C));
    cfg.blockDim = dim3((unsigned)(32 * group_warps(V.gi) * (V.W + 1)));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = c->stream;
    cfg.attrs = &at;
    cfg.numAttrs = V.C > 1 ? 1 : 0;
    TB_CUDA(cudaLaunchKernelEx(&cfg, k_wsor<S, STAGED>, P, V));
    TB_CHECK_LAUNCH(c);
    return TB_OK;
}

template <int S>
int launch_wsor(tb_ctx* c, const PlainDev& P, const Wave& V, size_t smem) {
    return V.staged > 1 ? launch_wsor_t<S, true>(c, P, V, smem) : launch_wsor_t<S, false>(c, P, V, smem);
}

// `itera` sweeps of sor at level l (poisson_par.f:167-226) for every active
// mode, the first with relaxation factor rf0.
int plain_sor(tb_ctx* c, const PlainDev& P, int l, int itera, double rf0, double rf) {
    const int n = c->g.ptsy[l], m = c->g.ptsx[l] - 2;
    cudaEvent_t ps = nullptr;
    if (tb_prof_begin(c, PROF_SOR, &ps)) return TB_ERR_CUDA;
    for (int done = 0; done < itera;) {
        Wave V;
        std::memset(&V, 0, sizeof V);
        V.l = l; V.ns = itera - done; V.rf0 = done ? rf : rf0; V.rf = rf;
        V.C = V.W = V.parity = 1;
        V.seq = m < 7;   // border stencils and wavefront want distinct lines
        // sweeps in flight: the first ends after m - 1 steps
        const int want = V.seq ? 1 : std::min(V.ns, (m - 1 + LAG - 1) / LAG);
        V.gi = plain_group(c, n, itera, want);
        const int G = group_warps(V.gi), S = rows_per_lane(n, G), NC = 32 * G;
        // one-warp groups: three to a CTA beside the border group, the SM's four sub-partitions
        if (want > 1) {
            const int most = G == 1 ? 3 : 1;
            if (want > most) {
                V.C = 2;
                while (V.C < MAX_CLUSTER && V.C * most < want) V.C *= 2;
            }
            V.W = std::min(most, (want + V.C - 1) / V.C);
        }
        auto bytes = [&]() { return (wave_lines(V, NC, S) + (size_t)6 * G * (V.W + 1)) * sizeof(double); };
        const size_t room = (size_t)226 * 1024, table = (size_t)tab_size(n, G) * sizeof(double);
        if (!V.seq && V.ns > V.C * V.W) {   // slots run several sweeps, or the launch fewer
            if (m - 1 <= LAG * V.C * V.W) V.parity = 2;
            if (V.parity == 1 || bytes() > room) { V.parity = 1; V.ns = V.C * V.W; }
        }
        while (bytes() > room && V.W > 1) { V.W--; V.ns = std::min(V.ns, V.C * V.W); }
        V.staged = bytes() + 2 * table <= room ? 2 : bytes() + table <= room ? 1 : 0;
        for (int chunks = (n - 1 + S - 1) / S; V.lv < 5 && (1 << V.lv) < chunks;) V.lv++;
        const size_t smem = bytes() + V.staged * table;
        int r;
        switch (S) {
            case 1: r = launch_wsor<1>(c, P, V, smem); break;
            case 2: r = launch_wsor<2>(c, P, V, smem); break;
            case 3: r = launch_wsor<3>(c, P, V, smem); break;
            case 4: r = launch_wsor<4>(c, P, V, smem); break;
            case 6: r = launch_wsor<6>(c, P, V, smem); break;
            case 8: r = launch_wsor<8>(c, P, V, smem); break;
            case 12: r = launch_wsor<12>(c, P, V, smem); break;
            default: r = launch_wsor<16>(c, P, V, smem); break;
        }
        if (r) return r;
        done += V.ns;
    }
    return tb_prof_end(c, PROF_SOR, ps);
}

}  // namespace

// Times `itera` sweeps at level l with each line group in `gis`, on the plain
// form's work arrays (rebuilt from uy by every solve), and keeps the fastest.
int tb_plain_tune(tb_ctx* c, int l, int itera, const int* gis, int ngis, int* best, float* best_ms) {
    if (!c->pl_fc) { tb_set_error("plain Poisson arrays missing"); return TB_ERR_STATE; }
    PlainDev P = make_plain(c);
    cudaEvent_t a, b;
    TB_CUDA(cudaEventCreate(&a));
    TB_CUDA(cudaEventCreate(&b));
    int* keep = itera == 1 ? &c->tune_pg1 : &c->tune_pg3;
    const int old = *keep;
    *best = -1;
    *best_ms = 1e30f;
    int r = TB_OK;
    for (int q = 0; q < ngis && !r; q++) {
        *keep = gis[q] + 1;
        k_pactivate<<<tb_blocks(c->g.K, 64), 64, 0, c->stream>>>(c->pstate, c->g.K);
        r = plain_sor(c, P, l, itera, 1.0, 1.0);   // warm-up
        if (r) break;
        cudaEventRecord(a, c->stream);
        for (int rep = 0; rep < 3 && !r; rep++) r = plain_sor(c, P, l, itera, 1.0, 1.0);
        cudaEventRecord(b, c->stream);
        float ms = 0.f;
        if (!r && cudaEventSynchronize(b) == cudaSuccess) cudaEventElapsedTime(&ms, a, b);
        if (!r && ms / 3 < *best_ms) { *best_ms = ms / 3; *best = gis[q]; }
    }
    *keep = (*best >= 0) ? *best + 1 : old;
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    if (!r) TB_CUDA(cudaGetLastError());
    return r;
}

// Line-contiguous real/imaginary multigrid arrays and line-solve tables of the plain form.
int tb_plain_setup(tb_ctx* c) {
    const int K = c->g.K, ny = c->g.ny, msh = c->g.msh;
    if (ny > 32 * 16) { tb_set_error("plain Poisson: ny above 512"); return TB_ERR_ARG; }
    const size_t w = (size_t)2 * K * c->g.lvl_elems;
    for (double** p : {&c->pl_fc, &c->pl_sc, &c->pl_fct}) {
        if (*p) cudaFree(*p);
        *p = nullptr;
        TB_CUDA(cudaMalloc(p, w * sizeof(double)));
        TB_CUDA(cudaMemset(*p, 0, w * sizeof(double)));
    }
    if (c->pl_def) cudaFree(c->pl_def);
    c->pl_def = nullptr;
    const size_t d = (size_t)2 * K * c->g.nx * c->g.ny;
    TB_CUDA(cudaMalloc(&c->pl_def, d * sizeof(double)));
    TB_CUDA(cudaMemset(c->pl_def, 0, d * sizeof(double)));
    if (!c->pl_maxsq) TB_CUDA(cudaMalloc(&c->pl_maxsq, K * sizeof(unsigned long long)));
    TB_CUDA(cudaMemset(c->pl_maxsq, 0, K * sizeof(unsigned long long)));
    // band LU of the y-line matrices (band5_poi, penta_par.f:308-364), factored
    // once per (type, level, mode), with the chunk tables of each line group
    const size_t bs = tab_block(ny);
    const PlainDev P = make_plain(c);
    std::vector<double> cf((size_t)24 * msh);
    TB_CUDA(cudaMemcpy(cf.data(), c->pcoef, cf.size() * sizeof(double), cudaMemcpyDeviceToHost));
    std::vector<double> all((size_t)NGROUP * 2 * msh * K * bs, 0.0), a;
    std::vector<double> L1(ny), L2(ny), U1(ny), U2(ny), ID(ny);
    for (int type = 0; type < 2; type++)
        for (int l = 0; l < msh; l++)
            for (int k = 0; k < K; k++) {
                tb_poisson_band_matrix(c, type, l + 1, k + 1, a);
                const int n = c->g.ptsy[l];
                tb_band5_factor(n, a, L1.data(), L2.data(), U1.data(), U2.data(), ID.data());
                for (int gi = 0; gi < NGROUP; gi++) {
                    const int G = group_warps(gi);
                    double* T = &all[((((size_t)gi * 2 + type) * msh + l) * K + k) * bs];
                    group_tables(n, rows_per_lane(n, G), G, L1.data(), L2.data(), U1.data(), U2.data(), ID.data(), &cf[24 * l],
                                 P.den[l], T);
                }
            }
    if (c->pl_tab) cudaFree(c->pl_tab);
    c->pl_tab = nullptr;
    TB_CUDA(cudaMalloc(&c->pl_tab, all.size() * sizeof(double)));
    TB_CUDA(cudaMemcpy(c->pl_tab, all.data(), all.size() * sizeof(double), cudaMemcpyHostToDevice));
    return TB_OK;
}

// poi_uy (poisson_par.f:6-64), plain FP64 form.
int tb_poi_uy_k(tb_ctx* c, const cplx* dwzdx, double erro) {
    if (!c->pl_fc) { tb_set_error("plain Poisson arrays missing (context not in the plain form)"); return TB_ERR_STATE; }
    PlainDev P = make_plain(c);
    const int K = c->g.K, msh = c->g.msh;
    cudaEvent_t pall = nullptr;
    if (tb_prof_begin(c, PROF_POISSON, &pall)) return TB_ERR_CUDA;
    const double stf_pow = tb_powi(c->cfg.stf, c->g.ny - 3);
    {
        dim3 grid(tb_blocks(c->g.nx, 32), tb_blocks(c->g.ny, 32), K), blk(32, 8);
        k_psource<<<grid, blk, 0, c->stream>>>(P, c->wx, dwzdx, c->uy, c->duexmdx, c->uyb, c->cfg.beta, c->cfg.dy,
                                               stf_pow, c->cfg.my_form);
        TB_CHECK_LAUNCH(c);
    }
    k_pactivate<<<tb_blocks(K, 64), 64, 0, c->stream>>>(c->pstate, K);
    TB_CHECK_LAUNCH(c);
    std::vector<int> hs(2 * K);
    const int vmax = c->cfg.max_vcycles;
    auto defect = [&](int l, double si) {
        const int per = (c->g.ptsx[l] - 2) * (c->g.ptsy[l] - 1);
        cudaEvent_t ps = nullptr;
        if (tb_prof_begin(c, PROF_DEFECT, &ps)) return TB_ERR_CUDA;
        k_pdefect<<<dim3(tb_blocks(per, 128), K), 128, 0, c->stream>>>(P, l, si);
        TB_CHECK_LAUNCH(c);
        return tb_prof_end(c, PROF_DEFECT, ps);
    };
    int r;
    for (int v = 1; v <= vmax; v++) {
        for (int l = 0; l < msh - 1; l++) {
            // the fine level's sweep that ends the cycle before goes ahead of this one's
            const int behind = (l == 0 && v > 1) ? 1 : 0;
            if ((r = plain_sor(c, P, l, 3 + behind, behind ? 1.0 : 1.2, 1.2))) return r;
            if ((r = defect(l, -1.0))) return r;
            if (l == 0) { k_pcheck<<<tb_blocks(K, 64), 64, 0, c->stream>>>(P, erro, v); TB_CHECK_LAUNCH(c); }
            const int per = c->g.ptsx[l + 1] * c->g.ptsy[l + 1];
            k_prestrict<<<dim3(tb_blocks(per, 128), 2 * K), 128, 0, c->stream>>>(P, l);
            TB_CHECK_LAUNCH(c);
            if ((r = defect(l + 1, 1.0))) return r;
        }
        if ((r = plain_sor(c, P, msh - 1, 60, 1.2, 1.2))) return r;
        for (int l = msh - 1; l >= 1; l--) {
            const int per = (c->g.ptsx[l] - 2) * c->g.ptsy[l];
            k_pcorrection<<<dim3(tb_blocks(per, 128), 2 * K), 128, 0, c->stream>>>(P, l);
            TB_CHECK_LAUNCH(c);
            const int perf = (c->g.ptsx[l - 1] - 2) * c->g.ptsy[l - 1];
            k_pintpol<<<dim3(tb_blocks(perf, 128), 2 * K), 128, 0, c->stream>>>(P, l);
            TB_CHECK_LAUNCH(c);
            if (l > 1 || v == vmax)
                if ((r = plain_sor(c, P, l - 1, 1, 1.0, 1.0))) return r;
        }
        TB_CUDA(cudaMemcpyAsync(hs.data(), c->pstate, 2 * K * sizeof(int), cudaMemcpyDeviceToHost, c->stream));
        TB_CUDA(cudaStreamSynchronize(c->stream));
        bool any = false;
        for (int k = 0; k < K; k++) any = any || hs[2 * k];
        if (!any) break;
    }
    {
        dim3 grid(tb_blocks(c->g.nx, 32), tb_blocks(c->g.ny, 32), K), blk(32, 8);
        k_pwrite_uy<<<grid, blk, 0, c->stream>>>(P, c->uy);
        TB_CHECK_LAUNCH(c);
    }
    if (tb_prof_end(c, PROF_POISSON, pall)) return TB_ERR_CUDA;
    std::vector<double> he(K);
    TB_CUDA(cudaMemcpyAsync(hs.data(), c->pstate, 2 * K * sizeof(int), cudaMemcpyDeviceToHost, c->stream));
    TB_CUDA(cudaMemcpyAsync(he.data(), c->perr, K * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
    TB_CUDA(cudaStreamSynchronize(c->stream));
    c->stats.noconv = 0;
    int nonfinite = 0;
    for (int k = 0; k < K && k < 256; k++) {
        int vc = hs[2 * k + 1];
        if (hs[2 * k]) { vc = vmax; c->stats.noconv++; }
        if (vc < 0) { nonfinite = 1; vc = -vc - 1; }
        c->stats.vcycles[k] = vc;
        c->stats.residual[k] = he[k];
        c->stats.total_vcycles += vc;
    }
    c->stats.solves++;
    if (nonfinite) { tb_set_error("poi_uy: non-finite defect"); return TB_ERR_NONFINITE; }
    return TB_OK;
}
