// tb_cycle.cuh -- the FP32 V-cycles of one FP64 correction (included by
// tb_mixed.cu): two kernels per level and the coarsest solve.
//
// A kernel per relaxation colour (91 launches a V-cycle) reads and writes its
// lines through L2 nine times a level, and a line's chain of loads and
// recurrences leaves the SMs waiting: 27.7 ms of a 68.9 ms step at 1025 x 193,
// 32 modes; one cluster per mode with a barrier per phase, the fields still in
// L2, was no faster (26.7 ms).  So a CTA keeps a strip of lines in registers
// through everything a level does on the way down (relaxation sweeps,
// residual, restriction) or up (prolongation, sweeps); only the right-hand side
// streams by, loaded one colour ahead: 19.1 ms, 13 launches a V-cycle.  What
// bounds these kernels is the latency of a colour's phases (recurrences, carry,
// barriers) with the one CTA an SM's registers hold.
//
// Layout.  A level's lines are split by colour: line i = 3t + c - 1 is
// element t of colour plane c (c = (i+1) mod 3); row j of plane c starts at
// off + (c*np + j + 1)*T.  One leading and trailing pad rows per plane, the
// columns beyond the domain and the Dirichlet points (row 0, lines 0 and
// nx-1) hold zeros that nothing writes.
//
// Strips (k_down, k_up).  Lane t of every warp holds the lines 3t-1, 3t, 3t+1
// of its strip, warp w the rows w S .. w S + S - 1 of them: e of 96 lines in
// the registers of one CTA.  A centre line's neighbours i+-1, i+-2 lie in the
// two other planes, in the same lane or one aside, so the x-stencils are
// shuffles.  A sweep spoils the strip's outer lanes (one on the left, two on
// the right), which the adjoining strips compute as their own: strips overlap
// instead of exchanging values, and e goes from one buffer to another.  Up to 7
// rows a warp the registers hold it all; k_down spills 0.4, 0.5 and 1.0 KB a thread
// at 9, 13 and 17 rows, and beyond (272 rows in all) tb_tall.cuh takes over.
//
// Line solves.  The NW warps own NW row chunks of S rows each.  Local
// recurrences with zero carry in registers, chunk-end states exchanged through
// shared memory, the warps' 2x2 chunk propagators chained in two levels
// (within groups of four warps, then over the groups), and the rows fixed up
// with precomputed homogeneous responses.  The row tables are the same for all
// lanes (broadcast reads).  Real and imaginary part go through the packed
// FP32 pairs of sm_100 (fma.rn.f32x2), whose coefficients are stored twice.
#pragma once
#include "tb_internal.h"

namespace mg {

constexpr int NW = 16;                 // warps per CTA = row chunks per line
constexpr int NT = 32 * NW;
constexpr int MAX_LEVELS = 16;
constexpr int DIRECT_LIMIT = 2048;     // largest directly solved level accepted
constexpr int ROW4 = 6;                // float4 per row of the line-solve tables (12 coefficients, twice)
constexpr int MATS = 2 * NW + NW / 4;  // propagators per direction: chunk, chunk prefix in its group, group
constexpr int PROP4 = 2 * 2 * MATS;    // float4 of propagators per line type and level
constexpr int RES4 = 4;                // float4 per residual row (8 coefficients, twice)
// Shared memory: the exchange buffer of the line solves (chunk states and
// group states of both directions), the centre and border tables with the
// residual rows, the chunks' two first and two last rows of each plane, the
// border lines' values and right-hand sides.
constexpr int XDIR4 = 32 * (NW + NW / 4);   // one direction
constexpr int TAB4 = 2 * XDIR4;        // float4 offset of the tables
constexpr int EDGE_C2 = 3 * NW * 4 * 32;

struct Level {
    int nx, n;          // lines, rows
    int T, np;          // global layout: row pitch, rows per plane
    int S;              // rows per chunk
    int semi;           // coarsening to the next level in x only
    int down, up;       // strips of k_down, k_up
    int tab;            // float4 offset of its tables in a mode's block: centre rows and propagators, border rows
                        // and propagators, residual rows
    int off;            // float2 offset in a mode's block
};

struct Cycle {
    float2 *ea, *eb, *r;   // e after the way down, after the way up; right-hand side
    const float4* tab;     // per mode: the levels' tables
    const float* ainv;     // (K, N, N) inverse of the coarsest operator per mode
    const int* state;      // per mode: [2k] active
    size_t elems, tab4;    // per-mode block sizes (float2, float4)
    int K, NL, N;
    int nu_pre, nu_post;
    Level lv[MAX_LEVELS];
};
// float4 of a level's line tables of one line type, and of all its tables
__host__ __device__ __forceinline__ int line4(const Level& L) { return ROW4 * NW * L.S + PROP4; }
__host__ __device__ __forceinline__ int level4(const Level& L) { return 2 * line4(L) + RES4 * L.n; }

// Offset of element (i, j) of a level in a mode's block.
__host__ __device__ __forceinline__ int el(const Level& L, int i, int j) {
    const int q = i + 1, t = q / 3;
    return L.off + ((q - 3 * t) * L.np + j + 1) * L.T + t;
}

// Strips of 32 elements over T: `nu` sweeps spoil nu lanes on the left and
// 2 nu on the right (and `more` on either side), except at the domain's ends.
__host__ __device__ __forceinline__ int strip_start(int q, int nu, int more) {   // first element whose result the strip keeps
    return q == 0 ? 0 : (32 - 2 * nu - more) + (q - 1) * (32 - 3 * nu - 2 * more);
}
inline int strips(int T, int nu, int more) {
    if (T <= 32) return 1;
    int q = 2;
    while (strip_start(q - 1, nu, more) + 32 - nu - more < T) q++;
    return q;
}

// Rows per chunk: the smallest instantiated S with NW * S >= n (n <= 272:
// taller levels are those of tb_tall.cuh).
inline int pick_rows(int n) {
    static const int opts[] = {2, 4, 5, 7, 9, 13};
    for (int s : opts)
        if (NW * s >= n) return s;
    return 17;
}

#ifdef __CUDACC__
// Pairs of FP32 values (re, im) in one 64-bit register.
typedef unsigned long long c2;
__device__ __forceinline__ c2 pk(float a, float b) {
    c2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 un(c2 a) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
    return r;
}
__device__ __forceinline__ c2 fma2(c2 a, c2 b, c2 c) {
    c2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ c2 mul2(c2 a, c2 b) {
    c2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ c2 add2(c2 a, c2 b) {
    c2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ c2 dup(float a) { return pk(a, a); }

// Tables in shared memory as pairs (coefficient q of a row at 2 q floats).
struct Tab {
    int o;
    __device__ __forceinline__ ulonglong2 two(int q) const {
        extern __shared__ float4 smem4[];
        return reinterpret_cast<const ulonglong2*>(smem4)[o + q];
    }
    __device__ __forceinline__ c2 one(int q, int h) const {
        extern __shared__ float4 smem4[];
        return reinterpret_cast<const c2*>(smem4)[2 * (o + q) + h];
    }
};

__device__ __forceinline__ void step2(c2& z0, c2& z1, const ulonglong2& b, const ulonglong2& m0, const ulonglong2& m1) {
    const c2 n0 = fma2(m0.y, z1, fma2(m0.x, z0, b.x));
    z1 = fma2(m1.y, z1, fma2(m1.x, z0, b.y));
    z0 = n0;
}

// State entering this warp's chunk from the chunk-end states (p1, p2) of the
// warps before it (after it for DOWN), in two levels: within the group of four
// warps, then over the groups' totals.  prop: the direction's propagators.
template <bool DOWN>
__device__ __forceinline__ void carry(const Tab& tab, int prop, c2 p1, c2 p2, c2& z0, c2& z1) {
    extern __shared__ float4 smem4[];
    ulonglong2* xch = reinterpret_cast<ulonglong2*>(smem4) + (DOWN ? XDIR4 : 0);
    ulonglong2* tot = xch + NW * 32;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, v = DOWN ? NW - 1 - w : w;   // place in the direction
    const int g = v >> 2, h = v & 3;
    auto mat = [&](int q, ulonglong2& m0, ulonglong2& m1) { m0 = tab.two(prop + 2 * q); m1 = tab.two(prop + 2 * q + 1); };
    xch[v * 32 + lane] = make_ulonglong2(p1, p2);
    __syncthreads();
    c2 l0 = 0, l1 = 0;
    ulonglong2 a0, a1;
    for (int q = 4 * g; q < v; q++) {
        mat(q, a0, a1);
        step2(l0, l1, xch[q * 32 + lane], a0, a1);
    }
    if (h == 3) {
        c2 t0 = l0, t1 = l1;
        mat(v, a0, a1);
        step2(t0, t1, make_ulonglong2(p1, p2), a0, a1);
        tot[g * 32 + lane] = make_ulonglong2(t0, t1);
    }
    __syncthreads();
    z0 = 0;
    z1 = 0;
    for (int q = 0; q < g; q++) {
        mat(2 * NW + q, a0, a1);
        step2(z0, z1, tot[q * 32 + lane], a0, a1);
    }
    mat(NW + v, a0, a1);
    step2(z0, z1, make_ulonglong2(l0, l1), a0, a1);
}

// Forward recurrence of one chunk, fed with the x-stencil sums of rows r0-1,
// r0, ... in order; y holds the right-hand sides of the chunk's rows.
template <int S>
struct Forward {
    const Tab& tab;
    int tr;
    c2 (&y)[S];
    c2 gm, g0, p1, p2;
    __device__ __forceinline__ Forward(const Tab& t, int r0, c2 (&yy)[S]) : tab(t), tr(ROW4 * r0), y(yy), gm(0), g0(0), p1(0), p2(0) {}
    __device__ __forceinline__ void feed(int q, c2 gp) {   // sum of row r0 - 1 + q
        if (q >= 2) {
            const int s = q - 2;
            const ulonglong2 a = tab.two(tr + ROW4 * s), b = tab.two(tr + ROW4 * s + 1);   // wm w0 | wp -l1
            c2 v = fma2(a.x, gm, y[s]);
            v = fma2(a.y, g0, v);
            v = fma2(b.x, gp, v);
            v = fma2(tab.one(tr + ROW4 * s + 2, 0), p2, v);                                // -l2
            v = fma2(b.y, p1, v);
            y[s] = v;
            p2 = p1; p1 = v;
        }
        gm = g0; g0 = gp;
    }
};

// The rest of the solve: y from the chunk's forward values to the solution.
// The tables give 0 on row 0 and on the pad rows.
template <int S>
__device__ __forceinline__ void finish_rows(const Tab& tab, c2 (&y)[S], c2 p1, c2 p2, int r0) {
    const int tr = ROW4 * r0, prop = ROW4 * NW * S;
    c2 z0, z1;
    carry<false>(tab, prop, p1, p2, z0, z1);
    p1 = 0; p2 = 0;
#pragma unroll
    for (int s = S - 1; s >= 0; s--) {
        const ulonglong2 b = tab.two(tr + ROW4 * s + 3), c = tab.two(tr + ROW4 * s + 4);   // h2/d -u1/d | -u2/d 1/d
        c2 v = mul2(c.y, y[s]);
        v = fma2(tab.one(tr + ROW4 * s + 2, 1), z0, v);                                    // h1/d
        v = fma2(b.x, z1, v);
        v = fma2(c.x, p2, v);
        v = fma2(b.y, p1, v);
        y[s] = v;
        p2 = p1; p1 = v;
    }
    carry<true>(tab, prop + 2 * MATS, p1, p2, z0, z1);
#pragma unroll
    for (int s = 0; s < S; s++) {
        const ulonglong2 k = tab.two(tr + ROW4 * s + 5);
        y[s] = fma2(k.y, z1, fma2(k.x, z0, y[s]));
    }
}

// ---- strips -----------------------------------------------------------------
// x-stencil sum of plane C's line in this lane, in units of 16: f[i-1] +
// f[i+1] - (f[i-2] + f[i+2]) / 16 (rhs_center, poisson_par.f:229-540), from
// the row's values of the three planes.
template <int C>
__device__ __forceinline__ c2 xsum(c2 f0, c2 f1, c2 f2, c2 m16) {
    if (C == 0) return add2(fma2(m16, f2, f1), __shfl_up_sync(0xffffffffu, fma2(m16, f1, f2), 1));
    if (C == 1) return fma2(m16, add2(__shfl_up_sync(0xffffffffu, f2, 1), __shfl_down_sync(0xffffffffu, f0, 1)), add2(f2, f0));
    return add2(fma2(m16, f0, f1), __shfl_down_sync(0xffffffffu, fma2(m16, f1, f0), 1));
}

template <int S>
struct Strip {
    c2 e[3][S];
    int lane, w, r0;
    int t;              // this lane's element
    int T, np, nx, n, Tn;
    bool ends;          // the strip holds an end of the domain (uniform over the CTA)
    bool lo, hi;        // which
    bool own;           // this lane holds a border line,
    int bp, bs;         // in this plane, of this side (0: line 1, 1: line nx-2)
    int cR;             // plane of line nx-2
    c2* edge;           // [plane][warp][first, second, last but one, last][lane]
    c2* bval;           // border lines' values, then their right-hand sides, [side][row]

    __device__ __forceinline__ void setup(const Level& L, int q, int nu, int more, c2* edge_, c2* bval_) {
        lane = threadIdx.x & 31; w = threadIdx.x >> 5; r0 = w * S;
        T = L.T; np = L.np; nx = L.nx; n = L.n; Tn = L.nx / 3 + 1;
        const int a = strip_start(q, nu, more) - (q ? nu + more : 0);
        t = a + lane;
        lo = a == 0; hi = 3 * (a + 31) + 1 > nx - 3; ends = lo || hi;
        cR = (nx - 1) % 3;
        const bool o1 = t == 0, o2 = t == (nx - 1) / 3;   // line 1 is in plane 2, line nx-2 in cR
        own = o1 || o2; bs = o2; bp = o2 ? cR : 2;
        edge = edge_; bval = bval_;
    }
    __device__ __forceinline__ c2* edges(int c, int ww, int q) const { return edge + ((c * NW + ww) * 4 + q) * 32; }
    // a plane's chunk-end rows for the warps above and below
    template <int C>
    __device__ __forceinline__ void publish() {
        edges(C, w, 0)[lane] = e[C][0];
        edges(C, w, 3)[lane] = e[C][S - 1];
    }
    // row -1 (UP false) or row S (UP true) of the chunk in a plane
    template <bool UP>
    __device__ __forceinline__ c2 beyond(int c) const {
        if (UP) return w < NW - 1 ? edges(c, w + 1, 0)[lane] : 0;
        return w > 0 ? edges(c, w - 1, 3)[lane] : 0;
    }
    template <int C>
    __device__ __forceinline__ void load(const c2* p) {   // p: the level's array
        const c2* q = p + (C * np + r0 + 1) * T + t;
        const bool ok = t < Tn;
#pragma unroll
        for (int s = 0; s < S; s++) e[C][s] = ok ? q[s * T] : 0;
    }
    // lines that are not centre lines keep what they had: the border lines
    // their last solution, the Dirichlet lines and those beyond 0
    template <int C>
    __device__ __forceinline__ void restore_ends() {
        const int i = 3 * t + C - 1;
        if (i >= 2 && i <= nx - 3) return;
        const bool b = own && bp == C;
        const c2* v = bval + bs * NW * S + r0;
#pragma unroll
        for (int s = 0; s < S; s++) e[C][s] = b ? v[s] : 0;
    }
    // one colour: e[C] holds the right-hand side; nxt is loaded once its old
    // values are dead
    template <int C>
    __device__ __forceinline__ void colour(const Tab& tab, const c2* rnext) {
        const c2 m16 = dup(-0.0625f);
        constexpr int A = C == 0 ? 1 : 0, B = C == 2 ? 1 : 2;
        auto sum = [&](c2 a, c2 b) { return C == 0 ? xsum<0>(0, a, b, m16) : C == 1 ? xsum<1>(a, 0, b, m16) : xsum<2>(a, b, 0, m16); };
        Forward<S> fw(tab, r0, e[C]);
        const c2 ha = beyond<true>(A), hb = beyond<true>(B);
        fw.feed(0, sum(beyond<false>(A), beyond<false>(B)));
#pragma unroll
        for (int s = 0; s < S; s++) fw.feed(s + 1, sum(e[A][s], e[B][s]));
        fw.feed(S + 1, sum(ha, hb));
        constexpr int N = (C + 1) % 3;
        if (rnext) load<N>(rnext);
        finish_rows<S>(tab, e[C], fw.p1, fw.p2, r0);
        if (ends) restore_ends<C>();
        publish<C>();
        __syncthreads();
    }
    // one-sided x-stencil of a border line (without its diagonal; the line
    // outside holds 0): -4 f[i+1] + 14 f[i+2] - 6 f[i+3] + f[i+4] (mirrored at
    // nx-2; rhs_border, poisson_par.f:229-540) from a row's values of the
    // three planes, valid in the lanes that hold a border line
    __device__ __forceinline__ c2 border_sum(c2 f0, c2 f1, c2 f2) const {
        const c2 a = dup(-4.f), b = dup(14.f), d = dup(-6.f);
        const unsigned all = 0xffffffffu;
        c2 g = 0;
        if (lo) {   // lines 2, 3, 4 are one lane up, line 5 two
            const c2 v = add2(fma2(a, f0, fma2(b, f1, mul2(d, f2))), __shfl_down_sync(all, f0, 1));
            g = __shfl_down_sync(all, v, 1);
        }
        if (hi) {
            c2 v;
            if (cR == 0) v = __shfl_up_sync(all, add2(fma2(a, f2, fma2(b, f1, mul2(d, f0))), __shfl_up_sync(all, f2, 1)), 1);
            else if (cR == 1) v = fma2(a, f0, __shfl_up_sync(all, fma2(b, f2, fma2(d, f1, f0)), 1));
            else v = fma2(a, f1, fma2(b, f0, __shfl_up_sync(all, fma2(d, f2, f1), 1)));
            if (bs) g = v;
        }
        return g;
    }
    // relax the border lines of the strip, both at once, each in its own
    // lane (line nx-2 may share lane 0 with line 1 only on grids below nx = 5);
    // r_0 is loaded once plane 0 is dead
    __device__ __forceinline__ void border(const Tab& tab, const c2* r) {
        c2 y[S];
        const c2* v = bval + (2 + bs) * NW * S + r0;
#pragma unroll
        for (int s = 0; s < S; s++) y[s] = own ? v[s] : 0;
        Forward<S> fw(tab, r0, y);
        fw.feed(0, border_sum(beyond<false>(0), beyond<false>(1), beyond<false>(2)));
#pragma unroll
        for (int s = 0; s < S; s++) fw.feed(s + 1, border_sum(e[0][s], e[1][s], e[2][s]));
        fw.feed(S + 1, border_sum(beyond<true>(0), beyond<true>(1), beyond<true>(2)));
        load<0>(r);
        finish_rows<S>(tab, y, fw.p1, fw.p2, r0);
        if (own) {
            c2* u = bval + bs * NW * S + r0;
#pragma unroll
            for (int s = 0; s < S; s++) {
                u[s] = y[s];
                if (bp == 1) e[1][s] = y[s];
                if (bp == 2) e[2][s] = y[s];
            }
        }
        publish<1>(); publish<2>();   // plane 0 follows with its colour
        __syncthreads();
    }
    // right-hand sides of the border lines into shared memory
    __device__ __forceinline__ void border_rhs(const c2* r) {
        if (!own) return;
        const c2* q = r + (bp * np + r0 + 1) * T + t;
        c2* u = bval + (2 + bs) * NW * S + r0;
#pragma unroll
        for (int s = 0; s < S; s++) u[s] = q[s * T];
    }
    // `nu` sweeps: the border lines, then the colours in order.  e of all planes
    // on entry and on return.
    __device__ __forceinline__ void sweeps(int nu, const Tab& tab, const Tab& btab, const c2* r) {
        if (ends) border_rhs(r);
        publish<0>(); publish<1>(); publish<2>();
        __syncthreads();
        if (!ends) load<0>(r);
        for (int q = 0; q < nu; q++) {
            if (ends) border(btab, r);
            colour<0>(tab, r);
            colour<1>(tab, r);
            colour<2>(tab, (!ends && q + 1 < nu) ? r : nullptr);
        }
    }
    __device__ __forceinline__ bool kept(int q, int nu, int more, int next) const {   // this strip's own elements
        return t >= strip_start(q, nu, more) && t < next && t < Tn;
    }
    template <int C>
    __device__ __forceinline__ void store(c2* p, bool ok) {
        const int i = 3 * t + C - 1;
        if (!ok || i < 1 || i > nx - 2) return;
        c2* q = p + (C * np + r0 + 1) * T + t;
#pragma unroll
        for (int s = 0; s < S; s++)
            if (r0 + s < n) q[s * T] = e[C][s];
    }
};

__device__ __forceinline__ c2* past_tables(const Level& L) {
    extern __shared__ float4 smem4[];
    return reinterpret_cast<c2*>(smem4 + TAB4 + level4(L));
}
inline size_t strip_bytes(const Level& L) {
    return ((size_t)TAB4 + level4(L)) * sizeof(float4) + ((size_t)EDGE_C2 + 4 * NW * L.S) * sizeof(float2);
}
// A level's tables into shared memory.
__device__ __forceinline__ void stage(const Level& L, const float4* tabg) {
    extern __shared__ float4 smem4[];
    for (int q = threadIdx.x; q < level4(L); q += NT) smem4[TAB4 + q] = __ldg(tabg + L.tab + q);
}

// Down a level: nu_pre sweeps from e = 0 (or from eb where `from`), e into ea,
// the restricted residual into r of the next level: full weighting in x
// (1/4, 1/2, 1/4) and, where the rows are halved too, in y (restrict,
// poisson_par.f:796-874; the top row from the fine top row alone).  The
// coarse lines of a lane follow from t's parity: t = 2m holds the coarse line
// 3m, t = 2m + 1 the coarse lines 3m + 1 and 3m + 2, whose outer fine lines
// are one lane aside.
template <int S>
__global__ void __launch_bounds__(NT, S <= 4 ? 2 : 1) k_down(const __grid_constant__ Cycle M, int l, int from) {
    const int k = blockIdx.y;
    if (!M.state[2 * k]) return;
    const Level &L = M.lv[l], &N = M.lv[l + 1];
    const float4* tabg = M.tab + (size_t)k * M.tab4;
    const c2* r = reinterpret_cast<const c2*>(M.r) + (size_t)k * M.elems + L.off;
    c2* rn = reinterpret_cast<c2*>(M.r) + (size_t)k * M.elems + N.off;
    c2* ea = reinterpret_cast<c2*>(M.ea) + (size_t)k * M.elems + L.off;
    stage(L, tabg);
    c2* sm = past_tables(L);
    extern __shared__ float4 smem4[];
    c2* strad = reinterpret_cast<c2*>(smem4);   // the exchange buffer, free after the sweeps
    Strip<S> X;
    X.setup(L, blockIdx.x, M.nu_pre, 1, sm, sm + EDGE_C2);
    const bool ok = X.kept(blockIdx.x, M.nu_pre, 1, blockIdx.x + 1 < L.down ? strip_start(blockIdx.x + 1, M.nu_pre, 1) : X.Tn);
    if (from) {
        const c2* eb = reinterpret_cast<const c2*>(M.eb) + (size_t)k * M.elems + L.off;
        X.template load<0>(eb); X.template load<1>(eb); X.template load<2>(eb);
    } else {
#pragma unroll
        for (int s = 0; s < S; s++) { X.e[0][s] = 0; X.e[1][s] = 0; X.e[2][s] = 0; }
    }
    const Tab tab{TAB4}, btab{TAB4 + line4(L)}, res{TAB4 + 2 * line4(L)};
    X.sweeps(M.nu_pre, tab, btab, r);
    X.template store<0>(ea, ok); X.template store<1>(ea, ok); X.template store<2>(ea, ok);
    // two rows of every plane around the chunk
    const int lane = X.lane, w = X.w, r0 = X.r0, t = X.t;
    __syncthreads();
#pragma unroll
    for (int c = 0; c < 3; c++) {
        X.edges(c, w, 0)[lane] = X.e[c][0];
        X.edges(c, w, 1)[lane] = X.e[c][S > 1 ? 1 : 0];
        X.edges(c, w, 2)[lane] = X.e[c][S > 1 ? S - 2 : 0];
        X.edges(c, w, 3)[lane] = X.e[c][S - 1];
    }
    __syncthreads();
    auto val = [&](int c, int s) -> c2 {   // row r0 + s of plane c, s = -2 .. S + 1
        if (s < 0) return w > 0 ? X.edges(c, w - 1, s + 4)[lane] : 0;
        if (s >= S) return w < NW - 1 ? X.edges(c, w + 1, s - S)[lane] : 0;
        return X.e[c][s];
    };
    const c2 m16 = dup(-0.0625f), k2 = dup(2.f);
    auto bx = [&](int s, c2 (&b)[3]) {     // x-stencil sums of the row, units of 16
        const c2 f0 = val(0, s), f1 = val(1, s), f2 = val(2, s);
        b[0] = xsum<0>(f0, f1, f2, m16); b[1] = xsum<1>(f0, f1, f2, m16); b[2] = xsum<2>(f0, f1, f2, m16);
        if (X.ends) {   // the border lines' one-sided stencils; + 15 f makes up for the folded diagonal (-15 instead of -30)
            const c2 g = X.border_sum(f0, f1, f2);
#pragma unroll
            for (int c = 0; c < 3; c++)
                if (X.own && X.bp == c) b[c] = mul2(dup(0.0625f), fma2(dup(15.f), c == 0 ? f0 : c == 1 ? f1 : f2, g));
        }
    };
    const bool odd = t & 1;
    const int Ia = odd ? (3 * t - 1) / 2 : 3 * t / 2, Ib = (3 * t + 1) / 2;   // coarse lines (b: odd lanes only)
    const bool oka = ok && Ia >= 1 && Ia <= N.nx - 2, okb = ok && odd && Ib >= 1 && Ib <= N.nx - 2;
    c2* pa = rn + ((Ia + 1) % 3 * N.np + 1) * N.T + (Ia + 1) / 3;   // row 0
    c2* pb = rn + ((Ib + 1) % 3 * N.np + 1) * N.T + (Ib + 1) / 3;
    c2 bm[3], b0[3], bp[3];
    bx(-1, bm);
    bx(0, b0);
    const int T = L.T;
    const c2* pr = r + (size_t)(r0 + 1) * T + t;
    const bool in = t < X.Tn;
    c2 aa = 0, ab = 0, ka = 0, kb = 0;   // coarse row under way; this chunk's share of the row before it
#pragma unroll
    for (int s = 0; s < S; s++) {
        const int j = r0 + s;
        bx(s + 1, bp);
        c2 d[3];
#pragma unroll
        for (int c = 0; c < 3; c++) d[c] = in ? pr[(c * L.np + s) * T] : 0;
        c2 va = 0, vb = 0;
        if (j >= 1 && j < L.n) {   // uniform over the warp
            const ulonglong2 a = res.two(RES4 * j), b = res.two(RES4 * j + 1), e = res.two(RES4 * j + 2), g = res.two(RES4 * j + 3);
#pragma unroll
            for (int c = 0; c < 3; c++) {
                c2 v = fma2(a.x, bm[c], d[c]);
                v = fma2(a.y, b0[c], v);
                v = fma2(b.x, bp[c], v);
                v = fma2(b.y, val(c, s - 2), v);
                v = fma2(e.x, val(c, s - 1), v);
                v = fma2(e.y, val(c, s), v);
                v = fma2(g.x, val(c, s + 1), v);
                d[c] = fma2(g.y, val(c, s + 2), v);
            }
        }
        const c2 up = __shfl_up_sync(0xffffffffu, d[2], 1), dn = __shfl_down_sync(0xffffffffu, d[0], 1);
        va = odd ? fma2(k2, d[0], add2(up, d[1])) : fma2(k2, d[1], add2(d[0], d[2]));
        vb = fma2(k2, d[2], add2(d[1], dn));
#pragma unroll
        for (int c = 0; c < 3; c++) { bm[c] = b0[c]; b0[c] = bp[c]; }
        if (j < 1 || j >= L.n) continue;
        if (L.semi) {
            if (oka) pa[j * N.T] = mul2(dup(0.25f), va);
            if (okb) pb[j * N.T] = mul2(dup(0.25f), vb);
        } else if (j == L.n - 1) {
            if (oka) pa[(N.n - 1) * N.T] = mul2(dup(0.25f), va);
            if (okb) pb[(N.n - 1) * N.T] = mul2(dup(0.25f), vb);
        } else if (j & 1) {        // completes coarse row (j-1)/2, begins (j+1)/2
            const int J = (j - 1) / 2;
            if (2 * J - 1 < r0) { ka = add2(aa, va); kb = add2(ab, vb); }   // it began in the chunk below
            else if (J >= 1) {
                if (oka) pa[J * N.T] = mul2(dup(0.0625f), add2(aa, va));
                if (okb) pb[J * N.T] = mul2(dup(0.0625f), add2(ab, vb));
            }
            aa = va; ab = vb;
        } else {
            aa = fma2(k2, va, aa); ab = fma2(k2, vb, ab);
        }
    }
    if (!L.semi) {
        // the coarse row that straddles the chunk's upper end: its rest comes
        // from the chunk above (whose first odd row completes it)
        strad[(w * 2) * 32 + lane] = ka;
        strad[(w * 2 + 1) * 32 + lane] = kb;
        __syncthreads();
        const int je = r0 + S, J = je / 2;   // rows 2J-1, 2J, 2J+1 with 2J-1 < je <= 2J+1
        if (w < NW - 1 && J >= 1 && J <= N.n - 2 && 2 * J - 1 >= r0 && 2 * J - 1 < je) {
            if (oka) pa[J * N.T] = mul2(dup(0.0625f), add2(aa, strad[((w + 1) * 2) * 32 + lane]));
            if (okb) pb[J * N.T] = mul2(dup(0.0625f), add2(ab, strad[((w + 1) * 2 + 1) * 32 + lane]));
        }
    }
}

// Up to a level: e = ea + interpolation of eb of the next level, linear in x
// and, where the rows are halved, in y (intpol, poisson_par.f:877-920), then
// nu_post sweeps, into eb.  With X, Y, Z the coarse planes 0, 1, 2 at (t+1)/2,
// t/2, t/2 the fine lines of lane t are (X+Y)/2, Y, (Y+Z)/2 for even and Z,
// (Z+X)/2, X for odd t.
template <int S>
__global__ void __launch_bounds__(NT, S <= 4 ? 2 : 1) k_up(const __grid_constant__ Cycle M, int l) {
    const int k = blockIdx.y;
    if (!M.state[2 * k]) return;
    const Level &L = M.lv[l], &N = M.lv[l + 1];
    const float4* tabg = M.tab + (size_t)k * M.tab4;
    const c2* r = reinterpret_cast<const c2*>(M.r) + (size_t)k * M.elems + L.off;
    const c2* ea = reinterpret_cast<const c2*>(M.ea) + (size_t)k * M.elems + L.off;
    const c2* en = reinterpret_cast<const c2*>(M.eb) + (size_t)k * M.elems + N.off;
    c2* eb = reinterpret_cast<c2*>(M.eb) + (size_t)k * M.elems + L.off;
    stage(L, tabg);
    c2* sm = past_tables(L);
    Strip<S> X;
    X.setup(L, blockIdx.x, M.nu_post, 0, sm, sm + EDGE_C2);
    const bool ok = X.kept(blockIdx.x, M.nu_post, 0, blockIdx.x + 1 < L.up ? strip_start(blockIdx.x + 1, M.nu_post, 0) : X.Tn);
    X.template load<0>(ea); X.template load<1>(ea); X.template load<2>(ea);
    const int t = X.t, r0 = X.r0;
    if (t < X.Tn) {
        const c2 half = dup(0.5f);
        const c2 *px = en + N.T + (t + 1) / 2, *py = en + (N.np + 1) * N.T + t / 2, *pz = en + (2 * N.np + 1) * N.T + t / 2;
        const bool odd = t & 1;
#pragma unroll
        for (int s = 0; s < S; s++) {
            const int j = r0 + s;
            if (j < L.n) {   // uniform over the warp
                c2 x, y, z;
                if (L.semi) { x = px[j * N.T]; y = py[j * N.T]; z = pz[j * N.T]; }
                else {
                    const int a = (j / 2) * N.T, b = ((j + 1) / 2) * N.T;
                    x = mul2(half, add2(px[a], px[b])); y = mul2(half, add2(py[a], py[b])); z = mul2(half, add2(pz[a], pz[b]));
                }
                X.e[0][s] = add2(X.e[0][s], odd ? z : mul2(half, add2(x, y)));
                X.e[1][s] = add2(X.e[1][s], odd ? mul2(half, add2(z, x)) : y);
                X.e[2][s] = add2(X.e[2][s], odd ? x : mul2(half, add2(y, z)));
            }
        }
    }
    __syncthreads();
    X.sweeps(M.nu_post, Tab{TAB4}, Tab{TAB4 + line4(L)}, r);
    X.template store<0>(eb, ok); X.template store<1>(eb, ok); X.template store<2>(eb, ok);
}

// Exact solve on the coarsest level: eb = A^{-1} r, four rows at a time per
// warp.  Unknown q is the interior point (1 + q / (n-1), 1 + q % (n-1)).
__global__ void __launch_bounds__(NT) k_direct(const __grid_constant__ Cycle M) {
    __shared__ c2 rs[DIRECT_LIMIT];
    const int k = blockIdx.y;
    if (!M.state[2 * k]) return;
    const Level& Z = M.lv[M.NL - 1];
    const int N = M.N, m = Z.n - 1, lane = threadIdx.x & 31;
    const c2* r = reinterpret_cast<const c2*>(M.r) + (size_t)k * M.elems;
    c2* e = reinterpret_cast<c2*>(M.eb) + (size_t)k * M.elems;
    const float* ainv = M.ainv + (size_t)k * N * N;
    auto at = [&](int q) { return el(Z, 1 + q / m, 1 + q % m); };
    for (int q = threadIdx.x; q < N; q += NT) rs[q] = r[at(q)];
    __syncthreads();
    constexpr int V = 4;
    const int p0 = V * (blockIdx.x * NW + (threadIdx.x >> 5));
    if (p0 >= N) return;
    const float* A[V];
    c2 s[V];
#pragma unroll
    for (int u = 0; u < V; u++) { A[u] = ainv + (size_t)min(p0 + u, N - 1) * N; s[u] = 0; }
#pragma unroll 4
    for (int q = lane; q < N; q += 32) {
        const c2 v = rs[q];
#pragma unroll
        for (int u = 0; u < V; u++) s[u] = fma2(dup(__ldg(A[u] + q)), v, s[u]);
    }
#pragma unroll
    for (int u = 0; u < V; u++) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s[u] = add2(s[u], __shfl_xor_sync(0xffffffffu, s[u], o));
        if (lane == 0 && p0 + u < N) e[at(p0 + u)] = s[u];
    }
}
#endif

}  // namespace mg
