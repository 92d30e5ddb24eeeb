// tb_xline.cuh -- one compact x-line solve on one warp (derparx/derparxx,
// derivs_par.f:80-113 with rhsx/rhsxx 259-397 and tridparx 775-858;
// filter_trid, filter_par.f:144-332), shared by the stage's batched lines
// (tb_deriv.cu) and the allocation-free filter (tb_noalloc.cu).
//
// An FP64 warp instruction holds its pipe for 64 cycles, so their number sets
// the time of a line.  The right-hand side is formed in units kappa in which
// one of its weights is 1 (D1: 1/(12 dx), D2: 3/(4 dx^2), filter: the
// centre weight), the forward sweep is unnormalised (v_i = t_i - l_i v_{i-1}),
// and kappa, 1/pivot and the chunk's response to its carry enter the
// backward sweep as row coefficients: x_i = c1_i v_i + c2_i V - g_i x_{i+1}.
// Per real value that is the stencil (3, 4 or 6 instructions), 1 forward, 3
// backward and 1 for the backward carry: 8, 9 and 11 in place of the 9, 11 and
// 12 of scaled right-hand side, normalised forward sweep and separate fix-up.
#pragma once
#include "tb_internal.h"

namespace xl {

// Row tables of one operator, element (q, lane) of row lane * S + q at
// q * 32 + lane, so that a warp reads a row of lanes at once:
//   l, c1, c2, g, hb    5 x S x 32
//   pf, pb              2 x 5 x 32 Kogge-Stone factors of the chunk responses
// Rows beyond the line hold zeros.
__host__ __device__ inline int table_size(int S) { return 5 * 32 * S + 320; }

enum Op { D1 = 0, D2 = 1, FILTER = 2 };

// Stencil weights of the filter in units of its centre weight (the others'
// are constants): interior w1, w2, w3 of f[i+-1], f[i+-2], f[i+-3] and the end
// rows' 1/16; w0 is the centre weight itself in these units (1, or 0 where it
// vanishes and the unit is 1).
struct Weights {
    double w0, w1, w2, w3, end;
};

template <class R> struct Cx;
template <> struct Cx<double> { using V = double2; };
template <> struct Cx<float> { using V = float2; };
template <class V, class R> __device__ __forceinline__ V cmul(R s, V a) { return V{s * a.x, s * a.y}; }
template <class V> __device__ __forceinline__ V cadd(V a, V b) { return V{a.x + b.x, a.y + b.y}; }
template <class V> __device__ __forceinline__ V csub(V a, V b) { return V{a.x - b.x, a.y - b.y}; }
template <class V, class R> __device__ __forceinline__ V cfma(R s, V a, V b) { return V{fma(s, a.x, b.x), fma(s, a.y, b.y)}; }

// A line staged in shared memory in lane chunks: row i at (i / S) * Sp + i % S
// (Sp = S rounded up to odd, so the accesses of consecutive lanes at the
// same chunk offset fall in distinct banks).
template <class V>
struct SmemLine {
    const V* F;
    int S, Sp;
    __device__ __forceinline__ V operator[](int i) const { return F[(i / S) * Sp + i % S]; }
};

// Right-hand side of a boundary row (rows 0-based) in units of kappa.
template <int OP, class R, class Line>
__device__ __forceinline__ typename Cx<R>::V end_row(const Line& f, int i, int n, const Weights& W) {
    using V = typename Cx<R>::V;
    const int m = n - 1;
    const bool low = i < 3;
    const int b = low ? 0 : m, e = low ? 1 : -1, r = low ? i : m - i;   // anchor, direction, distance from the end
    if (OP == D1) {
        if (r == 1) {
            V s = cmul((R)-406, f[b]); s = cfma((R)-300, f[b + e], s); s = cfma((R)760, f[b + 2 * e], s);
            s = cfma((R)-80, f[b + 3 * e], s); s = cfma((R)30, f[b + 4 * e], s); s = cfma((R)-4, f[b + 5 * e], s);
            return cmul((R)(0.1 * e), s);
        }
        if (low) {
            V s = cmul((R)-25, f[0]); s = cfma((R)48, f[1], s); s = cfma((R)-36, f[2], s); s = cfma((R)16, f[3], s);
            return cfma((R)-3, f[4], s);
        }
        V s = cmul((R)-74, f[m]); s = cfma((R)16, f[m - 1], s); s = cfma((R)72, f[m - 2], s); s = cfma((R)-16, f[m - 3], s);
        return cmul((R)-0.5, cfma((R)2, f[m - 4], s));
    } else if (OP == D2) {
        if (r == 0) {
            V s = cmul((R)9775, f[b]); s = cfma((R)-20285, f[b + e], s); s = cfma((R)11170, f[b + 2 * e], s);
            s = cfma((R)-550, f[b + 3 * e], s); s = cfma((R)-145, f[b + 4 * e], s); s = cfma((R)35, f[b + 5 * e], s);
            return cmul((R)(1.0 / 45.0), s);
        }
        V s = cmul((R)4834, f[b]); s = cfma((R)-8424, f[b + e], s); s = cfma((R)1890, f[b + 2 * e], s);
        s = cfma((R)2320, f[b + 3 * e], s); s = cfma((R)-810, f[b + 4 * e], s); s = cfma((R)216, f[b + 5 * e], s);
        return cmul((R)(1.0 / 270.0), cfma((R)-26, f[b + 6 * e], s));
    } else {
        const R w[3][5] = {{15, 4, -6, 4, -1}, {1, 12, 6, -4, 1}, {-1, 4, 10, 4, -1}};
        V s = cmul(w[r][0], f[b]);
#pragma unroll
        for (int q = 1; q < 5; q++) s = cfma(w[r][q], f[b + q * e], s);
        return cmul((R)W.end, s);
    }
}

template <class V> __device__ __forceinline__ V to_v(cplx c);
template <> __device__ __forceinline__ double2 to_v<double2>(cplx c) { return c; }
template <> __device__ __forceinline__ float2 to_v<float2>(cplx c) { return make_float2((float)c.x, (float)c.y); }
__device__ __forceinline__ cplx to_c(double2 v) { return v; }
__device__ __forceinline__ cplx to_c(float2 v) { return make_double2((double)v.x, (double)v.y); }

// The line f (n points) of one warp into o, rows from `first` on, in
// precision R: staged in shared memory (F: 32 x (S | 1) values) with coalesced
// loads; lane t owns rows [tS, tS + S) and runs the sweeps over its chunk with
// zero carry-in, the carries cross the lanes by a Kogge-Stone scan of the
// precomputed chunk responses.  T: the operator's tables; o may be f.
template <int OP, class R>
__device__ __forceinline__ void xline(const Weights& W, const R* __restrict__ T, int S, int n, const cplx* f, cplx* o, int first,
                                      typename Cx<R>::V* F) {
    using V = typename Cx<R>::V;
    const int lane = threadIdx.x & 31, Sp = S | 1;
    const R *Tl = T + lane, *Tc1 = Tl + 32 * S, *Tc2 = Tl + 64 * S, *Tg = Tl + 96 * S, *Thb = Tl + 128 * S;
    const R *Tpf = Tl + 160 * S, *Tpb = Tpf + 160;
    for (int i = lane; i < n; i += 32) F[(i / S) * Sp + i % S] = to_v<V>(f[i]);
    __syncwarp();
    const SmemLine<V> L{F, S, Sp};
    const int H = (OP == FILTER) ? 3 : 2;
    const int r0 = min(n, lane * S), r1 = min(n, r0 + S);
    V* Ul = F + lane * Sp;
    // Before any lane overwrites its rows, each takes what it reads outside
    // them or ahead of its own sweep: the right-hand sides of its boundary
    // rows (stencils reaching up to 6 rows in), the first window of its
    // interior rows, and the H rows after its chunk.
    const int ib0 = max(r0, H), ie = min(r1, n - H);   // the chunk's interior rows [ib0, ie)
    V rs0[3], rs1[3], hi[3], w[7];
#pragma unroll
    for (int q = 0; q < 3; q++) {
        rs0[q] = V{0, 0}; rs1[q] = V{0, 0}; hi[q] = V{0, 0};
        const int e = n - H + q;
        if (q < H && q >= r0 && q < r1) rs0[q] = end_row<OP, R>(L, q, n, W);
        if (q < H && e >= r0 && e < r1) rs1[q] = end_row<OP, R>(L, e, n, W);
        if (q < H && r1 + q < n) hi[q] = L[r1 + q];
    }
#pragma unroll
    for (int q = 0; q < 7; q++) w[q] = V{0, 0};
    if (ib0 < ie) {
#pragma unroll
        for (int q = 0; q < 2 * H; q++) w[q] = L[ib0 - H + q];
    }
    __syncwarp();
    // forward sweep over the chunk with zero carry-in
    V v = V{0, 0};
    auto fwd = [&](int i, V t) {
        const R l = Tl[32 * (i - r0)];
        v = V{fma(-l, v.x, t.x), fma(-l, v.y, t.y)};
        Ul[i - r0] = v;
    };
#pragma unroll
    for (int q = 0; q < 3; q++)
        if (q < H && q >= r0 && q < r1) fwd(q, rs0[q]);
    if (ib0 < ie) {
        const R w0 = (R)W.w0, w1 = (R)W.w1, w2 = (R)W.w2, w3 = (R)W.w3;
        int nc = (ib0 + H) / S, no = (ib0 + H) % S;   // chunk slot of row i + H
        for (int i = ib0; i < ie; i++) {
            const int d = i + H - r1;                 // >= 0: row i + H is after the chunk
            V h = hi[0];
            if (d == 1) h = hi[1];
            if (d == 2) h = hi[2];
            w[2 * H] = (d < 0) ? F[nc * Sp + no] : h;
            if (++no == S) { no = 0; nc++; }
            V t;
            if (OP == D1) t = cfma((R)28, csub(w[3], w[1]), csub(w[4], w[0]));
            else if (OP == D2) t = cfma((R)-34, w[2], cfma((R)16, cadd(w[3], w[1]), cadd(w[4], w[0])));
            else {
                t = cmul(w3, cadd(w[6], w[0]));
                t = cfma(w2, cadd(w[5], w[1]), t);
                t = cfma(w1, cadd(w[4], w[2]), t);
                t = (w0 == (R)1) ? cadd(w[3], t) : cfma(w0, w[3], t);
            }
            fwd(i, t);
#pragma unroll
            for (int q = 0; q < 2 * H; q++) w[q] = w[q + 1];
        }
    }
#pragma unroll
    for (int q = 0; q < 3; q++) {
        const int e = n - H + q;
        if (q < H && e >= r0 && e < r1) fwd(e, rs1[q]);
    }
    // forward carries: true chunk-end values by a scan, carry-in = previous lane's
    V b = v;
#pragma unroll
    for (int d = 0, off = 1; d < 5; d++, off <<= 1) {
        const R ox = __shfl_up_sync(0xffffffffu, b.x, off), oy = __shfl_up_sync(0xffffffffu, b.y, off);
        if (lane >= off) { const R m = Tpf[d * 32]; b.x = fma(m, ox, b.x); b.y = fma(m, oy, b.y); }
    }
    V Vin;
    Vin.x = __shfl_up_sync(0xffffffffu, b.x, 1); Vin.y = __shfl_up_sync(0xffffffffu, b.y, 1);
    if (lane == 0) Vin = V{0, 0};
    // backward sweep over the chunk (zero carry from the right)
    V x = V{0, 0};
    for (int q = r1 - r0 - 1; q >= 0; q--) {
        const R c1 = Tc1[32 * q], c2 = Tc2[32 * q], g = Tg[32 * q];
        const V u = Ul[q];
        x = V{fma(-g, x.x, fma(c1, u.x, c2 * Vin.x)), fma(-g, x.y, fma(c1, u.y, c2 * Vin.y))};
        Ul[q] = x;
    }
    // backward carries: true chunk-start values by a scan from the high lanes
    b = x;
#pragma unroll
    for (int d = 0, off = 1; d < 5; d++, off <<= 1) {
        const R ox = __shfl_down_sync(0xffffffffu, b.x, off), oy = __shfl_down_sync(0xffffffffu, b.y, off);
        if (lane + off < 32) { const R m = Tpb[d * 32]; b.x = fma(m, ox, b.x); b.y = fma(m, oy, b.y); }
    }
    V Xin;
    Xin.x = __shfl_down_sync(0xffffffffu, b.x, 1); Xin.y = __shfl_down_sync(0xffffffffu, b.y, 1);
    if (lane == 31) Xin = V{0, 0};
    for (int q = 0; q < r1 - r0; q++) {
        const R h = Thb[32 * q];
        const V u = Ul[q];
        Ul[q] = V{fma(h, Xin.x, u.x), fma(h, Xin.y, u.y)};
    }
    __syncwarp();
    for (int i = first + lane; i < n; i += 32) o[i] = to_c(F[(i / S) * Sp + i % S]);
    __syncwarp();
}

}  // namespace xl
