// tb_xline.cuh -- one compact x-line solve on two warps (derparx/derparxx,
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
// Per real value that is the stencil (3, 4 or 7 instructions), 1 forward, 3
// backward and 1 for the backward carry.  The rows at the ends of a line, whose
// stencils reach up to 6 rows in, are summed by one lane each at once.  The
// real and the imaginary part of a line are two problems on a warp each: as many
// lines as fit an SM's shared memory then bring twice the warps, which the pipe
// needs to stay full across a line's loads and carries (D1 at 1025 x 193 x 32: 303
// us and 69 % of the pipe with one warp a line, 261 us with two).
#pragma once
#include "tb_internal.h"

namespace xl {

// Row tables of one operator, element (q, lane) of row lane * S + q at
// q * 32 + lane, so that a warp reads a row of lanes at once:
//   l, c1, c2, g, hb    5 x S x 32
//   pf, pb              2 x 5 x 32 Kogge-Stone factors of the chunk responses
//   we          8 x 32: weights of end row e in lane e < 2H, then its scale
// Rows beyond the line hold zeros.
__host__ __device__ inline int table_size(int S) { return 5 * 32 * S + 320 + 256; }
// A line staged in shared memory: two planes in lane chunks, row i at (i / S) *
// (S | 1) + i % S (the odd stride keeps the lanes' accesses at one chunk offset in
// distinct banks), then the end rows' right-hand sides of each.
__host__ __device__ inline int line_size(int S) { return 64 * (S | 1) + 16; }

enum Op { D1 = 0, D2 = 1, FILTER = 2 };

// Stencil weights of the filter in units of its centre weight (the others'
// are constants): interior w1, w2, w3 of f[i+-1], f[i+-2], f[i+-3] and the end
// rows' 1/16; w0 is the centre weight itself in these units (1, or 0 where it
// vanishes and the unit is 1).
struct Weights {
    double w0, w1, w2, w3, end;
};
__host__ __device__ constexpr int ends(int op) { return op == FILTER ? 3 : 2; }   // end rows on either side

// Weight q of end row e < 2 ends(op) (the low end's first, both in row order) on the
// q-th point from its end, and for q = 7 the scale of their sum, in units of kappa.
__host__ __device__ inline double end_weight(int op, int e, int q, const Weights& W) {
    const int H = ends(op);
    if (e >= 2 * H) return 0.0;
    const bool low = e < H;
    const int r = low ? e : 2 * H - 1 - e;   // distance from the end
    if (op == D1) {
        const double w[3][8] = {{-25, 48, -36, 16, -3, 0, 0, 1.0}, {-406, -300, 760, -80, 30, -4, 0, 0.1},
                                {-74, 16, 72, -16, 2, 0, 0, -0.5}};
        if (r == 1) return q == 7 && !low ? -0.1 : w[1][q];
        return w[low ? 0 : 2][q];
    }
    if (op == D2) {
        const double w[2][8] = {{9775, -20285, 11170, -550, -145, 35, 0, 1.0 / 45.0},
                                {4834, -8424, 1890, 2320, -810, 216, -26, 1.0 / 270.0}};
        return w[r][q];
    }
    const double w[3][7] = {{15, 4, -6, 4, -1, 0, 0}, {1, 12, 6, -4, 1, 0, 0}, {-1, 4, 10, 4, -1, 0, 0}};
    return q == 7 ? W.end : w[r][q];
}

#ifdef __CUDACC__
// The part (0 real, 1 imaginary) of the line f (n points) into o, rows from
// `first` on, in precision R, by one warp of a pair that shares the staged line
// F and the named barrier `bar`.  Loads and stores are coalesced over the
// pair; lane t owns rows [tS, tS + S) and runs the sweeps over its chunk with zero
// carry-in, the carries cross the lanes by a Kogge-Stone scan of the precomputed
// chunk responses.  T: the operator's tables; o may be f.
template <int OP, class R>
__device__ __forceinline__ void xline(const Weights& W, const R* __restrict__ T, int S, int n, const cplx* f, cplx* o, int first,
                                      R* F, int part, int bar) {
    constexpr int H = ends(OP), TAPS = OP == FILTER ? 5 : OP == D1 ? 6 : 7;
    const int lane = threadIdx.x & 31, t64 = 32 * part + lane, Sp = S | 1, plane = 32 * Sp;
    const R *Tl = T + lane, *Tc1 = Tl + 32 * S, *Tc2 = Tl + 64 * S, *Tg = Tl + 96 * S, *Thb = Tl + 128 * S;
    const R *Tpf = Tl + 160 * S, *Tpb = Tpf + 160, *Twe = Tpb + 160;
    R *L = F + part * plane, *E = F + 2 * plane + 8 * part, *Ul = L + lane * Sp;
    auto pair_barrier = [&]() { asm volatile("bar.sync %0, 64;" ::"r"(bar) : "memory"); };
    auto row = [&](int i) { return L[(i / S) * Sp + i % S]; };
    const int dc = 64 / S, dr = 64 % S;
    {
        int c = t64 / S, r = t64 % S;
#pragma unroll 8
        for (int i = t64; i < n; i += 64) {
            const cplx v = f[i];
            F[c * Sp + r] = (R)v.x;
            F[plane + c * Sp + r] = (R)v.y;
            c += dc; r += dr;
            if (r >= S) { r -= S; c++; }
        }
    }
    pair_barrier();
    // Before any lane overwrites its rows: the end rows' right-hand sides, the
    // first window of the chunk and the H rows after it.
    const int r0 = min(n, lane * S), r1 = min(n, r0 + S);
    if (lane < 2 * H) {
        R s = 0;
#pragma unroll
        for (int q = 0; q < TAPS; q++) s = fma(Twe[32 * q], row(lane < H ? q : n - 1 - q), s);
        E[lane] = Twe[224] * s;
    }
    R hi[3], w[7];
#pragma unroll
    for (int q = 0; q < 3; q++) hi[q] = (q < H && r1 + q < n) ? row(r1 + q) : (R)0;
#pragma unroll
    for (int q = 0; q < 7; q++) {
        const int i = r0 - H + q;
        w[q] = (q < 2 * H && i >= 0 && i < n) ? row(i) : (R)0;
    }
    __syncwarp();
    // forward sweep over the chunk with zero carry-in
    R v = 0;
    const R w0 = (R)W.w0, w1 = (R)W.w1, w2 = (R)W.w2, w3 = (R)W.w3;
    for (int q = 0; q < r1 - r0; q++) {
        const int i = r0 + q, d = i + H - r1;   // d >= 0: row i + H is after the chunk
        R h = hi[0];
        if (d == 1) h = hi[1];
        if (d == 2) h = hi[2];
        w[2 * H] = (d < 0) ? Ul[q + H] : h;
        R t;
        if (OP == D1) t = fma((R)28, w[3] - w[1], w[4] - w[0]);
        else if (OP == D2) t = fma((R)-34, w[2], fma((R)16, w[3] + w[1], w[4] + w[0]));
        else {
            t = w3 * (w[6] + w[0]);
            t = fma(w2, w[5] + w[1], t);
            t = fma(w1, w[4] + w[2], t);
            t = fma(w0, w[3], t);
        }
        if (i < H || i >= n - H) t = E[i < H ? i : i - n + 2 * H];
        v = fma(-Tl[32 * q], v, t);
        Ul[q] = v;
#pragma unroll
        for (int e = 0; e < 2 * H; e++) w[e] = w[e + 1];
    }
    // forward carries: true chunk-end values by a scan, carry-in = previous lane's
    R b = v;
#pragma unroll
    for (int d = 0, off = 1; d < 5; d++, off <<= 1) {
        const R x = __shfl_up_sync(0xffffffffu, b, off);
        if (lane >= off) b = fma(Tpf[d * 32], x, b);
    }
    R Vin = __shfl_up_sync(0xffffffffu, b, 1);
    if (lane == 0) Vin = 0;
    // backward sweep over the chunk (zero carry from the right)
    R x = 0;
#pragma unroll 2
    for (int q = r1 - r0 - 1; q >= 0; q--) {
        x = fma(-Tg[32 * q], x, fma(Tc1[32 * q], Ul[q], Tc2[32 * q] * Vin));
        Ul[q] = x;
    }
    // backward carries: true chunk-start values by a scan from the high lanes
    b = x;
#pragma unroll
    for (int d = 0, off = 1; d < 5; d++, off <<= 1) {
        const R y = __shfl_down_sync(0xffffffffu, b, off);
        if (lane + off < 32) b = fma(Tpb[d * 32], y, b);
    }
    R Xin = __shfl_down_sync(0xffffffffu, b, 1);
    if (lane == 31) Xin = 0;
#pragma unroll 4
    for (int q = 0; q < r1 - r0; q++) Ul[q] = fma(Thb[32 * q], Xin, Ul[q]);
    pair_barrier();
    {
        int c = t64 / S, r = t64 % S;
#pragma unroll 8
        for (int i = t64; i < n; i += 64) {
            if (i >= first) o[i] = make_double2((double)F[c * Sp + r], (double)F[plane + c * Sp + r]);
            c += dc; r += dr;
            if (r >= S) { r -= S; c++; }
        }
    }
    pair_barrier();
}
#endif

}  // namespace xl
