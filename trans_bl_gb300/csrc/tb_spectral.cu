// tb_spectral.cu -- spanwise Fourier <-> physical transforms and the
// physical-space products of the stage.
//
// Convention of the reference (nlterms_par.f:303-428, Numerical-Recipes
// realft packing): a field with modes c_k, k = 0..K-1, has physical values
//     p_n = Re c_0 + (Im c_0 / 2) (-1)^n + sum_{k>=1} Re( c_k e^{-2 pi i k n / P} ),
// and the forward transform returns c_0 = (1/P) sum p_n, c_k = (2/P) sum p_n
// e^{+2 pi i k n / P}, zeroes components below 1e-14 and forces Im c_0 = 0.
// Both directions are computed here as a length-P/2 complex FFT plus the
// real-to-complex split, with exact twiddles from constant tables instead of
// the reference's rotation recurrence: one thread per (i, j) grid line, and two
// in k_les and k_cvirt at P = 128, where one line's values are more than a thread's
// registers.
//
// An FP64 warp instruction (comparisons included) holds its pipe for 64
// cycles, so the FP64 transforms are written for their number: a butterfly is
// six fused multiply-adds (twiddle w = m (1 + i r) or m (r + i), |r| <= 1: the factored
// butterfly of Linzer and Feig, "Implementation of efficient FFT algorithms on
// fused multiply-add architectures", IEEE Trans. Signal Process. 41, 1993), the
// split takes the modes k and P/2 - k together (12 in place of 28), its halves and
// the 1/P are left to the caller's factors, and values are compared as integers.
#include "tb_internal.h"
#include "tb_tc.cuh"
#include <cuda_bf16.h>
#include <cstring>
#include <algorithm>
#include <cmath>

#define TW_N 512
__constant__ double c_twr[TW_N], c_twi[TW_N];  // e^{-2 pi i t / TW_N}
__constant__ double c_lfm[TW_N / 2], c_lfr[TW_N / 2];   // the same as m (1 + i r) or m (r + i), see fft
__constant__ float c_twrf[TW_N], c_twif[TW_N]; // the same, rounded to FP32

namespace {

__device__ __forceinline__ double twr(int t) { return c_twr[t & (TW_N - 1)]; }
__device__ __forceinline__ double twi(int t) { return c_twi[t & (TW_N - 1)]; }
__device__ __forceinline__ float twr_f(int t) { return c_twrf[t & (TW_N - 1)]; }
__device__ __forceinline__ float twi_f(int t) { return c_twif[t & (TW_N - 1)]; }

template <int N>
__device__ __forceinline__ int brev(int i) {
    int r = 0;
#pragma unroll
    for (int b = 1; b < N; b <<= 1) { r = (r << 1) | (i & 1); i >>= 1; }
    return r;
}

// In-place radix-2 complex FFT of length N in FP32. SIGN = -1: sum X_k e^{-2 pi i km/N};
// SIGN = +1: sum X_k e^{+2 pi i km/N}.
template <int N, int SIGN>
__device__ __forceinline__ void cfft(float* re, float* im) {
#pragma unroll
    for (int i = 0; i < N; i++) {
        int j = brev<N>(i);
        if (j > i) {
            float t = re[i]; re[i] = re[j]; re[j] = t;
            t = im[i]; im[i] = im[j]; im[j] = t;
        }
    }
#pragma unroll
    for (int len = 2; len <= N; len <<= 1) {
        const int h = len / 2;
#pragma unroll
        for (int s = 0; s < N; s += len) {
#pragma unroll
            for (int q = 0; q < h; q++) {
                int a = s + q, b = a + h;
                float tr, ti;
                if (q == 0) {
                    tr = re[b]; ti = im[b];
                } else if (4 * q == len) {  // twiddle -SIGN*i ... e^{SIGN*i*pi/2} = SIGN*i
                    tr = (SIGN < 0) ? im[b] : -im[b];
                    ti = (SIGN < 0) ? -re[b] : re[b];
                } else {
                    float wr = twr_f(q * (TW_N / len));
                    float wi = (SIGN < 0) ? twi_f(q * (TW_N / len)) : -twi_f(q * (TW_N / len));
                    tr = wr * re[b] - wi * im[b];
                    ti = wr * im[b] + wi * re[b];
                }
                re[b] = re[a] - tr; im[b] = im[a] - ti;
                re[a] = re[a] + tr; im[a] = im[a] + ti;
            }
        }
    }
}

// |cos| >= |sin| of the angle 2 pi t / TW_N, 0 <= t < TW_N / 2.
__host__ __device__ constexpr bool lf_big(int t) { return t <= TW_N / 8 || t >= 3 * TW_N / 8; }

// The same in FP64, six fused multiply-adds a butterfly: w b = m u with
// u = (1 + i r) b or (r + i) b, and a +- m u.
template <int N, int SIGN>
__device__ __forceinline__ void fft(double* re, double* im) {
#pragma unroll
    for (int i = 0; i < N; i++) {
        int j = brev<N>(i);
        if (j > i) {
            double t = re[i]; re[i] = re[j]; re[j] = t;
            t = im[i]; im[i] = im[j]; im[j] = t;
        }
    }
#pragma unroll
    for (int len = 2; len <= N; len <<= 1) {
        const int h = len / 2;
#pragma unroll
        for (int s = 0; s < N; s += len) {
#pragma unroll
            for (int q = 0; q < h; q++) {
                const int a = s + q, b = a + h;
                const double ar = re[a], ai = im[a], br = re[b], bi = im[b];
                if (q == 0) {
                    re[b] = ar - br; im[b] = ai - bi;
                    re[a] = ar + br; im[a] = ai + bi;
                } else if (4 * q == len) {   // w = SIGN i
                    const double tr = (SIGN < 0) ? bi : -bi, ti = (SIGN < 0) ? -br : br;
                    re[b] = ar - tr; im[b] = ai - ti;
                    re[a] = ar + tr; im[a] = ai + ti;
                } else {
                    const int t = q * (TW_N / len);
                    const double m = c_lfm[t], r = c_lfr[t];
                    double ur, ui;
                    if (lf_big(t)) {
                        ur = fma(SIGN < 0 ? -r : r, bi, br);
                        ui = fma(SIGN < 0 ? r : -r, br, bi);
                    } else {   // SIGN > 0: conj(w) = m (r + i) with m -> -m, r -> -r
                        ur = fma(r, br, SIGN < 0 ? -bi : bi);
                        ui = fma(r, bi, SIGN < 0 ? br : -br);
                    }
                    re[b] = fma(-m, ur, ar); im[b] = fma(-m, ui, ai);
                    re[a] = fma(m, ur, ar); im[a] = fma(m, ui, ai);
                }
            }
        }
    }
}

// Components below 1e-14 -> 0, compared by their bits.
__device__ __forceinline__ double zap(double v) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
    return b < 0x3d06849b86a12b9bull ? 0.0 : v;   // 1e-14
}

// The K modes of a grid line at stride cs, zero beyond.
struct Modes {
    const cplx* f;
    size_t cs;
    int K;
    __device__ __forceinline__ cplx operator()(int k) const { return k < K ? f[(size_t)k * cs] : make_double2(0.0, 0.0); }
};

// Inverse split of the modes k and N - k, twice its value: Z_k and Z_{N-k} of
// the length-N transform; (wr, wi) = e^{-2 pi i k / P}.
__device__ __forceinline__ void split_in(cplx A, cplx B, double wr, double wi, double& zr, double& zi, double& yr, double& yi) {
    const double sr = A.x + B.x, si = A.y - B.y, dr = A.x - B.x, di = A.y + B.y;
    const double t1 = fma(wr, di, wi * dr), t2 = fma(wr, dr, -(wi * di));
    zr = sr - t1; zi = si + t2;
    yr = sr + t1; yi = t2 - si;
}
// Forward split: the modes k (a) and N - k (b), times P, of F_k and F_{N-k};
// (vr, vi) = e^{+2 pi i k / P}.
__device__ __forceinline__ void split_out(double fr, double fi, double gr, double gi, double vr, double vi, cplx& a, cplx& b) {
    const double sr = fr + gr, si = fi - gi, dr = fr - gr, di = fi + gi;
    const double t1 = fma(vr, di, vi * dr), t2 = fma(vi, di, -(vr * dr));
    a = make_double2(zap(sr + t1), zap(si + t2));
    b = make_double2(zap(sr - t1), zap(t2 - si));
}

// Fourier (load(k) gives mode k) -> twice the physical values p[0..P-1].
template <int P, class Load>
__device__ __forceinline__ void to_phys2(const Load& load, double* p) {
    constexpr int N = P / 2;
    double re[N], im[N];
    const cplx c0 = load(0);
    re[0] = fma(2.0, c0.x, c0.y); im[0] = fma(2.0, c0.x, -c0.y);
#pragma unroll
    for (int k = 1; 2 * k < N; k++)
        split_in(load(k), load(N - k), twr(k * (TW_N / P)), twi(k * (TW_N / P)), re[k], im[k], re[N - k], im[N - k]);
    if (N > 1) {
        const cplx c = load(N / 2);
        re[N / 2] = 2.0 * c.x; im[N / 2] = 2.0 * c.y;
    }
    fft<N, -1>(re, im);
#pragma unroll
    for (int m = 0; m < N; m++) { p[2 * m] = re[m]; p[2 * m + 1] = im[m]; }
}

// P^-1 times the physical values p[0..P-1] -> Fourier, store(k, mode k) for
// every k < P/2.
template <int P, class Store>
__device__ __forceinline__ void to_four(const double* p, const Store& store) {
    constexpr int N = P / 2;
    double re[N], im[N];
#pragma unroll
    for (int m = 0; m < N; m++) { re[m] = p[2 * m]; im[m] = p[2 * m + 1]; }
    fft<N, +1>(re, im);
    store(0, make_double2(zap(re[0] + im[0]), 0.0));
#pragma unroll
    for (int k = 1; 2 * k < N; k++) {
        cplx a, b;
        split_out(re[k], im[k], re[N - k], im[N - k], twr(k * (TW_N / P)), -twi(k * (TW_N / P)), a, b);
        store(k, a);
        store(N - k, b);
    }
    if (N > 1) store(N / 2, make_double2(zap(2.0 * re[N / 2]), zap(2.0 * im[N / 2])));
}

// A grid line on TP threads (lanes l and l ^ 16): thread p holds the values
// m = j TP + p, j < M, of the length-N transform, that is the physical points
// 2m and 2m + 1, and on the Fourier side the modes k of parity p.
template <int P>
struct Col {
    static constexpr int N = P / 2, TP = P >= 128 ? 2 : 1, M = N / TP;
    static constexpr int VAL = 2 * M, PER_BLOCK = 128 / TP;   // physical values of a thread; lines of a block
};
// The last stage over both threads' length-M transforms, thread p for the
// outputs k and k + M, k = 2i + p (positions i and M/2 + i).
template <int P, int SIGN>
__device__ __forceinline__ void join(int p, double* re, double* im) {
    constexpr int N = Col<P>::N, M = Col<P>::M;
    double xr[M], xi[M];
#pragma unroll
    for (int i = 0; i < M; i++) { xr[i] = re[i]; xi[i] = im[i]; }
#pragma unroll
    for (int i = 0; i < M / 2; i++) {
        const double sr = __shfl_xor_sync(0xffffffffu, p ? xr[2 * i] : xr[2 * i + 1], 16);
        const double si = __shfl_xor_sync(0xffffffffu, p ? xi[2 * i] : xi[2 * i + 1], 16);
        const double wr_ = p ? xr[2 * i + 1] : xr[2 * i], wi_ = p ? xi[2 * i + 1] : xi[2 * i];   // own
        const double er = p ? sr : wr_, ei = p ? si : wi_, orr = p ? wr_ : sr, oi = p ? wi_ : si;
        const int t = (2 * i + p) * (TW_N / N);
        const double c = twr(t), s = SIGN < 0 ? twi(t) : -twi(t);
        const double tr = fma(c, orr, -(s * oi)), ti = fma(c, oi, s * orr);
        re[i] = er + tr; im[i] = ei + ti;
        re[M / 2 + i] = er - tr; im[M / 2 + i] = ei - ti;
    }
}
template <int P, class Load>
__device__ __forceinline__ void col_phys2(const Load& load, int p, double* re, double* im) {
    constexpr int N = Col<P>::N, M = Col<P>::M;
    if constexpr (Col<P>::TP == 1) {
        double v[P];
        to_phys2<P>(load, v);
#pragma unroll
        for (int m = 0; m < N; m++) { re[m] = v[2 * m]; im[m] = v[2 * m + 1]; }
    } else {
        double yr[M / 2 + 1], yi[M / 2 + 1];   // Z_{N-k}
#pragma unroll
        for (int i = 0; i < M / 2; i++) {
            const int k = 2 * i + p, t = k * (TW_N / P);
            split_in(load(k), load(k ? N - k : 0), twr(t), twi(t), re[i], im[i], yr[i], yi[i]);
        }
        const cplx c0 = load(0), cm = load(N / 2);
        if (p == 0) { re[0] = fma(2.0, c0.x, c0.y); im[0] = fma(2.0, c0.x, -c0.y); }
        yr[M / 2] = 2.0 * cm.x; yi[M / 2] = 2.0 * cm.y;
#pragma unroll
        for (int q = M / 2; q < M; q++) {
            re[q] = p ? yr[M - 1 - q] : yr[M - q];
            im[q] = p ? yi[M - 1 - q] : yi[M - q];
        }
        fft<M, -1>(re, im);
        join<P, -1>(p, re, im);
    }
}
template <int P, class Store>
__device__ __forceinline__ void col_four(double* re, double* im, int p, const Store& store) {
    constexpr int N = Col<P>::N, M = Col<P>::M;
    if constexpr (Col<P>::TP == 1) {
        double v[P];
#pragma unroll
        for (int m = 0; m < N; m++) { v[2 * m] = re[m]; v[2 * m + 1] = im[m]; }
        to_four<P>(v, store);
    } else {
        fft<M, +1>(re, im);
        join<P, +1>(p, re, im);
#pragma unroll
        for (int i = 0; i < M / 2; i++) {
            const int k = 2 * i + p, t = k * (TW_N / P);
            const double gr = p ? re[M - 1 - i] : re[i ? M - i : 0], gi = p ? im[M - 1 - i] : im[i ? M - i : 0];
            cplx a, b;
            split_out(re[i], im[i], gr, gi, twr(t), -twi(t), a, b);
            if (k) {
                store(k, a);
                store(N - k, b);
            }
        }
        if (p == 0) {
            store(0, make_double2(zap(re[0] + im[0]), 0.0));
            store(N / 2, make_double2(zap(2.0 * re[M / 2]), zap(2.0 * im[M / 2])));
        }
    }
}

// ---------------------------------------------------------------------------
template <int P>
__global__ void __launch_bounds__(128) k_f_to_p(double* phys, const cplx* four, int n2, int K) {
    int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n2) return;
    double p[P];
    to_phys2<P>(Modes{four + q, (size_t)n2, K}, p);
#pragma unroll
    for (int z = 0; z < P; z++) phys[(size_t)q + (size_t)n2 * z] = 0.5 * p[z];
}
template <int P>
__global__ void __launch_bounds__(128) k_p_to_f(cplx* four, const double* phys, int n2, int K) {
    int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n2) return;
    double p[P];
#pragma unroll
    for (int z = 0; z < P; z++) p[z] = (1.0 / (double)P) * phys[(size_t)q + (size_t)n2 * z];
    to_four<P>(p, [&](int k, cplx v) { if (k < K) four[(size_t)q + (size_t)n2 * k] = v; });
}

// nlterms_fi (nlterms_par.f:41-86): a = uy wx - ux wy, b = ux wz - uz wx, c = uz wy - uy wz.
struct NlArgs {
    const cplx *ux, *uy, *uz, *wx, *wy, *wz;
    cplx *a, *b, *c;
    int n2, K;
};
template <int P>
__global__ void __launch_bounds__(128) k_nlterms(NlArgs A) {
    int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= A.n2) return;
    size_t cs = A.n2;
    const cplx* fs[6] = {A.ux, A.uy, A.uz, A.wx, A.wy, A.wz};
    double ph[6][P];
#pragma unroll
    for (int f = 0; f < 6; f++) to_phys2<P>(Modes{fs[f] + q, cs, A.K}, ph[f]);
    constexpr double sc = 0.25 / (double)P;   // the fields' factors 2 and the forward transform's 1 / P
#pragma unroll
    for (int z = 0; z < P; z++) {
        double ux = sc * ph[0][z], uy = sc * ph[1][z], uz = sc * ph[2][z], wx = ph[3][z], wy = ph[4][z], wz = ph[5][z];
        ph[0][z] = uy * wx - ux * wy;
        ph[1][z] = ux * wz - uz * wx;
        ph[2][z] = uz * wy - uy * wz;
    }
    cplx* outs[3] = {A.a, A.b, A.c};
#pragma unroll
    for (int f = 0; f < 3; f++) to_four<P>(ph[f], [&](int k, cplx v) { if (k < A.K) outs[f][q + cs * k] = v; });
}

// ---------------------------------------------------------------------------
// Mixed form of nlterms_fi.  With every field split into its spanwise mean
// M = Re c_0 (which carries the base flow) and its z-varying part d(z), a
// product such as uy wx transforms to
//   mode 0:   M_uy M_wx                 + T(d_uy d_wx)_0
//   mode k:   M_uy wx_k + M_wx uy_k     + T(d_uy d_wx)_k      (k >= 1)
// because T(M d)_k = M c_k(d) exactly (T the forward transform of the
// reference; d holds modes 1..K-1 and the packed Nyquist term).  The linear
// part, which dominates for a disturbance on a base flow, stays in FP64;
// only the quadratic disturbance term goes through FP32 transforms.
// Components below 1e-14 are zeroed and Im c_0 = 0, as nlterms_par.f does.

// z-varying part of a field (mean removed) -> physical p[0..P-1], FP32.
template <int P>
__device__ __forceinline__ void to_phys_dist(const cplx* __restrict__ cf, size_t cs, int K, float* p) {
    constexpr int N = P / 2;
    float re[N], im[N];
    float CN = (float)(0.5 * cf[0].y);
    re[0] = CN; im[0] = -CN;
#pragma unroll
    for (int k = 1; k < N; k++) {
        cplx A = (k < K) ? cf[(size_t)k * cs] : make_double2(0.0, 0.0);
        cplx Bc = (N - k < K) ? cf[(size_t)(N - k) * cs] : make_double2(0.0, 0.0);
        float Ar = (float)A.x, Ai = (float)A.y, Br = (float)Bc.x, Bi = -(float)Bc.y;
        float sr = 0.5f * (Ar + Br), si = 0.5f * (Ai + Bi);
        float dr = 0.5f * (Ar - Br), di = 0.5f * (Ai - Bi);
        float wr = twr_f(k * (TW_N / P)), wi = twi_f(k * (TW_N / P));
        re[k] = sr - (wr * di + wi * dr);
        im[k] = si + (wr * dr - wi * di);
    }
    cfft<N, -1>(re, im);
#pragma unroll
    for (int m = 0; m < N; m++) { p[2 * m] = re[m]; p[2 * m + 1] = im[m]; }
}

// physical p[0..P-1] -> modes 0..N-1 in FP32 (re[k], im[k]; Im c_0 = 0).
template <int P>
__device__ __forceinline__ void to_four_f(const float* p, float* cr, float* ci) {
    constexpr int N = P / 2;
    float re[N], im[N];
#pragma unroll
    for (int m = 0; m < N; m++) { re[m] = p[2 * m]; im[m] = p[2 * m + 1]; }
    cfft<N, +1>(re, im);
    const float invP = 1.0f / (float)P, two_P = 2.0f / (float)P;
    cr[0] = (re[0] + im[0]) * invP; ci[0] = 0.0f;
#pragma unroll
    for (int k = 1; k < N; k++) {
        float Fr = re[k], Fi = im[k], Gr = re[N - k], Gi = -im[N - k];
        float Er = 0.5f * (Fr + Gr), Ei = 0.5f * (Fi + Gi);
        float gr = Fr - Gr, gi = Fi - Gi;
        float Or = 0.5f * gi, Oi = -0.5f * gr;
        float vr = twr_f(k * (TW_N / P)), vi = -twi_f(k * (TW_N / P));
        cr[k] = two_P * (Er + (vr * Or - vi * Oi));
        ci[k] = two_P * (Ei + (vr * Oi + vi * Or));
    }
}

// Pass 1: one thread per (field f, point q): the FP32 physical disturbance
// d_f(z) into ph[(f * P + z) * n2 + q].
template <int P>
__global__ void __launch_bounds__(128) k_nl_phys(NlArgs A, float* __restrict__ ph) {
    const size_t n2 = A.n2;
    size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (t >= 6 * n2) return;
    const int f = (int)(t / n2);
    const size_t q = t - (size_t)f * n2;
    const cplx* F = (f == 0) ? A.ux : (f == 1) ? A.uy : (f == 2) ? A.uz : (f == 3) ? A.wx : (f == 4) ? A.wy : A.wz;
    float p[P];
    to_phys_dist<P>(F + q, n2, A.K, p);
    float* o = ph + (size_t)f * P * n2 + q;
#pragma unroll
    for (int z = 0; z < P; z++) o[(size_t)z * n2] = p[z];
}

// Pass 2: one thread per (output o, point q): the quadratic disturbance term
// through the FP32 forward transform, plus the FP64 mean terms.
// out = f[p1] f[q1] - f[p2] f[q2]: a = uy wx - ux wy, b = ux wz - uz wx, c = uz wy - uy wz.
template <int P>
__global__ void __launch_bounds__(128) k_nl_four(NlArgs A, const float* __restrict__ ph) {
    constexpr int N = P / 2;
    const size_t n2 = A.n2;
    size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (t >= 3 * n2) return;
    const int o = (int)(t / n2);
    const size_t q = t - (size_t)o * n2;
    const int p1 = (o == 0) ? 1 : (o == 1) ? 0 : 2, q1 = (o == 0) ? 3 : (o == 1) ? 5 : 4;
    const int p2 = (o == 0) ? 0 : (o == 1) ? 2 : 1, q2 = (o == 0) ? 4 : (o == 1) ? 3 : 5;
    const float *a1 = ph + (size_t)p1 * P * n2 + q, *b1 = ph + (size_t)q1 * P * n2 + q;
    const float *a2 = ph + (size_t)p2 * P * n2 + q, *b2 = ph + (size_t)q2 * P * n2 + q;
    float p[P];
#pragma unroll
    for (int z = 0; z < P; z++) {
        size_t zz = (size_t)z * n2;
        p[z] = a1[zz] * b1[zz] - a2[zz] * b2[zz];
    }
    float cr[N], ci[N];
    to_four_f<P>(p, cr, ci);
    auto fld = [&](int f) -> const cplx* {
        return (f == 0) ? A.ux : (f == 1) ? A.uy : (f == 2) ? A.uz : (f == 3) ? A.wx : (f == 4) ? A.wy : A.wz;
    };
    const cplx *P1 = fld(p1) + q, *Q1 = fld(q1) + q, *P2 = fld(p2) + q, *Q2 = fld(q2) + q;
    const double m1 = P1[0].x, n1 = Q1[0].x, m2 = P2[0].x, n2v = Q2[0].x;
    cplx* out = ((o == 0) ? A.a : (o == 1) ? A.b : A.c) + q;
    out[0] = make_double2(zap(m1 * n1 - m2 * n2v + (double)cr[0]), 0.0);
#pragma unroll
    for (int k = 1; k < N; k++) {
        if (k >= A.K) continue;
        size_t kk = (size_t)k * n2;
        cplx aq1 = Q1[kk], ap1 = P1[kk], aq2 = Q2[kk], ap2 = P2[kk];
        double vr = m1 * aq1.x + n1 * ap1.x - m2 * aq2.x - n2v * ap2.x + (double)cr[k];
        double vi = m1 * aq1.y + n1 * ap1.y - m2 * aq2.y - n2v * ap2.y + (double)ci[k];
        out[kk] = make_double2(zap(vr), zap(vi));
    }
}

// ---------------------------------------------------------------------------
// The same two passes on the tensor cores: the spanwise transforms of the
// disturbance as dense DFT-matrix GEMMs (tcgen05.mma, kind::f16), every FP32
// operand split into three BF16 parts (x = x0 + x1 + x2 exactly, 8 bits each)
// and the products compensated to FP32 accuracy,
//   a b ~ a0 b0 + (a0 b1 + a1 b0) + (a0 b2 + a1 b1 + a2 b0),
// accumulated in FP32 in tensor memory.  A tile is 128 points (one per
// thread and tensor-memory lane); per point the P "slots" hold Re c0 (0: the
// mean stays in FP64), Im c0 (the packed Nyquist term) and Re, Im of modes
// 1 .. P/2-1.  Pass 1: phys[pt][z] = sum_s slot[pt][s] Tinv[z][s]; pass 2:
// slot[pt][s] = sum_z prod[pt][z] Tfwd[s][z], the transforms to_phys_dist and
// to_four_f above written as matrices (tb_dft_matrices).
//
// Shared memory, K-major without swizzle: element (row r, k) of an operand
// with R rows sits at (k / 8) * (R * 16) + r * 16 + (k % 8) * 2 bytes, so a
// core matrix (8 rows x 8 k) is 128 contiguous bytes, core matrices
// adjacent in rows are 128 bytes apart and those adjacent in k R * 16 apart.
constexpr int TC_PARTS = 3;   // BF16 parts per FP32 operand

template <int P>
struct TcLayout {
    static constexpr int AB = 128 * P * 2, BB = P * P * 2;                 // bytes of one operand part
    static constexpr int A0 = 0, B0 = TC_PARTS * AB;                       // part p at A0 + p AB, B0 + p BB
    static constexpr int BAR = B0 + TC_PARTS * BB;                         // mbarrier, then the TMEM address
    static constexpr int BYTES = BAR + 16;
    static constexpr uint32_t NCOL = P < 32 ? 32 : P;                      // tensor-memory columns
    static constexpr uint32_t ID = tbtc::idesc_bf16_f32(128, P);
    // resident blocks per SM: shared memory (227 KB), tensor memory (512 columns), at most 8
    static constexpr int PER_SM_SMEM = (227 * 1024) / BYTES, PER_SM_TMEM = 512 / (int)NCOL;
    static constexpr int PER_SM0 = PER_SM_SMEM < PER_SM_TMEM ? PER_SM_SMEM : PER_SM_TMEM;
    static constexpr int PER_SM = PER_SM0 < 8 ? PER_SM0 : 8;
};

// x = x0 + x1 + x2 with BF16 parts (round to nearest at each step).
__device__ __forceinline__ void split_bf16(float x, unsigned short* p) {
#pragma unroll
    for (int q = 0; q < TC_PARTS; q++) {
        const __nv_bfloat16 b = __float2bfloat16_rn(x);
        p[q] = __bfloat16_as_ushort(b);
        x -= __bfloat162float(b);
    }
}

// Values 8 g0 .. 8 g0 + P/2 - 1 of row `row` of the A operand into its BF16 parts.
template <int P>
__device__ __forceinline__ void stage_row(unsigned char* sm, int row, int g0, const float* v) {
    using Lt = TcLayout<P>;
#pragma unroll
    for (int g = 0; g < P / 16; g++) {
        unsigned short h[TC_PARTS][8];
#pragma unroll
        for (int e = 0; e < 8; e++) {
            unsigned short p[TC_PARTS];
            split_bf16(v[8 * g + e], p);
#pragma unroll
            for (int q = 0; q < TC_PARTS; q++) h[q][e] = p[q];
        }
#pragma unroll
        for (int q = 0; q < TC_PARTS; q++) {
            uint4 H;
            H.x = h[q][0] | ((uint32_t)h[q][1] << 16); H.y = h[q][2] | ((uint32_t)h[q][3] << 16);
            H.z = h[q][4] | ((uint32_t)h[q][5] << 16); H.w = h[q][6] | ((uint32_t)h[q][7] << 16);
            *reinterpret_cast<uint4*>(sm + Lt::A0 + q * Lt::AB + (g0 + g) * 2048 + row * 16) = H;
        }
    }
}

// One thread issues the tile's MMAs (the six part products of order <= 2
// per 16-wide k-step) and commits them.
template <int P>
__device__ __forceinline__ void tile_mma(unsigned char* sm, uint32_t tmem, uint64_t* bar) {
    using Lt = TcLayout<P>;
    const uint32_t base = tbtc::smem_u32(sm);
#pragma unroll
    for (int ks = 0; ks < P / 16; ks++) {
        const uint32_t ao = ks * 2 * 2048, bo = ks * 2 * P * 16;
        uint64_t a[TC_PARTS], b[TC_PARTS];
#pragma unroll
        for (int q = 0; q < TC_PARTS; q++) {
            a[q] = tbtc::sdesc(base + Lt::A0 + q * Lt::AB + ao, 2048, 128);
            b[q] = tbtc::sdesc(base + Lt::B0 + q * Lt::BB + bo, P * 16, 128);
        }
        tbtc::mma_bf16(tmem, a[0], b[0], Lt::ID, ks > 0);
        tbtc::mma_bf16(tmem, a[0], b[1], Lt::ID, 1);
        tbtc::mma_bf16(tmem, a[1], b[0], Lt::ID, 1);
        tbtc::mma_bf16(tmem, a[0], b[2], Lt::ID, 1);
        tbtc::mma_bf16(tmem, a[1], b[1], Lt::ID, 1);
        tbtc::mma_bf16(tmem, a[2], b[0], Lt::ID, 1);
    }
    tbtc::mma_commit(bar);
}

// Set-up shared by both passes: the constant B operand (its BF16 parts) into
// shared memory, the mbarrier, and the tensor-memory columns.
template <int P>
__device__ __forceinline__ uint32_t tc_setup(unsigned char* sm, const uint16_t* mats) {
    using Lt = TcLayout<P>;
    const int t = threadIdx.x;
    for (int i = t; i < TC_PARTS * P * P / 8; i += blockDim.x)
        reinterpret_cast<uint4*>(sm + Lt::B0)[i] = reinterpret_cast<const uint4*>(mats)[i];
    uint64_t* bar = reinterpret_cast<uint64_t*>(sm + Lt::BAR);
    uint32_t* slot = reinterpret_cast<uint32_t*>(sm + Lt::BAR + 8);
    if (t == 0) tbtc::mbar_init(bar, 1);
    if ((t >> 5) == 0) {
        tbtc::tmem_alloc(slot, Lt::NCOL);
        tbtc::tmem_relinquish();
    }
    tbtc::fence_before_sync();
    __syncthreads();
    tbtc::fence_after_sync();
    return *slot;
}

// Issue, wait (bounded) and read: returns false (for the whole block) when
// the wait ran out, after which the caller stops issuing.
// TcCtl: the wait limit in polls and, for tests of the time-out path only,
// a switch that leaves the MMAs unissued so that the wait runs out.
struct TcCtl {
    uint32_t limit;
    int skip_mma;
};

template <int P>
__device__ __forceinline__ bool tc_run(unsigned char* sm, uint32_t tmem, uint32_t& phase, const TcCtl& ctl) {
    using Lt = TcLayout<P>;
    uint64_t* bar = reinterpret_cast<uint64_t*>(sm + Lt::BAR);
    tbtc::fence_async_smem();
    __syncthreads();
    if (threadIdx.x == 0 && !ctl.skip_mma) {
        tbtc::fence_after_sync();
        tile_mma<P>(sm, tmem, bar);
    }
    const bool ok = tbtc::mbar_wait(bar, phase, ctl.limit);
    tbtc::fence_after_sync();
    const bool all = !__syncthreads_or(!ok);
    if (all) phase ^= 1u;   // on a time-out `phase` stays that of the tile in flight
    return all;
}

template <int P>
__device__ __forceinline__ void tc_teardown(unsigned char* sm, uint32_t tmem, bool ok, uint32_t phase, int* err,
                                            const TcCtl& ctl) {
    using Lt = TcLayout<P>;
    if (!ok) {   // let the MMAs of the abandoned tile finish (bounded) before freeing their columns
        (void)tbtc::mbar_wait(reinterpret_cast<uint64_t*>(sm + Lt::BAR), phase, ctl.limit);
        if (threadIdx.x == 0) atomicExch(err, 1);
    }
    tbtc::fence_before_sync();
    __syncthreads();
    tbtc::fence_after_sync();
    if ((threadIdx.x >> 5) == 0) tbtc::tmem_dealloc(tmem, Lt::NCOL);
}

__device__ __forceinline__ const cplx* nl_field(const NlArgs& A, int f) {
    return (f == 0) ? A.ux : (f == 1) ? A.uy : (f == 2) ? A.uz : (f == 3) ? A.wx : (f == 4) ? A.wy : A.wz;
}

// Both passes take a tile of 128 points with two threads a point, one for the
// lower and one for the upper half of its slots or physical points: what they wait
// for is their loads, and shared memory holds few tiles per SM (one at P = 128).
// One thread a point took 4.3 ms (P = 128) and 1.01 ms (P = 64) for both passes at
// 1025 x 193 points; two take 2.57 and 0.81.
constexpr int TC_THREADS = 256;

// Columns of this thread's half of its point's row of tensor memory, with 8 of them (P =
// 16) out of the 16 that one load gives.
template <int P>
__device__ __forceinline__ void tmem_half(uint32_t tmem, int warp, int half, float* v) {
    constexpr int H = P / 2;
    const uint32_t lane = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    if constexpr (H < 16) {
        float w[16];
        tbtc::tmem_ld16(lane, w);
#pragma unroll
        for (int i = 0; i < H; i++) v[i] = half ? w[H + i] : w[i];
    } else {
#pragma unroll
        for (int c = 0; c < H; c += 16) tbtc::tmem_ld16(lane + half * H + c, v + c);
    }
}

// Pass 1 on the tensor cores: tile = (field f, 128 points) -> ph[(f P + z) n2 + q].
template <int P>
__global__ void __launch_bounds__(TC_THREADS) k_nl_phys_tc(NlArgs A, float* __restrict__ ph, const uint16_t* __restrict__ mats,
                                                           int* err, TcCtl ctl) {
    constexpr int H = P / 2;
    extern __shared__ __align__(1024) unsigned char sm[];
    const uint32_t tmem = tc_setup<P>(sm, mats);
    const int t = threadIdx.x & 127, half = threadIdx.x >> 7, warp = threadIdx.x >> 5;
    const size_t n2 = A.n2;
    const int tpf = (int)((n2 + 127) / 128), ntiles = 6 * tpf;
    uint32_t phase = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int f = tile / tpf;
        const size_t q = (size_t)(tile % tpf) * 128 + t;
        const cplx* F = nl_field(A, f) + q;
        float v[H];
#pragma unroll
        for (int i = 0; i < H / 2; i++) {
            const int k = half * (H / 2) + i;
            cplx c = make_double2(0.0, 0.0);
            if (k < A.K && q < n2) c = F[(size_t)k * n2];
            v[2 * i] = k ? (float)c.x : 0.f;
            v[2 * i + 1] = (float)c.y;
        }
        stage_row<P>(sm, t, half * (H / 8), v);
        if (!(ok = tc_run<P>(sm, tmem, phase, ctl))) break;
        tmem_half<P>(tmem, warp, half, v);
        if (q < n2) {
            float* o = ph + ((size_t)f * P + half * H) * n2 + q;
#pragma unroll
            for (int i = 0; i < H; i++) o[(size_t)i * n2] = v[i];
        }
        tbtc::fence_before_sync();
        __syncthreads();
    }
    tc_teardown<P>(sm, tmem, ok, phase, err, ctl);
}

// Pass 2 on the tensor cores: tile = (output o, 128 points); the quadratic
// disturbance term's slots plus the FP64 mean terms, as k_nl_four.
template <int P>
__global__ void __launch_bounds__(TC_THREADS) k_nl_four_tc(NlArgs A, const float* __restrict__ ph,
                                                           const uint16_t* __restrict__ mats, int* err, TcCtl ctl) {
    constexpr int H = P / 2;
    extern __shared__ __align__(1024) unsigned char sm[];
    const uint32_t tmem = tc_setup<P>(sm, mats);
    const int t = threadIdx.x & 127, half = threadIdx.x >> 7, warp = threadIdx.x >> 5;
    const size_t n2 = A.n2;
    const int tpf = (int)((n2 + 127) / 128), ntiles = 3 * tpf;
    uint32_t phase = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int o = tile / tpf;
        const size_t q = (size_t)(tile % tpf) * 128 + t;
        const int p1 = (o == 0) ? 1 : (o == 1) ? 0 : 2, q1 = (o == 0) ? 3 : (o == 1) ? 5 : 4;
        const int p2 = (o == 0) ? 0 : (o == 1) ? 2 : 1, q2 = (o == 0) ? 4 : (o == 1) ? 3 : 5;
        float v[H];
#pragma unroll
        for (int i = 0; i < H; i++) v[i] = 0.f;
        if (q < n2) {
            const size_t z0 = (size_t)half * H * n2 + q;
            const float *a1 = ph + (size_t)p1 * P * n2 + z0, *b1 = ph + (size_t)q1 * P * n2 + z0;
            const float *a2 = ph + (size_t)p2 * P * n2 + z0, *b2 = ph + (size_t)q2 * P * n2 + z0;
#pragma unroll
            for (int i = 0; i < H; i++) {
                const size_t zz = (size_t)i * n2;
                v[i] = a1[zz] * b1[zz] - a2[zz] * b2[zz];
            }
        }
        stage_row<P>(sm, t, half * (H / 8), v);
        if (!(ok = tc_run<P>(sm, tmem, phase, ctl))) break;
        tmem_half<P>(tmem, warp, half, v);
        if (q < n2) {
            const cplx *P1 = nl_field(A, p1) + q, *Q1 = nl_field(A, q1) + q, *P2 = nl_field(A, p2) + q, *Q2 = nl_field(A, q2) + q;
            const double m1 = P1[0].x, n1 = Q1[0].x, m2 = P2[0].x, n2v = Q2[0].x;
            cplx* out = ((o == 0) ? A.a : (o == 1) ? A.b : A.c) + q;
            if (half == 0) out[0] = make_double2(zap(m1 * n1 - m2 * n2v + (double)v[0]), 0.0);
#pragma unroll
            for (int i = 0; i < H / 2; i++) {
                const int k = half * (H / 2) + i;
                if (k == 0 || k >= A.K) continue;
                const size_t kk = (size_t)k * n2;
                const cplx aq1 = Q1[kk], ap1 = P1[kk], aq2 = Q2[kk], ap2 = P2[kk];
                const double vr = m1 * aq1.x + n1 * ap1.x - m2 * aq2.x - n2v * ap2.x + (double)v[2 * i];
                const double vi = m1 * aq1.y + n1 * ap1.y - m2 * aq2.y - n2v * ap2.y + (double)v[2 * i + 1];
                out[kk] = make_double2(zap(vr), zap(vi));
            }
        }
        tbtc::fence_before_sync();
        __syncthreads();
    }
    tc_teardown<P>(sm, tmem, ok, phase, err, ctl);
}

// Smagorinsky eddy viscosity and force nu_t lap(u) (les_par.f:6-211).
struct LesArgs {
    const cplx *dudx, *dvdx, *dwdx, *dudy, *dvdy, *dwdy;   // Fourier gradients
    const cplx *ux, *uy, *uz;                              // z-derivatives formed as -i k beta u
    const cplx *d2x[3], *d2y[3];                           // second derivatives of ux, uy, uz
    const double* k2b2;
    const cplx* wz;                                        // wall vorticity for y+
    cplx *fx, *fy, *fz;
    int nx, ny, n2, K, damping;
    double beta, Re, fac_y, dy, stf, Cs, Aplus, delta_les;
};
// Eddy viscosity and force of one grid line on Col<P>::TP threads, each with
// its share of the strain in shared memory.  The six distinct strain
// components are summed before their transforms: six of these, three of the
// Laplacian and three back, where the nine velocity gradients took fifteen.
// Bound by the FP64 pipe: 19.6 ms at 1025 x 193 x 64 (P = 128) with one thread a
// line and its arrays in local memory, 10.3 ms now.
template <int P>
__global__ void __launch_bounds__(128, 2) k_les(LesArgs A) {
    using CP = Col<P>;
    constexpr int M = CP::M;
    extern __shared__ double strain[];
    const int tid = threadIdx.x, p = CP::TP == 2 ? (tid >> 4) & 1 : 0;
    const int col = blockIdx.x * CP::PER_BLOCK + (CP::TP == 2 ? (tid >> 5) * 16 + (tid & 15) : tid);
    const bool in = col < A.n2;
    const int q = in ? col : A.n2 - 1;   // both threads of a line take part in its shuffles
    const size_t cs = A.n2;
    const int i = q % A.nx, j = q / A.nx;
    double y = (A.stf == 1.0) ? (double)j * A.dy : A.dy * (pow(A.stf, (double)j) - 1.0) / (A.stf - 1.0);
    double wz0 = (A.damping & 2) ? fabs(A.wz[i].x) : A.wz[i].x;
    double yplus = sqrt(A.Re * wz0 / sqrt(A.fac_y)) * y;
    double damp;
    if (A.damping & 1) {
        double e = 1.0 - exp(-yplus / A.Aplus);
        damp = e * e;
    } else {
        double ratio = fmin(yplus / A.Aplus, 100.0);
        ratio = ratio * ratio * ratio;
        damp = 1.0 - exp(-ratio);
    }
    const double cte = A.Cs * A.Cs * A.delta_les * A.delta_les * damp;
    double re[M], im[M];
    double* S = strain + tid;   // value v at v * 128
    // s_xx, s_yy, s_zz and twice s_xy, s_xz, s_yz: fields a (of 3: its z-derivative) + b
    for (int t = 0; t < 6; t++) {
        const cplx* a = (t == 0 ? A.dudx : t == 1 ? A.dvdy : t == 2 ? A.uz : t == 3 ? A.dudy : t == 4 ? A.ux : A.uy) + q;
        const cplx* b = t < 3 ? nullptr : (t == 3 ? A.dvdx : t == 4 ? A.dwdx : A.dwdy) + q;
        const bool dz = t == 2 || t > 3;
        col_phys2<P>([&](int k) {
            if (k >= A.K) return make_double2(0.0, 0.0);
            cplx v = a[(size_t)k * cs];
            if (dz) {   // -i (k-1) beta u  (main_par.f:1888)
                const double kb = -(double)k * A.beta;
                v = make_double2(-kb * v.y, kb * v.x);
            }
            if (b) { const cplx w = b[(size_t)k * cs]; v.x += w.x; v.y += w.y; }
            return v;
        }, p, re, im);
        const double f = t < 3 ? 1.0 : 0.5;
#pragma unroll
        for (int m = 0; m < M; m++) {
            const double u = f * re[m], w = f * im[m];
            S[(2 * m) * 128] = t ? fma(u, re[m], S[(2 * m) * 128]) : u * re[m];
            S[(2 * m + 1) * 128] = t ? fma(w, im[m], S[(2 * m + 1) * 128]) : w * im[m];
        }
    }
    // nu_t = cte sqrt(2 S); S is four times the sum of squares here, and the
    // factors 2 of the Laplacian and 1 / P of the transform back are taken along
    for (int v = 0; v < 2 * M; v++) S[v * 128] = (cte * (0.5 / (double)P)) * sqrt(0.5 * S[v * 128]);
    for (int f = 0; f < 3; f++) {
        const cplx* d2x = A.d2x[f] + q;
        const cplx* d2y = A.d2y[f] + q;
        const cplx* us = (f == 0 ? A.ux : f == 1 ? A.uy : A.uz) + q;
        cplx* out = (f == 0 ? A.fx : f == 1 ? A.fy : A.fz) + q;
        col_phys2<P>([&](int k) {
            if (k >= A.K) return make_double2(0.0, 0.0);
            const size_t o = (size_t)k * cs;
            const cplx a = d2x[o], b = d2y[o], u = us[o];
            const double kk = A.k2b2[k];
            return make_double2(fma(kk, u.x, a.x + b.x), fma(kk, u.y, a.y + b.y));
        }, p, re, im);
#pragma unroll
        for (int m = 0; m < M; m++) { re[m] *= S[(2 * m) * 128]; im[m] *= S[(2 * m + 1) * 128]; }
        col_four<P>(re, im, p, [&](int k, cplx v) { if (in && k < A.K) out[(size_t)k * cs] = v; });
    }
}

// Immersed-boundary feedback force (cvirt immersed_par.f:262-313):
// f = irf delta u in physical space, back to Fourier, Gibbs-filtered.
struct IbmArgs {
    const cplx *ux, *uy, *uz;
    const double* delta;
    const double* gibbs;
    cplx *fx, *fy, *fz;
    int n2, K, accumulate;
    double irf;
};
// The roughness touches few grid lines: a warp whose lines have delta = 0
// everywhere and finite velocities (which a NaN would have to reach) writes
// the zero force, or leaves what it would be added to, after one pass over
// delta and u: 0.36 ms at 1025 x 193 x 64, 6.3 ms with every line transformed.
template <int P>
__global__ void __launch_bounds__(128) k_cvirt(IbmArgs A) {
    using CP = Col<P>;
    constexpr int M = CP::M;
    const int tid = threadIdx.x, p = CP::TP == 2 ? (tid >> 4) & 1 : 0;
    const int col = blockIdx.x * CP::PER_BLOCK + (CP::TP == 2 ? (tid >> 5) * 16 + (tid & 15) : tid);
    const bool in = col < A.n2;
    const int q = in ? col : A.n2 - 1;
    const size_t cs = A.n2;
    const cplx* us[3] = {A.ux + q, A.uy + q, A.uz + q};
    cplx* outs[3] = {A.fx + q, A.fy + q, A.fz + q};
    const double* delta = A.delta + q;
    auto finite = [](double v) { return ((unsigned)__double2hiint(v) & 0x7ff00000u) != 0x7ff00000u; };
    bool work = !finite(A.irf);
#pragma unroll 8
    for (int z = p; z < P; z += CP::TP) work |= delta[cs * z] != 0.0;
    if (!__any_sync(0xffffffffu, work)) {
        for (int f = 0; f < 3; f++)
#pragma unroll 8
            for (int k = p; k < A.K; k += CP::TP) {
                const cplx v = us[f][cs * k];
                work |= !finite(v.x) || !finite(v.y);
            }
        if (!__any_sync(0xffffffffu, work)) {
            if (!A.accumulate && in)
                for (int f = 0; f < 3; f++)
                    for (int k = p; k < A.K && k < P / 2; k += CP::TP) outs[f][cs * k] = make_double2(0.0, 0.0);
            return;
        }
    }
    double re[M], im[M];
    const double sc = A.irf * (0.5 / (double)P);
    for (int f = 0; f < 3; f++) {
        col_phys2<P>(Modes{us[f], cs, A.K}, p, re, im);
#pragma unroll
        for (int m = 0; m < M; m++) {
            const size_t z = 2 * (size_t)(m * CP::TP + p);
            re[m] = sc * delta[cs * z] * re[m];
            im[m] = sc * delta[cs * (z + 1)] * im[m];
        }
        col_four<P>(re, im, p, [&](int k, cplx v) {
            if (!in || k >= A.K) return;
            v.x *= A.gibbs[k]; v.y *= A.gibbs[k];
            cplx* o = outs[f] + cs * k;
            if (A.accumulate) { const cplx w = *o; v.x += w.x; v.y += w.y; }
            *o = v;
        });
    }
}

// delta() (immersed_par.f:98-181): smoothed roughness indicator, filtered
// through p_to_f -> gibbs -> f_to_p.
template <int P>
__global__ void k_delta_filter(double* delta, const double* gibbs, int n2, int K) {
    int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n2) return;
    constexpr int N = P / 2;
    double p[P];
    cplx tmp[N];
#pragma unroll
    for (int z = 0; z < P; z++) p[z] = delta[(size_t)q + (size_t)n2 * z] * (1.0 / (double)P);
    to_four<P>(p, [&](int k, cplx v) { tmp[k] = k < K ? make_double2(gibbs[k] * v.x, gibbs[k] * v.y) : make_double2(0.0, 0.0); });
    to_phys2<P>([&](int k) { return tmp[k]; }, p);
#pragma unroll
    for (int z = 0; z < P; z++) delta[(size_t)q + (size_t)n2 * z] = 0.5 * p[z];
}

bool g_tw_ready[64] = {false};

int ensure_twiddles(tb_ctx* c) {
    int dev = c->device;
    if (dev >= 0 && dev < 64 && g_tw_ready[dev]) return TB_OK;
    double hr[TW_N], hi[TW_N], lm[TW_N / 2], lr[TW_N / 2];
    for (int t = 0; t < TW_N; t++) {
        long double ang = -2.0L * 3.141592653589793238462643383279502884L * (long double)t / (long double)TW_N;
        hr[t] = (double)cosl(ang);
        hi[t] = (double)sinl(ang);
    }
    TB_CUDA(cudaMemcpyToSymbol(c_twr, hr, sizeof hr));
    TB_CUDA(cudaMemcpyToSymbol(c_twi, hi, sizeof hi));
    for (int t = 0; t < TW_N / 2; t++) {
        const long double ang = -2.0L * 3.141592653589793238462643383279502884L * (long double)t / (long double)TW_N;
        const long double wr = cosl(ang), wi = sinl(ang);
        const bool big = lf_big(t);
        lm[t] = (double)(big ? wr : wi);
        lr[t] = (double)(big ? wi / wr : wr / wi);
    }
    TB_CUDA(cudaMemcpyToSymbol(c_lfm, lm, sizeof lm));
    TB_CUDA(cudaMemcpyToSymbol(c_lfr, lr, sizeof lr));
    float fr[TW_N], fi[TW_N];
    for (int t = 0; t < TW_N; t++) { fr[t] = (float)hr[t]; fi[t] = (float)hi[t]; }
    TB_CUDA(cudaMemcpyToSymbol(c_twrf, fr, sizeof fr));
    TB_CUDA(cudaMemcpyToSymbol(c_twif, fi, sizeof fi));
    if (dev >= 0 && dev < 64) g_tw_ready[dev] = true;
    return TB_OK;
}

#define TB_DISPATCH_P(P, ...)                                            \
    switch (P) {                                                         \
        case 2: { constexpr int PP = 2; __VA_ARGS__; } break;                   \
        case 4: { constexpr int PP = 4; __VA_ARGS__; } break;                   \
        case 8: { constexpr int PP = 8; __VA_ARGS__; } break;                   \
        case 16: { constexpr int PP = 16; __VA_ARGS__; } break;                 \
        case 32: { constexpr int PP = 32; __VA_ARGS__; } break;                 \
        case 64: { constexpr int PP = 64; __VA_ARGS__; } break;                 \
        case 128: { constexpr int PP = 128; __VA_ARGS__; } break;               \
        default: tb_set_error("kphys %d not supported", P); return TB_ERR_ARG; \
    }

}  // namespace

int tb_launch_f_to_p(tb_ctx* c, double* phys, const cplx* four) {
    int r = ensure_twiddles(c);
    if (r) return r;
    int n2 = (int)tb_n2(c);
    unsigned nb = tb_blocks(n2, 128);
    TB_DISPATCH_P(c->g.P, (k_f_to_p<PP><<<nb, 128, 0, c->stream>>>(phys, four, n2, c->g.K)));
    TB_CHECK_LAUNCH(c);
    return TB_OK;
}
int tb_launch_p_to_f(tb_ctx* c, cplx* four, const double* phys) {
    int r = ensure_twiddles(c);
    if (r) return r;
    int n2 = (int)tb_n2(c);
    unsigned nb = tb_blocks(n2, 128);
    TB_DISPATCH_P(c->g.P, (k_p_to_f<PP><<<nb, 128, 0, c->stream>>>(four, phys, n2, c->g.K)));
    TB_CHECK_LAUNCH(c);
    return TB_OK;
}
// ---- the DFT matrices of the tensor-core passes ------------------------------
static uint16_t bf16_bits(float f) {   // round to nearest even
    uint32_t u;
    std::memcpy(&u, &f, 4);
    u += 0x7FFFu + ((u >> 16) & 1u);
    return (uint16_t)(u >> 16);
}
static float bf16_value(uint16_t h) {
    uint32_t u = (uint32_t)h << 16;
    float f;
    std::memcpy(&f, &u, 4);
    return f;
}

// to_phys_dist and to_four_f in double precision on slot vectors, with the
// length-N complex transforms of cfft written as plain sums.
static const double TB_PI = 3.14159265358979323846;
static void host_cdft(int N, int sign, std::vector<double>& re, std::vector<double>& im) {
    std::vector<double> r(N, 0.0), i(N, 0.0);
    for (int m = 0; m < N; m++)
        for (int k = 0; k < N; k++) {
            const double a = sign * 2.0 * TB_PI * (double)((long)k * m % N) / N;
            r[m] += re[k] * std::cos(a) - im[k] * std::sin(a);
            i[m] += re[k] * std::sin(a) + im[k] * std::cos(a);
        }
    re = r;
    im = i;
}
static void host_phys_from_slots(int P, const double* s, double* p) {
    const int N = P / 2;
    std::vector<double> re(N), im(N);
    re[0] = 0.5 * s[1];
    im[0] = -0.5 * s[1];
    for (int k = 1; k < N; k++) {
        const double Ar = s[2 * k], Ai = s[2 * k + 1], Br = s[2 * (N - k)], Bi = -s[2 * (N - k) + 1];
        const double sr = 0.5 * (Ar + Br), si = 0.5 * (Ai + Bi), dr = 0.5 * (Ar - Br), di = 0.5 * (Ai - Bi);
        const double wr = std::cos(2.0 * TB_PI * k / P), wi = -std::sin(2.0 * TB_PI * k / P);
        re[k] = sr - (wr * di + wi * dr);
        im[k] = si + (wr * dr - wi * di);
    }
    host_cdft(N, -1, re, im);
    for (int m = 0; m < N; m++) { p[2 * m] = re[m]; p[2 * m + 1] = im[m]; }
}
static void host_slots_from_phys(int P, const double* p, double* s) {
    const int N = P / 2;
    std::vector<double> re(N), im(N);
    for (int m = 0; m < N; m++) { re[m] = p[2 * m]; im[m] = p[2 * m + 1]; }
    host_cdft(N, +1, re, im);
    s[0] = (re[0] + im[0]) / P;
    s[1] = 0.0;
    for (int k = 1; k < N; k++) {
        const double Fr = re[k], Fi = im[k], Gr = re[N - k], Gi = -im[N - k];
        const double Er = 0.5 * (Fr + Gr), Ei = 0.5 * (Fi + Gi), gr = Fr - Gr, gi = Fi - Gi;
        const double Or = 0.5 * gi, Oi = -0.5 * gr;
        const double vr = std::cos(2.0 * TB_PI * k / P), vi = std::sin(2.0 * TB_PI * k / P);
        s[2 * k] = 2.0 / P * (Er + (vr * Or - vi * Oi));
        s[2 * k + 1] = 2.0 / P * (Ei + (vr * Oi + vi * Or));
    }
}

// B operands of both passes, their TC_PARTS BF16 parts, in the K-major core
// layout of TcLayout: inverse (n = z, k = slot) then forward (n = slot, k = z).
void tb_dft_matrices(int P, std::vector<uint16_t>& out) {
    std::vector<double> Tinv((size_t)P * P), Tfwd((size_t)P * P), e(P), v(P);
    for (int s = 0; s < P; s++) {
        std::fill(e.begin(), e.end(), 0.0);
        e[s] = 1.0;
        host_phys_from_slots(P, e.data(), v.data());
        for (int z = 0; z < P; z++) Tinv[(size_t)z * P + s] = v[z];
        host_slots_from_phys(P, e.data(), v.data());   // e as a physical unit vector at z = s
        for (int q = 0; q < P; q++) Tfwd[(size_t)q * P + s] = v[q];
    }
    out.assign((size_t)2 * TC_PARTS * P * P, 0);
    auto put = [&](int first, const std::vector<double>& T) {   // T[n][k]
        for (int n = 0; n < P; n++)
            for (int k = 0; k < P; k++) {
                float x = (float)T[(size_t)n * P + k];
                const size_t o = (size_t)(k / 8) * (P * 8) + (size_t)n * 8 + (k % 8);
                for (int q = 0; q < TC_PARTS; q++) {
                    const uint16_t h = bf16_bits(x);
                    out[(size_t)(first + q) * P * P + o] = h;
                    x -= bf16_value(h);
                }
            }
    };
    put(0, Tinv);
    put(TC_PARTS, Tfwd);
}

// The two matrices in double precision, P x P row-major [n][k]: forward 0
// gives Tinv[z][slot], forward 1 gives Tfwd[slot][z].
extern "C" int tb_dft_matrix(int P, int forward, double* out) {
    if (!out || P < 4 || (P & (P - 1))) { tb_set_error("P must be a power of two >= 4"); return TB_ERR_ARG; }
    std::vector<double> e(P), v(P);
    for (int s = 0; s < P; s++) {
        std::fill(e.begin(), e.end(), 0.0);
        e[s] = 1.0;
        if (forward) {
            host_slots_from_phys(P, e.data(), v.data());
            for (int q = 0; q < P; q++) out[(size_t)q * P + s] = v[q];
        } else {
            host_phys_from_slots(P, e.data(), v.data());
            for (int z = 0; z < P; z++) out[(size_t)z * P + s] = v[z];
        }
    }
    return TB_OK;
}

static bool tc_form(const tb_ctx* c) {
    const int P = c->g.P;
    return c->cfg.precision == TB_FORM_MIXED && c->nl_tensor && (P == 16 || P == 32 || P == 64 || P == 128);
}

static bool g_tc_attr[64][4] = {{false}};

template <int P>
static int tc_attrs(int dev) {
    const int slot = P == 16 ? 0 : P == 32 ? 1 : P == 64 ? 2 : 3;
    if (dev >= 0 && dev < 64 && g_tc_attr[dev][slot]) return TB_OK;
    TB_CUDA(cudaFuncSetAttribute(k_nl_phys_tc<P>, cudaFuncAttributeMaxDynamicSharedMemorySize, TcLayout<P>::BYTES));
    TB_CUDA(cudaFuncSetAttribute(k_nl_four_tc<P>, cudaFuncAttributeMaxDynamicSharedMemorySize, TcLayout<P>::BYTES));
    if (dev >= 0 && dev < 64) g_tc_attr[dev][slot] = true;
    return TB_OK;
}

static int ensure_tc(tb_ctx* c) {
    if (!tc_form(c)) return TB_OK;
    int r;
    switch (c->g.P) {
        case 16: r = tc_attrs<16>(c->device); break;
        case 32: r = tc_attrs<32>(c->device); break;
        case 64: r = tc_attrs<64>(c->device); break;
        default: r = tc_attrs<128>(c->device); break;
    }
    if (r) return r;
    if (!c->dft_tc) {
        std::vector<uint16_t> m;
        tb_dft_matrices(c->g.P, m);
        TB_CUDA(cudaMalloc(&c->dft_tc, m.size() * sizeof(uint16_t)));
        TB_CUDA(cudaMemcpy(c->dft_tc, m.data(), m.size() * sizeof(uint16_t), cudaMemcpyHostToDevice));
    }
    if (!c->tc_err) {
        TB_CUDA(cudaMalloc(&c->tc_err, sizeof(int)));
        TB_CUDA(cudaMemset(c->tc_err, 0, sizeof(int)));
    }
    return TB_OK;
}

int tb_spectral_prepare(tb_ctx* c) {
    int r = ensure_twiddles(c);
    if (r) return r;
    if (c->cfg.precision == TB_FORM_MIXED && c->g.P >= 4 && !c->nl_phys)
        TB_CUDA(cudaMalloc(&c->nl_phys, (size_t)6 * c->g.P * tb_n2(c) * sizeof(float)));
    return ensure_tc(c);
}

int tb_tc_check(tb_ctx* c) {
    if (!c->tc_err) return TB_OK;
    int e = 0;
    TB_CUDA(cudaMemcpy(&e, c->tc_err, sizeof(int), cudaMemcpyDeviceToHost));
    if (e) {
        TB_CUDA(cudaMemset(c->tc_err, 0, sizeof(int)));
        tb_set_error("nlterms (tensor cores): a bounded wait for the MMAs ran out");
        return TB_ERR_TIMEOUT;
    }
    return TB_OK;
}

int tb_launch_nlterms(tb_ctx* c, cplx* a, cplx* b, cplx* cc) {
    int r = ensure_twiddles(c);
    if (r) return r;
    NlArgs A{c->ux, c->uy, c->uz, c->wx, c->wy, c->wz, a, b, cc, (int)tb_n2(c), c->g.K};
    cudaEvent_t ps = nullptr;
    if ((r = tb_prof_begin(c, PROF_NLTERMS, &ps))) return r;
    if (tc_form(c)) {
        if (!c->capturing && (r = tb_spectral_prepare(c))) return r;
        const int P = c->g.P, sms = c->sm_count > 0 ? c->sm_count : 148;
        const size_t tiles = (A.n2 + 127) / 128;
        // a time-out test shortens the wait to a few thousand polls and leaves the MMAs unissued
        const TcCtl ctl{c->tc_timeout_test ? 4096u : (1u << 22), c->tc_timeout_test};
        switch (P) {
#define TB_TC_CASE(PP)                                                                                        \
    case PP: {                                                                                                 \
        const int per = (c->tune_nl >= 1 && c->tune_nl <= TcLayout<PP>::PER_SM) ? c->tune_nl : TcLayout<PP>::PER_SM; \
        const size_t cap = (size_t)per * sms;                                                                  \
        const unsigned g1 = (unsigned)std::min<size_t>(6 * tiles, cap), g2 = (unsigned)std::min<size_t>(3 * tiles, cap); \
        k_nl_phys_tc<PP><<<g1, TC_THREADS, TcLayout<PP>::BYTES, c->stream>>>(A, c->nl_phys, c->dft_tc, c->tc_err, ctl);   \
        TB_CHECK_LAUNCH(c);                                                                                    \
        k_nl_four_tc<PP><<<g2, TC_THREADS, TcLayout<PP>::BYTES, c->stream>>>(A, c->nl_phys, c->dft_tc + TC_PARTS * PP * PP, \
                                                                      c->tc_err, ctl);                         \
        break;                                                                                                 \
    }
            TB_TC_CASE(16)
            TB_TC_CASE(32)
            TB_TC_CASE(64)
            TB_TC_CASE(128)
#undef TB_TC_CASE
        }
    } else if (c->cfg.precision == TB_FORM_MIXED && c->g.P >= 4) {
        size_t need = (size_t)6 * c->g.P * A.n2;
        if (!c->nl_phys) TB_CUDA(cudaMalloc(&c->nl_phys, need * sizeof(float)));
        TB_DISPATCH_P(c->g.P, (k_nl_phys<PP><<<tb_blocks(6 * (size_t)A.n2, 128), 128, 0, c->stream>>>(A, c->nl_phys)));
        TB_CHECK_LAUNCH(c);
        TB_DISPATCH_P(c->g.P, (k_nl_four<PP><<<tb_blocks(3 * (size_t)A.n2, 128), 128, 0, c->stream>>>(A, c->nl_phys)));
    } else {
        unsigned nb = tb_blocks(A.n2, 128);
        TB_DISPATCH_P(c->g.P, (k_nlterms<PP><<<nb, 128, 0, c->stream>>>(A)));
    }
    TB_CHECK_LAUNCH(c);
    return tb_prof_end(c, PROF_NLTERMS, ps);
}

int tb_launch_les(tb_ctx* c, cplx* fx, cplx* fy, cplx* fz) {
    int r = ensure_twiddles(c);
    if (r) return r;
    // Fourier-space derivatives: x (dudx, dvdx, dwdx, d2x u,v,w) and y (dudy, dvdy(fv), dwdy, d2y u,v,w)
    cplx** t = c->tmp;
    XJob xj[6] = {{c->ux, t[0], XOP_D1}, {c->uy, t[1], XOP_D1}, {c->uz, t[2], XOP_D1},
                  {c->ux, t[6], XOP_D2}, {c->uy, t[7], XOP_D2}, {c->uz, t[8], XOP_D2}};
    YJob yj[6] = {{c->ux, t[3], YOP_D1}, {c->uy, t[4], YOP_D1FV}, {c->uz, t[5], YOP_D1},
                  {c->ux, t[9], YOP_D2}, {c->uy, t[10], YOP_D2}, {c->uz, t[11], YOP_D2}};
    if ((r = tb_launch_xlines(c, xj, 6))) return r;
    if ((r = tb_launch_ylines(c, yj, 6))) return r;
    LesArgs A;
    A.dudx = t[0]; A.dvdx = t[1]; A.dwdx = t[2]; A.dudy = t[3]; A.dvdy = t[4]; A.dwdy = t[5];
    A.ux = c->ux; A.uy = c->uy; A.uz = c->uz;
    A.d2x[0] = t[6]; A.d2x[1] = t[7]; A.d2x[2] = t[8];
    A.d2y[0] = t[9]; A.d2y[1] = t[10]; A.d2y[2] = t[11];
    A.k2b2 = c->k2b2; A.wz = c->wz; A.fx = fx; A.fy = fy; A.fz = fz;
    A.nx = c->g.nx; A.ny = c->g.ny; A.n2 = (int)tb_n2(c); A.K = c->g.K; A.damping = c->cfg.les_damping;
    A.beta = c->cfg.beta; A.Re = c->cfg.Re; A.fac_y = c->cfg.fac_y; A.dy = c->cfg.dy; A.stf = c->cfg.stf;
    A.Cs = c->cfg.C_s; A.Aplus = c->cfg.A_plus;
    A.delta_les = std::pow(c->cfg.dx * c->cfg.dy * c->dz, 1.0 / 3.0);
    TB_DISPATCH_P(c->g.P, TB_CUDA(cudaFuncSetAttribute(k_les<PP>, cudaFuncAttributeMaxDynamicSharedMemorySize, Col<PP>::VAL * 128 * 8));
                          (k_les<PP><<<tb_blocks(A.n2, Col<PP>::PER_BLOCK), 128, Col<PP>::VAL * 128 * 8, c->stream>>>(A)));
    TB_CHECK_LAUNCH(c);
    return TB_OK;
}

int tb_launch_cvirt(tb_ctx* c, cplx* fx, cplx* fy, cplx* fz, bool accumulate) {
    int r = ensure_twiddles(c);
    if (r) return r;
    IbmArgs A{c->ux, c->uy, c->uz, c->delta_no, c->gibbs, fx, fy, fz, (int)tb_n2(c), c->g.K, accumulate ? 1 : 0,
              c->cfg.irf};
    TB_DISPATCH_P(c->g.P, (k_cvirt<PP><<<tb_blocks(A.n2, Col<PP>::PER_BLOCK), 128, 0, c->stream>>>(A)));
    TB_CHECK_LAUNCH(c);
    return TB_OK;
}

// Host construction of the roughness indicator (immersed_par.f:122-151),
// then the device-side Gibbs filtering of delta().
int tb_delta_setup(tb_ctx* c) {
    int r = ensure_twiddles(c);
    if (r) return r;
    int nx = c->g.nx, ny = c->g.ny, P = c->g.P;
    size_t n2 = tb_n2(c);
    std::vector<double> d(n2 * P, 0.0);
    const tb_config& cf = c->cfg;
    if (cf.ibm) {
        double sigx = 1.0, sigy = 1.0, dz = c->dz;
        for (int k = 1; k <= P; k++) {
            double z = (double)(k - 1) * dz;
            for (int j = 1; j <= ny; j++) {
                double y = (cf.stf == 1.0) ? (double)(j - 1) * cf.dy : cf.dy * (tb_powi(cf.stf, j - 1) - 1.0) / (cf.stf - 1.0);
                if (!(y <= cf.ibm_h)) continue;
                for (int i = 1; i <= nx; i++) {
                    double x = cf.x0 + (double)(i - 1) * cf.dx;
                    double dist = std::sqrt(tb_powi(x - cf.ibm_xc, 2) + tb_powi(z - cf.ibm_zc, 2));
                    double xs = cf.ibm_xc - (cf.ibm_R * (cf.ibm_xc - x)) / dist;
                    double zs = cf.ibm_zc - (cf.ibm_R * (cf.ibm_zc - z)) / dist;
                    double v = std::exp(-tb_powi((x - xs) / sigx / dz, 2) - tb_powi((z - zs) / sigy / dz, 2)) / (sigx * sigy);
                    if (dist < cf.ibm_R) v = 1.0;
                    if (v < 1e-14) v = 0.0;
                    d[(size_t)(i - 1) + (size_t)nx * (j - 1) + n2 * (k - 1)] = v;
                }
            }
        }
    }
    if (c->delta_no) cudaFree(c->delta_no);
    TB_CUDA(cudaMalloc(&c->delta_no, d.size() * sizeof(double)));
    TB_CUDA(cudaMemcpy(c->delta_no, d.data(), d.size() * sizeof(double), cudaMemcpyHostToDevice));
    if (cf.ibm) {
        unsigned nb = tb_blocks(n2, 128);
        TB_DISPATCH_P(P, (k_delta_filter<PP><<<nb, 128, 0, c->stream>>>(c->delta_no, c->gibbs, (int)n2, c->g.K)));
        TB_CHECK_LAUNCH(c);
    }
    return TB_OK;
}
