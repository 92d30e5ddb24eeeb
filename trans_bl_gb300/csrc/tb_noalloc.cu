// tb_noalloc.cu -- compact x-filter (filter_trid) on caller device buffers
// without any device allocation.
//
// Some hosts cannot call cudaMalloc once their time loop runs: a Fortran
// driver whose memory manager hands every free byte of the GPU to its own
// pool at start-up, or a real-time section where a device allocation (which
// may synchronise the whole device) is not allowed.  tb_filter_trid_noalloc
// serves them: the filtered lines are staged in a fixed scratch array that
// lives in the library's own device image instead of a per-context
// allocation.
//
//  - The lines are filtered in place, two warps per x-line staged in shared
//    memory (tb_xline.cuh).  The operator's row tables, built at every call, and
//    the pivots of lines where they do not settle sit in a file-scope __device__
//    array of 197 KB, which every GPU that loads this library keeps until the
//    process exits.  One call filters at most nx*ny*kfour = 2^21 - 4096 points
//    with nx <= 4096, the entry point's documented limits (larger grids: call once
//    per slice of Fourier modes, which the filter treats independently).
//  - The first call on a device (with that device current) looks up the
//    array's device address with cudaGetSymbolAddress and keeps it for the
//    device; make that first call before any stream capture.  The kept
//    address belongs to the device's primary context: after cudaDeviceReset
//    of that device it is stale, so a process that resets a device must not
//    call this entry point on it again.
//  - All calls share the one array: calls that overlap on the GPU (two
//    streams, or two host threads) race on it.  Every element the kernels read
//    is written earlier in the same call, so nothing needs clearing.
//  - One thread per line, dividing by the pivots and writing the sweeps through
//    the scratch, took 3720 us for three fields of 513 x 97 x 32 points; this
//    takes 291 us, the FP64 pipe's floor for 12 instructions a real value being 190.
#include "tb_internal.h"
#include "tb_xline.cuh"
#include <algorithm>
#include <atomic>

#define TB_NOALLOC_LINE_MAX 4096                                // longest line
#define TB_NOALLOC_FIELD_MAX ((1u << 21) - TB_NOALLOC_LINE_MAX)  // points per call

// the row tables of the longest line (xl::table_size), then its pivots
constexpr int TB_NOALLOC_TABLES = 5 * TB_NOALLOC_LINE_MAX + 320 + 256;
static __device__ __align__(256) double g_filter_scratch[TB_NOALLOC_TABLES + TB_NOALLOC_LINE_MAX];

namespace {

// Device address of the scratch per device ordinal, set by the first call on
// that device (concurrent first calls store the same value).
std::atomic<double*> g_scratch_addr[64];

// 1 / pivot of the Thomas factors of the filter's LHS (lhs_tridf
// filter_par.f:181), computed on the host and passed by value: rows first ..
// first + cnt - 1, then (`fill`) one value up to row nx - 5, since the pivots of
// the constant interior become constant (after ~65 rows at alpha_f = 0.48), and
// the last four rows.
constexpr int PIV = 440;   // kernel arguments are limited to 4 KB
struct Pivots {
    double ib[PIV], rest, tail[4];
    int first, cnt, fill;
    __device__ __forceinline__ double at(int i, int nx) const {
        return i < cnt ? ib[i] : i >= nx - 4 ? tail[i - (nx - 4)] : rest;
    }
};
// Lines whose pivots do not settle within PIV rows: through the scratch array.
__global__ void k_filter_pivots(double* piv, const __grid_constant__ Pivots P, int nx) {
    const int q = P.first + blockIdx.x * blockDim.x + threadIdx.x;
    if (q < P.first + P.cnt) piv[q] = P.ib[q - P.first];
    else if (P.fill && q < nx) piv[q] = q >= nx - 4 ? P.tail[q - (nx - 4)] : P.rest;
}

// The row tables of the filter (tb_xline.cuh) from its pivots (piv: null where
// P holds them all), one block.
__global__ void __launch_bounds__(512) k_filter_tables(double* T, const double* piv, const __grid_constant__ Pivots P, int nx, int S,
                                                       double alphaf, double kappa, xl::Weights wt) {
    const int tid = threadIdx.x, lane = tid & 31;
    auto pivot = [&](int i) { return piv ? piv[i] : P.at(i, nx); };
    auto off = [&](int i) { return (i >= 3 && i <= nx - 4) ? alphaf : 0.0; };   // off-diagonals of row i
    for (int e = tid; e < 32 * S; e += blockDim.x) {
        const int i = (e & 31) * S + (e >> 5);
        const bool in = i < nx;
        T[e] = (in && i) ? off(i) * pivot(i - 1) : 0.0;                         // l
        T[32 * S + e] = in ? kappa * pivot(i) : 0.0;                            // c1
        T[96 * S + e] = (in && i + 1 < nx) ? off(i) * pivot(i) : 0.0;          // g of row i + 1
    }
    if (tid < 256) T[160 * S + 320 + tid] = xl::end_weight(xl::FILTER, lane, tid >> 5, wt);
    __syncthreads();
    double* R = T + 160 * S;
    const int rows = max(0, min(nx, (lane + 1) * S) - lane * S);
    if (tid < 32) {          // responses of the forward sweep to the chunk's carry
        double h = 1.0;
        for (int q = 0; q < rows; q++) {
            h *= -T[32 * q + lane];
            T[64 * S + 32 * q + lane] = T[32 * S + 32 * q + lane] * h;          // c2
        }
        for (int q = rows; q < S; q++) T[64 * S + 32 * q + lane] = 0.0;
        for (int d = 0, o = 1; d < 5; d++, o <<= 1) {
            R[d * 32 + lane] = h;
            const double p = __shfl_up_sync(0xffffffffu, h, o);
            if (lane >= o) h *= p;
        }
    } else if (tid < 64) {   // of the backward sweep
        double h = 1.0;
        for (int q = S - 1; q >= rows; q--) T[128 * S + 32 * q + lane] = 0.0;
        for (int q = rows - 1; q >= 0; q--) {
            h *= -T[96 * S + 32 * q + lane];
            T[128 * S + 32 * q + lane] = h;                                     // hb
        }
        for (int d = 0, o = 1; d < 5; d++, o <<= 1) {
            R[160 + d * 32 + lane] = h;
            const double p = __shfl_down_sync(0xffffffffu, h, o);
            if (lane + o < 32) h *= p;
        }
    }
}

// The lines of nf fields in place, two warps per line, rows i >= 2 of the lines
// j >= 2 (filter_trid copies those back, filter_par.f:166-174).  `staged`: the
// tables fit shared memory beside the lines.
struct FilterArgs {
    double2* w[3];
    const double* T;
    xl::Weights wt;
    int nf, nx, ny, nlines, S, staged;
};
constexpr int FILTER_LINES = 8;   // per block at most
__global__ void __launch_bounds__(64 * FILTER_LINES) k_filter_lines(FilterArgs A) {
    extern __shared__ double fs[];
    const int pair = threadIdx.x >> 6, part = (threadIdx.x >> 5) & 1, W = blockDim.x >> 6, tsz = xl::table_size(A.S);
    const double* T = A.T;
    double* lines = fs;
    if (A.staged) {
        for (int q = threadIdx.x; q < tsz; q += blockDim.x) fs[q] = A.T[q];
        T = fs;
        lines = fs + tsz;
        __syncthreads();
    }
    double* F = lines + (size_t)pair * xl::line_size(A.S);
    for (int gw = pair * gridDim.x + blockIdx.x; gw < A.nf * A.nlines; gw += gridDim.x * W) {
        const int fld = gw / A.nlines, line = gw - fld * A.nlines;
        if (line % A.ny == 0) continue;
        double2* f = A.w[fld] + (size_t)line * A.nx;
        xl::xline<xl::FILTER, double>(A.wt, T, A.S, A.nx, f, f, 1, F, part, 1 + pair);
    }
}

int scratch_address(double** out) {
    int dev = 0;
    TB_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) { tb_set_error("device ordinal %d out of range", dev); return TB_ERR_ARG; }
    double* a = g_scratch_addr[dev].load(std::memory_order_acquire);
    if (!a) {
        void* p = nullptr;
        TB_CUDA(cudaGetSymbolAddress(&p, g_filter_scratch));
        a = static_cast<double*>(p);
        g_scratch_addr[dev].store(a, std::memory_order_release);
    }
    *out = a;
    return TB_OK;
}

}  // namespace

extern "C" int tb_filter_trid_noalloc(double* wx, double* wy, double* wz, int nx, int ny, int kfour, double alphaf,
                                      void* stream) {
    if (!wx || !wy || !wz) { tb_set_error("tb_filter_trid_noalloc: null field pointer"); return TB_ERR_ARG; }
    if (nx < 8 || nx > TB_NOALLOC_LINE_MAX || ny < 2 || kfour < 1) {
        tb_set_error("tb_filter_trid_noalloc: need 8 <= nx <= %d, ny >= 2, kfour >= 1", TB_NOALLOC_LINE_MAX);
        return TB_ERR_ARG;
    }
    size_t n3 = (size_t)nx * ny * kfour;
    if (n3 > TB_NOALLOC_FIELD_MAX) {
        tb_set_error("tb_filter_trid_noalloc: nx*ny*kfour = %zu exceeds the %u points of one call; "
                     "filter fewer Fourier modes per call", n3, (unsigned)TB_NOALLOC_FIELD_MAX);
        return TB_ERR_ARG;
    }
    double* T = nullptr;
    int r = scratch_address(&T);
    if (r) return r;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    double* piv = T + TB_NOALLOC_TABLES;
    auto off = [&](int i) { return (i >= 3 && i <= nx - 4) ? alphaf : 0.0; };
    Pivots P;
    double bet = 1.0;   // pivot of the row before
    bool through = false;
    for (int i = 0; i < nx;) {
        P.first = i; P.cnt = 0; P.fill = 0; P.rest = 0.0;
        for (; i < nx && P.cnt < PIV; i++) {
            if (i > 0) {
                const double b = 1.0 - off(i) * (off(i - 1) / bet);
                if (i > 4 && i < nx - 4 && b == bet) { P.fill = 1; break; }   // constant up to row nx - 5
                bet = b;
            }
            P.ib[P.cnt++] = 1.0 / bet;
        }
        if (P.fill) {
            P.rest = 1.0 / bet;
            for (int q = nx - 4; q < nx; q++) {
                bet = 1.0 - off(q) * (off(q - 1) / bet);
                P.tail[q - (nx - 4)] = 1.0 / bet;
            }
            i = nx;
        }
        if (through || i < nx) {
            through = true;
            k_filter_pivots<<<tb_blocks(P.fill ? nx - P.first : P.cnt, 256), 256, 0, st>>>(piv, P, nx);
            TB_CUDA(cudaGetLastError());
        }
    }
    const double af = (11.0 + 10.0 * alphaf) / 16.0;
    FilterArgs A;
    A.w[0] = reinterpret_cast<double2*>(wx); A.w[1] = reinterpret_cast<double2*>(wy); A.w[2] = reinterpret_cast<double2*>(wz);
    A.T = T;
    A.wt = tb_filter_weights(alphaf);
    A.nx = nx; A.ny = ny; A.nlines = ny * kfour; A.S = (nx + 31) / 32;
    k_filter_tables<<<1, 512, 0, st>>>(T, through ? piv : nullptr, P, nx, A.S, alphaf, af != 0.0 ? af : 1.0, A.wt);
    TB_CUDA(cudaGetLastError());
    // lines per block: two blocks per SM where the tables and four lines fit
    // half its shared memory, one with as many lines as fit otherwise; in fours, for
    // the SM's four sub-partitions
    const size_t tab = (size_t)xl::table_size(A.S) * sizeof(double), line = (size_t)xl::line_size(A.S) * sizeof(double);
    const size_t room = (size_t)226 * 1024;
    A.staged = tab + 2 * line <= room;
    const size_t t0 = A.staged ? tab : 0, half = (t0 + 4 * line + 1024 <= room / 2) ? room / 2 - 1024 : room;
    int W = (int)std::min<size_t>(FILTER_LINES, (half - t0) / line);
    if (W >= 4) W &= ~3;
    int dev = 0, sms = 0;
    TB_CUDA(cudaGetDevice(&dev));
    TB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    TB_CUDA(cudaFuncSetAttribute(k_filter_lines, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    // fields that share memory are filtered one after another, in order
    auto apart = [&](const double* a, const double* b) { return a + 2 * n3 <= b || b + 2 * n3 <= a; };
    const int batch = (apart(wx, wy) && apart(wx, wz) && apart(wy, wz)) ? 3 : 1;
    for (int q = 0; q < 3; q += batch) {
        A.nf = batch;
        if (q) A.w[0] = A.w[q];
        const unsigned nb = std::min<unsigned>(tb_blocks((size_t)batch * A.nlines, W), (unsigned)(2 * sms));
        k_filter_lines<<<nb, 64 * W, t0 + W * line, st>>>(A);
        TB_CUDA(cudaGetLastError());
    }
    return TB_OK;
}
