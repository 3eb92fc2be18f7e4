/* The CFAR detector's per-cell work on sm_100a (reference src/cfar.c:524-592,
 * the first half of one_frame): the conversion of each frame to linear power,
 * the average over k_frames frames, and each bin's test against alpha x T.
 *
 * One call covers every frame a process call brings, as a grid of (bins x
 * frames): the per-cell work of different frames is independent once the raw
 * ring holds the k - 1 frames before them. Every sum runs in the reference's
 * order (the k frames oldest first; the reference cells in table order), so
 * X, T and the threshold differ from the reference's only where the device
 * exp rounds the dB conversion differently in the last bit.
 *
 * The reference-cell table is cell-major (idx[q * nbins + i]), so the threads
 * of a warp, one bin each, read one table row with coalesced loads; the
 * frame's X row they index stays in L1 / L2. Each hit row is written twice:
 * as bytes (the W1 gate's layout) and as a bitmask from one warp ballot per
 * 32 bins, which is what the host tracker reads.
 */
#include <cuda_runtime.h>
#include <math.h>
#include <math_constants.h>
#include <stdint.h>

#include "internal.h"

namespace {

constexpr double kLn10Over10 = 0.23025850929940458;   /* ln(10) / 10 */
constexpr int kThreads = 256;

/* The three kernels below take one bin and FR consecutive frames a thread:
 * FR = 8 or 4 where that leaves two CTAs per SM, else 1 (a call of few cells
 * is bound by the latency of one thread's chain). The ring's remainder and the
 * reference-cell table's loads then serve FR frames: 47 us a pass of 2^20 cells
 * at one frame a thread, 36 here (4096 bins, CA over 32 cells, k 4); the cell
 * loads through L1 bound it. */
__device__ __forceinline__ double linear_of(float x, int units) {
    double v = (double)x;
    if (units == 0) {
        if (v < -300.0) v = -300.0;
        v = exp(v * kLn10Over10);
    } else if (v < 1e-30) {
        v = 1e-30;
    }
    return v;
}

template <int FR>
__global__ void __launch_bounds__(kThreads) cfar_raw_kernel(const float *__restrict__ frames, int units, int row0,
                                                            int nf, long long nbins, double *__restrict__ raw,
                                                            int ring) {
    const long long i = (long long)blockIdx.x * kThreads + threadIdx.x;
    if (i >= nbins) return;
    for (int j0 = blockIdx.y * FR; j0 < nf; j0 += gridDim.y * FR) {
        float x[FR];
#pragma unroll
        for (int u = 0; u < FR; ++u)
            if (j0 + u < nf) x[u] = __ldg(frames + (long long)(j0 + u) * nbins + i);
        int row = (int)(((long long)row0 + j0) % ring);
#pragma unroll
        for (int u = 0; u < FR; ++u) {
            if (j0 + u < nf) raw[(long long)row * nbins + i] = linear_of(x[u], units);
            if (++row == ring) row = 0;
        }
    }
}

/* X row of each tested frame: the mean of its raw row and the k - 1 before,
 * oldest first; row0: the ring row of the first tested frame's oldest. K > 0:
 * k known, the FR frames' raw rows read once (K a power of two, so the
 * product with 1 / K rounds as the quotient does); K = 0: any k, one frame. */
template <int K, int FR>
__global__ void __launch_bounds__(kThreads) cfar_mean_kernel(const double *__restrict__ raw, int ring, int row0,
                                                             int ntest, long long nbins, int k,
                                                             double *__restrict__ X) {
    const long long i = (long long)blockIdx.x * kThreads + threadIdx.x;
    const int j0 = blockIdx.y * FR;
    if (i >= nbins) return;
    int row = (int)(((long long)row0 + j0) % ring);
    if constexpr (K > 0) {
        double v[FR + K - 1];
#pragma unroll
        for (int u = 0; u < FR + K - 1; ++u) {
            if (j0 + u < ntest + K - 1) v[u] = raw[(long long)row * nbins + i];
            if (++row == ring) row = 0;
        }
#pragma unroll
        for (int u = 0; u < FR; ++u) {
            double s = 0.0;
#pragma unroll
            for (int r = 0; r < K; ++r) s = __dadd_rn(s, v[u + r]);
            if (j0 + u < ntest) X[(long long)(j0 + u) * nbins + i] = __dmul_rn(s, 1.0 / K);
        }
    } else {
        double s = 0.0;
        for (int r = 0; r < k; ++r) {
            s = __dadd_rn(s, raw[(long long)row * nbins + i]);
            if (++row == ring) row = 0;
        }
        X[(long long)j0 * nbins + i] = __ddiv_rn(s, (double)k);
    }
}

/* the k-th smallest (0-based) of a[0..n), NaN-free: Hoare's selection,
 * partitioning around the middle element; i and j stay inside [lo, hi]
 * because the pivot value stops both scans. The value is unique, whatever
 * order the cells came in. */
__device__ __forceinline__ double select_kth(double *a, int n, int k) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const double pivot = a[(lo + hi) >> 1];
        int i = lo, j = hi;
        while (i <= j) {
            while (a[i] < pivot) ++i;
            while (a[j] > pivot) --j;
            if (i <= j) {
                const double t = a[i];
                a[i] = a[j];
                a[j] = t;
                ++i;
                --j;
            }
        }
        if (k <= j) hi = j;
        else if (k >= i) lo = i;
        else break;
    }
    return a[k];
}

/* a bitonic network over P registers (every index a compile-time constant
 * once unrolled, so v stays in registers): ascending on return */
template <int LOGP>
__device__ __forceinline__ void bitonic_sort(double (&v)[1 << LOGP]) {
    constexpr int P = 1 << LOGP;
#pragma unroll
    for (int kk = 1; kk <= LOGP; ++kk) {
#pragma unroll
        for (int jj = kk - 1; jj >= 0; --jj) {
#pragma unroll
            for (int i = 0; i < P; ++i) {
                const int l = i ^ (1 << jj);
                if (l > i) {
                    const double a = v[i], b = v[l];
                    const bool swap = ((i >> kk) & 1) == 0 ? (a > b) : (a < b);
                    v[i] = swap ? b : a;
                    v[l] = swap ? a : b;
                }
            }
        }
    }
}

/* one testable bin's OS statistic over at most OSMAX cells of the row Xr: up
 * to 32 sorted in registers (padded with +inf, which sorts after every cell),
 * more gathered into a local array and selected */
template <int OSMAX>
__device__ __forceinline__ double os_stat(long long i, long long nbins, int N, int os_k,
                                          const int32_t *__restrict__ idx, const double *__restrict__ Xr) {
    bool has_nan = false;
    if constexpr (OSMAX == 32) {
        /* the os_k-th smallest; a NaN among the cells makes T NaN */
        double v[32];
#pragma unroll
        for (int q = 0; q < 32; ++q) {
            v[q] = q < N ? Xr[idx[(long long)q * nbins + i]] : CUDART_INF;
            has_nan |= isnan(v[q]);
        }
        bitonic_sort<5>(v);
        /* v[os_k - 1] by masks, not an index: a runtime index would move v
         * to local memory */
        unsigned long long pick = 0;
#pragma unroll
        for (int q = 0; q < 32; ++q)
            pick |= (unsigned long long)__double_as_longlong(v[q]) & (0ull - (unsigned long long)(q == os_k - 1));
        return has_nan ? CUDART_NAN : __longlong_as_double((long long)pick);
    } else {
        double v[OSMAX];
        for (int q = 0; q < N; ++q) {
            v[q] = Xr[idx[(long long)q * nbins + i]];
            has_nan |= isnan(v[q]);
        }
        return has_nan ? CUDART_NAN : select_kth(v, N, os_k - 1);
    }
}

/* s[f] = the sum over the reference cells q0 .. q1, in table order, of the
 * rows Xr + f * nbins: one table entry and FR values a step, four steps'
 * loads in flight */
template <int FR>
__device__ __forceinline__ void cell_sums(const double *const (&Xr)[FR], const int32_t *__restrict__ col,
                                          long long nbins, int q0, int q1, double (&s)[FR]) {
#pragma unroll
    for (int f = 0; f < FR; ++f) s[f] = 0.0;
#pragma unroll 4
    for (int q = q0; q < q1; ++q) {
        const int b = __ldg(col + (long long)q * nbins);
#pragma unroll
        for (int f = 0; f < FR; ++f) s[f] = __dadd_rn(s[f], Xr[f][b]);
    }
}

/* s / n, by the exact reciprocal where n is a power of two (the same bits) */
__device__ __forceinline__ double over(double s, int n) {
    return (n & (n - 1)) == 0 ? __dmul_rn(s, 1.0 / (double)n) : __ddiv_rn(s, (double)n);
}

/* OSMAX 0: the statistics that are sums, FR frames a thread; else the OS
 * statistic, FR = 1. X, noise, thr, hits and bits: rows of the first tested
 * frame. */
template <int OSMAX, int FR>
__global__ void __launch_bounds__(kThreads) cfar_cell_kernel(int ntest, long long nbins, int mode, int n_ref, int N,
                                                             int os_k, double alpha, double alpha_ca, double et,
                                                             const uint8_t *__restrict__ ok,
                                                             const uint8_t *__restrict__ sided,
                                                             const int32_t *__restrict__ idx,
                                                             const double *__restrict__ X,
                                                             double *__restrict__ noise, double *__restrict__ thr,
                                                             uint8_t *__restrict__ hits, uint32_t *__restrict__ bits,
                                                             long long words) {
    const long long i = (long long)blockIdx.x * kThreads + threadIdx.x;
    const int f0 = blockIdx.y * FR;
    const bool in = i < nbins, test = in && ok[i];
    double Z[FR], a = alpha, scale = et;
    const double *Xr[FR];
#pragma unroll
    for (int f = 0; f < FR; ++f)            /* frames past the last repeat it */
        Xr[f] = X + (long long)(f0 + f < ntest ? f0 + f : ntest - 1) * nbins;
    if (test) {
        if constexpr (OSMAX > 0) {
#pragma unroll
            for (int f = 0; f < FR; ++f) Z[f] = os_stat<OSMAX>(i, nbins, N, os_k, idx, Xr[f]);
        } else if ((mode == 2 || mode == 3) && sided[i]) {
            double L[FR], R[FR];
            cell_sums<FR>(Xr, idx + i, nbins, 0, n_ref, L);
            cell_sums<FR>(Xr, idx + i, nbins, n_ref, N, R);
#pragma unroll
            for (int f = 0; f < FR; ++f) {
                const double l = over(L[f], n_ref), r = over(R[f], n_ref);
                if (isnan(l) || isnan(r)) Z[f] = CUDART_NAN;
                else Z[f] = mode == 2 ? (l > r ? l : r) : (l < r ? l : r);
            }
        } else {
            cell_sums<FR>(Xr, idx + i, nbins, 0, N, Z);
#pragma unroll
            for (int f = 0; f < FR; ++f) Z[f] = over(Z[f], N);
            if (mode == 2 || mode == 3) {
                a = alpha_ca;
                scale = 1.0;
            }
        }
    }
#pragma unroll
    for (int f = 0; f < FR; ++f) {
        if (f0 + f >= ntest) break;
        const long long e = (long long)(f0 + f) * nbins + i;
        bool hit = false;
        if (test) {
            const double t = __dmul_rn(a, Z[f]);
            thr[e] = t;
            noise[e] = scale == 1.0 ? Z[f] : __ddiv_rn(Z[f], scale);
            hit = Xr[f][i] > t;
        } else if (in) {
            noise[e] = CUDART_NAN;
            thr[e] = CUDART_NAN;
        }
        if (in) hits[e] = hit;
        /* the row as a bitmask too: bin i is bit i % 32 of word i / 32 */
        const unsigned m = __ballot_sync(0xffffffffu, hit);
        if ((threadIdx.x & 31) == 0 && (i >> 5) < words) bits[(f0 + f) * words + (i >> 5)] = m;
    }
}

/* a pass's rows at its columns: rows of X and noise (row r of X / noise to
 * row r of Xc / Nc), then nraw raw rows from ring row rf0 on (to Rc) */
__global__ void __launch_bounds__(kThreads) cfar_gather_kernel(const double *__restrict__ X,
                                                               const double *__restrict__ noise, long long nbins,
                                                               int rows, const double *__restrict__ raw, int ring,
                                                               int rf0, int nraw, const int32_t *__restrict__ cols,
                                                               int ncol, double *__restrict__ Xc,
                                                               double *__restrict__ Nc, double *__restrict__ Rc) {
    const long long total = (long long)(rows + nraw) * ncol;
    for (long long e = (long long)blockIdx.x * kThreads + threadIdx.x; e < total;
         e += (long long)gridDim.x * kThreads) {
        const long long r = total <= 0xffffffffLL ? (unsigned)e / (unsigned)ncol : e / ncol, q = e - r * ncol;
        const long long b = cols[q];
        if (r < rows) {
            Xc[e] = X[r * nbins + b];
            Nc[e] = noise[r * nbins + b];
        } else {
            const int rr = (int)(r - rows);
            Rc[(long long)rr * ncol + q] = raw[(long long)(((unsigned)rf0 + (unsigned)rr) % (unsigned)ring) * nbins + b];
        }
    }
}

int grid_for(long long work) {
    long long g = (work + kThreads - 1) / kThreads;
    return (int)(g < 148LL * 16 ? (g < 1 ? 1 : g) : 148LL * 16);
}

}  // namespace

/* bins x (groups of fr frames), two CTAs on every SM: enough to take fr */
static bool wide_enough(long long nbins, long long nf, int fr) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    return (nbins + kThreads - 1) / kThreads * (nf / fr) >= 2LL * atkb_sm_count(dev);
}

extern "C" int atkb_cfar_raw(const float *frames, int units, long long f0, int nf, long long nbins, double *raw,
                             int ring, void *stream) {
    if (nf <= 0 || nbins <= 0) return ATKB_OK;
    cudaStream_t s = (cudaStream_t)stream;
    const unsigned bx = (unsigned)((nbins + kThreads - 1) / kThreads);
    const int row0 = (int)(f0 % ring);
    if (wide_enough(nbins, nf, 8))
        cfar_raw_kernel<8><<<dim3(bx, (unsigned)((nf + 7) / 8 < 65535 ? (nf + 7) / 8 : 65535)), kThreads, 0, s>>>(
            frames, units, row0, nf, nbins, raw, ring);
    else
        cfar_raw_kernel<1><<<dim3(bx, (unsigned)(nf < 65535 ? nf : 65535)), kThreads, 0, s>>>(frames, units, row0,
                                                                                              nf, nbins, raw, ring);
    return cudaGetLastError() == cudaSuccess ? ATKB_OK : ATKB_E_KERNEL;
}

extern "C" int atkb_cfar_test(const double *raw, int ring, long long f0, long long t0, int nf, long long nbins,
                              int k, int mode, int n_ref, int n_cells, int os_k, double alpha, double alpha_ca,
                              double et, const uint8_t *ok, const uint8_t *sided, const int32_t *idx, double *X,
                              double *noise, double *thr, uint8_t *hits, uint32_t *bits, long long words,
                              void *stream) {
    const long long ntest = f0 + nf - t0, r0 = t0 - f0;
    if (ntest <= 0) return ATKB_OK;
    if (ntest > 65535 || nbins <= 0) return ATKB_E_ARG;
    const unsigned bx = (unsigned)((nbins + kThreads - 1) / kThreads);
    const dim3 one(bx, (unsigned)ntest), four(bx, (unsigned)((ntest + 3) / 4)), eight(bx, (unsigned)((ntest + 7) / 8));
    cudaStream_t s = (cudaStream_t)stream;
    const int row0 = (int)((t0 - k + 1) % ring), n = (int)ntest;
    X += r0 * nbins;
    noise += r0 * nbins;
    thr += r0 * nbins;
    hits += r0 * nbins;
    bits += r0 * words;
    const bool w8 = wide_enough(nbins, ntest, 8);
    if (k == 1 && w8) cfar_mean_kernel<1, 8><<<eight, kThreads, 0, s>>>(raw, ring, row0, n, nbins, k, X);
    else if (k == 2 && w8) cfar_mean_kernel<2, 8><<<eight, kThreads, 0, s>>>(raw, ring, row0, n, nbins, k, X);
    else if (k == 4 && w8) cfar_mean_kernel<4, 8><<<eight, kThreads, 0, s>>>(raw, ring, row0, n, nbins, k, X);
    else if (k == 8 && w8) cfar_mean_kernel<8, 8><<<eight, kThreads, 0, s>>>(raw, ring, row0, n, nbins, k, X);
    else cfar_mean_kernel<0, 1><<<one, kThreads, 0, s>>>(raw, ring, row0, n, nbins, k, X);
#define CELLS(OSMAX, FR, GRID)                                                                                     \
    cfar_cell_kernel<OSMAX, FR><<<GRID, kThreads, 0, s>>>(n, nbins, mode, n_ref, n_cells, os_k, alpha, alpha_ca,   \
                                                          et, ok, sided, idx, X, noise, thr, hits, bits, words)
    if (mode != 1 && wide_enough(nbins, ntest, 4)) CELLS(0, 4, four);
    else if (mode != 1) CELLS(0, 1, one);
    else if (n_cells <= 32) CELLS(32, 1, one);
    else if (n_cells <= 64) CELLS(64, 1, one);
    else if (n_cells <= 512) CELLS(512, 1, one);
    else return ATKB_E_ARG;
#undef CELLS
    return cudaGetLastError() == cudaSuccess ? ATKB_OK : ATKB_E_KERNEL;
}

extern "C" int atkb_cfar_gather(const double *X, const double *noise, long long nbins, int rows, const double *raw,
                                int ring, long long rf0, int nraw, const int32_t *cols, int ncol, double *Xc,
                                double *Nc, double *Rc, void *stream) {
    if (ncol <= 0 || rows + nraw <= 0) return ATKB_OK;
    cfar_gather_kernel<<<grid_for((long long)(rows + nraw) * ncol), kThreads, 0, (cudaStream_t)stream>>>(
        X, noise, nbins, rows, raw, ring, (int)(rf0 % ring), nraw, cols, ncol, Xc, Nc, Rc);
    return cudaGetLastError() == cudaSuccess ? ATKB_OK : ATKB_E_KERNEL;
}
