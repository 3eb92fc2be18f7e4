/* Device-resident spectrum reduction on sm_100a (reference src/fft.c:154-164,
 * :176-295 atkdsp_spectrum_reduce, :315-430 atkdsp_spectrum_stats).
 *
 * Every frame of n samples (stride hop) of a device cf32 block is windowed
 * and transformed in double by n/8 threads of 8 points (a CTA of 512 threads
 * works on 4096/n frames at a time): the samples go straight into a radix-8
 * butterfly in registers, radix-8 Stockham passes exchange through shared
 * memory, and the last pass's bins are folded into accumulators that stay in
 * the thread's registers for all its frames (reduce: float max / min / sum of
 * |X|^2/n^2 from the float-rounded bin; stats: max and min in float -- the
 * rounding is monotonic, so the rounded extremes are the extremes rounded --
 * and sum P, sum P^2 in double). Each CTA takes a contiguous run of frames and
 * writes one partial line; a second kernel adds the lines in a fixed order and
 * converts to dB fftshifted, with the reference's rounded steps. Max and min
 * are exact in any order; the sums differ from a one-thread run only in their
 * rounding sequence.
 *
 * What bounds it: the double pipe (about 54 operations a point) and the three
 * shared-memory exchanges of 32 bytes a point at n 4096; HBM has a tenth of
 * the time. 2^24 samples, n 4096, hop 2048, Hann, the four statistics: 244 us
 * (69 GS/s), 710 us with the accumulators in shared memory and one thread per
 * bin merging the partial lines. A leg is multiplied by its whole twiddle once,
 * as in fft_r8: radix-2 steps with the twiddles folded into multiply-adds (and
 * a - w b formed as 2a minus the sum) take fewer operations, ran no faster
 * (248 us), and turned an infinite a into NaN.
 */
#include <cuda_runtime.h>
#include <atomic>
#include <stdint.h>

#include "fft_sm.cuh"
#include "internal.h"

#define SP_NT 512

namespace {

using namespace atkb_fft;

/* barrier of the G consecutive threads of a frame */
template <int G>
__device__ __forceinline__ void frame_sync() {
    if constexpr (G >= SP_NT) __syncthreads();
    else if constexpr (G <= 32) __syncwarp();
    else asm volatile("bar.sync %0, %1;" ::"r"(1 + (int)threadIdx.x / G), "n"(G) : "memory");
}

/* the passes after the first (which left Ns = 2^LOGNS) of one frame at sm, in
 * place; the last leaves bin lt + u*n/8 + r*Ns in v[u*R + r] */
template <int LOGN, int LOGNS>
struct SpecPass {
    static constexpr int REM = LOGN - LOGNS, LR = REM >= 3 ? 3 : REM, R = 1 << LR, U = 8 / R;
    static constexpr int N = 1 << LOGN, NS = 1 << LOGNS, NR = N / R, G = N / 8;
    static constexpr bool LAST = REM == LR;
    typedef SpecPass<LOGN, LAST ? LOGNS : LOGNS + LR> Next;
    static __device__ __forceinline__ void run(double2 *sm, double2 *v, const double2 *__restrict__ tw, int lt) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int j = lt + u * G, k = j & (NS - 1), a = swz(j) * 16;
#pragma unroll
            for (int r = 0; r < R; ++r) v[u * R + r] = swz_at<NR>(sm, a, r);
            dft_tw<R>(v + u * R, tw, k, LOGN - LOGNS - LR);
        }
        frame_sync<G>();                       /* every point of the frame is read */
        if constexpr (!LAST) {
            static_assert(U == 1, "a middle pass is radix 8");
            const int k = lt & (NS - 1), d = swz(((lt - k) << 3) + k) * 16;
#pragma unroll
            for (int r = 0; r < 8; ++r) swz_at<NS>(sm, d, r) = v[r];
            frame_sync<G>();
            Next::run(sm, v, tw, lt);
        }
    }
    /* of the last pass: where value i of v belongs */
    static __device__ __forceinline__ int bin(int i, int lt) {
        if constexpr (LAST) return lt + (i / R) * G + (i % R) * NS;
        else return Next::bin(i, lt);
    }
};

/* MODE 0 / 1 / 2: reduce with the max / min / average detector; 3: stats.
 * PER_SM CTAs an SM: at two the 64 registers spill a little, which a launch
 * that fills the chip with frames of 2048 or 4096 points (or 64) makes up for
 * and others do not: us at one / two, one detector, 2^23 samples, n 4096 hop
 * 2048 119 / 110, n 64 34 / 32, n 256 hop 128 63 / 73, n 1024 hop 512 89 / 94;
 * a single frame of 2048 points 11.2 / 12.5. */
template <int MODE, int LOGN, int PER_SM>
__global__ void __launch_bounds__(SP_NT, PER_SM)
spec_frames_kernel(const float2 *__restrict__ in, long long frames, long long hop, const float *__restrict__ win,
                   const double2 *__restrict__ tw, int per, void *__restrict__ part) {
    extern __shared__ double2 smem[];
    constexpr int N = 1 << LOGN, G = N / 8, NG = SP_NT / G;      /* threads a frame, frames at a time */
    typedef SpecPass<LOGN, 3> Rest;
    const int lt = (int)threadIdx.x & (G - 1), g = (int)threadIdx.x / G;
    double2 *sm = smem + g * N;
    const long long f0 = (long long)blockIdx.x * per, f1 = min(frames, f0 + per);
    const float inv2f = __fdiv_rn(1.0f, __fmul_rn((float)N, (float)N));
    const double inv2d = 1.0 / ((double)N * (double)N);
    float a0[8], a1[MODE == 3 ? 8 : 1];
    double su[MODE == 3 ? 8 : 1], s2[MODE == 3 ? 8 : 1];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        a0[i] = MODE == 1 ? __int_as_float(0x7f800000) : 0.0f;
        if (MODE == 3) {
            a1[i] = __int_as_float(0x7f800000);
            su[i] = s2[i] = 0.0;
        }
    }
    /* every group takes the same number of turns (the groups of a warp share
     * its barriers); one past the run's end transforms what it has and adds
     * nothing. Stats: the next frame's samples are loaded while this one is
     * transformed (at two CTAs an SM the registers are not there, and the
     * other CTA covers the wait). */
    const int turns = (int)((f1 - f0 + NG - 1) / NG);
    float2 x[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) x[r] = make_float2(0.0f, 0.0f);
    if (MODE == 3 && f0 + g < f1) {
#pragma unroll
        for (int r = 0; r < 8; ++r) x[r] = __ldg(in + (f0 + g) * hop + lt + r * G);
    }
    for (int turn = 0; turn < turns; ++turn) {
        const long long f = f0 + g + (long long)turn * NG;
        if (MODE < 3 && f < f1) {
#pragma unroll
            for (int r = 0; r < 8; ++r) x[r] = __ldg(in + f * hop + lt + r * G);
        }
        double2 v[8];
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            if (win) {
                const double h = (double)__ldg(win + lt + r * G);
                v[r] = make_double2(__dmul_rn((double)x[r].x, h), __dmul_rn((double)x[r].y, h));
            } else {
                v[r] = make_double2((double)x[r].x, (double)x[r].y);
            }
        }
        if (MODE == 3 && f + NG < f1) {
#pragma unroll
            for (int r = 0; r < 8; ++r) x[r] = __ldg(in + (f + NG) * hop + lt + r * G);
        }
        dft8(v, false);
        {
            const int d = swz(lt * 8) * 16;
#pragma unroll
            for (int r = 0; r < 8; ++r) swz_at<1>(sm, d, r) = v[r];
        }
        frame_sync<G>();
        Rest::run(sm, v, tw, lt);
        if (f < f1) {
            /* frame 0's power enters as it is (a NaN stays), others by comparison */
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                if (MODE < 3) {
                    const float re = __double2float_rn(v[i].x), im = __double2float_rn(v[i].y);
                    const float pw = __fmul_rn(__fadd_rn(__fmul_rn(re, re), __fmul_rn(im, im)), inv2f);
                    if (MODE == 2) a0[i] = __fadd_rn(a0[i], pw);
                    else if (f == 0 || (MODE == 0 ? pw > a0[i] : pw < a0[i])) a0[i] = pw;
                } else {
                    const double pw = __dmul_rn(__dadd_rn(__dmul_rn(v[i].x, v[i].x), __dmul_rn(v[i].y, v[i].y)), inv2d);
                    const float pf = __double2float_rn(pw);
                    if (f == 0 || pf > a0[i]) a0[i] = pf;
                    if (f == 0 || pf < a1[i]) a1[i] = pf;
                    su[i] = __dadd_rn(su[i], pw);
                    s2[i] = __dadd_rn(s2[i], __dmul_rn(pw, pw));
                }
            }
        }
    }
    /* the CTA's frame groups merged in order through shared memory, one plane
     * at a time, then its partial line (bins fftshifted). Groups past the
     * run's end hold no frame. */
    const int ng = (int)min((long long)NG, f1 - f0);
    __syncthreads();
    for (int pl = 0; pl < (MODE == 3 ? 4 : 1); ++pl) {
        double *q = (double *)smem;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int k = (Rest::bin(i, lt) + N / 2) & (N - 1);
            q[g * N + k] = MODE < 3 || pl == 0 ? (double)a0[i]
                         : pl == 1 ? (double)a1[MODE == 3 ? i : 0]
                         : pl == 2 ? su[MODE == 3 ? i : 0] : s2[MODE == 3 ? i : 0];
        }
        __syncthreads();
        for (int i = threadIdx.x; i < N; i += SP_NT) {
            double a = q[i];
            for (int e = 1; e < ng; ++e) {
                const double b = q[e * N + i];
                if (MODE == 0 || (MODE == 3 && pl == 0)) a = b > a ? b : a;
                else if (MODE == 1 || (MODE == 3 && pl == 1)) a = b < a ? b : a;
                else a = __dadd_rn(a, b);
            }
            ((double *)part)[((long long)blockIdx.x * (MODE == 3 ? 4 : 1) + pl) * N + i] = a;
        }
        __syncthreads();
    }
}

/* the partial lines merged, then dB (src/fft.c:280-290 and :405-426): reduce
 * -> o0; stats -> o0 max, o1 avg, o2 min, o3 kurtosis (NULL: skipped). A block
 * takes SF_BINS bins with SF_SL threads each: thread s adds the lines s, s +
 * SF_SL, ..., and the SF_SL sums are added in order. (One thread per bin over
 * all lines took 328 us at n 4096 and 293 lines; this takes a few.) */
#define SF_BINS 16
#define SF_SL 32
template <int MODE>
__global__ void __launch_bounds__(SF_BINS * SF_SL) spec_final_kernel(const double *__restrict__ part, int nblk, int n,
                                                                   long long frames, float *o0, float *o1, float *o2,
                                                                   float *o3) {
    constexpr int PL = MODE == 3 ? 4 : 1;
    __shared__ double red[PL][SF_SL][SF_BINS];
    const int c = threadIdx.x % SF_BINS, s = threadIdx.x / SF_BINS, i = blockIdx.x * SF_BINS + c;
    double a[PL];
#pragma unroll
    for (int p = 0; p < PL; ++p) {
        const int op = MODE == 3 ? (p < 2 ? p : 2) : MODE;
        a[p] = op == 1 ? __longlong_as_double(0x7ff0000000000000LL) : 0.0;
        if (i < n && s < nblk) {
            a[p] = part[((long long)s * PL + p) * n + i];
            for (int b = s + SF_SL; b < nblk; b += SF_SL) {
                const double v = part[((long long)b * PL + p) * n + i];
                a[p] = op == 0 ? (v > a[p] ? v : a[p]) : op == 1 ? (v < a[p] ? v : a[p]) : __dadd_rn(a[p], v);
            }
        }
        red[p][s][c] = a[p];
    }
    __syncthreads();
    if (s != 0 || i >= n) return;
    const int m = min(nblk, SF_SL);
#pragma unroll
    for (int p = 0; p < PL; ++p) {
        const int op = MODE == 3 ? (p < 2 ? p : 2) : MODE;
        for (int e = 1; e < m; ++e) {
            const double v = red[p][e][c];
            a[p] = op == 0 ? (v > a[p] ? v : a[p]) : op == 1 ? (v < a[p] ? v : a[p]) : __dadd_rn(a[p], v);
        }
    }
    if constexpr (MODE < 3) {
        const float scale = MODE == 2 ? __fdiv_rn(1.0f, (float)frames) : 1.0f;
        const float mag = __fsqrt_rn(__fmul_rn(__double2float_rn(a[0]), scale));
        o0[i] = __fmul_rn(20.0f, log10f(__fadd_rn(mag, 1e-12f)));
    } else {
        const double M = (double)frames, su = a[2], s2 = a[3];
        if (o0) o0[i] = __fmul_rn(10.0f, log10f(__fadd_rn(__double2float_rn(a[0]), 1e-12f)));
        if (o2) o2[i] = __fmul_rn(10.0f, log10f(__fadd_rn(__double2float_rn(a[1]), 1e-12f)));
        if (o1) o1[i] = __fmul_rn(10.0f, log10f(__fadd_rn(__double2float_rn(__ddiv_rn(su, M)), 1e-12f)));
        if (o3) {
            const double den = __dmul_rn(su, su);
            o3[i] = (frames < 2 || den <= 0.0) ? 1.0f : __double2float_rn(__ddiv_rn(__dmul_rn(M, s2), den));
        }
    }
}

template <int MODE, int LOGN>
int spec_run_n(const void *in, long long frames, long long hop, const float *win, const void *tw, int nblk, int per,
               void *part, float *o0, float *o1, float *o2, float *o3, cudaStream_t s) {
    constexpr int n = 1 << LOGN;
    constexpr int smem = SP_NT * 8 * 16;
    constexpr int full = MODE < 3 && (LOGN == 6 || LOGN >= 11) ? 2 : 1;
    /* the attribute is idempotent: concurrent first callers may both set it */
    static std::atomic<bool> configured[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return ATKB_E_NODEV;
    if (!configured[dev].load(std::memory_order_acquire)) {
        if (cudaFuncSetAttribute(spec_frames_kernel<MODE, LOGN, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 smem) != cudaSuccess ||
            cudaFuncSetAttribute(spec_frames_kernel<MODE, LOGN, full>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 smem) != cudaSuccess)
            return ATKB_E_KERNEL;
        configured[dev].store(true, std::memory_order_release);
    }
    const auto frames_kernel = nblk > atkb_sm_count(dev) ? spec_frames_kernel<MODE, LOGN, full>
                                                         : spec_frames_kernel<MODE, LOGN, 1>;
    frames_kernel<<<nblk, SP_NT, smem, s>>>((const float2 *)in, frames, hop, win, (const double2 *)tw, per, part);
    spec_final_kernel<MODE><<<(n + SF_BINS - 1) / SF_BINS, SF_BINS * SF_SL, 0, s>>>((const double *)part, nblk, n,
                                                                                   frames, o0, o1, o2, o3);
    return cudaGetLastError() == cudaSuccess ? ATKB_OK : ATKB_E_KERNEL;
}

template <int MODE>
int spec_launch(const void *in, long long frames, long long hop, int logn, const float *win, const void *tw,
                int nblk, int per, void *part, float *o0, float *o1, float *o2, float *o3, cudaStream_t s) {
    switch (logn) {
#define SPEC_N(L) case L: return spec_run_n<MODE, L>(in, frames, hop, win, tw, nblk, per, part, o0, o1, o2, o3, s);
        SPEC_N(4) SPEC_N(5) SPEC_N(6) SPEC_N(7) SPEC_N(8) SPEC_N(9) SPEC_N(10) SPEC_N(11) SPEC_N(12)
#undef SPEC_N
    default: return ATKB_E_ARG;
    }
}

}  // namespace

extern "C" int atkb_spec_launch(int mode, const void *in, long long frames, long long hop, int logn, const float *win,
                                const void *tw, int nblk, int per, void *part, float *o0, float *o1, float *o2,
                                float *o3, void *stream) {
    cudaStream_t s = (cudaStream_t)stream;
    switch (mode) {
    case 0: return spec_launch<0>(in, frames, hop, logn, win, tw, nblk, per, part, o0, o1, o2, o3, s);
    case 1: return spec_launch<1>(in, frames, hop, logn, win, tw, nblk, per, part, o0, o1, o2, o3, s);
    case 2: return spec_launch<2>(in, frames, hop, logn, win, tw, nblk, per, part, o0, o1, o2, o3, s);
    case 3: return spec_launch<3>(in, frames, hop, logn, win, tw, nblk, per, part, o0, o1, o2, o3, s);
    default: return ATKB_E_ARG;
    }
}
