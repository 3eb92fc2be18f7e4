/* Small calls of the filterbank: one CTA per hop. */
#include <cuda_runtime.h>
#include <stdint.h>
#include <atomic>
#include "internal.h"

namespace {

#include "pfb_dev.cuh"
#include "pfb_generic.cuh"

/* ---- small calls: one CTA per hop ------------------------------------------
 * A call of a few dozen to a few hundred hops cannot fill the tile kernel: its
 * tiles of 4096 points are too few for the SMs, and one tile's fold and passes
 * take ~20 us of latency. Here every hop of every job gets its own CTA
 * (power-of-two nchan 16..1024 on the fast plan), and the jobs' state carries
 * one CTA each after them:
 *   fold    thread per branch q, k ascending, a rounded multiply then a
 *           rounded add: the bits of every tile shape's fold;
 *   FFT     the bank's own plan, pass by pass between two shared-memory
 *           buffers: the first pass (radix plan.radix[0], Ns = 1) without
 *           twiddles, the others with tw_powers of the bank's per-pass table
 *           and cmul, the last fused with finish_bin -- the arithmetic of the
 *           tile kernel's passes, so the outputs equal the tile path's bits.
 * NTH threads: two branches each from nchan 256 on, so that a thread's loads
 * are one or two rounds of memory latency. The uniform bounds checks are the
 * tile kernel's (window, output, carry). */
#define HOPS_MAXM 1024

template <int NTH, int R>
__device__ __forceinline__ void hop_pass(const double2 *__restrict__ src, double2 *__restrict__ dst, int M, int Ns,
                                         const double2 *__restrict__ tw, bool first) {
    const int MR = M / R;
    for (int j = threadIdx.x; j < MR; j += NTH) {
        const int k = j & (Ns - 1);
        double2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = src[j + r * MR];
        if (!first) {
            double2 w[R];
            tw_powers<R>(__ldg(tw + k), w);
#pragma unroll
            for (int r = 1; r < R; ++r) v[r] = cmul(v[r], w[r]);
        }
        dftR<R>(v);
        const int d = (j - k) * R + k;
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (IDX_OK(d + r * Ns < M)) dst[d + r * Ns] = v[r];
    }
}

template <int NTH, int R>
__device__ __forceinline__ void hop_pass_last(const double2 *__restrict__ src, int M, int Ns,
                                              const double2 *__restrict__ tw, bool first, const atkb_bank &B,
                                              const atkb_job &J, long long t) {
    const int MR = M / R;                       /* == Ns */
    const double2 *twd = (const double2 *)B.twd;
    const float2 *cal = (const float2 *)J.cal;
    float2 *out = (float2 *)J.out;
    const int osm = B.os - 1;
    const int s = (int)(J.b0 + t + 1) & osm;
    for (int j = threadIdx.x; j < MR; j += NTH) {
        double2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = src[j + r * MR];
        if (!first) {
            double2 w[R];
            tw_powers<R>(__ldg(tw + j), w);
#pragma unroll
            for (int r = 1; r < R; ++r) v[r] = cmul(v[r], w[r]);
        }
        dftR<R>(v);
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int kb = j + r * Ns;
            if (IDX_OK(kb < M && J.out_col + t < J.ldo))
                out[(long long)kb * J.ldo + J.out_col + t] = finish_bin(v[r], kb, s, M, osm + 1, B.hop, true, twd, cal);
        }
    }
}

template <int NTH>
__device__ __forceinline__ void hop_carry(const atkb_carry &C, float cre, float cim, int *counters) {
    const long long from = C.from, len = C.len;
    if (from < 0 || len < 0 || from + len > C.nsrc || len > C.cap) {
        if (threadIdx.x == 0) atomicOr((unsigned *)&counters[ATKB_FAULT_WORD], ATKB_FAULT_CARRY);
        return;
    }
    const Src src{(const float2 *)C.state, C.in, C.head, C.in_kind, cre, cim, C.kscale};
    float2 *dst = (float2 *)C.dst;
    carry_copy<NTH>(src, dst, from, len);
}

/* hop t of job J (its int16 constants cre, cim); buf: 2 * nchan points */
template <int NTH>
__device__ __forceinline__ void hop_run(const atkb_job &J, float cre, float cim, long long t, double2 *buf,
                                        atkb_bank &SB, int *counters) {
    {
        static_assert(sizeof(atkb_bank) % 4 == 0, "word copies");
        const int *bs = (const int *)J.bank;
        int *bd = (int *)&SB;
        for (int w = threadIdx.x; w < (int)(sizeof(atkb_bank) / 4); w += NTH) bd[w] = bs[w];
    }
    __syncthreads();
    const int M = SB.nchan;
    /* uniform across the CTA: a shape this kernel does not run, a window past
     * the job's samples or a column past the row stride skips the hop */
    {
        unsigned bad = 0, dyn_smem;
        asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn_smem));
        if (t >= J.hops || t * SB.hop + SB.L > J.nsrc) bad |= ATKB_FAULT_WINDOW;
        if (J.out_col + t + 1 > J.ldo) bad |= ATKB_FAULT_OUTPUT;
        if (!SB.plan.fast || M > HOPS_MAXM || M < 16 || 32u * (unsigned)M > dyn_smem) bad |= ATKB_FAULT_INDEX;
        for (int p = 0; p < SB.plan.npass; ++p)
            if (SB.plan.radix[p] != 2 && SB.plan.radix[p] != 4 && SB.plan.radix[p] != 8) bad |= ATKB_FAULT_INDEX;
        if (bad) {
            if (threadIdx.x == 0) atomicOr((unsigned *)&counters[ATKB_FAULT_WORD], bad);
            return;
        }
    }
    /* the fold, one branch per thread and step, eight taps' loads in flight */
    {
        const Src src{(const float2 *)J.state, J.in, J.head, J.in_kind, cre, cim, J.kscale};
        const float *taps = SB.taps;
        const int K = SB.K;
        const long long base = t * SB.hop;
        for (int q = threadIdx.x; q < M; q += NTH) {
            float fr = -0.0f, fi = -0.0f;
            for (int k0 = 0; k0 < K; k0 += 8) {
                float h[8];
                float2 x[8];
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    if (k0 + u < K && IDX_OK(base + (long long)(k0 + u) * M + q < J.nsrc)) {
                        h[u] = __ldg(taps + (long long)(k0 + u) * M + q);
                        x[u] = src.at(base + (long long)(k0 + u) * M + q);
                    }
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    if (k0 + u < K) {
                        fr = __fadd_rn(fr, __fmul_rn(h[u], x[u].x));
                        fi = __fadd_rn(fi, __fmul_rn(h[u], x[u].y));
                    }
            }
            buf[q] = make_double2((double)fr, (double)fi);
        }
    }
    __syncthreads();
    /* the plan's passes */
    const double2 *wp = (const double2 *)SB.wpass;
    double2 *cur = buf, *nxt = buf + M;
    int Ns = 1;
    for (int p = 0; p < SB.plan.npass; ++p) {
        const int R = SB.plan.radix[p];
        const double2 *tw = wp + SB.plan.twoff[p];
        const bool first = p == 0;
        if (p == SB.plan.npass - 1) {
            if (R == 8) hop_pass_last<NTH, 8>(cur, M, Ns, tw, first, SB, J, t);
            else if (R == 4) hop_pass_last<NTH, 4>(cur, M, Ns, tw, first, SB, J, t);
            else hop_pass_last<NTH, 2>(cur, M, Ns, tw, first, SB, J, t);
        } else {
            if (R == 8) hop_pass<NTH, 8>(cur, nxt, M, Ns, tw, first);
            else if (R == 4) hop_pass<NTH, 4>(cur, nxt, M, Ns, tw, first);
            else hop_pass<NTH, 2>(cur, nxt, M, Ns, tw, first);
            __syncthreads();
            double2 *x = cur;
            cur = nxt;
            nxt = x;
        }
        Ns *= R;
    }
}

/* njobs jobs of m hops each from a device table */
template <int NTH>
__global__ void __launch_bounds__(NTH)
pfb_hops_kernel(const atkb_job *__restrict__ jobs, const atkb_carry *__restrict__ carries, int njobs, int m,
                int *counters) {
    extern __shared__ double2 hop_buf[];
    __shared__ atkb_bank SB;
    const int b = blockIdx.x;
    if (b >= njobs * m) {                       /* a state carry */
        if (b - njobs * m < njobs) {
            const atkb_carry &C = carries[b - njobs * m];
            hop_carry<NTH>(C, C.cre, C.cim, counters);
        }
        return;
    }
    const atkb_job &J = jobs[b / m];
    hop_run<NTH>(J, J.cre, J.cim, b % m, hop_buf, SB, counters);
}

/* one job from the launch's own parameters: no table, no copy before it. The
 * int16 constants of a device-held offset are derived by each CTA. */
template <int NTH>
__global__ void __launch_bounds__(NTH)
pfb_hops1_kernel(const __grid_constant__ atkb_job J, const __grid_constant__ atkb_carry C, int m, int *counters) {
    extern __shared__ double2 hop_buf[];
    __shared__ atkb_bank SB;
    float cre = J.cre, cim = J.cim;
    if (J.doff) doff_consts(J.doff, J.kscale, cre, cim);
    if ((int)blockIdx.x >= m) hop_carry<NTH>(C, cre, cim, counters);
    else hop_run<NTH>(J, cre, cim, blockIdx.x, hop_buf, SB, counters);
}

/* The same for a bank on the generic plan (any other nchan up to 6400): a CTA
 * takes GH consecutive hops, as many as hold about 1024 points, of one job;
 * every call of a single handle comes here, whatever its size, since no tile
 * shares samples between hops anyway. One kernel for a table of jobs (m hops
 * each) and for one job from the launch's parameters. Bound by the latency of
 * the passes' shared-memory round trips: four CTAs of 256 threads per SM hide
 * it (one CTA of 144 registers a thread: 121 us for nchan 1000, 2x, 12 taps,
 * 500,003 samples; this one 37.5; the tile kernel's generic branch 94.0). */
template <int NTH>
__device__ __forceinline__ void generic_cta(const atkb_job &J, float cre, float cim, long long h0, int gh,
                                            atkb_bank &SB, int *counters) {
    extern __shared__ double2 hop_buf[];
    const int *bs = (const int *)J.bank;
    for (int w = threadIdx.x; w < (int)(sizeof(atkb_bank) / 4); w += NTH) ((int *)&SB)[w] = bs[w];
    __syncthreads();
    const long long left = J.hops - h0;
    const int nvalid = (int)(left < gh ? left : gh);
    unsigned bad = 0, dyn_smem;
    asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn_smem));
    if (nvalid <= 0) return;
    if ((h0 + nvalid - 1) * SB.hop + SB.L > J.nsrc) bad |= ATKB_FAULT_WINDOW;
    if (J.out_col + h0 + nvalid > J.ldo) bad |= ATKB_FAULT_OUTPUT;
    if (SB.plan.big || 32ll * nvalid * SB.nchan > (long long)dyn_smem) bad |= ATKB_FAULT_INDEX;
    if (bad) {
        if (threadIdx.x == 0) atomicOr((unsigned *)&counters[ATKB_FAULT_WORD], bad);
        return;
    }
    generic_tile<NTH>(J, SB, cre, cim, h0, nvalid, hop_buf);
}

template <int NTH>
__global__ void __launch_bounds__(NTH, 1024 / NTH)
pfb_generic_kernel(const atkb_job *__restrict__ jobs, const atkb_carry *__restrict__ carries, int njobs, int groups,
                   int gh, int *counters) {
    __shared__ atkb_bank SB;
    const int b = blockIdx.x;
    if (b >= njobs * groups) {                  /* a state carry */
        if (b - njobs * groups < njobs) {
            const atkb_carry &C = carries[b - njobs * groups];
            hop_carry<NTH>(C, C.cre, C.cim, counters);
        }
        return;
    }
    const atkb_job &J = jobs[b / groups];
    generic_cta<NTH>(J, J.cre, J.cim, (long long)(b % groups) * gh, gh, SB, counters);
}

template <int NTH>
__global__ void __launch_bounds__(NTH, 1024 / NTH)
pfb_generic1_kernel(const __grid_constant__ atkb_job J, const __grid_constant__ atkb_carry C, int groups, int gh,
                    int *counters) {
    __shared__ atkb_bank SB;
    float cre = J.cre, cim = J.cim;
    if (J.doff) doff_consts(J.doff, J.kscale, cre, cim);
    if ((int)blockIdx.x >= groups) hop_carry<NTH>(C, cre, cim, counters);
    else generic_cta<NTH>(J, cre, cim, (long long)blockIdx.x * gh, gh, SB, counters);
}

}  // namespace

/* threads of a hop's CTA: two branches each, 64 to 512 */
static int hops_threads(int nchan) { return nchan <= 128 ? 64 : nchan <= 256 ? 128 : nchan <= 512 ? 256 : 512; }

/* the small-call kernel: njobs jobs of m hops each, then their carries */
extern "C" int atkb_pfb_hops(const atkb_job *d_jobs, const atkb_carry *d_carry, int njobs, int m, int nchan,
                             int *d_counters, void *stream) {
    if (njobs < 1 || m < 0) return ATKB_E_ARG;
    const long long grid = (long long)njobs * m + njobs;
    if (grid > 0x7fffffffLL) return ATKB_E_ARG;
    const size_t smem = (size_t)nchan * 32;
    cudaStream_t st = (cudaStream_t)stream;
    atkb_range_push("atkdsp small call");
    switch (hops_threads(nchan)) {
    case 64: pfb_hops_kernel<64><<<(unsigned)grid, 64, smem, st>>>(d_jobs, d_carry, njobs, m, d_counters); break;
    case 128: pfb_hops_kernel<128><<<(unsigned)grid, 128, smem, st>>>(d_jobs, d_carry, njobs, m, d_counters); break;
    case 256: pfb_hops_kernel<256><<<(unsigned)grid, 256, smem, st>>>(d_jobs, d_carry, njobs, m, d_counters); break;
    default: pfb_hops_kernel<512><<<(unsigned)grid, 512, smem, st>>>(d_jobs, d_carry, njobs, m, d_counters); break;
    }
    atkb_range_pop();
    return cudaGetLastError() == cudaSuccess ? ATKB_OK : ATKB_E_KERNEL;
}

extern "C" int atkb_pfb_hops1(const atkb_job *J, const atkb_carry *C, int m, int nchan, int *d_counters,
                              void *stream) {
    if (m < 0) return ATKB_E_ARG;
    const size_t smem = (size_t)nchan * 32;
    cudaStream_t st = (cudaStream_t)stream;
    atkb_range_push("atkdsp small call");
    switch (hops_threads(nchan)) {
    case 64: pfb_hops1_kernel<64><<<m + 1, 64, smem, st>>>(*J, *C, m, d_counters); break;
    case 128: pfb_hops1_kernel<128><<<m + 1, 128, smem, st>>>(*J, *C, m, d_counters); break;
    case 256: pfb_hops1_kernel<256><<<m + 1, 256, smem, st>>>(*J, *C, m, d_counters); break;
    default: pfb_hops1_kernel<512><<<m + 1, 512, smem, st>>>(*J, *C, m, d_counters); break;
    }
    atkb_range_pop();
    return cudaGetLastError() == cudaSuccess ? ATKB_OK : ATKB_E_KERNEL;
}

/* hops a generic CTA takes: about 1024 points (nchan 24 43 hops, 1000 one);
 * fewer when a launch of m hops would leave less than two CTAs an SM */
static int generic_hops(int dev, int nchan, long long m) {
    const long long wave = 2LL * atkb_sm_count(dev);
    long long gh = 1024 / nchan;
    if (gh > (m + wave - 1) / wave) gh = (m + wave - 1) / wave;
    return gh < 1 ? 1 : (int)gh;
}

template <int NTH>
static int generic_launch(const atkb_job *jobs, const atkb_carry *carries, bool one, int njobs, int m, int nchan,
                          int *d_counters, cudaStream_t st) {
    /* the attributes are idempotent: concurrent first callers may both set them */
    static std::atomic<bool> configured[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return ATKB_E_NODEV;
    if (!configured[dev].load(std::memory_order_acquire)) {
        const int most = 6400 * 32;
        if (cudaFuncSetAttribute(pfb_generic_kernel<NTH>, cudaFuncAttributeMaxDynamicSharedMemorySize, most) != cudaSuccess ||
            cudaFuncSetAttribute(pfb_generic1_kernel<NTH>, cudaFuncAttributeMaxDynamicSharedMemorySize, most) != cudaSuccess)
            return ATKB_E_KERNEL;
        configured[dev].store(true, std::memory_order_release);
    }
    const int gh = generic_hops(dev, nchan, (long long)m * njobs), groups = (m + gh - 1) / gh;
    const long long grid = (long long)njobs * groups + njobs;
    if (grid > 0x7fffffffLL) return ATKB_E_ARG;
    const size_t smem = (size_t)nchan * gh * 32;
    if (one) pfb_generic1_kernel<NTH><<<(unsigned)grid, NTH, smem, st>>>(*jobs, *carries, groups, gh, d_counters);
    else pfb_generic_kernel<NTH><<<(unsigned)grid, NTH, smem, st>>>(jobs, carries, njobs, groups, gh, d_counters);
    return cudaGetLastError() == cudaSuccess ? ATKB_OK : ATKB_E_KERNEL;
}

extern "C" int atkb_pfb_generic(const atkb_job *jobs, const atkb_carry *carries, int one, int njobs, int m, int nchan,
                                int *d_counters, void *stream) {
    if (njobs < 1 || m < 0 || nchan < 2 || nchan > 6400) return ATKB_E_ARG;
    atkb_range_push("atkdsp generic hops");
    const int rc = nchan <= 1024 ? generic_launch<256>(jobs, carries, one != 0, njobs, m, nchan, d_counters, (cudaStream_t)stream)
                                 : generic_launch<512>(jobs, carries, one != 0, njobs, m, nchan, d_counters, (cudaStream_t)stream);
    atkb_range_pop();
    return rc;
}

extern "C" unsigned atkb_pfb_hops_fault(void) {
#ifdef ATKB_DEBUG_BOUNDS
    return take_debug_fault();
#else
    return 0;
#endif
}

extern "C" int atkb_pfb_hops_ok(const atkb_bank *B) {
    if (!B->plan.fast || B->plan.big || B->nchan < 16 || B->nchan > HOPS_MAXM) return 0;
    for (int p = 0; p < B->plan.npass; ++p)
        if (B->plan.radix[p] != 2 && B->plan.radix[p] != 4 && B->plan.radix[p] != 8) return 0;
    return 1;
}

