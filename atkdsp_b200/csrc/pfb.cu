/* The polyphase filterbank on sm_100a.
 *
 * What one hop computes (reference src/channelizer.c:235-292):
 *   window   w = s[h*hop, h*hop + L),  s = history ++ leftover ++ input
 *   fold     f[q] = sum_{k ascending} taps[k*M + q] * w[k*M + q]   (float,
 *            one rounded multiply then one rounded add per tap -- the
 *            reference's pinned C99 build does exactly this, so the fold is
 *            bit-identical)
 *   FFT      X = DFT_M(f) in DOUBLE (the reference runs pocketfft in double;
 *            a float FFT misses the 1e-5 per-channel bar at M >= 1024)
 *   rotate   y[k] = X[k] * twd[(-k*shift) mod M], shift = ((b+1)*hop) mod M,
 *            with the reference's own double table (cos, sin)(2 pi j / M)
 *   cal      y[k] *= cal[k] (double), then one rounding to float
 *   out      channel-major: out[k*ldo + h]
 *
 * Kernel layout (B200-first):
 *   - ONE persistent kernel over a device job list. A job is a run of hops of
 *     one element stream (a handle's element, one stream of a batch, or one
 *     served block); a tile is tile_hops consecutive hops of a job. CTAs
 *     (512 threads, 2 per SM) claim tiles from an atomic counter; warp 0
 *     claims and looks up the next tile while the CTA works on the current
 *     one. CTAs out of tiles copy the state carries (each job's tail into
 *     its other state buffer, which no tile reads). The launch shape is
 *     fixed (CUDA graph friendly) and the counters reset themselves when the
 *     last CTA leaves.
 *   - Fast path (M a power of two, 16..4096): a tile is 4096 complex points
 *     (tile_hops = 4096/M), 512 threads x 8 points. For oversample 1/2/4 and
 *     M <= 2048 each thread folds two consecutive hops over the even or odd
 *     branches (the paired fold: every sample and tap load serves both
 *     hops) into a radix-4 first Stockham pass in registers; otherwise one
 *     hop's 8 branches into a radix-8 first pass. Small M stages the tile
 *     window in shared memory with cp.async first. The FFT runs in double,
 *     radix-8 passes in place in shared memory (XOR swizzle, one twiddle
 *     load per butterfly, group barriers), the last pass fused with the
 *     rotation, cal, rounding and the transpose to channel-major; each
 *     channel gets a run of tile_hops consecutive outputs.
 *   - Any other M up to 6400: single handles have kernels of their own
 *     (hops.cu); a batch's tiles run the same passes here (pfb_generic.cuh).
 */
#include <atomic>
#include "pfb_kernel.cuh"

namespace {

#include "pfb_generic.cuh"

/* Every shape's tile, and the generic banks', is a function of its own, so
 * that each gets the 64 registers for itself: with all of them inline one
 * allocation served 50 shapes with 1.5 to 1.9 KB of spills, and a change in
 * any one (the generic branch above all) moved the others. us, all inline /
 * apart: 64 uneven streams 1068 / 1062, another 64 1231 / 1211, 256 of them
 * 5209 / 5169. The generic tile loads one tap at a time: eight in flight need
 * more registers than are left (six scales of 8 to 256 channels, chunks of
 * 65,536 samples: 1255 MS/s at eight, 1450 at one). */
__device__ __noinline__ void tile_generic(const atkb_job &__restrict__ J, const atkb_bank &__restrict__ B,
                                          long long h0, int nvalid) {
    extern __shared__ double2 sm[];
    generic_tile<NT, 1>(J, B, J.cre, J.cim, h0, nvalid, sm);
}

template <int KEY>
__device__ __noinline__ void tile_of(const atkb_job &__restrict__ J, const atkb_bank &__restrict__ B, long long h0,
                                     int nvalid) {
    extern __shared__ double2 sm[];
    run_tile<KEY>(J, B, h0, nvalid, sm, (float2 *)sm);
}

struct AllShapes {
    static __device__ __forceinline__ void carry(const Src &src, float2 *dst, long long from, long long len) {
        carry_runs<NT>(src, dst, from, len);
    }
    static __device__ __forceinline__ void run(int key, const atkb_job &J, const atkb_bank &SB, long long h0,
                                               int nvalid, double2 *, float2 *) {
        switch (key) {
#define T(K) case K: tile_of<K>(J, SB, h0, nvalid); break;
#define EACH(S) T(S + 4) T(S + 5) T(S + 6) T(S + 7) T(S + 8) T(S + 9) T(S + 10)
        EACH(0) T(11) EACH(16) EACH(32) EACH(48) T(16 + 11) T(32 + 11) T(48 + 11)
        T(12) T(16 + 12) T(32 + 12) T(48 + 12) EACH(80) EACH(96)
#undef T
#undef EACH
        case -1: break;                      /* a tile to skip */
        default: tile_generic(J, SB, h0, nvalid); break;
        }
    }
};

__global__ void __launch_bounds__(NT, 2)
pfb_tiles_kernel(const atkb_job *__restrict__ jobs, const int *__restrict__ tile_start,
                 const atkb_carry *__restrict__ carries, int njobs, const int *__restrict__ d_njobs,
                 int *counters) {
    tiles_loop<AllShapes>(jobs, tile_start, carries, njobs, d_njobs, counters);
}

/* ---- large filterbanks: nchan beyond one CTA's shared memory --------------
 * A power of two above 4096 or any other nchan above 6400 has no in-CTA tile:
 * a hop's M points (16 M bytes in double) do not fit beside a second buffer.
 * Such a filterbank runs one hop chunk at a time through device scratch:
 *   fold      one thread per (hop, branch), the reference's operation order
 *             (a rounded multiply, then a rounded add, k ascending);
 *   FFT       the plan's Stockham passes, each one kernel over the chunk,
 *             ping-ponging between the two scratch halves (mixed radix 2, 3,
 *             4, 8, 16, and a direct DFT for any other prime factor);
 *   epilogue  rotation, cal and rounding as the tile kernel does them, written
 *             channel-major (a warp's lanes on consecutive hops of a channel).
 * Slower than the tile kernel (every pass goes through HBM), but any nchan
 * the reference accepts runs, with the same results. */
__global__ void __launch_bounds__(256)
big_fold_kernel(const atkb_job J, const float *__restrict__ taps, int M, int K, int hop, long long h0, int nh,
                double2 *__restrict__ F) {
    float cre = J.cre, cim = J.cim;
    if (J.doff) doff_consts(J.doff, J.kscale, cre, cim);
    const Src src{(const float2 *)J.state, J.in, J.head, J.in_kind, cre, cim, J.kscale};
    const long long total = (long long)nh * M;
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total;
         e += (long long)gridDim.x * blockDim.x) {
        const int t = (int)(e / M);
        const int q = (int)(e - (long long)t * M);
        const long long base = (h0 + t) * (long long)hop + q;
        float h = __ldg(taps + q);
        float2 x = src.at(base);
        float fr = __fmul_rn(h, x.x), fi = __fmul_rn(h, x.y);
        for (int k = 1; k < K; ++k) {
            h = __ldg(taps + (long long)k * M + q);
            x = src.at(base + (long long)k * M);
            fr = __fadd_rn(fr, __fmul_rn(h, x.x));
            fi = __fadd_rn(fi, __fmul_rn(h, x.y));
        }
        F[e] = make_double2((double)fr, (double)fi);
    }
}

__global__ void __launch_bounds__(256)
big_pass_kernel(const double2 *__restrict__ src, double2 *__restrict__ dst, int M, int Ns, int R, int nh,
                const double2 *__restrict__ W) {
    const int MR = M / R;
    const int NsR = Ns * R;
    const int stride = M / NsR;
    const long long total = (long long)nh * MR;
    for (long long bi = (long long)blockIdx.x * blockDim.x + threadIdx.x; bi < total;
         bi += (long long)gridDim.x * blockDim.x) {
        const int tt = (int)(bi / MR);
        const int j = (int)(bi - (long long)tt * MR);
        const int k = j % Ns;
        const double2 *s = src + (long long)tt * M + j;
        double2 *d = dst + (long long)tt * M + (long long)(j - k) * R + k;
        if (R == 2 || R == 3 || R == 4 || R == 8 || R == 16) {
            double2 v[16];
            for (int r = 0; r < R; ++r) {
                v[r] = s[(long long)r * MR];
                if (r) v[r] = cmul(v[r], __ldg(W + (long long)r * k * stride));
            }
            if (R == 2) dft2(v[0], v[1]);
            else if (R == 3) dft3(v[0], v[1], v[2]);
            else if (R == 4) dft4(v[0], v[1], v[2], v[3]);
            else if (R == 8) dft8(v);
            else dft16(v);
            for (int r = 0; r < R; ++r) d[(long long)r * Ns] = v[r];
        } else {
            /* direct DFT with the twiddle folded in: W_{NsR}^{r (k + o Ns)} */
            for (int o = 0; o < R; ++o) {
                double2 acc = make_double2(0.0, 0.0);
                for (int r = 0; r < R; ++r) {
                    const long long ex = ((long long)r * (k + (long long)o * Ns)) % NsR;
                    const double2 w = __ldg(W + ex * stride);
                    const double2 x = s[(long long)r * MR];
                    acc.x += x.x * w.x - x.y * w.y;
                    acc.y += x.x * w.y + x.y * w.x;
                }
                d[(long long)o * Ns] = acc;
            }
        }
    }
}

__global__ void __launch_bounds__(256)
big_out_kernel(const double2 *__restrict__ X, const atkb_job J, const double2 *__restrict__ twd, int M, int os,
               int hop, long long h0, int nh) {
    const float2 *cal = (const float2 *)J.cal;
    float2 *out = (float2 *)J.out;
    const long long total = (long long)nh * M;
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total;
         e += (long long)gridDim.x * blockDim.x) {
        const int kb = (int)(e / nh);
        const int tt = (int)(e - (long long)kb * nh);
        double2 v = X[(long long)tt * M + kb];
        const long long b = J.b0 + h0 + tt;
        const int s = (int)((b + 1) % os);
        const int jr = (int)(((long long)kb * s) % os);
        v = cmul_rn(v, __ldg(twd + (jr ? M - jr * hop : 0)));
        if (cal) {
            const float2 c = __ldg(cal + kb);
            v = cmul_rn(v, make_double2((double)c.x, (double)c.y));
        }
        out[(long long)kb * J.ldo + J.out_col + h0 + tt] = make_float2(__double2float_rn(v.x), __double2float_rn(v.y));
    }
}


}  // namespace

extern "C" int atkb_pfb_max_smem(void) { return 200 * 1024; }

namespace {
/* the kernel a launch of bank B's tiles alone takes: its shape's own where
 * there is one, else (and for B NULL, any mix of banks) the one of every
 * shape. The largest shared memory it may be given is set on first use; the
 * attribute is idempotent, concurrent first callers may both set it. */
const void *tile_kernel(const atkb_bank *B) {
    static std::atomic<unsigned char> configured[64][128];
    const void *fn = B ? atkb_pfb_one(atkb_tile_key(B)) : nullptr;
    const int key = fn ? atkb_tile_key(B) : 0;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64 || key < 0 || key >= 128) return nullptr;
    if (!fn) fn = (const void *)pfb_tiles_kernel;
    if (!configured[dev][key].load(std::memory_order_acquire)) {
        if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, atkb_pfb_max_smem()) != cudaSuccess)
            return nullptr;
        configured[dev][key].store(1, std::memory_order_release);
    }
    return fn;
}

int launch_tiles(const atkb_job *d_jobs, const int *d_tile_start, const atkb_carry *d_carry, int njobs,
                 const int *d_njobs, int *d_counters, int grid, int smem_bytes, const atkb_bank *B, bool dependent,
                 void *stream) {
    if (njobs <= 0) return ATKB_OK;
    const void *fn = tile_kernel(B);
    if (!fn) return ATKB_E_KERNEL;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(grid < 1 ? 1 : grid));
    cfg.blockDim = dim3(NT);
    cfg.dynamicSmemBytes = (size_t)smem_bytes;
    cfg.stream = (cudaStream_t)stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = dependent ? 1 : 0;
    void *args[] = {&d_jobs, &d_tile_start, &d_carry, &njobs, &d_njobs, &d_counters};
    atkb_range_push("atkdsp tile kernel launch");
    const cudaError_t e = cudaLaunchKernelExC(&cfg, fn, args);
    atkb_range_pop();
    return e == cudaSuccess && cudaGetLastError() == cudaSuccess ? ATKB_OK : ATKB_E_KERNEL;
}
}  // namespace

extern "C" int atkb_pfb_grid(int dev, int smem_bytes, const atkb_bank *B) {
    int per_sm = 0;
    const void *fn = tile_kernel(B);
    if (!fn) return -1;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, NT, smem_bytes) != cudaSuccess ||
        per_sm < 1)
        per_sm = 1;
    return per_sm * atkb_sm_count(dev);
}

extern "C" int atkb_pfb_launch(const atkb_job *d_jobs, const int *d_tile_start, const atkb_carry *d_carry,
                               int njobs, int *d_counters, int grid, int smem_bytes, const atkb_bank *B, void *stream) {
    return launch_tiles(d_jobs, d_tile_start, d_carry, njobs, NULL, d_counters, grid, smem_bytes, B, false, stream);
}

extern "C" int atkb_pfb_launch_n(const atkb_job *d_jobs, const int *d_tile_start, const atkb_carry *d_carry,
                                 int njobs, const int *d_njobs, int *d_counters, int grid, int smem_bytes,
                                 void *stream) {
    return launch_tiles(d_jobs, d_tile_start, d_carry, njobs, d_njobs, d_counters, grid, smem_bytes, NULL, false,
                        stream);
}

/* atkb_pfb_launch as a programmatic dependent launch: its CTAs may start
 * while the previous kernel on the stream (conv_from_offset_kernel) runs,
 * and wait for that kernel's completion before reading the table */
extern "C" int atkb_pfb_launch_pdl(const atkb_job *d_jobs, const int *d_tile_start, const atkb_carry *d_carry,
                                   int njobs, int *d_counters, int grid, int smem_bytes, const atkb_bank *B,
                                   void *stream) {
    return launch_tiles(d_jobs, d_tile_start, d_carry, njobs, NULL, d_counters, grid, smem_bytes, B, true, stream);
}

extern "C" long long atkb_pfb_big_hops(int nchan) {
    const long long h = (1LL << 20) / nchan;
    return h < 1 ? 1 : h;
}

extern "C" int atkb_pfb_big(const atkb_job *J, const atkb_bank *B, long long h0, int nh, void *scratch,
                            int grid, void *stream) {
    if (nh <= 0) return ATKB_OK;
    cudaStream_t st = (cudaStream_t)stream;
    const int M = B->nchan;
    double2 *A = (double2 *)scratch, *Bf = A + (size_t)nh * M;
    if (grid < 1) grid = 1;
    atkb_range_push("atkdsp large-filterbank chunk");
    big_fold_kernel<<<grid, 256, 0, st>>>(*J, B->taps, M, B->K, B->hop, h0, nh, A);
    int Ns = 1;
    double2 *cur = A, *nxt = Bf;
    for (int p = 0; p < B->plan.npass; ++p) {
        const int R = B->plan.radix[p];
        big_pass_kernel<<<grid, 256, 0, st>>>(cur, nxt, M, Ns, R, nh, (const double2 *)B->wfull);
        Ns *= R;
        double2 *t = cur; cur = nxt; nxt = t;
    }
    big_out_kernel<<<grid, 256, 0, st>>>(cur, *J, (const double2 *)B->twd, M, B->os, B->hop, h0, nh);
    atkb_range_pop();
    return cudaGetLastError() == cudaSuccess ? ATKB_OK : ATKB_E_KERNEL;
}

extern "C" unsigned atkb_pfb_debug_fault(void) {
#ifdef ATKB_DEBUG_BOUNDS
    return take_debug_fault() | atkb_pfb_one_fault() | atkb_pfb_hops_fault();
#else
    return 0;
#endif
}

extern "C" int atkb_pfb_debug_build(void) {
#ifdef ATKB_DEBUG_BOUNDS
    return 1;
#else
    return 0;
#endif
}
