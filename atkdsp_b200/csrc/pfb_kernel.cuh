/* The filterbank's persistent tile kernel: the tile shapes and the loop over
 * tiles and carries. Instantiated for every shape at once (pfb.cu: batches,
 * the server, any mix of banks) and for one shape each (pfb_one.cu: launches
 * of a single bank). The shapes' arithmetic is the same in both, so are the
 * bits. */
#ifndef ATKB_PFB_KERNEL_CUH
#define ATKB_PFB_KERNEL_CUH

#include <cuda_runtime.h>
#include <stdint.h>
#include "internal.h"

/* the fast path's tile: 4096 complex points, PTS per thread (ATKB_PTS in
 * internal.h: 8 points -> 512 threads at <= 64 registers, 32 warps per SM) */
#define PTS ATKB_PTS
#define LOGP (PTS == 16 ? 4 : 3)
#define TILE_POINTS 4096
#define NT (TILE_POINTS / PTS)


/* which tile a bank's hops run through: 16 * shape + log2(nchan), shape 0 one
 * hop per thread (at nchan 4096: 0 the two-hop tile, 1-3 its paired fold at
 * oversample 1, 2, 4), 1-3 the paired fold at oversample 1, 2, 4, 5 and 6 the
 * quad fold at 1 and 2; 0 for a generic bank, which has no tile here */
__host__ __device__ inline int atkb_tile_key(const atkb_bank *B) {
    if (!B->plan.fast) return 0;
    const int o = B->os == 1 ? 0 : B->os == 2 ? 1 : 2;
    const int shape = B->plan.quad ? 5 + o : B->plan.pair || (B->logm == 12 && B->plan.ptaps) ? 1 + o : 0;
    return 16 * shape + B->logm;
}

namespace {


#include "pfb_dev.cuh"

/* ---- fast path: nchan = 2^n, 16 <= nchan <= 4096 ------------------------- */
/* Shared-memory index swizzle for the 16-byte complex doubles: the low LOGP
 * index bits are XORed with the next LOGP. The first pass stores at a stride
 * of PTS (or 4) elements across lanes; swizzled, every 8-lane wavefront lands
 * on 8 distinct 16-byte slots, and the unit-stride accesses of later passes
 * stay conflict-free too (a XOR with a per-block constant permutes the
 * slots). */
__device__ __forceinline__ int SW(int i) { return i ^ ((i >> LOGP) & (PTS - 1)); }

/* Barrier over the G consecutive threads that share a hop group (G a power of
 * two): a warp sync up to 32 threads, a named barrier (ids 1..NT/G) up to
 * the CTA, __syncthreads for the whole CTA. Memory ordering among the
 * participants is that of bar.sync / bar.warp.sync. */
template <int G>
__device__ __forceinline__ void group_sync() {
    static_assert((G & (G - 1)) == 0 && G <= NT, "group size");
    if constexpr (G >= NT) {
        __syncthreads();
    } else if constexpr (G <= 32) {
        __syncwarp();
    } else {
        static_assert(NT / G <= 15, "named barrier ids 1..15");
        asm volatile("bar.sync %0, %1;" ::"r"(1 + (int)threadIdx.x / G), "r"(G) : "memory");
    }
}

/* Butterfly u of this thread in a pass with U butterflies per thread:
 * warp w owns butterflies [32 w U, 32 (w + 1) U), lanes consecutive, so a
 * warp's butterflies are the same hops as its threads' points in a radix-PTS
 * pass (M/PTS consecutive threads per hop) and lanes read consecutive j. */
template <int U>
__device__ __forceinline__ int bfly(int u) {
    return (((int)threadIdx.x & ~31) * U) + u * 32 + ((int)threadIdx.x & 31);
}

/* One in-place Stockham pass over a 4096-point tile (NT threads x PTS
 * points): every index is a compile-time shift or mask. tw holds
 * W_{Ns R}^{k} at k (tw_powers forms the other powers). G is the group whose barrier
 * suffices (a multiple of the M/PTS threads of one hop): with bfly's
 * numbering the pass reads and writes only its group's hops. */
template <int LOGM, int R, int LOGNS, int G = NT>
__device__ __forceinline__ void pass_c(double2 *sm, const double2 *__restrict__ tw) {
    constexpr int M = 1 << LOGM;
    constexpr int NS = 1 << LOGNS;
    constexpr int LOGR = R == 16 ? 4 : R == 8 ? 3 : R == 4 ? 2 : 1;
    constexpr int LOGMR = LOGM - LOGR;
    constexpr int MR = 1 << LOGMR;
    constexpr int U = PTS / R;
    double2 v[U][R];
    int dst[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int bi = bfly<U>(u);
        const int tt = bi >> LOGMR;
        const int j = bi & (MR - 1);
        const int k = j & (NS - 1);
        const int base = (tt << LOGM) + j;
#pragma unroll
        for (int r = 0; r < R; ++r) v[u][r] = sm[SW(base + r * MR)];
        double2 w[R];
        tw_powers<R>(__ldg(tw + k), w);
#pragma unroll
        for (int r = 1; r < R; ++r) v[u][r] = cmul(v[u][r], w[r]);
        dst[u] = (tt << LOGM) + ((j - k) << LOGR) + k;
    }
    group_sync<G>();
#pragma unroll
    for (int u = 0; u < U; ++u) {
        dftR<R>(v[u]);
#pragma unroll
        for (int r = 0; r < R; ++r) sm[SW(dst[u] + r * NS)] = v[u][r];
    }
    group_sync<G>();
}

/* The last Stockham pass fused with the epilogue: after the butterflies every
 * output is a final bin (j + r*Ns of hop tt), rotated, calibrated, rounded and
 * written straight into the padded channel-major tile. The loads read only
 * this thread's group's hops (so the previous pass may end on a group
 * barrier); the tile_out stores overlap every group's points, hence the
 * CTA-wide barrier between them. */
template <int LOGM, int R, int LOGNS>
__device__ __forceinline__ void pass_last(double2 *sm, const double2 *__restrict__ tw,
                                          float2 *tile_out, const atkb_bank &B, const atkb_job &J,
                                          long long h0) {
    constexpr int M = 1 << LOGM;
    constexpr int NS = 1 << LOGNS;
    constexpr int LOGR = R == 16 ? 4 : R == 8 ? 3 : R == 4 ? 2 : 1;
    constexpr int LOGMR = LOGM - LOGR;          /* == LOGNS: Ns * R == M */
    constexpr int MR = 1 << LOGMR;
    constexpr int U = PTS / R;
    constexpr int NH = 1 << (12 - LOGM);
    double2 v[U][R];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int bi = bfly<U>(u);
        const int tt = bi >> LOGMR;
        const int j = bi & (MR - 1);
        const int base = (tt << LOGM) + j;
#pragma unroll
        for (int r = 0; r < R; ++r) v[u][r] = sm[SW(base + r * MR)];
        double2 w[R];
        tw_powers<R>(__ldg(tw + j), w);
#pragma unroll
        for (int r = 1; r < R; ++r) v[u][r] = cmul(v[u][r], w[r]);
    }
    __syncthreads();
    const double2 *twd = (const double2 *)B.twd;
    const float2 *cal = (const float2 *)J.cal;
    /* os divides M, a power of two here: every "mod os" is a mask */
    const int osm = B.os - 1, hop = B.hop;
    const int s0 = (int)(J.b0 + h0 + 1) & osm;
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int bi = bfly<U>(u);
        const int tt = bi >> LOGMR;
        const int j = bi & (MR - 1);
        const int s = (s0 + tt) & osm;
        dftR<R>(v[u]);
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int kb = j + r * NS;
            tile_out[kb * (NH + 1) + tt] = finish_bin(v[u][r], kb, s, M, osm + 1, hop, true, twd, cal);
        }
    }
    __syncthreads();
}

/* The fold of one hop's PTS branches q = j + r*M/PTS (r < PTS), straight
 * into the registers of the first radix-PTS butterfly. Taps come from the
 * bank's permuted copy: float4 loads whose addresses are consecutive across
 * the lanes (branches j) of a warp.
 * MODE 0: the tile's windows lie wholly in one cf32 buffer, read through
 * `lin` (offset to this thread's first sample); MODE 1: the same in raw int16
 * I/Q converted on the fly; MODE 2: each sample from the state or the input
 * by index. */
template <int LOGM, int MODE>
__device__ __forceinline__ void foldP(double2 *v, const atkb_job &J, const atkb_bank &B,
                                      long long h0, int tt, int j, const void *lin) {
    constexpr int M = 1 << LOGM;
    constexpr int MP = M >> LOGP;
    const float4 *tq = (const float4 *)B.tapsP + j;
    float fr[PTS], fi[PTS];
    const float2 *xk = (const float2 *)lin;
    const short2 *xk16 = (const short2 *)lin;
    const float cre = J.cre, cim = J.cim, ks = J.kscale;
    const Src src{(const float2 *)J.state, J.in, J.head, J.in_kind, J.cre, J.cim, J.kscale};
    const long long base = (h0 + tt) * (long long)B.hop + j;
#pragma unroll
    for (int q = 0; q < PTS / 4; ++q) {
        const float4 h = __ldg(tq + q * MP);
        const float hh[4] = {h.x, h.y, h.z, h.w};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int r = 4 * q + c;
            const float2 x = MODE == 0 ? __ldg(xk + r * MP)
                           : MODE == 1 ? conv16(__ldg(xk16 + r * MP), cre, cim, ks)
                                       : src.at(base + r * MP);
            fr[r] = __fmul_rn(hh[c], x.x);
            fi[r] = __fmul_rn(hh[c], x.y);
        }
    }
    for (int k = 1; k < B.K; ++k) {
        tq += MP * (PTS / 4);
        xk += M;
        xk16 += M;
#pragma unroll
        for (int q = 0; q < PTS / 4; ++q) {
            const float4 h = __ldg(tq + q * MP);
            const float hh[4] = {h.x, h.y, h.z, h.w};
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int r = 4 * q + c;
                const float2 x = MODE == 0 ? __ldg(xk + r * MP)
                               : MODE == 1 ? conv16(__ldg(xk16 + r * MP), cre, cim, ks)
                                           : src.at(base + (long long)k * M + r * MP);
                fr[r] = __fadd_rn(fr[r], __fmul_rn(hh[c], x.x));
                fi[r] = __fadd_rn(fi[r], __fmul_rn(hh[c], x.y));
            }
        }
    }
#pragma unroll
    for (int r = 0; r < PTS; ++r) v[r] = make_double2((double)fr[r], (double)fi[r]);
}

/* ---- the staged fold for small nchan ----------------------------------------
 * With nchan <= 512 a tile spans many hops whose windows overlap heavily (each
 * staged sample is used 6-20 times). The whole tile window is copied once into
 * shared memory with asynchronous copies (cp.async: no registers held while
 * the copies fly), then folded from there. Layout: logical sample i of the
 * window lives at i + (i / hop) * (M/16), a pad of M/16 samples after every
 * hop-long block, so the lanes of a warp (several hops x M/16 branches) hit
 * distinct banks. */
__device__ __forceinline__ void cp_async8(void *smem, const void *gmem) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

/* physical size (in samples) of a staged window of W samples */
__device__ __forceinline__ int staged_size(int W, int logs, int MR) { return W + ((W - 1) >> logs) * MR + MR; }

template <int LOGM, int LOGOS>
__device__ __forceinline__ void foldP_staged(double2 *v, const atkb_bank &B, int tt, int j,
                                             const float2 *xs) {
    constexpr int M = 1 << LOGM;
    constexpr int MP = M >> LOGP;
    constexpr int OS = 1 << LOGOS;
    constexpr int HOP = M >> LOGOS;
    /* logical tt*hop + k*M + j + r*MP  ->  physical, with (i / hop) = tt + k*os + (r*os)/PTS */
    const float2 *xb = xs + tt * (HOP + MP) + j;
    const float4 *tq = (const float4 *)B.tapsP + j;
    float fr[PTS], fi[PTS];
#pragma unroll
    for (int q = 0; q < PTS / 4; ++q) {
        const float4 h = __ldg(tq + q * MP);
        const float hh[4] = {h.x, h.y, h.z, h.w};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int r = 4 * q + c;
            const float2 x = xb[r * MP + ((r * OS) >> LOGP) * MP];
            fr[r] = __fmul_rn(hh[c], x.x);
            fi[r] = __fmul_rn(hh[c], x.y);
        }
    }
    for (int k = 1; k < B.K; ++k) {
        tq += MP * (PTS / 4);
        xb += M + OS * MP;
#pragma unroll
        for (int q = 0; q < PTS / 4; ++q) {
            const float4 h = __ldg(tq + q * MP);
            const float hh[4] = {h.x, h.y, h.z, h.w};
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int r = 4 * q + c;
                const float2 x = xb[r * MP + ((r * OS) >> LOGP) * MP];
                fr[r] = __fadd_rn(fr[r], __fmul_rn(hh[c], x.x));
                fi[r] = __fadd_rn(fi[r], __fmul_rn(hh[c], x.y));
            }
        }
    }
#pragma unroll
    for (int r = 0; r < PTS; ++r) v[r] = make_double2((double)fr[r], (double)fi[r]);
}

/* copy the tile window s[h0*hop, h0*hop + W) into the padded shared layout */
__device__ __forceinline__ void stage_window(float2 *xs, const atkb_job &J, long long g0, int W,
                                             int logs, int MR) {
    const float2 *st = (const float2 *)J.state;
    const float2 *in = (const float2 *)J.in;
    for (int i = threadIdx.x; i < W; i += NT) {
        const long long g = g0 + i;
        const float2 *src = g < J.head ? st + g : in + (g - J.head);
        if (IDX_OK(i + (i >> logs) * MR < 8192 && g < J.nsrc)) cp_async8(xs + i + (i >> logs) * MR, src);
    }
    cp_async_wait_all();
    __syncthreads();
}

template <int LOGM>
__device__ __forceinline__ bool fold_tile_staged(double2 *v, const atkb_job &J, const atkb_bank &B,
                                                 long long h0, int nvalid, int tt, int j, double2 *sm) {
    constexpr int M = 1 << LOGM;
    constexpr int MR = M >> LOGP;
    if constexpr (LOGM > 9) {
        return false;
    } else {
        const int os = B.os;
        if (J.in_kind || B.plan.nostage || (os != 1 && os != 2 && os != 4)) return false;
        const int logs = LOGM - (os == 1 ? 0 : os == 2 ? 1 : 2);
        const long long Wl = (long long)(nvalid - 1) * B.hop + B.L;
        if (Wl > 8192) return false;
        const int W = (int)Wl;
        if (staged_size(W, logs, MR) > 8192) return false;     /* sm holds 8192 float2 */
        float2 *xs = (float2 *)sm;
        stage_window(xs, J, h0 * (long long)B.hop, W, logs, MR);
        if (tt < nvalid) {
            if (os == 1) foldP_staged<LOGM, 0>(v, B, tt, j, xs);
            else if (os == 2) foldP_staged<LOGM, 1>(v, B, tt, j, xs);
            else foldP_staged<LOGM, 2>(v, B, tt, j, xs);
        } else {
#pragma unroll
            for (int r = 0; r < PTS; ++r) v[r] = make_double2(0.0, 0.0);
        }
        __syncthreads();              /* the window is dead; sm becomes the FFT tile */
        return true;
    }
}

/* ---- the paired fold: oversample 1, 2 or 4, nchan <= 2048 -------------------
 * Thread (pair p, parity c, branch j) folds hops ta = 2p and tb = 2p + 1 of
 * the tile over the four branches j + r*MP with r = c + 2i, i = 0..3
 * (MP = M/8). Slot u = 8k + r of hop ta's window (sample u*MP + j, tap
 * k*M + r*MP + j) is slot u - 8/os of hop tb's: every sample the thread loads
 * feeds both hops, and each float4 of taps (row k, parity c) serves hop ta in
 * row k and hop tb in rows k and k + 1. Against one hop and eight branches per
 * thread this halves the loads of samples and taps per output. Slots stream in
 * ascending order, so every branch still sums its taps k ascending; the sums
 * start from -0.0f, and -0 + p == p for every p, so the first product enters
 * unchanged as in the reference's loop. */
__device__ __forceinline__ void mac(float2 &a, float h, float2 x) {
    a.x = __fadd_rn(a.x, __fmul_rn(h, x.x));
    a.y = __fadd_rn(a.y, __fmul_rn(h, x.y));
}

/* sample loaders: at(k, i) is slot 8k + c + 2i of hop ta's window */
template <int LOGM>
struct PairLin {                       /* cf32, the tile's windows in one buffer */
    const float2 *p;
    __device__ __forceinline__ float2 at(int k, int i) const {
        return __ldg(p + ((long long)k << LOGM) + 2 * i * (1 << (LOGM - LOGP)));
    }
};
template <int LOGM>
struct PairLin16 {                     /* raw int16 I/Q, converted on the fly */
    const short2 *p;
    float cre, cim, ks;
    __device__ __forceinline__ float2 at(int k, int i) const {
        return conv16(__ldg(p + ((long long)k << LOGM) + 2 * i * (1 << (LOGM - LOGP))), cre, cim, ks);
    }
};
template <int LOGM>
struct PairMixed {                     /* cf32 state / input by index */
    const float2 *st, *in;
    long long g, head;
    __device__ __forceinline__ float2 at(int k, int i) const {
        const long long pos = g + ((long long)k << LOGM) + 2 * i * (1 << (LOGM - LOGP));
        return __ldg(pos < head ? st + pos : in + (pos - head));
    }
};
template <int LOGM>
struct PairMixed16 {                   /* cf32 state / raw int16 input by index */
    const float2 *st;
    const short2 *in;
    long long g, head;
    float cre, cim, ks;
    __device__ __forceinline__ float2 at(int k, int i) const {
        const long long pos = g + ((long long)k << LOGM) + 2 * i * (1 << (LOGM - LOGP));
        return pos < head ? __ldg(st + pos) : conv16(__ldg(in + (pos - head)), cre, cim, ks);
    }
};
template <int LOGM, int LOGOS>
struct PairStaged {                    /* the padded shared-memory window */
    const float2 *p;                   /* at slot c of hop ta, row 0 */
    __device__ __forceinline__ float2 at(int k, int i) const {
        constexpr int MP = 1 << (LOGM - LOGP);
        constexpr int LOGD = 3 - LOGOS;             /* slot shift 8/os = 2^LOGD */
        return p[k * ((1 << LOGM) + (MP << LOGOS)) + (2 * i + (i >> (LOGD - 1))) * MP];
    }
};

/* Taps a turn of the paired fold's loop in the kernels of one shape
 * (pfb_one.cu); 0 leaves it to the compiler, as in the kernel of every shape.
 * us left to it / as here, 3,000,001 samples: nchan 4096 4x 12 taps 189 / 177,
 * 4x 16 199 / 189, 2x 16 97.4 / 94.6; 2048 1x 12 taps 45.4 / 43.3; nchan 16 4x 5
 * taps 115 / 110, 4x 16 137 / 134. The other shapes' loops are as good as any. */
__host__ __device__ constexpr int fold_unroll(int logm, int logos) {
#ifdef ONE_LOGM
    if (logm == 4) return logos > 0 ? 2 : 0;
    return (logm == 12 && logos > 0) || (logm == 11 && logos == 0) ? 1 : 0;
#else
    return 0;
#endif
}

template <int LOGM, int LOGOS, class LD>
__device__ __forceinline__ void fold_pair(float2 (&a)[4], float2 (&b)[4], const float4 *tq, int K,
                                          bool tb_ok, const LD &ld) {
    constexpr int MP = 1 << (LOGM - LOGP);
    constexpr int D2 = 4 >> LOGOS;     /* hop tb's taps trail hop ta's by D2 entries */
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        a[i] = make_float2(-0.0f, -0.0f);
        b[i] = make_float2(-0.0f, -0.0f);
    }
    float4 pv = __ldg(tq);
    {
        const float h[4] = {pv.x, pv.y, pv.z, pv.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 x = ld.at(0, i);
            mac(a[i], h[i], x);
            if (i >= D2) mac(b[i - D2], h[i - D2], x);
        }
    }
    auto step = [&](int k) {
        const float4 cv = __ldg(tq + k * 2 * MP);
        const float h[4] = {cv.x, cv.y, cv.z, cv.w};
        const float g[4] = {pv.x, pv.y, pv.z, pv.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 x = ld.at(k, i);
            mac(a[i], h[i], x);
            if (i >= D2) mac(b[i - D2], h[i - D2], x);
            else mac(b[i - D2 + 4], g[i - D2 + 4], x);
        }
        pv = cv;
    };
    constexpr int U = fold_unroll(LOGM, LOGOS);
    if constexpr (U == 0) {
        for (int k = 1; k < K; ++k) step(k);
    } else {
#pragma unroll U
        for (int k = 1; k < K; ++k) step(k);
    }
    if (tb_ok) {                       /* the slots past hop ta's window */
        const float g[4] = {pv.x, pv.y, pv.z, pv.w};
#pragma unroll
        for (int i = 0; i < D2; ++i) mac(b[i - D2 + 4], g[i - D2 + 4], ld.at(K, i));
    }
}

/* radix-4 first pass (Ns = 1) of one hop's four even or odd branches:
 * branch j + (c + 2i)*MP is point jp + i*M/4 of the hop, jp = j + c*MP */
template <int LOGM>
__device__ __forceinline__ void first_pass4(const float2 (&f)[4], double2 *sm, int t, int jp) {
    double2 v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = make_double2((double)f[i].x, (double)f[i].y);
    dft4(v[0], v[1], v[2], v[3]);
#pragma unroll
    for (int i = 0; i < 4; ++i)
        if (IDX_OK((t << LOGM) + jp * 4 + i < TILE_POINTS)) sm[SW((t << LOGM) + jp * 4 + i)] = v[i];
}

/* the paired fold of hops ta, ta + 1 (parity c, branch j) from global memory;
 * the window source (input, state, or both by index) is chosen per tile */
template <int LOGM, int LOGOS>
__device__ __forceinline__ void fold_pair_global(float2 (&a)[4], float2 (&b)[4], const atkb_job &J,
                                                 const atkb_bank &B, long long h0, int nvalid, int ta,
                                                 int c, int j, bool tb_ok) {
    constexpr int MP = 1 << (LOGM - LOGP);
    constexpr int HOP = (1 << LOGM) >> LOGOS;
    const float4 *tq = (const float4 *)B.tapsP + c * MP + j;
    const long long w0 = h0 * (long long)HOP;
    const long long w1 = (h0 + nvalid - 1) * (long long)HOP + B.L;
    const long long off = (h0 + ta) * (long long)HOP + c * MP + j;
    if (w0 >= J.head) {
        if (J.in_kind) {
            const PairLin16<LOGM> ld{(const short2 *)J.in + (off - J.head), J.cre, J.cim, J.kscale};
            fold_pair<LOGM, LOGOS>(a, b, tq, B.K, tb_ok, ld);
        } else {
            const PairLin<LOGM> ld{(const float2 *)J.in + (off - J.head)};
            fold_pair<LOGM, LOGOS>(a, b, tq, B.K, tb_ok, ld);
        }
    } else if (w1 <= J.head) {
        const PairLin<LOGM> ld{(const float2 *)J.state + off};
        fold_pair<LOGM, LOGOS>(a, b, tq, B.K, tb_ok, ld);
    } else {
        if (J.in_kind) {
            const PairMixed16<LOGM> ld{(const float2 *)J.state, (const short2 *)J.in, off, J.head,
                                       J.cre, J.cim, J.kscale};
            fold_pair<LOGM, LOGOS>(a, b, tq, B.K, tb_ok, ld);
        } else {
            const PairMixed<LOGM> ld{(const float2 *)J.state, (const float2 *)J.in, off, J.head};
            fold_pair<LOGM, LOGOS>(a, b, tq, B.K, tb_ok, ld);
        }
    }
}

template <int LOGM, int LOGOS>
__device__ __forceinline__ void fold_tile_pair(const atkb_job &J, const atkb_bank &B, long long h0,
                                               int nvalid, double2 *sm) {
    constexpr int M = 1 << LOGM;
    constexpr int LOGMP = LOGM - LOGP;
    constexpr int MP = 1 << LOGMP;
    constexpr int HOP = M >> LOGOS;
    const int tid = threadIdx.x;
    const int j = tid & (MP - 1);
    const int c = (tid >> LOGMP) & 1;
    const int ta = (tid >> (LOGMP + 1)) * 2;
    const bool ta_ok = ta < nvalid, tb_ok = ta + 1 < nvalid;
    const float4 *tq = (const float4 *)B.tapsP + c * MP + j;
    float2 a[4], b[4];
    if constexpr (LOGM <= 9) {
        /* small nchan: the whole tile window through shared memory (as in
         * fold_tile_staged; logical sample i at i + (i / hop) * MP) */
        const long long Wl = (long long)(nvalid - 1) * HOP + B.L;
        if (!J.in_kind && !B.plan.nostage && Wl <= 8192 && staged_size((int)Wl, LOGM - LOGOS, MP) <= 8192) {
            float2 *xs = (float2 *)sm;
            stage_window(xs, J, h0 * (long long)HOP, (int)Wl, LOGM - LOGOS, MP);
            if (ta_ok) {
                const PairStaged<LOGM, LOGOS> ld{xs + ta * (HOP + MP) + j + c * MP};
                fold_pair<LOGM, LOGOS>(a, b, tq, B.K, tb_ok, ld);
            } else {
#pragma unroll
                for (int i = 0; i < 4; ++i) a[i] = b[i] = make_float2(0.0f, 0.0f);
            }
            __syncthreads();          /* the window is dead; sm becomes the FFT tile */
            /* the first pass inside this branch: merging the sums of both
             * branches ahead of one first pass cost ~1 KB of spills */
            first_pass4<LOGM>(a, sm, ta, j + c * MP);
            first_pass4<LOGM>(b, sm, ta + 1, j + c * MP);
            return;
        }
    }
    if (ta_ok) fold_pair_global<LOGM, LOGOS>(a, b, J, B, h0, nvalid, ta, c, j, tb_ok);
    if (!ta_ok) {
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = b[i] = make_float2(0.0f, 0.0f);
    }
    first_pass4<LOGM>(a, sm, ta, j + c * MP);
    first_pass4<LOGM>(b, sm, ta + 1, j + c * MP);
}

/* the Stockham passes after the first (which left Ns = 2^LOGNS): radix PTS
 * while more than LOGP index bits remain, then the last pass (radix 2, 4 or
 * 8) fused with the epilogue; P indexes the plan's twiddle offsets */
template <int LOGM, int LOGNS, int P, int G = NT>
__device__ __forceinline__ void fft_rest(double2 *sm, const double2 *wp, const int *twoff,
                                         float2 *tile_out, const atkb_bank &B, const atkb_job &J,
                                         long long h0) {
    if constexpr (LOGM - LOGNS > LOGP) {
        pass_c<LOGM, PTS, LOGNS, G>(sm, wp + twoff[P]);
        fft_rest<LOGM, LOGNS + LOGP, P + 1, G>(sm, wp, twoff, tile_out, B, J, h0);
    } else {
        pass_last<LOGM, (1 << (LOGM - LOGNS)), LOGNS>(sm, wp + twoff[P], tile_out, B, J, h0);
    }
}

/* write a finished tile: thread -> (channel kb0 + u*MP, hop t2), runs of NH
 * consecutive hops per channel */
template <int LOGM>
__device__ __forceinline__ void write_tile(const atkb_job &J, long long h0, int nvalid,
                                           const float2 *tile_out) {
    constexpr int LOGNH = 12 - LOGM;
    constexpr int NH = 1 << LOGNH;
    constexpr int MP = (1 << LOGM) >> LOGP;
    const int tid = threadIdx.x;
    const int t2 = tid & (NH - 1);
    if (t2 < nvalid) {
        const int kb0 = tid >> LOGNH;
        float2 *o = (float2 *)J.out + (J.out_col + h0 + t2) + (long long)kb0 * J.ldo;
        const long long step = (long long)MP * J.ldo;
#pragma unroll 4
        for (int u = 0; u < PTS; ++u) {
            const int row = kb0 + u * MP;
            if (IDX_OK(row < (1 << LOGM) && J.out_col + h0 + t2 < J.ldo &&
                       row * (NH + 1) + t2 < TILE_POINTS * 2))
                *o = tile_out[row * (NH + 1) + t2];
            o += step;
        }
    }
}

/* W2 fused into the epilogue: the tile's power per channel, sum over its
 * valid hops t of |y|^2 in double from the rounded outputs (the reference's
 * W2 sum, src/channelizer.c:459-461, for these hops), written to the job's
 * partial buffer at row h0 / tile_hops. A second kernel adds the tiles' rows
 * in tile order (atkb_w2_finish). tile_out stays intact until the barrier
 * that opens the next tile. */
template <int LOGM>
__device__ __forceinline__ void w2_partial(const atkb_job &J, long long h0, int nvalid, const float2 *tile_out) {
    constexpr int M = 1 << LOGM;
    constexpr int NH = 1 << (12 - LOGM);
    double *row = J.w2 + (h0 / NH) * M;
    for (int kb = threadIdx.x; kb < M; kb += NT) {
        double s = 0.0;
        for (int t = 0; t < nvalid; ++t) {
            const float2 y = tile_out[kb * (NH + 1) + t];
            s += (double)y.x * y.x + (double)y.y * y.y;
        }
        row[kb] = s;
    }
}

/* ---- the quad fold: oversample 1 or 2, nchan <= 1024 --------------------------
 * Thread (quad g, class c, branch j) folds the four hops ta + t (ta = 4g,
 * t = 0..3) of the tile over the two branches q0 = j + c*MP and q1 = q0 + M/2
 * (MP = M/8, c = 0..3). In hop ta's frame its samples are the slots
 * u = 4v + c (sample u*MP + j, tap u*MP + j), v = 0 .. 2K-1; hop ta + t sees
 * the same sample at slot u - t*8/os, i.e. at v - t*D with D = 2/os, which
 * keeps the class c. So every sample the thread loads feeds all four hops,
 * and each tap it loads serves the four hops in turn through a window of
 * W = 4*D taps held in registers: per input sample position one 8-byte
 * sample load, one 4-byte tap load and four complex multiply-adds (against
 * one tap load per two multiply-adds in the paired fold). Branch q_i of hop t
 * sums its taps in slot order -- k ascending, a rounded multiply then a
 * rounded add, from -0.0f -- like every other fold here, so all tile shapes
 * give the reference's bits. The two branches feed a radix-2
 * first Stockham pass (Ns = 1: points q0 and q0 + M/2 of each hop). */
template <int LOGM>
struct QuadLin {                       /* cf32, the quad's windows in one buffer */
    const float2 *p;                   /* at slot c of hop ta, branch j */
    __device__ __forceinline__ float2 at(int v) const { return __ldg(p + (long long)v * (1 << (LOGM - 1))); }
};
template <int LOGM>
struct QuadLin16 {                     /* raw int16 I/Q, converted on the fly */
    const short2 *p;
    float cre, cim, ks;
    __device__ __forceinline__ float2 at(int v) const {
        return conv16(__ldg(p + (long long)v * (1 << (LOGM - 1))), cre, cim, ks);
    }
};
template <int LOGM>
struct QuadMixed {                     /* cf32 state / input by index */
    const float2 *st, *in;
    long long g, head;
    __device__ __forceinline__ float2 at(int v) const {
        const long long pos = g + (long long)v * (1 << (LOGM - 1));
        return __ldg(pos < head ? st + pos : in + (pos - head));
    }
};
template <int LOGM>
struct QuadMixed16 {                   /* cf32 state / raw int16 input by index */
    const float2 *st;
    const short2 *in;
    long long g, head;
    float cre, cim, ks;
    __device__ __forceinline__ float2 at(int v) const {
        const long long pos = g + (long long)v * (1 << (LOGM - 1));
        return pos < head ? __ldg(st + pos) : conv16(__ldg(in + (pos - head)), cre, cim, ks);
    }
};

/* acc[t][i]: hop ta + t, branch q_i. tq: this thread's 2K taps at stride MP
 * (tap v of class c, branch j). nq: valid hops of the quad (1..4). */
template <int LOGOS, class LD>
__device__ __forceinline__ void fold_quad(float2 (&acc)[4][2], const float *__restrict__ tq, int MP, int K,
                                          int nq, const LD &ld) {
    constexpr int D = 2 >> LOGOS;      /* v-shift per hop */
    constexpr int W = 4 * D;           /* tap window (a power of two) */
    const int V = 2 * K;               /* taps per class */
    const int vend = V + (nq - 1) * D; /* one past the last sample position */
#pragma unroll
    for (int t = 0; t < 4; ++t) acc[t][0] = acc[t][1] = make_float2(-0.0f, -0.0f);
    float T[W];
#pragma unroll
    for (int w = 0; w < W; ++w) T[w] = 0.0f;
    for (int v0 = 0; v0 < vend; v0 += W) {
        if (v0 >= W - D && v0 + W <= V && nq == 4) {
            /* every hop in its window: no conditions */
#pragma unroll
            for (int s = 0; s < W; ++s) {
                const int v = v0 + s;
                T[s] = __ldg(tq + (long long)v * MP);
                const float2 x = ld.at(v);
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    const int sv = (s - t * D) & (W - 1);       /* slot of tap v - t*D */
                    const int par = LOGOS ? ((s - t) & 1) : (s & 1);
                    mac(acc[t][par], T[sv], x);
                }
            }
        } else {
#pragma unroll
            for (int s = 0; s < W; ++s) {
                const int v = v0 + s;
                if (v < V) T[s] = __ldg(tq + (long long)v * MP);
                if (v < vend) {
                    const float2 x = ld.at(v);
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        const int vt = v - t * D;
                        const int sv = (s - t * D) & (W - 1);
                        const int par = LOGOS ? ((s - t) & 1) : (s & 1);
                        if (t < nq && vt >= 0 && vt < V) mac(acc[t][par], T[sv], x);
                    }
                }
            }
        }
    }
}

/* the radix-2 first pass (Ns = 1) of one hop: points q0 and q0 + M/2 in,
 * 2*q0 + {0, 1} out */
template <int LOGM>
__device__ __forceinline__ void first_pass2(float2 a, float2 b, double2 *sm, int t, int q0) {
    double2 x0 = make_double2((double)a.x, (double)a.y), x1 = make_double2((double)b.x, (double)b.y);
    dft2(x0, x1);
    if (IDX_OK((t << LOGM) + 2 * q0 + 1 < TILE_POINTS)) {
        sm[SW((t << LOGM) + 2 * q0)] = x0;
        sm[SW((t << LOGM) + 2 * q0 + 1)] = x1;
    }
}

template <int LOGM, int LOGOS>
__device__ __forceinline__ void fold_tile_quad(const atkb_job &J, const atkb_bank &B, long long h0,
                                               int nvalid, double2 *sm) {
    constexpr int M = 1 << LOGM;
    constexpr int LOGMP = LOGM - LOGP;
    constexpr int MP = 1 << LOGMP;
    constexpr int HOP = M >> LOGOS;
    static_assert(PTS == 8 && LOGM <= 10 && LOGOS <= 1, "quad fold: PTS 8, four hops a tile");
    const int tid = threadIdx.x;
    const int j = tid & (MP - 1);
    const int c = (tid >> LOGMP) & 3;
    const int ta = (tid >> (LOGMP + 2)) * 4;
    const int nq = min(4, nvalid - ta);
    float2 acc[4][2];
    if (nq > 0) {
        const float *tq = B.tapsQ + (long long)c * (2 * B.K) * MP + j;
        const long long w0 = h0 * (long long)HOP;
        const long long w1 = (h0 + nvalid - 1) * (long long)HOP + B.L;
        const long long off = (h0 + ta) * (long long)HOP + c * MP + j;
        if (w0 >= J.head) {
            if (J.in_kind) {
                const QuadLin16<LOGM> ld{(const short2 *)J.in + (off - J.head), J.cre, J.cim, J.kscale};
                fold_quad<LOGOS>(acc, tq, MP, B.K, nq, ld);
            } else {
                const QuadLin<LOGM> ld{(const float2 *)J.in + (off - J.head)};
                fold_quad<LOGOS>(acc, tq, MP, B.K, nq, ld);
            }
        } else if (w1 <= J.head) {
            const QuadLin<LOGM> ld{(const float2 *)J.state + off};
            fold_quad<LOGOS>(acc, tq, MP, B.K, nq, ld);
        } else if (J.in_kind) {
            const QuadMixed16<LOGM> ld{(const float2 *)J.state, (const short2 *)J.in, off, J.head,
                                       J.cre, J.cim, J.kscale};
            fold_quad<LOGOS>(acc, tq, MP, B.K, nq, ld);
        } else {
            const QuadMixed<LOGM> ld{(const float2 *)J.state, (const float2 *)J.in, off, J.head};
            fold_quad<LOGOS>(acc, tq, MP, B.K, nq, ld);
        }
    } else {
#pragma unroll
        for (int t = 0; t < 4; ++t) acc[t][0] = acc[t][1] = make_float2(0.0f, 0.0f);
    }
#pragma unroll
    for (int t = 0; t < 4; ++t) first_pass2<LOGM>(acc[t][0], acc[t][1], sm, ta + t, j + c * MP);
}

template <int LOGM, int LOGOS>
__device__ void tile_quad(const atkb_job &J, const atkb_bank &B, long long h0, int nvalid, double2 *sm,
                          float2 *tile_out) {
    constexpr int M = 1 << LOGM;
    fold_tile_quad<LOGM, LOGOS>(J, B, h0, nvalid, sm);
    /* a quad's M/2 threads hold its four hops' points through the passes
     * before the last (bfly gives each hop M/8 consecutive threads) */
    constexpr int G0 = M / 2;
    constexpr int G = G0 < 32 ? 32 : G0 > NT ? NT : G0;
    group_sync<G>();
    fft_rest<LOGM, 1, 1, G>(sm, (const double2 *)B.wpass, B.plan.twoff, tile_out, B, J, h0);
    write_tile<LOGM>(J, h0, nvalid, tile_out);
    if (J.w2) w2_partial<LOGM>(J, h0, nvalid, tile_out);
}

/* fold + first Stockham pass (Ns = 1, radix PTS, no twiddles) of one hop
 * and PTS branches per thread, into the tile's shared points */
template <int LOGM>
__device__ __forceinline__ void fold_first_unpaired(const atkb_job &J, const atkb_bank &B, long long h0,
                                                    int nvalid, double2 *sm) {
    constexpr int MP = (1 << LOGM) >> LOGP;
    const int tid = threadIdx.x;
    const int tt = tid >> (LOGM - LOGP);
    const int j = tid & (MP - 1);
    double2 v[PTS];
    if (!fold_tile_staged<LOGM>(v, J, B, h0, nvalid, tt, j, sm)) {
        if (tt < nvalid) {
            const long long w0 = h0 * (long long)B.hop;                       /* first window start */
            const long long w1 = (h0 + nvalid - 1) * (long long)B.hop + B.L;  /* last window end */
            const long long off = (h0 + tt) * (long long)B.hop + j;
            if (w0 >= J.head) {
                if (J.in_kind)
                    foldP<LOGM, 1>(v, J, B, h0, tt, j, (const short2 *)J.in + (off - J.head));
                else
                    foldP<LOGM, 0>(v, J, B, h0, tt, j, (const float2 *)J.in + (off - J.head));
            } else if (w1 <= J.head) {
                foldP<LOGM, 0>(v, J, B, h0, tt, j, (const float2 *)J.state + off);
            } else {
                foldP<LOGM, 2>(v, J, B, h0, tt, j, nullptr);
            }
        } else {
#pragma unroll
            for (int r = 0; r < PTS; ++r) v[r] = make_double2(0.0, 0.0);
        }
    }
    dftR<PTS>(v);
#pragma unroll
    for (int r = 0; r < PTS; ++r) sm[SW((tt << LOGM) + j * PTS + r)] = v[r];
}

/* nchan 4096: a tile is two hops, computed in turn. Hop a's outputs wait in
 * a side buffer (4096 float2 after the FFT tile, 96 KB in all) while hop b
 * is computed, so the write covers two hops per channel: lanes 2l and 2l+1
 * write the two adjacent outputs of one channel, half the sectors of
 * single-hop writes (a single hop's 4096 outputs land in 4096 rows). */
__device__ void tile_4096x2(const atkb_job &J, const atkb_bank &B, long long h0, int nvalid, double2 *sm) {
    constexpr int LOGM = 12;
    constexpr int M = 1 << LOGM;
    constexpr int MP = M >> LOGP;
    static_assert(NT == MP, "one thread per branch group");
    float2 *tile_out = (float2 *)sm;       /* pass_last: hop at tile_out[kb * 2] */
    float2 *side = (float2 *)(sm + M);
    const double2 *wp = (const double2 *)B.wpass;
    const int tid = threadIdx.x;
#pragma unroll 1
    for (int sub = 0; sub < 2 && sub < nvalid; ++sub) {
        fold_first_unpaired<LOGM>(J, B, h0 + sub, 1, sm);
        __syncthreads();
        fft_rest<LOGM, LOGP, 1, NT>(sm, wp, B.plan.twoff, tile_out, B, J, h0 + sub);
        if (sub == 0) {
#pragma unroll
            for (int u = 0; u < PTS; ++u) side[tid + u * MP] = tile_out[(tid + u * MP) * 2];
            __syncthreads();                 /* read before hop b's first pass */
        }
    }
    const int t2 = tid & 1;
    if (t2 < nvalid) {
        const int kb0 = tid >> 1;
        float2 *o = (float2 *)J.out + (J.out_col + h0 + t2) + (long long)kb0 * J.ldo;
        const long long step = (long long)(NT / 2) * J.ldo;
#pragma unroll 4
        for (int u = 0; u < 2 * PTS; ++u) {
            const int kb = kb0 + u * (NT / 2);
            *o = t2 ? tile_out[kb * 2] : side[kb];
            o += step;
        }
    }
}

/* nchan 4096 at oversample 1/2/4: the same two-hop tile with the paired
 * fold. Thread j folds both hops over the even branches, then over the odd
 * ones (each sample and tap loaded once for the two hops); the even sums
 * wait in the side buffer, so each hop's 8 branches meet in registers for a
 * radix-8 first pass (the 4-pass plan). Hop b's sums wait in the side
 * buffer while hop a is transformed; then hop a's outputs take their place. */
template <int LOGOS>
__device__ void tile_4096x2_pair(const atkb_job &J, const atkb_bank &B, long long h0, int nvalid,
                                 double2 *sm) {
    constexpr int LOGM = 12;
    constexpr int M = 1 << LOGM;
    constexpr int MP = M >> LOGP;
    static_assert(NT == MP && PTS == 8, "one thread per branch group");
    float2 *tile_out = (float2 *)sm;       /* pass_last: hop at tile_out[kb * 2] */
    float2 *side = (float2 *)(sm + M);     /* [8][MP] float2, slot (row, j) owned by thread j */
    const double2 *wp = (const double2 *)B.wpass;
    const int j = threadIdx.x;
    const bool tb_ok = nvalid > 1;
    float2 a[4], b[4];
    fold_pair_global<LOGM, LOGOS>(a, b, J, B, h0, nvalid, 0, 0, j, tb_ok);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        side[i * MP + j] = a[i];           /* rows 0-3: hop a, even branches */
        side[(4 + i) * MP + j] = b[i];     /* rows 4-7: hop b, even branches */
    }
    fold_pair_global<LOGM, LOGOS>(a, b, J, B, h0, nvalid, 0, 1, j, tb_ok);
    {
        double2 v[PTS];                    /* branch r = c + 2i of hop a */
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 e = side[i * MP + j];
            v[2 * i] = make_double2((double)e.x, (double)e.y);
            v[2 * i + 1] = make_double2((double)a[i].x, (double)a[i].y);
            side[i * MP + j] = b[i];       /* rows 0-3 now: hop b, odd branches */
        }
        dftR<PTS>(v);
#pragma unroll
        for (int r = 0; r < PTS; ++r) sm[SW(j * PTS + r)] = v[r];
    }
    __syncthreads();
    fft_rest<LOGM, LOGP, 1, NT>(sm, wp, B.plan.twoff, tile_out, B, J, h0);
    if (tb_ok) {
        double2 v[PTS];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 e = side[(4 + i) * MP + j], o = side[i * MP + j];
            v[2 * i] = make_double2((double)e.x, (double)e.y);
            v[2 * i + 1] = make_double2((double)o.x, (double)o.y);
        }
#pragma unroll
        for (int u = 0; u < PTS; ++u) side[u * MP + j] = tile_out[(j + u * MP) * 2];   /* hop a's outputs */
        __syncthreads();                   /* tile_out read before hop b's first pass */
        dftR<PTS>(v);
#pragma unroll
        for (int r = 0; r < PTS; ++r) sm[SW(j * PTS + r)] = v[r];
        __syncthreads();
        fft_rest<LOGM, LOGP, 1, NT>(sm, wp, B.plan.twoff, tile_out, B, J, h0 + 1);
    } else {
#pragma unroll
        for (int u = 0; u < PTS; ++u) side[u * MP + j] = tile_out[(j + u * MP) * 2];
        __syncthreads();
    }
    const int tid = threadIdx.x;
    const int t2 = tid & 1;
    if (t2 < nvalid) {
        const int kb0 = tid >> 1;
        float2 *o = (float2 *)J.out + (J.out_col + h0 + t2) + (long long)kb0 * J.ldo;
        const long long step = (long long)(NT / 2) * J.ldo;
#pragma unroll 4
        for (int u = 0; u < 2 * PTS; ++u) {
            const int kb = kb0 + u * (NT / 2);
            *o = t2 ? tile_out[kb * 2] : side[kb];
            o += step;
        }
    }
}

/* LOGOS < 0: one hop and PTS branches per thread, first pass radix PTS;
 * LOGOS = log2(os) in 0..2: the paired fold, first pass radix 4 */
template <int LOGM, int LOGOS>
__device__ void tile_fast(const atkb_job &J, const atkb_bank &B, long long h0, int nvalid,
                          double2 *sm, float2 *tile_out) {
    constexpr int M = 1 << LOGM;
    constexpr int LOGNH = 12 - LOGM;
    constexpr int NH = 1 << LOGNH;
    constexpr int MP = M >> LOGP;
    static_assert(LOGM > LOGP, "the fast path needs nchan > PTS");
    const int tid = threadIdx.x;

    if constexpr (LOGOS >= 0) {
        static_assert(PTS == 8 && LOGM <= 11 && LOGOS <= 2, "paired fold: PTS 8, two hops a tile");
        fold_tile_pair<LOGM, LOGOS>(J, B, h0, nvalid, sm);
    } else {
        fold_first_unpaired<LOGM>(J, B, h0, nvalid, sm);
    }
    /* from here to the last pass each hop group (the threads of a hop pair,
     * or of one hop) touches only its own points: group barriers suffice.
     * The region was last used by the previous tile's write, fenced by the
     * CTA-wide barrier that ends every tile. */
    constexpr int G0 = (LOGOS >= 0 ? M / 4 : M / PTS);
    constexpr int G = G0 < 32 ? 32 : G0 > NT ? NT : G0;
    group_sync<G>();

    fft_rest<LOGM, (LOGOS >= 0 ? 2 : LOGP), 1, G>(sm, (const double2 *)B.wpass, B.plan.twoff, tile_out, B,
                                                   J, h0);

    write_tile<LOGM>(J, h0, nvalid, tile_out);
    if (J.w2) w2_partial<LOGM>(J, h0, nvalid, tile_out);
}

/* The CTA's next tile (warp 0, all lanes): claim it from the counter, find
 * its job (the last whose first tile <= tile) by a 32-ary search over the
 * tile prefix table, and copy the job and its bank into shared slot `slot`
 * with asynchronous copies that land while the CTA works on the current
 * tile (the caller waits for them before the next barrier). */
__device__ __forceinline__ void cp_async4(void *smem, const void *gmem) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(sa), "l"(gmem) : "memory");
}

__device__ __forceinline__ void fetch_tile(const atkb_job *__restrict__ jobs, const int *__restrict__ tile_start,
                                           int njobs, int total, int *counters, int *s_tile, int *s_local,
                                           atkb_job *s_job, atkb_bank *s_bank, int slot) {
    static_assert(sizeof(atkb_job) % 4 == 0 && sizeof(atkb_bank) % 4 == 0, "word copies");
    const int lane = threadIdx.x & 31;
    int tile = 0;
    if (lane == 0) tile = atomicAdd(&counters[0], 1);
    tile = __shfl_sync(0xffffffffu, tile, 0);
    if (lane == 0) s_tile[slot] = tile;
    if (tile >= total) return;
    int lo = 0, hi = njobs - 1;                  /* tile_start[lo] <= tile throughout */
    while (lo < hi) {
        const int step = (hi - lo + 32) >> 5;    /* ceil(span / 32) */
        const int idx = lo + lane * step;
        const bool ok = idx <= hi && tile_start[idx] <= tile;
        const unsigned m = __ballot_sync(0xffffffffu, ok);
        lo += (31 - __clz(m)) * step;            /* lane 0 is always set */
        hi = min(hi, lo + step - 1);
    }
    const int *js = (const int *)(jobs + lo);
    int *jd = (int *)(s_job + slot);
    for (int w = lane; w < (int)(sizeof(atkb_job) / 4); w += 32) cp_async4(jd + w, js + w);
    const int *bs = (const int *)jobs[lo].bank;
    int *bd = (int *)(s_bank + slot);
    for (int w = lane; w < (int)(sizeof(atkb_bank) / 4); w += 32) cp_async4(bd + w, bs + w);
    if (lane == 0) s_local[slot] = tile - tile_start[lo];
}

/* RUN::run(key, ...) does one tile, or nothing for key -1, a tile to skip;
 * RUN::carry copies (part of) a state carry */
template <class RUN>
__device__ __forceinline__ void tiles_loop(const atkb_job *__restrict__ jobs, const int *__restrict__ tile_start,
                                           const atkb_carry *__restrict__ carries, int njobs,
                                           const int *__restrict__ d_njobs, int *counters) {
    extern __shared__ double2 sm[];
    /* launched as a programmatic dependent of the kernel that fills the job
     * table (atkb_pfb_launch_pdl): wait for it before the first read; a no-op
     * for an ordinary launch */
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (d_njobs) njobs = min(njobs, *d_njobs);      /* a server round: count set per launch */
    unsigned dyn_smem;
    asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn_smem));
    const int total_tiles = njobs > 0 ? tile_start[njobs] : 0;
    /* two slots: warp 0 fetches tile i+1 into one while the CTA works on
     * tile i from the other */
    __shared__ int s_tile[2], s_local[2];
    __shared__ atkb_bank s_bank[2];
    __shared__ atkb_job s_job[2];
    if (threadIdx.x < 32) fetch_tile(jobs, tile_start, njobs, total_tiles, counters, s_tile, s_local, s_job, s_bank, 0);
    for (int slot = 0;; slot ^= 1) {
        if (threadIdx.x < 32) cp_async_wait_all();  /* this slot's copies, issued by warp 0 */
        __syncthreads();
        const int tile = s_tile[slot];
        if (tile >= total_tiles) break;
        if (threadIdx.x < 32)
            fetch_tile(jobs, tile_start, njobs, total_tiles, counters, s_tile, s_local, s_job, s_bank, slot ^ 1);
        const atkb_job &J = s_job[slot];
        const atkb_bank &SB = s_bank[slot];
        const long long h0 = (long long)s_local[slot] * SB.tile_hops;
        const long long left = J.hops - h0;
        const int nvalid = (int)(left < SB.tile_hops ? left : SB.tile_hops);
        int key = atkb_tile_key(&SB);
        /* a launch with less dynamic shared memory than the bank's tile needs
         * skips the tile (its outputs stay unwritten) instead of running off
         * the end of shared memory */
        if ((unsigned)SB.smem_bytes > dyn_smem) key = -1;
        /* bounds, uniform across the CTA: the tile's last window must end
         * within the job's samples and its columns within the output rows */
        {
            unsigned bad = 0;
            if ((h0 + nvalid - 1) * (long long)SB.hop + SB.L > J.nsrc || h0 + nvalid > J.hops) bad |= ATKB_FAULT_WINDOW;
            if (J.out_col + h0 + nvalid > J.ldo) bad |= ATKB_FAULT_OUTPUT;
            if (bad) {
                if (threadIdx.x == 0) atomicOr((unsigned *)&counters[ATKB_FAULT_WORD], bad);
                key = -1;
            }
        }
        float2 *to = (float2 *)sm;
        RUN::run(key, J, SB, h0, nvalid, sm, to);
        /* the barrier at the top of the loop fences this tile's reads of sm
         * and of its slot from the next tile's writes */
    }
    /* this CTA's tiles are done: a programmatic dependent (the W2 finish of
     * atkdsp_gpu_pfb_process_w12) may be scheduled once every CTA is here; it
     * waits for this grid's completion before it reads anything */
    asm volatile("griddepcontrol.launch_dependents;");
    /* then the state carries, an eighth of a job's per claim where the jobs are
     * few (else a whole one), the CTA's threads copying its part of
     * s[from, from + len) into the other state buffer (no tile reads it). One
     * CTA for a whole carry set the time of short launches with long prototypes:
     * nchan 2048, 1x, 40 taps, 262,147 samples 42.7 us, so 27.7. */
    const int sh = njobs <= ATKB_FEW_JOBS ? ATKB_CARRY_SPLIT : 0;
    __shared__ int s_carry;
    for (;;) {
        if (threadIdx.x == 0) s_carry = atomicAdd(&counters[2], 1);
        __syncthreads();
        const int ci = s_carry;
        __syncthreads();                  /* read before thread 0 claims again */
        if (ci >> sh >= njobs) break;
        const atkb_carry &C = carries[ci >> sh];
        const Src src{(const float2 *)C.state, C.in, C.head, C.in_kind, C.cre, C.cim, C.kscale};
        float2 *dst = (float2 *)C.dst;
        const long long from = C.from, len = C.len;
        if (from < 0 || len < 0 || from + len > C.nsrc || len > C.cap) {   /* uniform: skip it */
            if (threadIdx.x == 0) atomicOr((unsigned *)&counters[ATKB_FAULT_WORD], ATKB_FAULT_CARRY);
            continue;
        }
        const long long part = (len + (1 << sh) - 1) >> sh, at = part * (ci & ((1 << sh) - 1));
        if (at < len) RUN::carry(src, dst + at, from + at, min(part, len - at));
    }
    if (threadIdx.x == 0) {
        __threadfence();
        const int done = atomicAdd(&counters[1], 1);
        if (done == (int)gridDim.x - 1) {      /* the last CTA out resets */
            atomicExch(&counters[0], 0);
            atomicExch(&counters[2], 0);
            atomicExch(&counters[1], 0);
        }
    }
}

/* the tile of one key */
template <int KEY>
__device__ __forceinline__ void run_tile(const atkb_job &J, const atkb_bank &SB, long long h0, int nvalid, double2 *sm,
                                         float2 *to) {
    constexpr int L = KEY & 15, SHAPE = KEY >> 4;
    if constexpr (L == 12) {
        if constexpr (SHAPE == 0) tile_4096x2(J, SB, h0, nvalid, sm);
        else tile_4096x2_pair<SHAPE - 1>(J, SB, h0, nvalid, sm);
    } else if constexpr (SHAPE >= 5) {
        tile_quad<L, SHAPE - 5>(J, SB, h0, nvalid, sm, to);
    } else {
        tile_fast<L, SHAPE - 1>(J, SB, h0, nvalid, sm, to);
    }
}

}  // namespace

#endif
