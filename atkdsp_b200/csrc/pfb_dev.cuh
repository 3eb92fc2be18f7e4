/* Device helpers of the filterbank's kernels (pfb.cu, hops.cu): complex
 * doubles, small DFTs, sample sources and the epilogue of one bin. Both
 * translation units use these very operations, so their outputs agree bit for
 * bit. Include inside a namespace. */
#ifndef ATKB_PFB_DEV_CUH
#define ATKB_PFB_DEV_CUH

/* Per-thread index checks of the debug build (ATKB_DEBUG_BOUNDS): an index
 * outside its buffer sets a bit of g_atkb_debug_fault and the access is
 * skipped; atkb_pfb_debug_fault reads and clears the word. In the normal
 * build IDX_OK is constant true and costs nothing. */
#ifdef ATKB_DEBUG_BOUNDS
__device__ unsigned g_atkb_debug_fault;
__device__ __forceinline__ bool idx_ok(bool ok) {
    if (!ok) atomicOr(&g_atkb_debug_fault, ATKB_FAULT_INDEX);
    return ok;
}
#define IDX_OK(c) idx_ok(c)
[[maybe_unused]] inline unsigned take_debug_fault() {
    unsigned v = 0, z = 0;
    if (cudaMemcpyFromSymbol(&v, g_atkb_debug_fault, sizeof v) != cudaSuccess) return ATKB_FAULT_INDEX;
    if (v) cudaMemcpyToSymbol(g_atkb_debug_fault, &z, sizeof z);
    return v;
}
#else
#define IDX_OK(c) true
#endif

__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
/* multiply by -i */
__device__ __forceinline__ double2 cmi(double2 a) { return make_double2(a.y, -a.x); }

/* the reference's rotation / cal product: one rounding per multiply and add */
__device__ __forceinline__ double2 cmul_rn(double2 a, double2 b) {
    return make_double2(__dsub_rn(__dmul_rn(a.x, b.x), __dmul_rn(a.y, b.y)),
                        __dadd_rn(__dmul_rn(a.x, b.y), __dmul_rn(a.y, b.x)));
}

#define C16_1 0.92387953251128675613   /* cos(pi/8) */
#define S16_1 0.38268343236508977173   /* sin(pi/8) */
#define SQH   0.70710678118654752440   /* sqrt(1/2) */

/* forward DFTs, e^{-2 pi i nk/R} */
__device__ __forceinline__ void dft2(double2 &a, double2 &b) {
    const double2 t = a;
    a = cadd(t, b);
    b = csub(t, b);
}

__device__ __forceinline__ void dft4(double2 &v0, double2 &v1, double2 &v2, double2 &v3) {
    const double2 t0 = cadd(v0, v2), t1 = csub(v0, v2);
    const double2 t2 = cadd(v1, v3), t3 = cmi(csub(v1, v3));
    v0 = cadd(t0, t2);
    v2 = csub(t0, t2);
    v1 = cadd(t1, t3);
    v3 = csub(t1, t3);
}

__device__ __forceinline__ void dft8(double2 *v) {
    /* n = 2 n1 + n2, k = k1 + 4 k2 */
    double2 a0 = v[0], a1 = v[2], a2 = v[4], a3 = v[6];
    double2 b0 = v[1], b1 = v[3], b2 = v[5], b3 = v[7];
    dft4(a0, a1, a2, a3);
    dft4(b0, b1, b2, b3);
    b1 = make_double2(SQH * (b1.x + b1.y), SQH * (b1.y - b1.x));      /* W8^1 */
    b2 = cmi(b2);                                                     /* W8^2 */
    b3 = make_double2(SQH * (b3.y - b3.x), -SQH * (b3.x + b3.y));     /* W8^3 */
    v[0] = cadd(a0, b0); v[4] = csub(a0, b0);
    v[1] = cadd(a1, b1); v[5] = csub(a1, b1);
    v[2] = cadd(a2, b2); v[6] = csub(a2, b2);
    v[3] = cadd(a3, b3); v[7] = csub(a3, b3);
}

__device__ __forceinline__ void dft16(double2 *v) {
    /* n = 4 n1 + n2, k = k1 + 4 k2: radix-4 columns, W16^(n2 k1), radix-4
     * rows, all in place; the rows leave y[k1 + 4 k2] at v[4 k1 + k2], and a
     * final renaming (free once unrolled) restores natural order */
#pragma unroll
    for (int n2 = 0; n2 < 4; ++n2) dft4(v[n2], v[4 + n2], v[8 + n2], v[12 + n2]);
    v[4 * 1 + 1] = cmul(v[4 * 1 + 1], make_double2(C16_1, -S16_1));
    v[4 * 2 + 1] = cmul(v[4 * 2 + 1], make_double2(SQH, -SQH));
    v[4 * 3 + 1] = cmul(v[4 * 3 + 1], make_double2(S16_1, -C16_1));
    v[4 * 1 + 2] = cmul(v[4 * 1 + 2], make_double2(SQH, -SQH));
    v[4 * 2 + 2] = cmi(v[4 * 2 + 2]);
    v[4 * 3 + 2] = cmul(v[4 * 3 + 2], make_double2(-SQH, -SQH));
    v[4 * 1 + 3] = cmul(v[4 * 1 + 3], make_double2(S16_1, -C16_1));
    v[4 * 2 + 3] = cmul(v[4 * 2 + 3], make_double2(-SQH, -SQH));
    v[4 * 3 + 3] = cmul(v[4 * 3 + 3], make_double2(-C16_1, S16_1));
#pragma unroll
    for (int k1 = 0; k1 < 4; ++k1) dft4(v[4 * k1], v[4 * k1 + 1], v[4 * k1 + 2], v[4 * k1 + 3]);
    /* transpose the 4x4 index grid */
    double2 t;
    t = v[1]; v[1] = v[4]; v[4] = t;
    t = v[2]; v[2] = v[8]; v[8] = t;
    t = v[3]; v[3] = v[12]; v[12] = t;
    t = v[6]; v[6] = v[9]; v[9] = t;
    t = v[7]; v[7] = v[13]; v[13] = t;
    t = v[11]; v[11] = v[14]; v[14] = t;
}

__device__ __forceinline__ void dft3(double2 &a, double2 &b, double2 &c) {
    const double S3 = 0.86602540378443864676;   /* sin(2 pi / 3) */
    const double2 s = cadd(b, c), d = csub(b, c);
    const double2 m = make_double2(a.x - 0.5 * s.x, a.y - 0.5 * s.y);
    const double2 r = make_double2(S3 * d.y, -S3 * d.x);  /* -i sin(2pi/3) (b - c) */
    a = cadd(a, s);
    b = cadd(m, r);
    c = csub(m, r);
}

template <int R>
__device__ __forceinline__ void dftR(double2 *v) {
    if (R == 2) dft2(v[0], v[1]);
    else if (R == 4) dft4(v[0], v[1], v[2], v[3]);
    else if (R == 8) dft8(v);
    else if (R == 16) dft16(v);
}

/* int16 I/Q -> cf32 exactly as the unpack front end does, (float(v) - c) * k
 * with rounded operations (reference src/convert.c:64-73), in the fused form
 * the host prepares: nc = -(c * k) with k a power of two, one rounding */
__device__ __forceinline__ float2 conv16(short2 v, float ncre, float ncim, float k) {
    return make_float2(__fmaf_rn((float)v.x, k, ncre), __fmaf_rn((float)v.y, k, ncim));
}

/* one element of the stream s = state[0, head) ++ in[0, ...); `in` is cf32 or
 * raw int16 I/Q converted on the fly */
struct Src {
    const float2 *st;
    const void *in;
    long long head;
    int kind;
    float cre, cim, k;
    __device__ __forceinline__ float2 at(long long i) const {
        if (i < head) return __ldg(st + i);
        if (kind) return conv16(__ldg((const short2 *)in + (i - head)), cre, cim, k);
        return __ldg((const float2 *)in + (i - head));
    }
};

/* The int16 constants from an offset held in device memory (a job's or a
 * carry's doff): atkb_job_conv's -((off / k) * k), off the double rounded to
 * float, by the same IEEE float operations as the host. */
__device__ __forceinline__ void doff_consts(const double *doff, float k, float &cre, float &cim) {
    cre = -__fmul_rn(__fdiv_rn(__double2float_rn(__ldg(doff)), k), k);
    cim = -__fmul_rn(__fdiv_rn(__double2float_rn(__ldg(doff + 1)), k), k);
}

/* the twiddles of one butterfly, w[r] = W^(r k) for r = 1 .. R-1, from the
 * one table entry w1 = W^k: squares and products (each power carries at most
 * two double roundings more than a table entry, ~1e-16 relative) instead of
 * R-1 table loads, so a pass reads Ns table entries, not (R-1)*Ns */
__device__ __forceinline__ double2 csq(double2 a) {
    return make_double2(a.x * a.x - a.y * a.y, 2.0 * a.x * a.y);
}
template <int R>
__device__ __forceinline__ void tw_powers(double2 w1, double2 *w) {
    w[1] = w1;
    if constexpr (R > 2) {
        w[2] = csq(w1);
        w[3] = cmul(w[2], w1);
    }
    if constexpr (R > 4) {
        w[4] = csq(w[2]);
        w[5] = cmul(w[4], w1);
        w[6] = csq(w[3]);
        w[7] = cmul(w[4], w[3]);
    }
}

/* Rotation to input sample 0 and cal for bin kb of a hop whose (b + 1) mod os
 * is s, then one rounding to float (reference src/channelizer.c:270-292). */
__device__ __forceinline__ float2 finish_bin(double2 X, int kb, int s, int M, int os, int hop,
                                             bool os_pow2, const double2 *twd, const float2 *cal) {
    const int jr = os_pow2 ? ((kb * s) & (os - 1)) : ((kb * s) % os);
    X = cmul_rn(X, __ldg(twd + (jr ? M - jr * hop : 0)));
    if (cal) {
        const float2 c = __ldg(cal + kb);
        X = cmul_rn(X, make_double2((double)c.x, (double)c.y));
    }
    return make_float2(__double2float_rn(X.x), __double2float_rn(X.y));
}

/* dst[0, len) = s[from, from + len), eight loads in flight per thread before
 * their stores (a load-store loop would wait one memory round trip per
 * step: the compiler cannot tell dst from the sources) */
template <int T>
__device__ __forceinline__ void carry_copy(const Src &src, float2 *dst, long long from, long long len) {
    for (long long i0 = threadIdx.x; i0 < len; i0 += 8LL * T) {
        float2 v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const long long i = i0 + (long long)u * T;
            if (i < len) v[u] = src.at(from + i);
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const long long i = i0 + (long long)u * T;
            if (i < len) dst[i] = v[u];
        }
    }
}

/* the same, each source a run of its own: with the source chosen per sample its
 * branches can keep a thread's loads apart, a memory round trip each. (The
 * kernels of one shape keep the form above: this one moves the registers of
 * their tile code, 2 to 10 % of some shapes.) */
template <int T, class AT>
__device__ __forceinline__ void copy_run(float2 *dst, long long n, const AT &at) {
    for (long long i0 = threadIdx.x; i0 < n; i0 += 8LL * T) {
        float2 v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const long long i = i0 + (long long)u * T;
            if (i < n) v[u] = at(i);
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const long long i = i0 + (long long)u * T;
            if (i < n) dst[i] = v[u];
        }
    }
}
template <int T>
__device__ __forceinline__ void carry_runs(const Src &src, float2 *dst, long long from, long long len) {
    const long long left = src.head - from, n = left < 0 ? 0 : left < len ? left : len;
    const float2 *st = src.st + from;
    copy_run<T>(dst, n, [=](long long i) { return __ldg(st + i); });
    if (n == len) return;
    dst += n;
    if (src.kind) {
        const short2 *in = (const short2 *)src.in + (from + n - src.head);
        const float cre = src.cre, cim = src.cim, k = src.k;
        copy_run<T>(dst, len - n, [=](long long i) { return conv16(__ldg(in + i), cre, cim, k); });
    } else {
        const float2 *in = (const float2 *)src.in + (from + n - src.head);
        copy_run<T>(dst, len - n, [=](long long i) { return __ldg(in + i); });
    }
}

#endif
