/* Any nchan >= 2 whose hop fits a CTA's shared memory twice: a run of hops
 * through fold, mixed-radix Stockham passes between two buffers, epilogue.
 * Include after pfb_dev.cuh inside a namespace.
 *
 * Radices 2, 3, 4, 5, 7 and 8 are butterflies in registers (the radix a
 * template argument); any other prime factor is a direct DFT. */
#ifndef ATKB_PFB_GENERIC_CUH
#define ATKB_PFB_GENERIC_CUH

__device__ __forceinline__ void dft5(double2 *v) {
    const double C1 = 0.30901699437494742410, C2 = -0.80901699437494742410;   /* cos(2 pi / 5), cos(4 pi / 5) */
    const double S1 = 0.95105651629515357212, S2 = 0.58778525229247312917;    /* sin */
    const double2 a1 = cadd(v[1], v[4]), d1 = csub(v[1], v[4]), a2 = cadd(v[2], v[3]), d2 = csub(v[2], v[3]);
    const double2 m1 = make_double2(v[0].x + C1 * a1.x + C2 * a2.x, v[0].y + C1 * a1.y + C2 * a2.y);
    const double2 m2 = make_double2(v[0].x + C2 * a1.x + C1 * a2.x, v[0].y + C2 * a1.y + C1 * a2.y);
    const double2 n1 = make_double2(S1 * d1.y + S2 * d2.y, -(S1 * d1.x + S2 * d2.x));
    const double2 n2 = make_double2(S2 * d1.y - S1 * d2.y, -(S2 * d1.x - S1 * d2.x));
    v[0] = cadd(v[0], cadd(a1, a2));
    v[1] = cadd(m1, n1);
    v[4] = csub(m1, n1);
    v[2] = cadd(m2, n2);
    v[3] = csub(m2, n2);
}

__device__ __forceinline__ void dft7(double2 *v) {
    const double C[3] = {0.62348980185873353053, -0.22252093395631440429, -0.90096886790241912624};
    const double S[3] = {0.78183148246802980871, 0.97492791218182360702, 0.43388373911755812048};
    double2 a[3], d[3];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        a[r] = cadd(v[r + 1], v[6 - r]);
        d[r] = csub(v[r + 1], v[6 - r]);
    }
    const double2 z = v[0];
    v[0] = cadd(z, cadd(a[0], cadd(a[1], a[2])));
#pragma unroll
    for (int k = 1; k <= 3; ++k) {
        double2 m = z, n = make_double2(0.0, 0.0);
#pragma unroll
        for (int r = 1; r <= 3; ++r) {
            const int e = (r * k) % 7, i = (e <= 3 ? e : 7 - e) - 1;
            const double c = C[i], s = e <= 3 ? S[i] : -S[i];
            m.x += c * a[r - 1].x;
            m.y += c * a[r - 1].y;
            n.x += s * d[r - 1].y;
            n.y -= s * d[r - 1].x;
        }
        v[k] = cadd(m, n);
        v[7 - k] = csub(m, n);
    }
}

template <int R>
__device__ __forceinline__ void dft_any(double2 *v) {
    if constexpr (R == 3) dft3(v[0], v[1], v[2]);
    else if constexpr (R == 5) dft5(v);
    else if constexpr (R == 7) dft7(v);
    else dftR<R>(v);
}

/* one radix-R pass of nh hops; W: the nchan-point table W^j */
template <int NTH, int R>
__device__ __forceinline__ void generic_pass(const double2 *__restrict__ src, double2 *__restrict__ dst, int M, int Ns,
                                             int nh, const double2 *__restrict__ W) {
    const unsigned MR = (unsigned)M / R, stride = (unsigned)M / (unsigned)(Ns * R);
    for (unsigned bi = threadIdx.x; bi < nh * MR; bi += NTH) {
        const unsigned tt = bi / MR, j = bi - tt * MR, k = j % (unsigned)Ns;
        const double2 *s = src + tt * M + j;
        double2 *d = dst + tt * M + (j - k) * R + k;
        double2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = s[r * MR];
        if (Ns > 1) {
            const unsigned e = k * stride;
#pragma unroll
            for (int r = 1; r < R; ++r) v[r] = cmul(v[r], __ldg(W + r * e));
        }
        dft_any<R>(v);
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (IDX_OK((j - k) * R + k + r * Ns < (unsigned)M)) d[r * Ns] = v[r];
    }
}

/* a prime factor without a butterfly: the direct DFT with the twiddle folded
 * in, W_{Ns R}^{r (k + o Ns)}, the exponent kept below Ns R by subtraction */
template <int NTH>
__device__ __noinline__ void direct_pass(const double2 *__restrict__ src, double2 *__restrict__ dst, int M, int Ns,
                                         int R, int nh, const double2 *__restrict__ W) {
    const unsigned MR = (unsigned)M / R, NsR = (unsigned)(Ns * R), stride = (unsigned)M / NsR;
    for (unsigned bi = threadIdx.x; bi < (unsigned)nh * M; bi += NTH) {
        const unsigned tt = bi / (unsigned)M, c = bi - tt * M, o = c / MR, j = c - o * MR, k = j % (unsigned)Ns;
        const double2 *s = src + tt * M + j;
        const unsigned inc = k + o * Ns;
        unsigned e = 0;
        double2 acc = make_double2(0.0, 0.0);
        for (int r = 0; r < R; ++r) {
            const double2 w = __ldg(W + e * stride), x = s[r * MR];
            acc.x += x.x * w.x - x.y * w.y;
            acc.y += x.x * w.y + x.y * w.x;
            e += inc;
            if (e >= NsR) e -= NsR;
        }
        if (IDX_OK(e < NsR && (j - k) * R + k + o * Ns < (unsigned)M)) dst[tt * M + (j - k) * R + k + o * Ns] = acc;
    }
}

/* hops h0 .. h0 + nvalid of job J (int16 constants cre, cim) through `sm`
 * (2 * nvalid * nchan points) by NTH threads */
template <int NTH, int U = 8>
__device__ __forceinline__ void generic_tile(const atkb_job &J, const atkb_bank &B, float cre, float cim, long long h0,
                                          int nvalid, double2 *sm) {
    const int M = B.nchan, K = B.K;
    double2 *cur = sm, *nxt = sm + nvalid * M;
    const Src src{(const float2 *)J.state, J.in, J.head, J.in_kind, cre, cim, J.kscale};
    const float *taps = B.taps;
    for (unsigned e = threadIdx.x; e < (unsigned)(nvalid * M); e += NTH) {
        const unsigned tt = e / (unsigned)M, q = e - tt * M;
        const long long base = (h0 + tt) * (long long)B.hop + q;
        float fr = -0.0f, fi = -0.0f;
        for (int k0 = 0; k0 < K; k0 += U) {            /* U taps' loads in flight */
            float h[U];
            float2 x[U];
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (k0 + u < K && IDX_OK(base + (k0 + u) * M < J.nsrc)) {
                    h[u] = __ldg(taps + (k0 + u) * M + q);
                    x[u] = src.at(base + (k0 + u) * M);
                }
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (k0 + u < K) {
                    fr = __fadd_rn(fr, __fmul_rn(h[u], x[u].x));
                    fi = __fadd_rn(fi, __fmul_rn(h[u], x[u].y));
                }
        }
        cur[e] = make_double2((double)fr, (double)fi);
    }
    __syncthreads();
    const double2 *W = (const double2 *)B.wfull;
    int Ns = 1;
    for (int p = 0; p < B.plan.npass; ++p) {
        const int R = B.plan.radix[p];
        switch (R) {
        case 2: generic_pass<NTH, 2>(cur, nxt, M, Ns, nvalid, W); break;
        case 3: generic_pass<NTH, 3>(cur, nxt, M, Ns, nvalid, W); break;
        case 4: generic_pass<NTH, 4>(cur, nxt, M, Ns, nvalid, W); break;
        case 5: generic_pass<NTH, 5>(cur, nxt, M, Ns, nvalid, W); break;
        case 7: generic_pass<NTH, 7>(cur, nxt, M, Ns, nvalid, W); break;
        case 8: generic_pass<NTH, 8>(cur, nxt, M, Ns, nvalid, W); break;
        default: direct_pass<NTH>(cur, nxt, M, Ns, R, nvalid, W); break;
        }
        __syncthreads();
        Ns *= R;
        double2 *t = cur;
        cur = nxt;
        nxt = t;
    }
    const double2 *twd = (const double2 *)B.twd;
    const float2 *cal = (const float2 *)J.cal;
    float2 *out = (float2 *)J.out;
    const unsigned os = (unsigned)B.os, s0 = (unsigned)((J.b0 + h0 + 1) % B.os);
    for (unsigned e = threadIdx.x; e < (unsigned)(nvalid * M); e += NTH) {
        const unsigned kb = e / (unsigned)nvalid, tt = e - kb * nvalid;
        double2 X = cur[tt * M + kb];
        const unsigned s = (s0 + tt) % os, jr = (unsigned)(((unsigned long long)kb * s) % os);
        X = cmul_rn(X, __ldg(twd + (jr ? M - (int)jr * B.hop : 0)));
        if (cal) {
            const float2 c = __ldg(cal + kb);
            X = cmul_rn(X, make_double2((double)c.x, (double)c.y));
        }
        if (IDX_OK(kb < (unsigned)M && J.out_col + h0 + tt < J.ldo))
            out[(long long)kb * J.ldo + J.out_col + h0 + tt] =
                make_float2(__double2float_rn(X.x), __double2float_rn(X.y));
    }
}

#endif
