// fft_smem.cuh — the project's own shared-memory FFT for sm_100a.
//
// Batched complex FFTs of one runtime length L per call, data resident in
// shared memory, mixed-radix Stockham autosort passes (radix 2..16 in registers,
// any other prime factor by a direct small DFT), natural-order output.  A signal
// is stored at padded indices (FftPlan::at).  Twiddles of pass s come from a
// table in [r][k] order (pass_tables), the zero-padding pre/post twiddles
// W_{2L}^n of the pruned 2L-point transforms from a table of
// exp(-2 pi i k / (2L)), k < 2L.
//
// What bounds it and why it is laid out so: a pass moves every value through
// shared memory once each way, so the composite radices (16, 12, 10, 6) save whole
// passes and their barriers (1536 = 16*12*8 is 3 passes instead of 4, 50 = 10*5 is 2
// instead of 3); the [r][k] tables let a warp read consecutive twiddles (the
// strided reads of one exp(-2 pi i k / 2L) table cost up to 28 L1 wavefronts per
// load and more than the data itself); one pad slot per 128 bytes spreads the
// first pass's stride-P writes over all banks; the runtime divisions by m and ns
// are multiplications by a reciprocal formed once per pass.
#pragma once
#include "types.cuh"

namespace llg {

template <typename R>
struct __align__(2 * sizeof(R)) cx {
    R re, im;
};

template <typename R>
__device__ __forceinline__ cx<R> mkc(R a, R b) {
    cx<R> r;
    r.re = a;
    r.im = b;
    return r;
}
template <typename R>
__device__ __forceinline__ cx<R> operator+(cx<R> a, cx<R> b) { return mkc(a.re + b.re, a.im + b.im); }
template <typename R>
__device__ __forceinline__ cx<R> operator-(cx<R> a, cx<R> b) { return mkc(a.re - b.re, a.im - b.im); }
template <typename R>
__device__ __forceinline__ cx<R> cmul(cx<R> a, cx<R> b) {
    return mkc(a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re);
}
// a * conj(b)
template <typename R>
__device__ __forceinline__ cx<R> cmulc(cx<R> a, cx<R> b) {
    return mkc(a.re * b.re + a.im * b.im, a.im * b.re - a.re * b.im);
}
template <typename R>
__device__ __forceinline__ cx<R> cscale(cx<R> a, R s) { return mkc(a.re * s, a.im * s); }
template <typename R>
__device__ __forceinline__ cx<R> conjc(cx<R> a) { return mkc(a.re, -a.im); }
// multiply by -i (forward) or +i (inverse)
template <typename R>
__device__ __forceinline__ cx<R> rot(cx<R> a, bool inv) { return inv ? mkc(-a.im, a.re) : mkc(a.im, -a.re); }

// twiddle W_L^idx = tw2[2*idx] (forward), conj for inverse
template <typename R>
__device__ __forceinline__ cx<R> twl(const cx<R>* tw2, int idx, bool inv) {
    cx<R> w = tw2[2 * idx];
    return inv ? conjc(w) : w;
}

template <typename R>
__device__ __forceinline__ void bfly2(cx<R>* v) {
    cx<R> a = v[0], b = v[1];
    v[0] = a + b;
    v[1] = a - b;
}
template <typename R>
__device__ __forceinline__ void bfly4(cx<R>* v, bool inv) {
    cx<R> s02 = v[0] + v[2], d02 = v[0] - v[2];
    cx<R> s13 = v[1] + v[3], d13 = v[1] - v[3];
    cx<R> r = rot(d13, inv);
    v[0] = s02 + s13;
    v[1] = d02 + r;
    v[2] = s02 - s13;
    v[3] = d02 - r;
}
template <typename R>
__device__ __forceinline__ void bfly8(cx<R>* v, bool inv) {
    const R h = (R)0.70710678118654752440;
    cx<R> e[4] = {v[0], v[2], v[4], v[6]};
    cx<R> o[4] = {v[1], v[3], v[5], v[7]};
    bfly4(e, inv);
    bfly4(o, inv);
    // o[q] *= w8^q
    cx<R> o1, o3;
    if (!inv) {
        o1 = mkc((o[1].re + o[1].im) * h, (o[1].im - o[1].re) * h);
        o3 = mkc((o[3].im - o[3].re) * h, (-o[3].re - o[3].im) * h);
    } else {
        o1 = mkc((o[1].re - o[1].im) * h, (o[1].re + o[1].im) * h);
        o3 = mkc((-o[3].re - o[3].im) * h, (o[3].re - o[3].im) * h);
    }
    cx<R> o2 = rot(o[2], inv);
    v[0] = e[0] + o[0];
    v[4] = e[0] - o[0];
    v[1] = e[1] + o1;
    v[5] = e[1] - o1;
    v[2] = e[2] + o2;
    v[6] = e[2] - o2;
    v[3] = e[3] + o3;
    v[7] = e[3] - o3;
}
template <typename R>
__device__ __forceinline__ void bfly3(cx<R>* v, bool inv) {
    const R s3 = (R)0.86602540378443864676;  // sqrt(3)/2
    cx<R> s = v[1] + v[2], d = v[1] - v[2];
    cx<R> t = mkc(v[0].re - (R)0.5 * s.re, v[0].im - (R)0.5 * s.im);
    cx<R> r = rot(cscale(d, s3), inv);
    v[0] = v[0] + s;
    v[1] = t + r;
    v[2] = t - r;
}
template <typename R>
__device__ __forceinline__ void bfly5(cx<R>* v, bool inv) {
    const R c1 = (R)0.30901699437494742410, c2 = (R)-0.80901699437494742410;
    const R s1 = (R)0.95105651629515357212, s2 = (R)0.58778525229247312917;
    cx<R> a1s = v[1] + v[4], a1d = v[1] - v[4];
    cx<R> a2s = v[2] + v[3], a2d = v[2] - v[3];
    cx<R> x0 = v[0];
    cx<R> p1 = mkc(x0.re + c1 * a1s.re + c2 * a2s.re, x0.im + c1 * a1s.im + c2 * a2s.im);
    cx<R> p2 = mkc(x0.re + c2 * a1s.re + c1 * a2s.re, x0.im + c2 * a1s.im + c1 * a2s.im);
    cx<R> q1 = mkc(s1 * a1d.re + s2 * a2d.re, s1 * a1d.im + s2 * a2d.im);
    cx<R> q2 = mkc(s2 * a1d.re - s1 * a2d.re, s2 * a1d.im - s1 * a2d.im);
    cx<R> r1 = rot(q1, inv), r2 = rot(q2, inv);  // -i*q (fwd)
    v[0] = x0 + a1s + a2s;
    v[1] = p1 + r1;
    v[4] = p1 - r1;
    v[2] = p2 + r2;
    v[3] = p2 - r2;
}

template <typename R>
__device__ __forceinline__ void bfly16(cx<R>* v, bool inv) {
    // 4 x 4: input n = 4 n1 + n2, output k = k1 + 4 k2, internal twiddles W_16^{n2 k1}
    constexpr double c[10] = {1.0, 0.92387953251128675613, 0.70710678118654752440, 0.38268343236508977173, 0.0,
                              0.0, -0.70710678118654752440, 0.0, 0.0, -0.92387953251128675613};
    constexpr double s[10] = {0.0, 0.38268343236508977173, 0.70710678118654752440, 0.92387953251128675613, 1.0,
                              0.0, 0.70710678118654752440, 0.0, 0.0, -0.38268343236508977173};
    cx<R> y[16];
#pragma unroll
    for (int n2 = 0; n2 < 4; ++n2) {
        cx<R> a[4] = {v[n2], v[4 + n2], v[8 + n2], v[12 + n2]};
        bfly4(a, inv);
#pragma unroll
        for (int k1 = 0; k1 < 4; ++k1) {
            const int e = n2 * k1;
            if (e == 0) y[n2 * 4 + k1] = a[k1];
            else if (e == 4) y[n2 * 4 + k1] = rot(a[k1], inv);
            else {
                const R wr = (R)c[e], wi = inv ? (R)s[e] : (R)-s[e];
                y[n2 * 4 + k1] = mkc(a[k1].re * wr - a[k1].im * wi, a[k1].re * wi + a[k1].im * wr);
            }
        }
    }
#pragma unroll
    for (int k1 = 0; k1 < 4; ++k1) {
        cx<R> b[4] = {y[k1], y[4 + k1], y[8 + k1], y[12 + k1]};
        bfly4(b, inv);
#pragma unroll
        for (int k2 = 0; k2 < 4; ++k2) v[k1 + 4 * k2] = b[k2];
    }
}

__host__ __device__ constexpr int inv_mod(int a, int n) {
    for (int x = 1; x < n; ++x)
        if ((a * x) % n == 1) return x;
    return 1;
}

// In-register DFT of P points, natural order; coprime composites by the
// Good-Thomas prime-factor mapping (no internal twiddles).
template <typename R, int P>
__device__ __forceinline__ void bfly(cx<R>* v, bool inv);
template <typename R, int N1, int N2>
__device__ __forceinline__ void bfly_pfa(cx<R>* v, bool inv) {
    constexpr int N = N1 * N2, A = N2 * inv_mod(N2 % N1, N1), B = N1 * inv_mod(N1 % N2, N2);
    cx<R> t[N];
#pragma unroll
    for (int n2 = 0; n2 < N2; ++n2) {
        cx<R> x[N1];
#pragma unroll
        for (int n1 = 0; n1 < N1; ++n1) x[n1] = v[(N2 * n1 + N1 * n2) % N];
        bfly<R, N1>(x, inv);
#pragma unroll
        for (int k1 = 0; k1 < N1; ++k1) t[k1 * N2 + n2] = x[k1];
    }
#pragma unroll
    for (int k1 = 0; k1 < N1; ++k1) {
        cx<R> x[N2];
#pragma unroll
        for (int n2 = 0; n2 < N2; ++n2) x[n2] = t[k1 * N2 + n2];
        bfly<R, N2>(x, inv);
#pragma unroll
        for (int k2 = 0; k2 < N2; ++k2) v[(A * k1 + B * k2) % N] = x[k2];
    }
}
template <typename R, int P>
__device__ __forceinline__ void bfly(cx<R>* v, bool inv) {
    if constexpr (P == 2) bfly2(v);
    if constexpr (P == 3) bfly3(v, inv);
    if constexpr (P == 4) bfly4(v, inv);
    if constexpr (P == 5) bfly5(v, inv);
    if constexpr (P == 6) bfly_pfa<R, 2, 3>(v, inv);
    if constexpr (P == 8) bfly8(v, inv);
    if constexpr (P == 10) bfly_pfa<R, 2, 5>(v, inv);
    if constexpr (P == 12) bfly_pfa<R, 4, 3>(v, inv);
    if constexpr (P == 16) bfly16(v, inv);
}

// Quotient by a divisor fixed over a loop: exact for value * divisor < 2^32 (both
// stay far below 2^16 here).
struct FastDiv {
    uint32_t mul;
    int d;
    __device__ __forceinline__ explicit FastDiv(int div) : mul(0xffffffffu / (uint32_t)div + 1u), d(div) {}
    __device__ __forceinline__ int quot(int v) const { return d == 1 ? v : (int)__umulhi((uint32_t)v, mul); }
};

template <typename R, int P, bool INV>
__device__ __forceinline__ void stockham_pass_fixed(const cx<R>* __restrict__ a, cx<R>* __restrict__ b, int nsig,
                                                    const FftPlan& plan, int ns, const cx<R>* __restrict__ tw) {
    const int m = plan.L / P, LP = plan.stride();
    const int total = nsig * m;
    const FastDiv dm(m), dns(ns);
    for (int t = threadIdx.x; t < total; t += blockDim.x) {
        const int sig = dm.quot(t);
        const int j = t - sig * m;
        const int q = dns.quot(j);
        const int k = j - q * ns;
        const cx<R>* in = a + sig * LP;
        cx<R> v[P];
#pragma unroll
        for (int r = 0; r < P; ++r) v[r] = in[plan.at(j + r * m)];
        if (ns > 1) {
#pragma unroll
            for (int r = 1; r < P; ++r) {
                const cx<R> w = tw[r * ns + k];
                v[r] = INV ? cmulc(v[r], w) : cmul(v[r], w);
            }
        }
        bfly<R, P>(v, INV);
        cx<R>* out = b + sig * LP;
        const int o = q * ns * P + k;
#pragma unroll
        for (int r = 0; r < P; ++r) out[plan.at(o + r * ns)] = v[r];
    }
}

// Any prime radix p: one output per thread iteration, direct p-term sum.
template <typename R, bool INV>
__device__ void stockham_pass_generic(const cx<R>* __restrict__ a, cx<R>* __restrict__ b, int nsig,
                                      const FftPlan& plan, int p, int ns, const cx<R>* __restrict__ tw,
                                      const cx<R>* __restrict__ tw2) {
    const int L = plan.L, m = L / p, LP = plan.stride();
    const int total = nsig * L;
    for (int e = threadIdx.x; e < total; e += blockDim.x) {
        const int sig = e / L;
        const int rem = e - sig * L;
        const int q = rem / m;
        const int j = rem - q * m;
        const int k = j % ns;
        const cx<R>* in = a + sig * LP;
        cx<R> acc = in[plan.at(j)];
        int qr = 0;   // (q * r) mod p
        for (int r = 1; r < p; ++r) {
            cx<R> x = in[plan.at(j + r * m)];
            if (k > 0) x = INV ? cmulc(x, tw[r * ns + k]) : cmul(x, tw[r * ns + k]);
            qr += q;
            if (qr >= p) qr -= p;
            if (qr) x = cmul(x, twl(tw2, qr * m, INV));
            acc = acc + x;
        }
        b[sig * LP + plan.at((j / ns) * ns * p + k + q * ns)] = acc;
    }
}

// Runs the plan on nsig signals (plan.stride() apart) in `a` (scratch `b`, same
// size).  `tw` holds the plan's pass tables, `tw2` exp(-2 pi i k / (2L)).  Returns
// the buffer holding the result.  Ends with __syncthreads().
template <typename R, bool INV>
__device__ cx<R>* fft_smem(cx<R>* a, cx<R>* b, int nsig, const FftPlan& plan, const cx<R>* __restrict__ tw,
                           const cx<R>* __restrict__ tw2) {
    int ns = 1;
    for (int s = 0; s < plan.npass; ++s) {
        const int p = plan.radix[s];
        switch (p) {
            case 2: stockham_pass_fixed<R, 2, INV>(a, b, nsig, plan, ns, tw); break;
            case 3: stockham_pass_fixed<R, 3, INV>(a, b, nsig, plan, ns, tw); break;
            case 4: stockham_pass_fixed<R, 4, INV>(a, b, nsig, plan, ns, tw); break;
            case 5: stockham_pass_fixed<R, 5, INV>(a, b, nsig, plan, ns, tw); break;
            case 6: stockham_pass_fixed<R, 6, INV>(a, b, nsig, plan, ns, tw); break;
            case 8: stockham_pass_fixed<R, 8, INV>(a, b, nsig, plan, ns, tw); break;
            case 10: stockham_pass_fixed<R, 10, INV>(a, b, nsig, plan, ns, tw); break;
            case 12: stockham_pass_fixed<R, 12, INV>(a, b, nsig, plan, ns, tw); break;
            case 16: stockham_pass_fixed<R, 16, INV>(a, b, nsig, plan, ns, tw); break;
            default: stockham_pass_generic<R, INV>(a, b, nsig, plan, p, ns, tw, tw2); break;
        }
        __syncthreads();
        cx<R>* t = a;
        a = b;
        b = t;
        if (s > 0) tw += p * ns;   // pass 0 has no table
        ns *= p;
    }
    return a;
}

// Pass tables of a plan: for every pass s >= 1 (radix p, stride ns = product of the
// earlier radices) W_{ns p}^{k r} at [r * ns + k], r < p, k < ns, pass after pass.
// Fewer than 2L entries.  Entry e; false past the end.
__device__ __forceinline__ bool pass_table_entry(const FftPlan& plan, int e, double* c, double* s) {
    if (plan.npass == 0) return false;
    int ns = plan.radix[0];
    for (int q = 1; q < plan.npass; ++q) {
        const int p = plan.radix[q], n = p * ns;
        if (e < n) {
            const long long r = e / ns, k = e % ns;
            sincospi(2.0 * (double)((k * r) % n) / (double)n, s, c);
            *s = -*s;
            return true;
        }
        e -= n;
        ns = n;
    }
    return false;
}

}  // namespace llg
