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
// Rounded operations that the compiler may not fuse or reorder: the transforms and
// the local field terms spell out every product, sum and fused multiply-add that
// could be contracted in more than one way, so a value has the same bits whichever
// kernel (and whichever surrounding code) forms it.
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float sub_rn(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ double sub_rn(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }

// Complex sums.  In FP32 one packed instruction (add / sub / fma .f32x2, sm_100) forms
// both parts, each rounded as the scalar operation rounds it: the sums are most of a
// transform's instructions, and the passes of a 1024 x 1024 film went from 769 to 747 us
// per step (column 51.2 -> 48.5 us) with the same bits.
__device__ __forceinline__ unsigned long long pk(cx<float> a) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a.re), "f"(a.im));
    return r;
}
__device__ __forceinline__ cx<float> upk(unsigned long long v) {
    cx<float> r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.re), "=f"(r.im) : "l"(v));
    return r;
}
__device__ __forceinline__ cx<float> operator+(cx<float> a, cx<float> b) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pk(a)), "l"(pk(b)));
    return upk(r);
}
__device__ __forceinline__ cx<float> operator-(cx<float> a, cx<float> b) {
    unsigned long long r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pk(a)), "l"(pk(b)));
    return upk(r);
}
__device__ __forceinline__ cx<double> operator+(cx<double> a, cx<double> b) {
    return mkc(__dadd_rn(a.re, b.re), __dadd_rn(a.im, b.im));
}
__device__ __forceinline__ cx<double> operator-(cx<double> a, cx<double> b) {
    return mkc(__dsub_rn(a.re, b.re), __dsub_rn(a.im, b.im));
}
// a + p h with real h, one rounding per part
__device__ __forceinline__ cx<float> caxpy(cx<float> p, float h, cx<float> a) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(pk(p)), "l"(pk(mkc(h, h))), "l"(pk(a)));
    return upk(r);
}
__device__ __forceinline__ cx<double> caxpy(cx<double> p, double h, cx<double> a) {
    return mkc(__fma_rn(p.re, h, a.re), __fma_rn(p.im, h, a.im));
}
template <typename R>
__device__ __forceinline__ cx<R> cmul(cx<R> a, cx<R> b) {
    return mkc(fma_rn(a.re, b.re, -mul_rn(a.im, b.im)), fma_rn(a.re, b.im, mul_rn(a.im, b.re)));
}
// a * conj(b)
template <typename R>
__device__ __forceinline__ cx<R> cmulc(cx<R> a, cx<R> b) {
    return mkc(fma_rn(a.re, b.re, mul_rn(a.im, b.im)), fma_rn(a.im, b.re, -mul_rn(a.re, b.im)));
}
// p a + q b with real p, q (a bin of the kernel product)
template <typename R>
__device__ __forceinline__ cx<R> cmix(R p, cx<R> a, R q, cx<R> b) {
    return mkc(fma_rn(p, a.re, mul_rn(q, b.re)), fma_rn(p, a.im, mul_rn(q, b.im)));
}
template <typename R>
__device__ __forceinline__ cx<R> cscale(cx<R> a, R s) { return mkc(mul_rn(a.re, s), mul_rn(a.im, s)); }
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
// a + / - (-i b) (forward) or a + / - (+i b) (inverse): the parts cross over, scalar sums
template <typename R>
__device__ __forceinline__ void cross_sums(cx<R> a, cx<R> b, bool inv, cx<R>* plus, cx<R>* minus) {
    const cx<R> p = mkc(add_rn(a.re, b.im), sub_rn(a.im, b.re)), q = mkc(sub_rn(a.re, b.im), add_rn(a.im, b.re));
    *plus = inv ? q : p;
    *minus = inv ? p : q;
}
template <typename R>
__device__ __forceinline__ void bfly4(cx<R>* v, bool inv) {
    const cx<R> s02 = v[0] + v[2], d02 = v[0] - v[2];
    const cx<R> s13 = v[1] + v[3], d13 = v[1] - v[3];
    v[0] = s02 + s13;
    v[2] = s02 - s13;
    cross_sums(d02, d13, inv, &v[1], &v[3]);
}
template <typename R>
__device__ __forceinline__ void bfly8(cx<R>* v, bool inv) {
    const R h = (R)0.70710678118654752440;
    cx<R> e[4] = {v[0], v[2], v[4], v[6]};
    cx<R> o[4] = {v[1], v[3], v[5], v[7]};
    bfly4(e, inv);
    bfly4(o, inv);
    // odd outputs times w8^q; the sqrt(1/2) of q = 1, 3 goes into the multiply-adds
    const cx<R> p1 = inv ? mkc(sub_rn(o[1].re, o[1].im), add_rn(o[1].re, o[1].im))
                         : mkc(add_rn(o[1].re, o[1].im), sub_rn(o[1].im, o[1].re));
    const cx<R> p3 = inv ? mkc(-add_rn(o[3].re, o[3].im), sub_rn(o[3].re, o[3].im))
                         : mkc(sub_rn(o[3].im, o[3].re), -add_rn(o[3].re, o[3].im));
    v[0] = e[0] + o[0];
    v[4] = e[0] - o[0];
    v[1] = caxpy(p1, h, e[1]);
    v[5] = caxpy(p1, -h, e[1]);
    cross_sums(e[2], o[2], inv, &v[2], &v[6]);
    v[3] = caxpy(p3, h, e[3]);
    v[7] = caxpy(p3, -h, e[3]);
}
template <typename R>
__device__ __forceinline__ void bfly3(cx<R>* v, bool inv) {
    const R s3 = (R)0.86602540378443864676;  // sqrt(3)/2
    const cx<R> s = v[1] + v[2], d = rot(v[1] - v[2], inv);
    const cx<R> t = caxpy(s, (R)-0.5, v[0]);
    v[0] = v[0] + s;
    v[1] = caxpy(d, s3, t);
    v[2] = caxpy(d, -s3, t);
}
template <typename R>
__device__ __forceinline__ void bfly5(cx<R>* v, bool inv) {
    const R c1 = (R)0.30901699437494742410, c2 = (R)-0.80901699437494742410;
    const R s1 = (R)0.95105651629515357212, s2 = (R)0.58778525229247312917;
    const cx<R> a1s = v[1] + v[4], a1d = rot(v[1] - v[4], inv);   // -i d (forward)
    const cx<R> a2s = v[2] + v[3], a2d = rot(v[2] - v[3], inv);
    const cx<R> x0 = v[0];
    const cx<R> p1 = caxpy(a2s, c2, caxpy(a1s, c1, x0)), p2 = caxpy(a2s, c1, caxpy(a1s, c2, x0));
    const cx<R> q1 = caxpy(a2d, s2, cscale(a1d, s1)), q2 = caxpy(a2d, -s1, cscale(a1d, s2));
    v[0] = x0 + a1s + a2s;
    v[1] = p1 + q1;
    v[4] = p1 - q1;
    v[2] = p2 + q2;
    v[3] = p2 - q2;
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
                y[n2 * 4 + k1] = cmul(a[k1], mkc(wr, wi));
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
// Fewer than 2L entries.  Entry e is exp(-2 pi i num / den); false past the end.
__device__ __forceinline__ bool pass_table_entry(const FftPlan& plan, int e, int* num, int* den) {
    if (plan.npass == 0) return false;
    int ns = plan.radix[0];
#pragma unroll 1
    for (int q = 1; q < plan.npass; ++q) {
        const int p = plan.radix[q], n = p * ns;
        if (e < n) {
            const int r = e / ns;
            *num = (e - r * ns) * r;   // k r < n
            *den = n;
            return true;
        }
        e -= n;
        ns = n;
    }
    return false;
}

}  // namespace llg
