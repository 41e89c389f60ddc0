// fast_kernels.cuh — register-FFT versions of the three evaluation passes for
// power-of-two film sizes (16..2048).  Same data layout, same algorithm and
// same epilogue as field_kernels.cuh; the transforms use GroupFFT (fft_reg.cuh)
// with per-pass twiddle tables and the W_{2L}^n pre-twiddles resident in
// shared memory.
#pragma once
#include "field_kernels.cuh"
#include "fft_reg.cuh"
#include "async_copy.cuh"

namespace llg {

// Row passes: T rows per block; signals: T packed xy rows and T/2 packed z
// row pairs, each as an even-bin and an odd-bin transform (s = 2g + parity).
// Registers per thread that let `blocks` blocks of `threads` threads reside on
// one SM.  The register file is split over the SM's four sub-partitions (16384
// 32-bit registers each) and a warp takes its registers from the sub-partition it
// is scheduled on, so the sub-partition with the most warps sets the bound: 112
// registers allow two 192-thread blocks, not three (18 warps put five on one
// sub-partition; 96 registers are needed).
constexpr int regs_for_blocks(int threads, int blocks) {
    const int warps = blocks * ((threads + 31) / 32);
    const int per_partition = (warps + 3) / 4;
    const int r = (16384 / (32 * per_partition)) / 8 * 8;
    return r > 255 ? 255 : r;
}

template <typename R, int L, int V = 0>
struct RowCfg {
    using P = FPlan<R, L, V>;
    static constexpr int G = P::G, E = P::E;
    static constexpr int T = (64 / G) < 2 ? 2 : 64 / G;
    static constexpr int NGRP = T + T / 2;
    static constexpr int NSIG = 2 * NGRP;
    static constexpr int THREADS = NSIG * G;
    // register caps (regs_for_blocks): one resident block at least (REGCAP); the
    // FP32 forward and lean inverse passes of 192-thread blocks capped for three
    // resident blocks, plan 1 (half the registers per thread) for two (MAXREG);
    // the fused pass and the inverse passes with an epilogue, 192-thread FP32
    // blocks, for two (REG2: they hold a transform and a stencil at once; the
    // smaller cap only spilled without adding a block)
    static constexpr int REGCAP = regs_for_blocks(THREADS, 1);
    static constexpr int MAXREG = V == 1 ? regs_for_blocks(THREADS, 2)
                                         : (sizeof(R) == 4 && THREADS <= 192) ? regs_for_blocks(THREADS, 3) : REGCAP;
    static constexpr int REG2 = V == 1 ? regs_for_blocks(THREADS, 2)
                                       : (sizeof(R) == 4 && THREADS <= 192) ? regs_for_blocks(THREADS, 2) : REGCAP;
    static constexpr int BUF = Pad<R, L, V>::size;
    static constexpr int SMEM_CX = NSIG * BUF + TwTab<R, L, V>::size + L;
    // the staged spectrum (swizzled slots, stage_slot) lives in the signal buffers
    static constexpr int STAGE_CX = ((3 * (L + 1) * T * (int)sizeof(cx<R>) / 16 + 7) / 8 * 8) * (16 / (int)sizeof(cx<R>));
    static_assert(STAGE_CX <= NSIG * BUF, "staged spectrum does not fit the signal buffers");
    static constexpr size_t SMEM = sizeof(cx<R>) * (size_t)SMEM_CX;
};

// Column pass: NC columns per block, six signals per column (3 components x
// even / odd ky bins).  Shared memory: the signal exchange buffers, the pass
// tables and pre-twiddles, and the staging areas that the bulk copies of the
// next item's spectrum columns (Xst, [3][NC][L]) and folded kernel columns
// (Kst, [NC][L+1]) land in while the current item is transformed.  The LEAN form
// reads the tables and the kernel columns from global memory (through L1) and
// keeps only the signal buffers and Xst in shared memory, so that more blocks fit
// per SM.
template <typename R, int L, int V = 0, bool LEAN = false>
struct ColCfg {
    using P = FPlan<R, L, V>;
    static constexpr int G = P::G, E = P::E;
    static constexpr int NC = (32 / G) < 1 ? 1 : 32 / G;
    static constexpr int NSIG = 6 * NC;
    static constexpr int THREADS = NSIG * G;
    static constexpr int BUF = Pad<R, L, V>::size;
    static constexpr size_t al16(size_t b) { return (b + 15) / 16 * 16; }
    static constexpr size_t OFF_TW = al16(sizeof(cx<R>) * (size_t)NSIG * BUF);
    static constexpr size_t OFF_PRE = al16(OFF_TW + (LEAN ? 0 : sizeof(cx<R>) * (size_t)TwTab<R, L, V>::size));
    static constexpr size_t OFF_XST = al16(OFF_PRE + (LEAN ? 0 : sizeof(cx<R>) * (size_t)L));
    static constexpr size_t OFF_KST = al16(OFF_XST + sizeof(cx<R>) * 3 * (size_t)NC * L);
    static constexpr size_t SMEM = al16(OFF_KST + (LEAN ? 0 : sizeof(r4<R>) * (size_t)NC * (L + 1)));
    // register cap: two resident blocks for plan 1 (half the registers per thread) and
    // for the 192-thread FP32 blocks (three for their lean form; their shared memory
    // allows as many), one block otherwise
    static constexpr int MAXREG =
        regs_for_blocks(THREADS, V == 1 ? 2 : (sizeof(R) == 4 && THREADS <= 192) ? (LEAN ? 3 : 2) : 1);
};

// Staged spectrum of a row block, [c][k][r] in 16-byte pieces (PER complex values).
// A warp of the inverse transform reads one row of every other k, pieces 2 T / PER
// slots apart: without more, 8 (two rows per block in FP32) to all 32 of its lanes
// (eight rows and more) fall on the same banks.  The slot of a piece is XOR-swizzled
// within its group of eight by bits of the group's number, as many as it takes: one
// or two for two rows, three for more, which leaves at most 4 wavefronts.  The slots of
// a group stay in the group, so the staging area needs the piece count rounded up to
// a multiple of eight.
template <typename R, int T>
__host__ __device__ __forceinline__ int stage_slot(int p) {
    return p ^ ((p >> 3) & (T > 2 ? 7 : sizeof(R) == 4 ? 1 : 3));
}
template <typename R, int T>
__host__ __device__ __forceinline__ int stage_index(int e) {
    constexpr int PER = 16 / (int)sizeof(cx<R>);
    return stage_slot<R, T>(e / PER) * PER + e % PER;
}

template <typename R>
__device__ __forceinline__ void load_tables(cx<R>* twp, const cx<R>* __restrict__ gtwp, int ntwp, cx<R>* pre,
                                            const cx<R>* __restrict__ gpre, int L) {
    for (int i = threadIdx.x; i < ntwp; i += blockDim.x) twp[i] = gtwp[i];
    for (int i = threadIdx.x; i < L; i += blockDim.x) pre[i] = gpre[i];
}

// Barrier over the threads of the block's transforms: all of them, or the first
// THREADS of a block that has as many again (XT = 2; barrier 15).
template <int THREADS, int XT>
__device__ __forceinline__ void fft_sync() {
    if constexpr (XT == 1) __syncthreads();
    else asm volatile("bar.sync 15, %0;" ::"n"(THREADS) : "memory");
}

// Stages the spectrum of a block's rows, [c][k][r] in swizzled 16-byte pieces with
// contiguous T-row chunks per (c, k), into the signal buffers (free here).
template <typename R, int L, int V, int NT = RowCfg<R, L, V>::THREADS>   // NT: threads of the block
__device__ __forceinline__ void row_stage_spectrum(const cx<R>* __restrict__ X, cx<R>* stg, int ny, int j0) {
    using C = RowCfg<R, L, V>;
    constexpr int T = C::T, PER = 16 / (int)sizeof(cx<R>), TP = T / PER;
    for (int p = threadIdx.x; p < 3 * (L + 1) * TP; p += NT) {
        const int ck = p / TP, r = p % TP * PER;
        cx<R>* dst = stg + stage_slot<R, T>(p) * PER;
        if (j0 + r < ny) {
            cp_async16(dst, X + (size_t)ck * ny + j0 + r);
        } else {
#pragma unroll
            for (int q = 0; q < PER; ++q) dst[q] = mkc((R)0, (R)0);
        }
    }
    cp_async_wait_all();
}

// Inputs of a group's inverse transform from the staged spectrum: signal g < T is
// x + i y of row g, the others z of two rows; the group of parity par takes the bins
// k = 2 (t + G r) + par.  Bins up to L are stored, the ones above are conjugates of
// bin 2L - k: r < E / 2 lies below L for every thread and r >= E / 2 above, but for
// k = L itself (r = E / 2, t = 0, even bins), whose mirror image it is, unconjugated.
// So each r has one address, a constant away from the thread's first (the swizzle of
// a slot depends on the bits below 2 G T / PER pieces only).
template <typename R, int L, int V>
__device__ __forceinline__ void row_load_inverse(const cx<R>* stg, cx<R> (&v)[RowCfg<R, L, V>::E], int t, int g, int par) {
    using C = RowCfg<R, L, V>;
    constexpr int G = C::G, E = C::E, T = C::T, K1 = L + 1, PER = 16 / (int)sizeof(cx<R>);
    static_assert((2 * G * T / PER) % (T == 2 ? 32 : 64) == 0, "swizzle strides");
    static_assert(E >= 2 && G * E == L, "bins of a thread");
    const int kb = 2 * t + par;
    const int ca = g < T ? 0 : 2, cb = g < T ? 1 : 2;             // the two real fields of the signal
    const int ra = g < T ? g : 2 * (g - T), rb = g < T ? g : ra + 1;
    const cx<R>* lo_a = stg + stage_index<R, T>((ca * K1 + kb) * T + ra);
    const cx<R>* lo_b = stg + stage_index<R, T>((cb * K1 + kb) * T + rb);
    const cx<R>* hi_a = stg + stage_index<R, T>((ca * K1 + (2 * L - kb)) * T + ra);
    const cx<R>* hi_b = stg + stage_index<R, T>((cb * K1 + (2 * L - kb)) * T + rb);
#pragma unroll
    for (int r = 0; r < E; ++r) {
        const int off = 2 * G * r * T;
        cx<R> a, b;
        if (r < E / 2) {
            a = lo_a[off];
            b = lo_b[off];
        } else {
            a = hi_a[-off];
            b = hi_b[-off];
            if (!(r == E / 2 && kb == 0)) {   // above the last stored bin
                a = conjc(a);
                b = conjc(b);
            }
        }
        v[r] = mkc(a.re - b.im, a.im + b.re);
    }
}

// Hermitian bins of the block's rows from the forward transforms in the signal
// buffers.  The two real fields of a signal come from the same two values, so each
// value is read once; PER consecutive rows of one (component, kx) make one 16-byte
// store into the column-major spectrum.
template <typename R, int L, int V, int NT = RowCfg<R, L, V>::THREADS>
__device__ __forceinline__ void row_store_spectrum(const cx<R>* buf, cx<R>* __restrict__ X, int ny, int j0) {
    using C = RowCfg<R, L, V>;
    constexpr int T = C::T, E = C::E, BUF = C::BUF, K1 = L + 1;
    constexpr int PER = 16 / (int)sizeof(cx<R>), TP = T / PER;
    const size_t plane = (size_t)K1 * ny;
    for (int e = threadIdx.x; e < K1 * TP; e += NT) {
        const int k = e / TP, r0 = e % TP * PER;
        if (j0 + r0 >= ny) continue;
        // bins k and 2L - k (mod 2L) have the parity of k
        const int km = k ? 2 * L - k : 0;
        const cx<R>* bk = buf + (k & 1) * BUF + padi<E>(k >> 1);
        const cx<R>* bm = buf + (k & 1) * BUF + padi<E>(km >> 1);
        auto first = [](cx<R> zk, cx<R> zm) { return mkc((R)0.5 * (zk.re + zm.re), (R)0.5 * (zk.im - zm.im)); };
        auto second = [](cx<R> zk, cx<R> zm) { return mkc((R)0.5 * (zk.im + zm.im), (R)0.5 * (zm.re - zk.re)); };
        cx<R>* dst = X + (size_t)k * ny + j0 + r0;
        Vec16<R> px, py, pz;
#pragma unroll
        for (int q = 0; q < PER; ++q) {
            const int r = r0 + q;
            const cx<R> zk = bk[2 * r * BUF], zm = bm[2 * r * BUF];
            const cx<R> x = first(zk, zm), y = second(zk, zm);
            px.v[2 * q] = x.re; px.v[2 * q + 1] = x.im;
            py.v[2 * q] = y.re; py.v[2 * q + 1] = y.im;
            // z of rows 2p, 2p + 1 share a signal (and, with PER = 2, this iteration)
            const cx<R> wk = bk[2 * (T + r / 2) * BUF], wm = bm[2 * (T + r / 2) * BUF];
            const cx<R> z = (r & 1) ? second(wk, wm) : first(wk, wm);
            pz.v[2 * q] = z.re; pz.v[2 * q + 1] = z.im;
        }
        stv(reinterpret_cast<R*>(dst), px);
        stv(reinterpret_cast<R*>(dst + plane), py);
        stv(reinterpret_cast<R*>(dst + 2 * plane), pz);
    }
}

// ---------------------------------------------------------------------------
template <typename R, int L, int V>
__global__ void __launch_bounds__(RowCfg<R, L, V>::THREADS) __maxnreg__((RowCfg<R, L, V>::MAXREG)) k_row_forward_fast(const FilmDev* __restrict__ films,
                                                                            const WorkItem* __restrict__ items,
                                                                            int nitems, EvalSpec spec) {
    using C = RowCfg<R, L, V>;
    using FFT = GroupFFT<R, L, false, V>;
    constexpr int G = C::G, E = C::E, T = C::T, BUF = C::BUF;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cx<R>* buf = reinterpret_cast<cx<R>*>(smem_raw);
    cx<R>* twp = buf + C::NSIG * BUF;
    cx<R>* pre = twp + TwTab<R, L, V>::size;
    const int tid = threadIdx.x, s = tid / G, t = tid % G, g = s >> 1, par = s & 1;
    bool tables = false;
    for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
        const WorkItem w = items[it];
        const FilmDev& F = films[w.film];
        const StepState* st = F.st;
        if (skip_item(spec, st)) continue;
        const bool do_fft = spec.demag && F.demag_mat;
        if (do_fft && !tables) {
            load_tables<R>(twp, reinterpret_cast<const cx<R>*>(F.twp_row[V]), TwTab<R, L, V>::size, pre,
                           reinterpret_cast<const cx<R>*>(F.tw_row), L);
            tables = true;
        }
        const int ny = F.ny, n = L * ny;
        const int j0 = w.blk * T;
        const int cur = st->cur;
        const R* __restrict__ m0 = mbuf<R>(F, MB_M0, cur);
        R* __restrict__ ms = mbuf<R>(F, spec.m_in, cur);
        const double dt = st->dt;
        const R* kp[6];
        R cq[6];
#pragma unroll
        for (int q = 0; q < 6; ++q) {
            kp[q] = q < spec.nterm ? kbuf<R>(F, spec.kidx[q], cur) : nullptr;
            cq[q] = q < spec.nterm ? (R)(dt * spec.a[q]) : (R)0;
        }
        const R Ms = (R)F.ms;
        // m_s = normalize(m0 + sum_q dt*a_q*k_q), W cells per step, the three
        // components together; the state goes to m_s and,
        // scaled by Ms, to the signal slots: x, y of row r in buffer 2r (re, im); z of
        // rows 2p, 2p+1 in buffer 2(T+p) (re, im).
        constexpr int W = 2, NV = T * L / W;
        using VW = VecW<R, W>;
        for (int e = tid; e < NV; e += C::THREADS) {
            const int c0 = e * W, r = c0 / L, i0 = c0 - r * L, j = j0 + r;
            VW a[3];
            if (j < ny) {
                const int idx = j * L + i0;
                if (spec.nterm > 0) {
#pragma unroll
                    for (int c = 0; c < 3; ++c) a[c] = ldw<R, W>(m0 + c * n + idx);
#pragma unroll
                    for (int h = 0; h < 6; h += 2) {   // two torques in flight at a time
                        VW ka[2][3];
#pragma unroll
                        for (int q = h; q < h + 2; ++q)
                            if (q < spec.nterm)
#pragma unroll
                                for (int c = 0; c < 3; ++c) ka[q - h][c] = ldw<R, W>(kp[q] + c * n + idx);
#pragma unroll
                        for (int q = h; q < h + 2; ++q)
                            if (q < spec.nterm)
#pragma unroll
                                for (int c = 0; c < 3; ++c)
#pragma unroll
                                    for (int l = 0; l < W; ++l)
                                        a[c].v[l] = fma_rn(cq[q], ka[q - h][c].v[l], a[c].v[l]);
                    }
#pragma unroll
                    for (int l = 0; l < W; ++l) {
                        R v3[3] = {a[0].v[l], a[1].v[l], a[2].v[l]};
                        if (cell_inside(F, idx + l)) normalize3(v3);
                        else { v3[0] = (R)0; v3[1] = (R)0; v3[2] = (R)0; }   // vacuum pinned at m = 0
#pragma unroll
                        for (int c = 0; c < 3; ++c) a[c].v[l] = v3[c];
                    }
#pragma unroll
                    for (int c = 0; c < 3; ++c) stw<R, W>(ms + c * n + idx, a[c]);
                } else {
#pragma unroll
                    for (int c = 0; c < 3; ++c) a[c] = ldw<R, W>(ms + c * n + idx);
                }
            } else {   // rows past the film are zero in the transform
#pragma unroll
                for (int c = 0; c < 3; ++c)
#pragma unroll
                    for (int l = 0; l < W; ++l) a[c].v[l] = (R)0;
            }
            if (do_fft) {
#pragma unroll
                for (int l = 0; l < W; ++l) {
                    buf[(2 * r) * BUF + padi<E>(i0 + l)] = mkc(Ms * a[0].v[l], Ms * a[1].v[l]);
                    cx<R>* z = &buf[(2 * (T + r / 2)) * BUF + padi<E>(i0 + l)];
                    *((r & 1) ? &z->im : &z->re) = Ms * a[2].v[l];
                }
            }
        }
        if (!do_fft) continue;
        __syncthreads();
        cx<R> v[E];
        {
            const cx<R>* zb = buf + (2 * g) * BUF;
#pragma unroll
            for (int r = 0; r < E; ++r) {
                const int nn = t + G * r;
                cx<R> x = zb[padi<E>(nn)];
                v[r] = par ? cmul(x, pre[nn]) : x;
            }
        }
        __syncthreads();
        FFT::run(v, t, buf + s * BUF, twp);
        __syncthreads();
#pragma unroll
        for (int i = 0; i < E; ++i) buf[s * BUF + padi<E>(FFT::out_index(t, i))] = v[i];
        __syncthreads();
        cx<R>* __restrict__ X = reinterpret_cast<cx<R>*>(F.X);
        row_store_spectrum<R, L, V>(buf, X, ny, j0);
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// Column pass.  Item = NC consecutive kx columns of one film.  Per column: the
// pruned forward y-transforms of the three components (even and odd ky bins as
// two length-L transforms, odd ones pre-twiddled by W_{2L}^n), the product with
// the real kernel planes (Bx = Kxx Mx + Kxy My, By = Kxy Mx + Kyy My,
// Bz = Kzz Mz; demag_fft_uniform.rs:700-742), and the pruned inverse keeping
// the L physical rows.  The spectrum and kernel columns of the block's next item
// are fetched by bulk copies while this item is transformed.
template <typename R, int L>
__device__ __forceinline__ bool col_item_has(const FilmDev* __restrict__ films, const WorkItem* __restrict__ items,
                                             int nitems, const EvalSpec& spec, int it) {
    return it < nitems && spec.demag && films[items[it].film].demag_mat;
}

template <typename R, int L, int V>
__device__ __forceinline__ void col_issue_x(const FilmDev* __restrict__ films, const WorkItem* __restrict__ items,
                                            int it, cx<R>* xst, uint64_t* bar) {
    using C = ColCfg<R, L, V>;
    const WorkItem w = items[it];
    const FilmDev& F = films[w.film];
    const int K1 = F.nx + 1, kx0 = w.blk * C::NC;
    const int nv = min(C::NC, K1 - kx0);
    const uint32_t bytes = (uint32_t)(sizeof(cx<R>) * (size_t)nv * L);
    const cx<R>* X = reinterpret_cast<const cx<R>*>(F.X);
    mbar_arrive_expect_tx(bar, 3 * bytes);
#pragma unroll
    for (int c = 0; c < 3; ++c) bulk_copy_g2s(xst + (size_t)c * C::NC * L, X + ((size_t)c * K1 + kx0) * L, bytes, bar);
}

template <typename R, int L, int V>
__device__ __forceinline__ void col_issue_k(const FilmDev* __restrict__ films, const WorkItem* __restrict__ items,
                                            int it, r4<R>* kst, uint64_t* bar) {
    using C = ColCfg<R, L, V>;
    const WorkItem w = items[it];
    const FilmDev& F = films[w.film];
    const int K1 = F.nx + 1, kx0 = w.blk * C::NC;
    const int nv = min(C::NC, K1 - kx0);
    const uint32_t bytes = (uint32_t)(sizeof(r4<R>) * (size_t)nv * (L + 1));
    mbar_arrive_expect_tx(bar, bytes);
    bulk_copy_g2s(kst, reinterpret_cast<const r4<R>*>(F.Khat) + (size_t)kx0 * (L + 1), bytes, bar);
}

template <typename R, int L, int V, bool LEAN>
__global__ void __launch_bounds__(ColCfg<R, L, V, LEAN>::THREADS) __maxnreg__((ColCfg<R, L, V, LEAN>::MAXREG)) k_column_fast(
    const FilmDev* __restrict__ films, const WorkItem* __restrict__ items, int nitems, EvalSpec spec) {
    using C = ColCfg<R, L, V, LEAN>;
    using FF = GroupFFT<R, L, false, V>;
    using FI = GroupFFT<R, L, true, V>;
    constexpr int G = C::G, E = C::E, BUF = C::BUF, NC = C::NC;
    constexpr int ny = L;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ uint64_t bars[2];   // 0: spectrum columns, 1: kernel columns
    __shared__ int s_timeout;
    cx<R>* buf = reinterpret_cast<cx<R>*>(smem_raw);
    const cx<R>* twp = reinterpret_cast<const cx<R>*>(smem_raw + C::OFF_TW);
    const cx<R>* pre = reinterpret_cast<const cx<R>*>(smem_raw + C::OFF_PRE);
    cx<R>* xst = reinterpret_cast<cx<R>*>(smem_raw + C::OFF_XST);
    r4<R>* kst = reinterpret_cast<r4<R>*>(smem_raw + C::OFF_KST);
    const int tid = threadIdx.x, s = tid / G, t = tid % G;
    const int cl = s / 6, comp = (s % 6) >> 1, par = s & 1;
    if (tid == 0) {
        mbar_init(&bars[0], 1);
        mbar_init(&bars[1], 1);
        s_timeout = 0;
        mbar_init_fence();
    }
    __syncthreads();
    const int it0 = blockIdx.x;
    if (tid == 0 && col_item_has<R, L>(films, items, nitems, spec, it0)) {
        col_issue_x<R, L, V>(films, items, it0, xst, &bars[0]);
        if (!LEAN) col_issue_k<R, L, V>(films, items, it0, kst, &bars[1]);
    }
    uint32_t phase = 0;
    bool tables = false;
    for (int it = it0; it < nitems; it += gridDim.x) {
        const int nxt = it + gridDim.x;
        const bool has = col_item_has<R, L>(films, items, nitems, spec, it);
        const bool has_next = col_item_has<R, L>(films, items, nitems, spec, nxt);
        if (!has) {   // nothing was fetched for this item (uniform over the block)
            if (tid == 0 && has_next) {
                fence_async_smem();
                col_issue_x<R, L, V>(films, items, nxt, xst, &bars[0]);
                if (!LEAN) col_issue_k<R, L, V>(films, items, nxt, kst, &bars[1]);
            }
            continue;
        }
        const WorkItem w = items[it];
        const FilmDev& F = films[w.film];
        if constexpr (LEAN) {
            twp = reinterpret_cast<const cx<R>*>(F.twp_col[V]);
            pre = reinterpret_cast<const cx<R>*>(F.tw_col);
        } else if (!tables) {
            load_tables<R>(const_cast<cx<R>*>(twp), reinterpret_cast<const cx<R>*>(F.twp_col[V]), TwTab<R, L, V>::size,
                           const_cast<cx<R>*>(pre), reinterpret_cast<const cx<R>*>(F.tw_col), L);
            tables = true;
        }
        const bool okx = mbar_wait(&bars[0], phase);
        const bool okk = LEAN ? true : mbar_wait(&bars[1], phase);
        if (!(okx && okk)) s_timeout = 1;
        phase ^= 1u;
        __syncthreads();   // tables, staged columns, timeout flag
        if (s_timeout) {
            // a copy that never completed: report and leave without touching its buffers again
            if (tid == 0) atomicExch(const_cast<int*>(&F.st->err_code), kErrAsyncTimeout);
            return;
        }
        const bool run = !skip_item(spec, F.st);
        const int K1 = F.nx + 1;
        const int kx = w.blk * NC + cl;
        const bool valid = kx < K1;
        cx<R> v[E];
        if (run) {
#pragma unroll
            for (int r = 0; r < E; ++r) {
                const int nn = t + G * r;
                const cx<R> x = valid ? xst[((size_t)comp * NC + cl) * L + nn] : mkc((R)0, (R)0);
                v[r] = par ? cmul(x, pre[nn]) : x;
            }
        }
        __syncthreads();   // staged spectrum consumed
        if (tid == 0 && has_next) {
            fence_async_smem();
            col_issue_x<R, L, V>(films, items, nxt, xst, &bars[0]);
        }
        if (run) {
            FF::run(v, t, buf + s * BUF, twp);
            group_sync<G>();
#pragma unroll
            for (int i = 0; i < E; ++i) buf[s * BUF + padi<E>(FF::out_index(t, i))] = v[i];
            __syncthreads();   // all components of the column transformed
            const r4<R>* kc = LEAN ? reinterpret_cast<const r4<R>*>(F.Khat) + (size_t)(valid ? kx : 0) * (L + 1)
                                   : kst + (size_t)cl * (L + 1);
            const cx<R>* sx = buf + (6 * cl + 0 + par) * BUF;
            const cx<R>* sy = buf + (6 * cl + 2 + par) * BUF;
            const cx<R>* sz = buf + (6 * cl + 4 + par) * BUF;
#pragma unroll
            for (int r = 0; r < E; ++r) {
                const int kk = t + G * r;
                const int ky = 2 * kk + par;
                // the kernel spectrum is even in ky except Kxy, which is odd; the
                // column is parity-split (khat_index): ky and L2 - ky have the parity
                // of this signal, so a warp reads consecutive entries
                const bool up = ky > ny;
                const r4<R> K = kc[par ? (up ? ny / 2 + L - kk : ny / 2 + 1 + kk) : (up ? L - kk : kk)];
                const R kxy = up ? -K.y : K.y;
                const int pi = padi<E>(kk);
                cx<R> out;
                if (comp == 0) {
                    const cx<R> Mx = sx[pi], My = sy[pi];
                    out = cmix(K.x, Mx, kxy, My);
                } else if (comp == 1) {
                    const cx<R> Mx = sx[pi], My = sy[pi];
                    out = cmix(kxy, Mx, K.z, My);
                } else {
                    const cx<R> Mz = sz[pi];
                    out = cscale(Mz, K.w);
                }
                v[r] = out;
            }
        }
        __syncthreads();   // products formed: the signal buffers and staged kernel are free
        if (!LEAN && tid == 0 && has_next) {
            fence_async_smem();
            col_issue_k<R, L, V>(films, items, nxt, kst, &bars[1]);
        }
        if (run) {
            FI::run(v, t, buf + s * BUF, twp);
            group_sync<G>();
            if (par) {
#pragma unroll
                for (int i = 0; i < E; ++i) buf[s * BUF + padi<E>(FI::out_index(t, i))] = v[i];
            }
            __syncthreads();   // odd-bin results visible to the even-bin groups
            if (!par && valid) {
                cx<R>* __restrict__ X = reinterpret_cast<cx<R>*>(F.X);
                const cx<R>* ob = buf + (s + 1) * BUF;
#pragma unroll
                for (int i = 0; i < E; ++i) {
                    const int nn = FI::out_index(t, i);
                    X[((size_t)comp * K1 + kx) * ny + nn] = v[i] + cmulc(ob[padi<E>(nn)], pre[nn]);
                }
            }
        }
    }
}

// ---------------------------------------------------------------------------
// MODE 0: full epilogue; 1: no epilogue, the demag field is written to the film's
// bdem planes for k_stage_torque; 2: the minimiser epilogue (RHS_MINIMIZE).
// The minimiser's FP64 cell update is a long dependent chain: in launches with at most
// one block per SM (inverse_xt_ok, chosen by the launch as for k_row_fused) the block has
// as many threads again (XT = 2), which take no part in the transforms but halve the cells
// per thread of the epilogue (an iteration of one 256 x 256 film, 64 blocks: 36 us, with
// the one-fold form 44 before this form).  With more blocks than SMs two blocks of the
// one-fold form share an SM, which keeps its threads busy in the transforms too: 16 such
// films 144 us per iteration, with the two-fold form 225; 64 films of 64 x 64 55 and 77.
template <typename R, int L, int V>
__host__ __device__ constexpr bool inverse_xt_ok() {
    return sizeof(R) == 4 && V == 0 && L <= 256 && RowCfg<R, L, V>::THREADS <= 192;
}
template <typename R, int L, int MODE, int V, int XT = 1>
__global__ void __launch_bounds__(RowCfg<R, L, V>::THREADS * XT) __maxnreg__((MODE == 1 ? RowCfg<R, L, V>::MAXREG : RowCfg<R, L, V>::REG2)) k_row_inverse_fast(const FilmDev* __restrict__ films,
                                                                            const WorkItem* __restrict__ items,
                                                                            int nitems, EvalSpec spec) {
    using C = RowCfg<R, L, V>;
    constexpr int NT = C::THREADS * XT;
    using FI = GroupFFT<R, L, true, V>;
    constexpr int G = C::G, E = C::E, T = C::T, BUF = C::BUF;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ double sm_red[32 * RED_NSLOT];
    cx<R>* buf = reinterpret_cast<cx<R>*>(smem_raw);
    cx<R>* twp = buf + C::NSIG * BUF;
    cx<R>* pre = twp + TwTab<R, L, V>::size;
    const int tid = threadIdx.x, s = tid / G, t = tid % G, g = s >> 1, par = s & 1;
    bool tables = false;
    for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
        const WorkItem w = items[it];
        const FilmDev& F = films[w.film];
        StepState* st = F.st;
        if (skip_item(spec, st)) continue;
        const bool do_fft = spec.demag && F.demag_mat;
        if (do_fft && !tables) {
            load_tables<R>(twp, reinterpret_cast<const cx<R>*>(F.twp_row[V]), TwTab<R, L, V>::size, pre,
                           reinterpret_cast<const cx<R>*>(F.tw_row), L);
            tables = true;
            __syncthreads();
        }
        const int ny = F.ny;
        const int j0 = w.blk * T;
        if (do_fft) {
            const cx<R>* __restrict__ X = reinterpret_cast<const cx<R>*>(F.X);
            row_stage_spectrum<R, L, V, NT>(X, buf, ny, j0);
            __syncthreads();
            if (XT == 1 || tid < C::THREADS) {   // threads of the transforms
                cx<R> v[E];
                row_load_inverse<R, L, V>(buf, v, t, g, par);
                fft_sync<C::THREADS, XT>();
                FI::run(v, t, buf + s * BUF, twp);
                fft_sync<C::THREADS, XT>();
                if (par) {
#pragma unroll
                    for (int i = 0; i < E; ++i) buf[s * BUF + padi<E>(FI::out_index(t, i))] = v[i];
                }
                fft_sync<C::THREADS, XT>();
                if (!par) {
                    const cx<R>* ob = buf + (s + 1) * BUF;
                    cx<R>* db = buf + s * BUF;
#pragma unroll
                    for (int i = 0; i < E; ++i) {
                        const int nn = FI::out_index(t, i);
                        db[padi<E>(nn)] = v[i] + cmulc(ob[padi<E>(nn)], pre[nn]);
                    }
                }
            }
            __syncthreads();
        }
        // demag field of row r, cell i: xy rows in buffer 2r, z pairs in buffer 2(T + r/2)
        auto dfield = [&](int r, int i, int c) -> R {
            if (c < 2) {
                const cx<R> z = buf[(2 * r) * BUF + padi<E>(i)];
                return c == 0 ? z.re : z.im;
            }
            const cx<R> z = buf[(2 * (T + r / 2)) * BUF + padi<E>(i)];
            return (r & 1) ? z.im : z.re;
        };
        if constexpr (MODE == 1) {
            // demag field only, for the streaming torque kernel
            if (do_fft) {
                constexpr int W = Vec16<R>::W;
                const int n = F.nx * ny;
                R* __restrict__ bd = reinterpret_cast<R*>(F.bdem);
                for (int e = tid; e < T * L / W; e += C::THREADS) {
                    const int c0 = e * W, r = c0 / L, i0 = c0 - r * L, j = j0 + r;
                    if (j >= ny) continue;
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        Vec16<R> o;
#pragma unroll
                        for (int l = 0; l < W; ++l) o.v[l] = dfield(r, i0 + l, c);
                        stv(bd + c * n + j * L + i0, o);
                    }
                }
            }
        } else {
            row_epilogue<R, MODE == 2>(F, spec, st, w.blk, T, do_fft, dfield, sm_red);
        }
        __syncthreads();
    }
}

// Pass twiddle tables [r][k] for GroupFFT<R, L>.
template <typename R, int L, int V>
__global__ void k_pass_tables(cx<R>* out) {
    using P = FPlan<R, L, V>;
    using TT = TwTab<R, L, V>;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < TT::size; e += gridDim.x * blockDim.x) {
        long long k, r, N;
        if (e < TT::size1) {
            r = e / TT::ns1;
            k = e % TT::ns1;
            N = (long long)TT::ns1 * P::RAD1;
        } else {
            const int f = e - TT::size1;
            r = f / TT::ns2;
            k = f % TT::ns2;
            N = (long long)TT::ns2 * P::RAD2;
        }
        double sn, cs;
        sincospi(2.0 * (double)((k * r) % N) / (double)N, &sn, &cs);
        out[e] = mkc((R)cs, (R)(-sn));
    }
}

}  // namespace llg
