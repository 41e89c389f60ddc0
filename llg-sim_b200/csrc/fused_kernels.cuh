// fused_kernels.cuh — one row pass that ends RK stage s and starts stage s+1
// (register-FFT path, power-of-two nx).
//
// Per block of T rows it does, in shared memory and registers:
//   1. the inverse x transform of the block's spectrum rows (the last third of
//      stage s's field evaluation, as k_row_inverse_fast),
//   2. per cell: the local terms (Zeeman, exchange, anisotropy, DMI in the
//      reference's order; cells away from edges and vacuum by the ghost-free
//      path with the same arithmetic) plus the demag field, the torque k_s (llg_rhs /
//      llg_rhs_relax, llg.rs:20-50), stored for the later combinations and the
//      error norm, and at once the stage s+1 state
//        m_{s+1} = normalize(m0 + sum_q dt*a_q k_q)   (llg.rs:869-942 / 296-309)
//      with k_s taken from registers (it is always the last term of the next
//      combination in both tableaux),
//   3. the zero-padded forward x transform of Ms*m_{s+1} and the store of its
//      Hermitian bins (the first third of stage s+1, as k_row_forward_fast).
// An RK45 attempt is then one row-forward pass, six column passes, five fused
// row passes and the last stage's row inverse, instead of three passes per
// evaluation.  The arithmetic of every value is the one of the unfused passes
// (same operations in the same order), so both paths give the same bits.
#pragma once
#include "fast_kernels.cuh"

namespace llg {

// si: stage s (inverse half: m_in, k_out, rhs, field terms); sf: stage s+1
// (forward half: m_in receives m_{s+1}, the combination kidx / a with
// sf.kidx[sf.nterm - 1] == si.k_out).  Both carry the same request gate.
// XT = 2: the block has as many threads again, which take no part in the transforms
// but halve the cells per thread of step 2 — for launches with at most one block per
// SM, where latency is all that counts and the threads would be free anyway.
template <typename R, int L, int V>
__host__ __device__ constexpr bool fused_xt_ok() {   // one block of twice the threads at 168 registers, groups within a warp
    return V == 0 && RowCfg<R, L, V>::THREADS <= 192 && RowCfg<R, L, V>::G <= 32;
}
template <typename R, int L, int V, int XT>
__global__ void __launch_bounds__(RowCfg<R, L, V>::THREADS * XT) __maxnreg__((XT == 1 ? RowCfg<R, L, V>::REG2 : regs_for_blocks(2 * RowCfg<R, L, V>::THREADS, 1))) k_row_fused(
    const FilmDev* __restrict__ films, const WorkItem* __restrict__ items, int nitems, EvalSpec si, EvalSpec sf) {
    using C = RowCfg<R, L, V>;
    using FF = GroupFFT<R, L, false, V>;
    using FI = GroupFFT<R, L, true, V>;
    constexpr int G = C::G, E = C::E, T = C::T, BUF = C::BUF, NT = C::THREADS * XT;
    // phase 2 takes W cells per step of its loop, two in FP32 and one in FP64 (the same
    // registers): with EARLY the stencil, m0 and the previous torques of a step are all
    // loaded before any arithmetic, one memory round trip per step instead of one per
    // term.  Plan 1 and the FP64 blocks of 384 threads before doubling (L = 1024) have too
    // few registers for that: they load the torques where they are used and take the
    // general path for interior cells too.  The cap of the one-fold block decides: FP64
    // blocks doubled to 384 threads keep the early loads at 168 registers and spill for
    // it (80 to 104 bytes of stores).
    constexpr int W = sizeof(R) == 4 ? 2 : 1, NV = T * L / W;
    using VW = VecW<R, W>;
    constexpr bool EARLY = V == 0 && (sizeof(R) == 4 || C::REG2 > 200);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cx<R>* buf = reinterpret_cast<cx<R>*>(smem_raw);
    cx<R>* twp = buf + C::NSIG * BUF;
    cx<R>* pre = twp + TwTab<R, L, V>::size;
    const int tid = threadIdx.x, s = tid / G, t = tid % G, g = s >> 1, par = s & 1;
    // signal slot of component c of row r, cell i: x, y of row r in buffer 2r
    // (re, im); z of rows 2p, 2p+1 in buffer 2(T+p) (re, im).  The inverse
    // transform leaves the demag field there and the forward one takes M there.
    auto slot = [&](int c, int r, int i) -> R* {
        cx<R>* z = c < 2 ? &buf[(2 * r) * BUF + padi<E>(i)] : &buf[(2 * (T + r / 2)) * BUF + padi<E>(i)];
        return (c == 0 || (c == 2 && (r & 1) == 0)) ? &z->re : &z->im;
    };
    const bool fft = XT == 1 || tid < C::THREADS;   // threads of the transforms
    bool tables = false;
    for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
        const WorkItem w = items[it];
        const FilmDev& F = films[w.film];
        StepState* st = F.st;
        if (skip_item(si, st)) continue;   // uniform over the block
        const bool do_fft = si.demag && F.demag_mat;
        if (do_fft && !tables) {
            load_tables<R>(twp, reinterpret_cast<const cx<R>*>(F.twp_row[V]), TwTab<R, L, V>::size, pre,
                           reinterpret_cast<const cx<R>*>(F.tw_row), L);
            tables = true;
            __syncthreads();
        }
        const int ny = F.ny, n = L * ny;
        const int j0 = w.blk * T;
        const int cur = st->cur;
        cx<R>* __restrict__ X = reinterpret_cast<cx<R>*>(F.X);
        if (do_fft) {
            // ---- 1. inverse transform of stage s (k_row_inverse_fast) ----
            row_stage_spectrum<R, L, V, NT>(X, buf, ny, j0);
            __syncthreads();
            if (fft) {
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
        // ---- 2. torque of stage s and state of stage s+1, W cells per step ----
        {
            const R* __restrict__ msb = mbuf<R>(F, si.m_in, cur);
            const R* __restrict__ m0 = mbuf<R>(F, MB_M0, cur);
            R* __restrict__ kout = kbuf<R>(F, si.k_out, cur);
            R* __restrict__ mnext = mbuf<R>(F, sf.m_in, cur);
            const double dt = st->dt;
            const R gam = (R)F.gamma, alp = (R)F.alpha;
            const R denom = (R)1 + alp * alp;
            const R pref = si.rhs == RHS_LLG ? -gam / denom : -gam * alp / denom;
            const R c1 = si.rhs == RHS_LLG ? (R)1 : (R)0;
            const R c2 = si.rhs == RHS_LLG ? alp : (R)1;
            const int nq = sf.nterm - 1;   // terms read from HBM; the last one is k_s
            const R* kp[5];
            R cq[6];
#pragma unroll
            for (int q = 0; q < 5; ++q) kp[q] = q < nq ? kbuf<R>(F, sf.kidx[q], cur) : nullptr;
#pragma unroll
            for (int q = 0; q < 6; ++q) cq[q] = q < sf.nterm ? (R)(dt * sf.a[q]) : (R)0;
            const R cs = (R)(dt * sf.a[nq]);   // k_s coefficient
            const R Ms = (R)F.ms;
            const LocalCoef<R> cf = local_coef<R>(F, si.dmi != 0);
            for (int e = tid; e < NV; e += NT) {
                const int c0 = e * W, r = c0 / L, i0 = c0 - r * L, j = j0 + r;
                if (j >= ny) {   // rows past the film are zero in the forward transform
                    if (do_fft)
#pragma unroll
                        for (int l = 0; l < W; ++l)
#pragma unroll
                            for (int c = 0; c < 3; ++c) *slot(c, r, i0 + l) = (R)0;
                    continue;
                }
                const int base = j * L + i0;
                // stencil of m_s: centre, the rows below / above, one x halo on each side;
                // m0 and the torques of the combination
                VW cen[3], dn[3], upv[3], a[3], kq[EARLY ? 5 : 1][3];
                R hl[3], hr[3];
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    cen[c] = ldw<R, W>(msb + c * n + base);
                    if (j > 0) dn[c] = ldw<R, W>(msb + c * n + base - L);
                    if (j + 1 < ny) upv[c] = ldw<R, W>(msb + c * n + base + L);
                    hl[c] = i0 > 0 ? msb[c * n + base - 1] : (R)0;
                    hr[c] = i0 + W < L ? msb[c * n + base + W] : (R)0;
                }
                if constexpr (EARLY) {
#pragma unroll
                    for (int c = 0; c < 3; ++c) a[c] = ldw<R, W>(m0 + c * n + base);
#pragma unroll
                    for (int q = 0; q < 5; ++q)
                        if (q < nq)
#pragma unroll
                            for (int c = 0; c < 3; ++c) kq[q][c] = ldw<R, W>(kp[q] + c * n + base);
                }
                const bool inner = EARLY && cf.mask == nullptr && j > 0 && j + 1 < ny && i0 > 0 && i0 + W < L;
                VW ko[3];
#pragma unroll
                for (int l = 0; l < W; ++l) {
                    const int i = i0 + l;
                    const R mc[3] = {cen[0].v[l], cen[1].v[l], cen[2].v[l]};
                    auto nb = [&](int d, R* o) {
#pragma unroll
                        for (int c = 0; c < 3; ++c) {
                            if (d == 0) o[c] = l > 0 ? cen[c].v[l > 0 ? l - 1 : 0] : hl[c];
                            else if (d == 1) o[c] = l < W - 1 ? cen[c].v[l < W - 1 ? l + 1 : 0] : hr[c];
                            else if (d == 2) o[c] = dn[c].v[l];
                            else o[c] = upv[c].v[l];
                        }
                    };
                    R b[3];
                    if (inner) local_field_interior<R>(cf, nb, mc, b);
                    else local_field_c<R>(cf, nb, i, j, mc, b);
                    if (do_fft) {
#pragma unroll
                        for (int c = 0; c < 3; ++c) b[c] += *slot(c, r, i);
                    }
                    R k[3];
                    torque_cell<R>(mc, b, pref, c1, c2, k);
#pragma unroll
                    for (int c = 0; c < 3; ++c) ko[c].v[l] = k[c];
                }
#pragma unroll
                for (int c = 0; c < 3; ++c) stw<R, W>(kout + c * n + base, ko[c]);
                // m_{s+1} = normalize(m0 + sum_q dt*a_q k_q), terms in the tableau's order
                if constexpr (!EARLY) {
#pragma unroll
                    for (int c = 0; c < 3; ++c) a[c] = ldw<R, W>(m0 + c * n + base);
                }
#pragma unroll
                for (int q = 0; q < 5; ++q) {
                    if (q < nq) {
#pragma unroll
                        for (int c = 0; c < 3; ++c) {
                            const VW kv = EARLY ? kq[EARLY ? q : 0][c] : ldw<R, W>(kp[q] + c * n + base);
#pragma unroll
                            for (int l = 0; l < W; ++l) a[c].v[l] = fma_rn(cq[q], kv.v[l], a[c].v[l]);
                        }
                    }
                }
#pragma unroll
                for (int c = 0; c < 3; ++c)
#pragma unroll
                    for (int l = 0; l < W; ++l) a[c].v[l] = fma_rn(cs, ko[c].v[l], a[c].v[l]);
#pragma unroll
                for (int l = 0; l < W; ++l) {
                    R v3[3] = {a[0].v[l], a[1].v[l], a[2].v[l]};
                    if (coef_inside(cf, base + l)) normalize3(v3);
                    else { v3[0] = (R)0; v3[1] = (R)0; v3[2] = (R)0; }   // vacuum pinned at m = 0
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        a[c].v[l] = v3[c];
                        if (do_fft) *slot(c, r, i0 + l) = Ms * v3[c];
                    }
                }
#pragma unroll
                for (int c = 0; c < 3; ++c) stw<R, W>(mnext + c * n + base, a[c]);
            }
        }
        if (!do_fft) continue;
        __syncthreads();
        // ---- 3. forward transform of stage s+1 (k_row_forward_fast) ----
        if (fft) {
            cx<R> v[E];
            const cx<R>* zb = buf + (2 * g) * BUF;
#pragma unroll
            for (int r = 0; r < E; ++r) {
                const int nn = t + G * r;
                const cx<R> x = zb[padi<E>(nn)];
                v[r] = par ? cmul(x, pre[nn]) : x;
            }
            fft_sync<C::THREADS, XT>();
            FF::run(v, t, buf + s * BUF, twp);
            fft_sync<C::THREADS, XT>();
#pragma unroll
            for (int i = 0; i < E; ++i) buf[s * BUF + padi<E>(FF::out_index(t, i))] = v[i];
        }
        __syncthreads();
        row_store_spectrum<R, L, V, NT>(buf, X, ny, j0);
        __syncthreads();
    }
}

// The same row pass for films whose nx has no register FFT: the transforms of the
// generic kernels (shared-memory Stockham) around one cell per thread and step.  It
// replaces two launches by one; its loads of a step are all in flight together, and
// the field and torque arithmetic needs neither the reductions nor the FP64 of the
// full epilogue.  Same operations in the same order as the unfused kernels.
// NT threads: 512 in FP32 for launches with at most one block per SM (two rows of up to
// 256 cells are then one step), else 256 and two blocks per SM (one in FP64, whose
// butterflies need the registers).
template <typename R, int NT>
__global__ void __launch_bounds__(NT, sizeof(R) == 4 && NT == 256 ? 2 : 1) k_row_fused_generic(const FilmDev* __restrict__ films,
                                                              const WorkItem* __restrict__ items, int nitems,
                                                              EvalSpec si, EvalSpec sf) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cx<R>* sm = reinterpret_cast<cx<R>*>(smem_raw);
    for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
        const WorkItem w = items[it];
        const FilmDev& F = films[w.film];
        const StepState* st = F.st;
        if (skip_item(si, st)) continue;   // uniform over the block
        const bool do_fft = si.demag && F.demag_mat;
        const int nx = F.nx, ny = F.ny, n = nx * ny, T = F.rows_per_block, j0 = w.blk * T;
        const int cur = st->cur;
        const FftPlan& PL = F.plan_row;
        const int LP = PL.stride();
        cx<R>* A = nullptr;   // signals of the forward transform, in the half D does not use
        const R* D = do_fft ? generic_rows_inverse<R>(F, sm, j0, &A) : nullptr;
        const R* __restrict__ msb = mbuf<R>(F, si.m_in, cur);
        const R* __restrict__ m0 = mbuf<R>(F, MB_M0, cur);
        R* __restrict__ kout = kbuf<R>(F, si.k_out, cur);
        R* __restrict__ mnext = mbuf<R>(F, sf.m_in, cur);
        const double dt = st->dt;
        const R gam = (R)F.gamma, alp = (R)F.alpha;
        const R denom = (R)1 + alp * alp;
        const R pref = si.rhs == RHS_LLG ? -gam / denom : -gam * alp / denom;
        const R c1 = si.rhs == RHS_LLG ? (R)1 : (R)0;
        const R c2 = si.rhs == RHS_LLG ? alp : (R)1;
        const int nq = sf.nterm - 1;   // terms read from HBM; the last one is k_s
        const R* kp[5];
        R cq[5];
#pragma unroll
        for (int q = 0; q < 5; ++q) {
            kp[q] = q < nq ? kbuf<R>(F, sf.kidx[q], cur) : nullptr;
            cq[q] = q < nq ? (R)(dt * sf.a[q]) : (R)0;
        }
        const R cs = (R)(dt * sf.a[nq]);
        const R Ms = (R)F.ms;
        const LocalCoef<R> cf = local_coef<R>(F, si.dmi != 0);
        for (int e = threadIdx.x; e < T * nx; e += blockDim.x) {
            const int r = e / nx, i = e - r * nx, j = j0 + r;
            R v[3] = {(R)0, (R)0, (R)0};   // rows past the film are zero in the forward transform
            if (j < ny) {
                const int idx = j * nx + i;
                R a[3], kq[5][3], mc[3], b[3], k[3];
#pragma unroll
                for (int c = 0; c < 3; ++c) a[c] = m0[c * n + idx];
#pragma unroll
                for (int q = 0; q < 5; ++q)
                    if (q < nq)
#pragma unroll
                        for (int c = 0; c < 3; ++c) kq[q][c] = kp[q][c * n + idx];
                ld3(msb, n, idx, mc);
                local_field_c<R>(
                    cf,
                    [&](int d, R* o) {
                        ld3(msb, n, d == 0 ? idx - 1 : d == 1 ? idx + 1 : d == 2 ? idx - nx : idx + nx, o);
                    },
                    i, j, mc, b);
                if (do_fft) {
#pragma unroll
                    for (int c = 0; c < 3; ++c) b[c] += D[(r * 3 + c) * nx + i];
                }
                torque_cell<R>(mc, b, pref, c1, c2, k);
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    kout[c * n + idx] = k[c];
                    v[c] = a[c];
                }
#pragma unroll
                for (int q = 0; q < 5; ++q)
                    if (q < nq)
#pragma unroll
                        for (int c = 0; c < 3; ++c) v[c] = fma_rn(cq[q], kq[q][c], v[c]);
#pragma unroll
                for (int c = 0; c < 3; ++c) v[c] = fma_rn(cs, k[c], v[c]);
                if (coef_inside(cf, idx)) normalize3(v);
                else { v[0] = (R)0; v[1] = (R)0; v[2] = (R)0; }   // vacuum pinned at m = 0
#pragma unroll
                for (int c = 0; c < 3; ++c) mnext[c * n + idx] = v[c];
            }
            if (do_fft) {
                A[(2 * r) * LP + PL.at(i)] = mkc(Ms * v[0], Ms * v[1]);
                cx<R>* zp = &A[(2 * (T + r / 2)) * LP + PL.at(i)];
                if ((r & 1) == 0) {
                    zp->re = Ms * v[2];
                    if (r + 1 >= T) zp->im = (R)0;
                } else {
                    zp->im = Ms * v[2];
                }
            }
        }
        if (!do_fft) continue;
        __syncthreads();
        generic_rows_forward<R>(F, A, A == sm ? sm + 2 * (T + (T + 1) / 2) * LP : sm, j0);
        __syncthreads();
    }
}

}  // namespace llg
