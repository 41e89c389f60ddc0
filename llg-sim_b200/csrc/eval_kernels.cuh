// eval_kernels.cuh — instantiation and launch of the per-evaluation kernels:
// register-FFT kernels for power-of-two sizes, generic shared-memory Stockham
// kernels otherwise.  Included by one compilation unit per precision
// (eval_f32.cu, eval_f64.cu), which the build compiles side by side.
#pragma once
#include "build_api.h"
#include "fast_kernels.cuh"
#include "fused_kernels.cuh"
#include "stage_kernels.cuh"

#include <algorithm>
#include <cstdlib>

namespace llg {

namespace {

template <typename R, typename F>
bool dispatch_L(int L, F&& f) {
    switch (L) {
        case 16: f(std::integral_constant<int, 16>{}); return true;
        case 32: f(std::integral_constant<int, 32>{}); return true;
        case 64: f(std::integral_constant<int, 64>{}); return true;
        case 128: f(std::integral_constant<int, 128>{}); return true;
        case 256: f(std::integral_constant<int, 256>{}); return true;
        case 512: f(std::integral_constant<int, 512>{}); return true;
        case 1024: f(std::integral_constant<int, 1024>{}); return true;
        case 2048: f(std::integral_constant<int, 2048>{}); return true;
        default: return false;
    }
}

// f(L, V) for a power-of-two length L and radix plan V that exist (FPlan::ok).
template <typename R, typename F>
bool dispatch_LV(int L, int V, F&& f) {
    bool done = false;
    dispatch_L<R>(L, [&](auto LC) {
        constexpr int LL = decltype(LC)::value;
        if (V == 0) {
            f(LC, std::integral_constant<int, 0>{});
            done = true;
        } else if constexpr (FPlan<R, LL, 1>::ok) {
            f(LC, std::integral_constant<int, 1>{});
            done = true;
        }
    });
    return done;
}

constexpr size_t kStaticSmemCol = 64;   // mbarriers and the timeout flag of k_column_fast

// Intermediate RK stages need only the torque: no reductions, error norm or
// field output.
bool lean_epilogue(const EvalSpec& e) {
    return e.err == ERR_NONE && !e.reduce && e.local && (e.rhs == RHS_LLG || e.rhs == RHS_RELAX);
}
constexpr int log2_of(int v) { return v <= 1 ? 0 : 1 + log2_of(v / 2); }
int stage_grid(long long work) {
    return (int)std::max(1LL, std::min((work + 255) / 256, 148LL * 8));
}

// The last RK45 stage of a run (no reductions): torque plus the error norm.
bool lean_err45_epilogue(const EvalSpec& e) {
    return e.err == ERR_RK45 && !e.reduce && e.local && e.rhs == RHS_LLG && e.k_out != KB_NONE;
}

}  // namespace

template <typename R>
FastCfg fast_config(int nx, int ny) {
    FastCfg c{};
    for (int v = 0; v < 2; ++v) {
        bool okr = dispatch_LV<R>(nx, v, [&](auto LC, auto VC) {
            constexpr int L = decltype(LC)::value, V = decltype(VC)::value;
            c.T[v] = RowCfg<R, L, V>::T;
            c.row_threads[v] = RowCfg<R, L, V>::THREADS;
            c.smem_row[v] = RowCfg<R, L, V>::SMEM;
            c.twp_row_size[v] = TwTab<R, L, V>::size;
        });
        bool okc = dispatch_LV<R>(ny, v, [&](auto LC, auto VC) {
            constexpr int L = decltype(LC)::value, V = decltype(VC)::value;
            c.NC[v] = ColCfg<R, L, V>::NC;
            c.col_threads[v] = ColCfg<R, L, V>::THREADS;
            c.smem_col[v] = ColCfg<R, L, V>::SMEM;
            c.twp_col_size[v] = TwTab<R, L, V>::size;
        });
        // The register-FFT row kernels move the spectrum of consecutive rows as 16-byte
        // pieces of the column-major X[c][kx][j]: in FP32 a piece is two rows, so the
        // column stride ny must be even for every piece to start on a 16-byte boundary.
        c.ok_row[v] = okr && c.smem_row[v] <= kSmemMax && (sizeof(R) == 8 || ny % 2 == 0);
        c.ok_col[v] = okc && c.smem_col[v] + kStaticSmemCol <= kSmemMax;
    }
    return c;
}

template <typename R>
cudaError_t build_pass_tables(void* out, int L_, int v, cudaStream_t s) {
    cudaError_t err = cudaSuccess;
    dispatch_LV<R>(L_, v, [&](auto LC, auto VC) {
        constexpr int L = decltype(LC)::value, V = decltype(VC)::value;
        if (TwTab<R, L, V>::size > 0) {
            k_pass_tables<R, L, V><<<(TwTab<R, L, V>::size + 255) / 256, 256, 0, s>>>(reinterpret_cast<cx<R>*>(out));
            err = cudaGetLastError();
        }
    });
    return err;
}

// Opts a kernel into the largest dynamic shared memory it can have beside its static
// part; an error where `need` exceeds that.  The limit is state of the process: set to
// one engine's size it refused the launches of a live engine with longer films.
static cudaError_t allow_max_smem(const void* kernel, size_t need) {
    cudaFuncAttributes fa;
    cudaError_t e = cudaFuncGetAttributes(&fa, kernel);
    if (e != cudaSuccess) return e;
    const size_t most = kSmemMax - fa.sharedSizeBytes;
    if (need > most) return cudaErrorInvalidValue;
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
}

template <typename R>
cudaError_t prepare_eval_kernels(size_t smem_row, size_t smem_col) {
    constexpr int NT = sizeof(R) == 4 ? 512 : 256;
    for (const void* f : {(const void*)k_row_forward<R>, (const void*)k_row_inverse<R, false>,
                          (const void*)k_row_inverse<R, true>, (const void*)k_row_fused_generic<R, 256>,
                          (const void*)k_row_fused_generic<R, NT>})
        if (cudaError_t e = allow_max_smem(f, smem_row)) return e;
    if (cudaError_t e = allow_max_smem((const void*)k_column<R>, smem_col)) return e;
    // fast kernels: every instantiation whose shared memory fits; the whole unified
    // L1/shared array as shared memory, so that occupancy is bounded by registers
    // and the blocks' own shared memory only
    auto set_all = [&](auto LC, auto VC) {
        constexpr int L = decltype(LC)::value, V = decltype(VC)::value;
        auto both = [](const void* f, int bytes) {
            cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
            cudaFuncSetAttribute(f, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
        };
        if constexpr (RowCfg<R, L, V>::SMEM <= kSmemMax) {
            constexpr int sm = (int)RowCfg<R, L, V>::SMEM;
            both((const void*)k_row_forward_fast<R, L, V>, sm);
            both((const void*)k_row_inverse_fast<R, L, 0, V>, sm);
            both((const void*)k_row_inverse_fast<R, L, 1, V>, sm);
            both((const void*)k_row_inverse_fast<R, L, 2, V>, sm);
            if constexpr (inverse_xt_ok<R, L, V>()) both((const void*)k_row_inverse_fast<R, L, 2, V, 2>, sm);
            both((const void*)k_row_fused<R, L, V, 1>, sm);
            if constexpr (fused_xt_ok<R, L, V>()) both((const void*)k_row_fused<R, L, V, 2>, sm);
        }
        if constexpr (ColCfg<R, L, V>::SMEM + kStaticSmemCol <= kSmemMax) {
            both((const void*)k_column_fast<R, L, V, false>, (int)ColCfg<R, L, V, false>::SMEM);
            both((const void*)k_column_fast<R, L, V, true>, (int)ColCfg<R, L, V, true>::SMEM);
        }
    };
    for (int L : {16, 32, 64, 128, 256, 512, 1024, 2048})
        for (int v = 0; v < 2; ++v) dispatch_LV<R>(L, v, set_all);
    return cudaGetLastError();
}

template <typename R>
cudaError_t launch_one(int which, const EvalSpec& spec, const LaunchGeom& g, cudaStream_t s, int* nk) {
    int count = 0;
    auto row = [&](auto kernel, int grid, int block, size_t smem) {
        kernel<<<grid, block, smem, s>>>(g.films, g.row_items, g.n_row_items, spec);
        ++count;
    };
    auto col = [&](auto kernel, int block, size_t smem) {
        kernel<<<g.grid_col, block, smem, s>>>(g.films, g.col_items, g.n_col_items, spec);
        ++count;
    };
    if (which == 0 || which == 2) {
        if (g.fast_row) {
            dispatch_LV<R>(g.fast_row, g.row_var, [&](auto LC, auto VC) {
                constexpr int L = decltype(LC)::value, V = decltype(VC)::value;
                if constexpr (RowCfg<R, L, V>::SMEM <= kSmemMax) {
                    using C = RowCfg<R, L, V>;
                    if (which == 0) {
                        row(k_row_forward_fast<R, L, V>, g.grid_row, C::THREADS, C::SMEM);
                    } else if (lean_epilogue(spec) || lean_err45_epilogue(spec)) {
                        // transform only, then the torque epilogue as a streaming kernel
                        constexpr int LOG_L = log2_of(L), LOG_T = log2_of(C::T);
                        row(k_row_inverse_fast<R, L, 1, V>, g.grid_rinv, C::THREADS, C::SMEM);
                        const int grid = stage_grid((long long)g.n_row_items * C::T * L);
                        auto torque = lean_err45_epilogue(spec) ? k_stage_torque<R, true> : k_stage_torque<R, false>;
                        torque<<<grid, 256, 0, s>>>(g.films, g.row_items, g.n_row_items, LOG_L, LOG_T, spec);
                        ++count;
                    } else if (spec.rhs == RHS_MINIMIZE) {
                        if constexpr (inverse_xt_ok<R, L, V>()) {
                            if (g.n_row_items <= g.nsm) {   // one block per SM at most
                                row(k_row_inverse_fast<R, L, 2, V, 2>, g.n_row_items, 2 * C::THREADS, C::SMEM);
                                return;
                            }
                        }
                        row(k_row_inverse_fast<R, L, 2, V>, g.grid_rfull, C::THREADS, C::SMEM);
                    } else {
                        row(k_row_inverse_fast<R, L, 0, V>, g.grid_rfull, C::THREADS, C::SMEM);
                    }
                }
            });
        } else if (which == 0) {
            row(k_row_forward<R>, g.grid_row, 256, g.smem_row);
        } else {
            row(spec.rhs == RHS_MINIMIZE ? k_row_inverse<R, true> : k_row_inverse<R, false>, g.grid_row, 256,
                g.smem_row);
        }
    } else if (g.fast_col) {
        // col_var = 2 * radix plan + lean form
        dispatch_LV<R>(g.fast_col, g.col_var / 2, [&](auto LC, auto VC) {
            constexpr int L = decltype(LC)::value, V = decltype(VC)::value;
            if constexpr (ColCfg<R, L, V>::SMEM + kStaticSmemCol <= kSmemMax) {
                using Staged = ColCfg<R, L, V, false>;
                using Lean = ColCfg<R, L, V, true>;
                if (g.col_var % 2) col(k_column_fast<R, L, V, true>, Lean::THREADS, Lean::SMEM);
                else col(k_column_fast<R, L, V, false>, Staged::THREADS, Staged::SMEM);
            }
        });
    } else {
        col(k_column<R>, 256, g.smem_col);
    }
    if (nk) *nk += count;
    return cudaGetLastError();
}

template <typename R>
bool can_fuse(const EvalSpec& si, const EvalSpec& sf, const LaunchGeom& g) {
    return g.fuse_rows && lean_epilogue(si) && si.k_out != KB_NONE && !si.skip_if_fsal &&
           !sf.skip_if_fsal && sf.nterm >= 1 && sf.nterm <= 6 && sf.kidx[sf.nterm - 1] == si.k_out &&
           sf.req == si.req && sf.demag == si.demag && sf.m_in != si.m_in;
}

template <typename R>
cudaError_t launch_fused(const EvalSpec& si, const EvalSpec& sf, const LaunchGeom& g, cudaStream_t s, int* nk) {
    if (!g.fast_row) {
        if (sizeof(R) == 4 && g.n_row_items <= g.nsm)
            k_row_fused_generic<R, sizeof(R) == 4 ? 512 : 256><<<g.n_row_items, sizeof(R) == 4 ? 512 : 256, g.smem_row, s>>>(
                g.films, g.row_items, g.n_row_items, si, sf);
        else
            k_row_fused_generic<R, 256><<<g.grid_fused, 256, g.smem_row, s>>>(g.films, g.row_items, g.n_row_items, si,
                                                                            sf);
    }
    dispatch_LV<R>(g.fast_row, g.row_var, [&](auto LC, auto VC) {
        constexpr int L = decltype(LC)::value, V = decltype(VC)::value;
        if constexpr (RowCfg<R, L, V>::SMEM <= kSmemMax) {
            using C = RowCfg<R, L, V>;
            if constexpr (fused_xt_ok<R, L, V>()) {
                if (g.n_row_items <= g.nsm) {   // one block per SM at most
                    k_row_fused<R, L, V, 2><<<g.n_row_items, 2 * C::THREADS, C::SMEM, s>>>(g.films, g.row_items,
                                                                                          g.n_row_items, si, sf);
                    return;
                }
            }
            k_row_fused<R, L, V, 1><<<g.grid_fused, C::THREADS, C::SMEM, s>>>(g.films, g.row_items, g.n_row_items, si,
                                                                              sf);
        }
    });
    if (nk) *nk += 1;
    return cudaGetLastError();
}

template <typename R>
void fast_occupancy(int nx, int ny, int row_var, int col_var, int* fwd_blocks_per_sm, int* inv_blocks_per_sm,
                    int* full_blocks_per_sm, int* fused_blocks_per_sm, int* col_blocks_per_sm) {
    *fwd_blocks_per_sm = *inv_blocks_per_sm = *full_blocks_per_sm = *fused_blocks_per_sm = *col_blocks_per_sm = 1;
    dispatch_LV<R>(nx, row_var, [&](auto LC, auto VC) {
        constexpr int L = decltype(LC)::value, V = decltype(VC)::value;
        if constexpr (RowCfg<R, L, V>::SMEM <= kSmemMax) {
            using C = RowCfg<R, L, V>;
            int a = 1, b = 1, c = 1, d = 1;
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, k_row_forward_fast<R, L, V>, C::THREADS, C::SMEM);
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_row_inverse_fast<R, L, 1, V>, C::THREADS, C::SMEM);
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&c, k_row_inverse_fast<R, L, 0, V>, C::THREADS, C::SMEM);
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&d, k_row_fused<R, L, V, 1>, C::THREADS, C::SMEM);
            *fwd_blocks_per_sm = std::max(1, a);
            *inv_blocks_per_sm = std::max(1, b);
            *full_blocks_per_sm = std::max(1, c);
            *fused_blocks_per_sm = std::max(1, d);
        }
    });
    dispatch_LV<R>(ny, col_var / 2, [&](auto LC, auto VC) {
        constexpr int L = decltype(LC)::value, V = decltype(VC)::value;
        if constexpr (ColCfg<R, L, V>::SMEM + kStaticSmemCol <= kSmemMax) {
            int a = 1;
            if (col_var % 2)
                cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, k_column_fast<R, L, V, true>,
                                                              ColCfg<R, L, V, true>::THREADS,
                                                              ColCfg<R, L, V, true>::SMEM);
            else
                cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, k_column_fast<R, L, V, false>,
                                                              ColCfg<R, L, V, false>::THREADS,
                                                              ColCfg<R, L, V, false>::SMEM);
            *col_blocks_per_sm = std::max(1, a);
        }
    });
}

}  // namespace llg
