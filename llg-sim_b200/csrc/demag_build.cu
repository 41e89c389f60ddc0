// demag_build.cu — FP64 construction of the demag kernel on the GPU.
//
// Follows Demag2D::new for open boundaries (demag_fft_uniform.rs:470-634):
//   1. quadrant kernel K = mu0*N(sx, sy) for 0 <= sx < nx, 0 <= sy < ny by the
//      MuMax-like face-charge integration (kernel_2d_components_mumax_like /
//      mumax_like_h_from_unit_m, demag_fft_uniform.rs:1076-1253) — one warp per
//      displacement, the integration points split over the lanes;
//   2. reflection onto the 2nx x 2ny padded grid with exact parity, Kxy zero on
//      the axes, Nyquist planes zero (demag_fft_uniform.rs:1013-1072);
//   3. FP64 2-D FFT of the four planes (rows then columns, the project's
//      shared-memory FFT in double precision);
//   4. extraction of the real parts on kx in [0,nx], ky in [0,ny], scaled by
//      1/(px*py) and cast to the solver precision.
// Each integration sample differences two charge/(4 pi r^3) pole terms that
// cancel at large r, so all of this stays FP64.
#include <algorithm>
#include <vector>

#include "build_api.h"
#include "fft_smem.cuh"
#include "field_kernels.cuh"

namespace llg {

namespace {

constexpr double kPi = 3.14159265358979323846;

__device__ __forceinline__ double delta_cell(long long d) {
    double a = (double)(d < 0 ? -d : d);
    if (a > 0.0) a -= 1.0;
    return a;
}
__device__ __forceinline__ long long mumax_n(double x) { return (long long)floor(fmax(x, 1.0) + 0.5); }

// One warp integrates the field of unit magnetisation along `u` of the source
// cell at r_center (mumax_like_h_from_unit_m, demag_fft_uniform.rs:1139-1242).
__device__ void warp_h_from_unit_m(int u, const double* rc, const double* cell, const long long* disp, double accuracy,
                                   double* h_out) {
    const int lane = threadIdx.x & 31;
    const int v = (u + 1) % 3, w = (u + 2) % 3;
    const double lmin = fmin(fmin(cell[0], cell[1]), cell[2]);
    const double dxm = delta_cell(disp[0]) * cell[0];
    const double dym = delta_cell(disp[1]) * cell[1];
    const double dzm = delta_cell(disp[2]) * cell[2];
    double d = sqrt(dxm * dxm + dym * dym + dzm * dzm);
    if (d == 0.0) d = lmin;
    const double max_size = d / accuracy;
    const long long nx = mumax_n(cell[0] / max_size);
    const long long ny = mumax_n(cell[1] / max_size);
    const long long nz = mumax_n(cell[2] / max_size);
    const long long nv = 2 * mumax_n(cell[v] / max_size);
    const long long nw = 2 * mumax_n(cell[w] / max_size);
    const double scale = 1.0 / (double)(nv * nw * nx * ny * nz);
    const double charge = cell[v] * cell[w] * scale;
    const double pu1 = 0.5 * cell[u], pu2 = -pu1;
    const long long total = nv * nw * nx * ny * nz;
    double h0 = 0.0, h1 = 0.0, h2 = 0.0;
    for (long long t = lane; t < total; t += 32) {
        long long q = t;
        const long long az = q % nz; q /= nz;
        const long long ay = q % ny; q /= ny;
        const long long ax = q % nx; q /= nx;
        const long long jw = q % nw;
        const long long iv = q / nw;
        double pole[3];
        pole[v] = -0.5 * cell[v] + cell[v] / (2.0 * (double)nv) + (double)iv * (cell[v] / (double)nv);
        pole[w] = -0.5 * cell[w] + cell[w] / (2.0 * (double)nw) + (double)jw * (cell[w] / (double)nw);
        const double rx = rc[0] - 0.5 * cell[0] + cell[0] / (2.0 * (double)nx) + (double)ax * (cell[0] / (double)nx);
        const double ry = rc[1] - 0.5 * cell[1] + cell[1] / (2.0 * (double)ny) + (double)ay * (cell[1] / (double)ny);
        const double rz = rc[2] - 0.5 * cell[2] + cell[2] / (2.0 * (double)nz) + (double)az * (cell[2] / (double)nz);
        pole[u] = pu1;
        const double r1x = rx - pole[0], r1y = ry - pole[1], r1z = rz - pole[2];
        const double r1 = sqrt(r1x * r1x + r1y * r1y + r1z * r1z);
        const double q1 = charge / (4.0 * kPi * r1 * r1 * r1);
        pole[u] = pu2;
        const double r2x = rx - pole[0], r2y = ry - pole[1], r2z = rz - pole[2];
        const double r2 = sqrt(r2x * r2x + r2y * r2y + r2z * r2z);
        const double q2 = -charge / (4.0 * kPi * r2 * r2 * r2);
        h0 += r1x * q1 + r2x * q2;
        h1 += r1y * q1 + r2y * q2;
        h2 += r1z * q1 + r2z * q2;
    }
    for (int o = 16; o > 0; o >>= 1) {
        h0 += __shfl_xor_sync(0xffffffffu, h0, o);
        h1 += __shfl_xor_sync(0xffffffffu, h1, o);
        h2 += __shfl_xor_sync(0xffffffffu, h2, o);
    }
    h_out[0] = h0;
    h_out[1] = h1;
    h_out[2] = h2;
}

__global__ void k_kernel_quadrant(int nx, int ny, double dx, double dy, double dz, double accuracy,
                                  double* __restrict__ quad) {
    const long long wid = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (wid >= (long long)nx * ny) return;
    const int sy = (int)(wid / nx), sx = (int)(wid % nx);
    const double rc[3] = {(double)sx * dx, (double)sy * dy, 0.0};
    const double cell[3] = {dx, dy, dz};
    const long long disp[3] = {sx, sy, 0};
    double hx[3], hy[3], hz[3];
    warp_h_from_unit_m(0, rc, cell, disp, accuracy, hx);
    warp_h_from_unit_m(1, rc, cell, disp, accuracy, hy);
    warp_h_from_unit_m(2, rc, cell, disp, accuracy, hz);
    if ((threadIdx.x & 31) == 0) {
        const double mu0 = 4.0 * kPi * 1e-7;  // params.rs:15
        double* o = quad + wid * 4;
        o[0] = mu0 * hx[0];
        o[1] = mu0 * hy[0];
        o[2] = mu0 * hy[1];
        o[3] = mu0 * hz[2];
    }
}

__global__ void k_kernel_expand(int nx, int ny, const double* __restrict__ quad, cx<double>* __restrict__ planes) {
    const int px = 2 * nx, py = 2 * ny;
    const long long np = (long long)px * py;
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < np; e += (long long)gridDim.x * blockDim.x) {
        const int ix = (int)(e % px), iy = (int)(e / px);
        double v[4] = {0.0, 0.0, 0.0, 0.0};
        if (ix != nx && iy != ny) {
            const int sx = ix < nx ? ix : ix - px;
            const int sy = iy < ny ? iy : iy - py;
            const int ax = sx < 0 ? -sx : sx, ay = sy < 0 ? -sy : sy;
            const double* q = quad + ((long long)ay * nx + ax) * 4;
            v[0] = q[0];
            v[2] = q[2];
            v[3] = q[3];
            v[1] = (sx == 0 || sy == 0) ? 0.0 : ((sx < 0) != (sy < 0) ? -q[1] : q[1]);
        }
        for (int c = 0; c < 4; ++c) planes[c * np + e] = mkc(v[c], 0.0);
    }
}

template <typename R>
__global__ void k_kernel_extract(int nx, int ny, const cx<double>* __restrict__ planes, double scale,
                                 r4<R>* __restrict__ khat, double* __restrict__ k64, bool split) {
    const int px = 2 * nx, py = 2 * ny;
    const long long np = (long long)px * py;
    const int total = (nx + 1) * (ny + 1);
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < total; e += gridDim.x * blockDim.x) {
        const int kx = e / (ny + 1), ky = e % (ny + 1);
        const int slot = split ? kx * (ny + 1) + khat_index(ky, ny) : e;
        double v[4];
        for (int c = 0; c < 4; ++c) v[c] = planes[c * np + (long long)ky * px + kx].re;
        r4<R> o;
        o.x = (R)(v[0] * scale);
        o.y = (R)(v[1] * scale);
        o.z = (R)(v[2] * scale);
        o.w = (R)(v[3] * scale);
        khat[slot] = o;
        // export layout [c][ky][kx]
        for (int c = 0; c < 4; ++c) k64[((long long)c * (ny + 1) + ky) * (nx + 1) + kx] = v[c];
    }
}

// Periodic images (build_kernel_realspace_pbc, demag_fft_uniform.rs:941-1005):
// one warp per displacement (sx, sy) in [-sx_max, sx_max] x [-sy_max, sy_max].
__global__ void k_kernel_displacements(int sx_max, int sy_max, double dx, double dy, double dz, double accuracy,
                                       double* __restrict__ comp) {
    const long long nsx = 2LL * sx_max + 1, nsy = 2LL * sy_max + 1;
    const long long wid = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (wid >= nsx * nsy) return;
    const long long sx = wid % nsx - sx_max, sy = wid / nsx - sy_max;
    const double rc[3] = {(double)sx * dx, (double)sy * dy, 0.0};
    const double cell[3] = {dx, dy, dz};
    const long long disp[3] = {sx, sy, 0};
    double hx[3], hy[3], hz[3];
    warp_h_from_unit_m(0, rc, cell, disp, accuracy, hx);
    warp_h_from_unit_m(1, rc, cell, disp, accuracy, hy);
    warp_h_from_unit_m(2, rc, cell, disp, accuracy, hz);
    if ((threadIdx.x & 31) == 0) {
        const double mu0 = 4.0 * kPi * 1e-7;  // params.rs:15
        double* o = comp + wid * 4;
        o[0] = mu0 * hx[0];
        o[1] = mu0 * hy[0];
        o[2] = mu0 * hy[1];
        o[3] = mu0 * hz[2];
    }
}

// Wrapped sums of the images into the px x py bins, per bin in the reference's
// accumulation order (sy ascending, then sx ascending); Kxy zero on the axes.
__global__ void k_kernel_wrap(int sx_max, int sy_max, int px, int py, const double* __restrict__ comp,
                              cx<double>* __restrict__ planes) {
    const long long nsx = 2LL * sx_max + 1;
    const long long np = (long long)px * py;
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < np; e += (long long)gridDim.x * blockDim.x) {
        const int ix = (int)(e % px), iy = (int)(e / px);
        double v[4] = {0.0, 0.0, 0.0, 0.0};
        // smallest sy >= -sy_max with sy = iy (mod py)
        long long sy0 = iy - ((iy + (long long)sy_max) / py) * py;
        long long sx0 = ix - ((ix + (long long)sx_max) / px) * px;
        for (long long sy = sy0; sy <= sy_max; sy += py)
            for (long long sx = sx0; sx <= sx_max; sx += px) {
                const double* kc = comp + ((sy + sy_max) * nsx + (sx + sx_max)) * 4;
                for (int c = 0; c < 4; ++c) v[c] += kc[c];
            }
        if (ix == 0 || iy == 0) v[1] = 0.0;
        for (int c = 0; c < 4; ++c) planes[c * np + e] = mkc(v[c], 0.0);
    }
}

}  // namespace

template <typename R>
__global__ void k_twiddles(cx<R>* tw, int L2) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < L2; k += gridDim.x * blockDim.x) {
        double s, c;
        sincospi(2.0 * (double)k / (double)L2, &s, &c);
        tw[k] = mkc((R)c, (R)(-s));
    }
}

// In-place transforms of ns signals per block (fewer in the last block of a row of tiles).
// rows: a signal is contiguous and threads run along it; else the signals are adjacent
// columns and threads run along them, so that each row of a tile is ns contiguous elements
// (whole 32-byte sectors in FP64 instead of half ones).
template <typename R>
__global__ void __launch_bounds__(256) k_fft_strided(cx<R>* data, FftPlan plan, const cx<R>* tw, const cx<R>* tw2,
                                                     long long elem_stride, int nsig_a, long long stride_a,
                                                     long long stride_b, int ns, int rows, int inverse) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int L = plan.L, LP = plan.stride();
    cx<R>* A = reinterpret_cast<cx<R>*>(smem_raw);
    cx<R>* B = A + (size_t)ns * LP;
    const int tiles_a = (nsig_a + ns - 1) / ns;
    const int a0 = (int)(blockIdx.x % tiles_a) * ns, nv = min(ns, nsig_a - a0);
    cx<R>* d = data + a0 * stride_a + (long long)(blockIdx.x / tiles_a) * stride_b;
    for (int e = threadIdx.x; e < nv * L; e += blockDim.x) {
        const int t = rows ? e % L : e / nv, c = rows ? e / L : e % nv;
        A[(size_t)c * LP + plan.at(t)] = d[c * stride_a + t * elem_stride];
    }
    __syncthreads();
    cx<R>* res = inverse ? fft_smem<R, true>(A, B, nv, plan, tw, tw2) : fft_smem<R, false>(A, B, nv, plan, tw, tw2);
    for (int e = threadIdx.x; e < nv * L; e += blockDim.x) {
        const int t = rows ? e % L : e / nv, c = rows ? e / L : e % nv;
        d[c * stride_a + t * elem_stride] = res[(size_t)c * LP + plan.at(t)];
    }
}

template __global__ void k_twiddles<float>(cx<float>*, int);
template __global__ void k_twiddles<double>(cx<double>*, int);

template <typename R>
__global__ void k_pass_tables_smem(FftPlan plan, cx<R>* out) {
    int num, den;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; pass_table_entry(plan, e, &num, &den);
         e += gridDim.x * blockDim.x) {
        double s, c;
        sincospi(2.0 * (double)num / (double)den, &s, &c);
        out[e] = mkc((R)c, (R)-s);
    }
}

static constexpr int kRadices[] = {16, 12, 10, 8, 6, 5, 4, 3, 2};   // radices with a register butterfly

// Radix plans of the generic Stockham transform of length L: the fewest passes over
// the radices with a register butterfly (16, 12, 10, 8, 6, 5, 4, 3, 2; a larger
// prime factor is a pass of its own), each multiset of radices in descending and in
// ascending order, the ones with the smallest sum of radices (fewest registers and
// the most even split) first.
std::vector<FftPlan> plan_candidates(int L) {
    std::vector<int> primes;   // factors without a register butterfly
    int r = L;
    for (int f : {2, 3, 5})
        while (r % f == 0) r /= f;
    for (int f = 7; r > 1; f += 2)
        while (r % f == 0) {
            primes.push_back(f);
            r /= f;
        }
    int smooth = L;
    for (int p : primes) smooth /= p;
    std::vector<std::vector<int>> best;
    std::vector<int> cur;
    auto search = [&](auto&& self, int rest, int max_radix, size_t depth) -> void {
        if (rest == 1) {
            if (cur.size() == depth) best.push_back(cur);
            return;
        }
        if (cur.size() >= depth) return;
        for (int p : kRadices)
            if (p <= max_radix && rest % p == 0) {
                cur.push_back(p);
                self(self, rest / p, p, depth);
                cur.pop_back();
            }
    };
    for (size_t depth = 0; best.empty() && depth <= (size_t)kMaxRadices; ++depth) search(search, smooth, 16, depth);
    std::stable_sort(best.begin(), best.end(), [](const std::vector<int>& a, const std::vector<int>& b) {
        int sa = 0, sb = 0;
        for (int x : a) sa += x;
        for (int x : b) sb += x;
        return sa < sb;
    });
    std::vector<FftPlan> out;
    auto add = [&](std::vector<int> rad) {
        rad.insert(rad.end(), primes.begin(), primes.end());
        FftPlan p{};
        p.L = L;
        p.sh = 30;
        p.npass = (int)rad.size();
        for (size_t i = 0; i < rad.size(); ++i) p.radix[i] = rad[i];
        for (const FftPlan& q : out)
            if (std::equal(q.radix, q.radix + q.npass, p.radix)) return;
        out.push_back(p);
    };
    for (size_t i = 0; i < best.size() && i < 3; ++i) {
        add(best[i]);
        std::reverse(best[i].begin(), best[i].end());
        add(best[i]);
    }
    return out;
}

namespace {
// Descending radices of the 2-3-5-smooth `rest` in exactly `depth` passes with the
// smallest sum (the first such in search order, as in plan_candidates).
void best_radices(int rest, int max_radix, int n, int depth, int sum, int* cur, int* best, int* best_sum) {
    if (rest == 1) {
        if (n == depth && sum < *best_sum) {
            *best_sum = sum;
            std::copy(cur, cur + n, best);
        }
        return;
    }
    if (n >= depth) return;
    for (int p : kRadices)
        if (p <= max_radix && rest % p == 0) {
            cur[n] = p;
            best_radices(rest / p, p, n + 1, depth, sum + p, cur, best, best_sum);
        }
}
}  // namespace

// plan_candidates(L)[0] without allocations (plans are also formed per call).
FftPlan make_plan(int L) {
    FftPlan p{};
    p.L = L;
    p.sh = 30;
    int smooth = L;
    for (int f : {2, 3, 5})
        while (smooth % f == 0) smooth /= f;
    int rest = smooth;
    smooth = L / smooth;
    int cur[kMaxRadices], best_sum = 1 << 30;
    for (int depth = 0; depth <= kMaxRadices && best_sum == 1 << 30; ++depth) {
        best_radices(smooth, 16, 0, depth, 0, cur, p.radix, &best_sum);
        p.npass = depth;
    }
    for (int f = 7; rest > 1; f += 2)
        while (rest % f == 0) {
            p.radix[p.npass++] = f;
            rest /= f;
        }
    return p;
}

FftPlan padded_plan(FftPlan p, bool fp64, int buffers, size_t smem_max) {
    const size_t elem = fp64 ? sizeof(cx<double>) : sizeof(cx<float>);
    p.sh = fp64 ? 3 : 4;
    if (elem * (size_t)buffers * p.stride() > smem_max) p.sh = 30;
    return p;
}

int fft_block_threads(const FftPlan& plan, int nsig, int sweeps, int most) {
    int best = 128;
    long long best_cost = 0;
    for (int nt = 128; nt <= most; nt += 32) {
        long long cost = ((long long)sweeps * plan.L + nt - 1) / nt;
        for (int q = 0; q < plan.npass; ++q) {
            const long long n = (long long)nsig * (plan.L / plan.radix[q]);
            cost += (n + nt - 1) / nt * plan.radix[q];
        }
        if (best_cost == 0 || cost < best_cost) {
            best_cost = cost;
            best = nt;
        }
    }
    return best;
}

cudaError_t launch_pass_tables(const FftPlan& plan, void* out, bool fp64, cudaStream_t s) {
    const int blocks = (2 * plan.L + 255) / 256;
    if (fp64) k_pass_tables_smem<double><<<blocks, 256, 0, s>>>(plan, reinterpret_cast<cx<double>*>(out));
    else k_pass_tables_smem<float><<<blocks, 256, 0, s>>>(plan, reinterpret_cast<cx<float>*>(out));
    return cudaGetLastError();
}

cudaError_t launch_twiddles(void* tw, int L2, bool fp64, cudaStream_t s) {
    int blocks = (L2 + 255) / 256;
    if (fp64) k_twiddles<double><<<blocks, 256, 0, s>>>(reinterpret_cast<cx<double>*>(tw), L2);
    else k_twiddles<float><<<blocks, 256, 0, s>>>(reinterpret_cast<cx<float>*>(tw), L2);
    return cudaGetLastError();
}

template <typename R>
cudaError_t launch_fft_strided(void* data, const FftPlan& base, const void* tw, const void* tw2, long long elem_stride, int nsig_a,
                               long long stride_a, int nsig_b, long long stride_b, bool inverse, cudaStream_t s) {
    constexpr bool fp64 = sizeof(R) == 8;
    const bool rows = elem_stride == 1;
    int ns = 1;
    // Signals per block: as many as leave 2.5 blocks per SM and three of them room in the
    // shared memory of one (128 threads at 122 registers: four fit the registers).  FP64
    // pass, us, with one signal of 256 threads per block and now: 300 x 300 rows 18.6 and
    // 8.4, 512 x 512 27.0 and 14.6, columns 20.6 and 8.9, 32.4 and 16.1; a launch of fewer
    // blocks than SMs keeps 256 threads (rows of 2000 x 40: 11.5, with 128 15.4).
    int dev = 0, nsm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    auto smem_of = [&](int n) { return 2 * (size_t)n * padded_plan(base, fp64, 2 * n, kSmemMax).stride() * sizeof(cx<R>); };
    auto blocks_of = [&](int n) { return (nsig_a + n - 1) / n * nsig_b; };
    while (ns < 8 && smem_of(2 * ns) <= 74 * 1024 && 2 * blocks_of(2 * ns) >= 5 * nsm) ns *= 2;

    const FftPlan plan = padded_plan(base, fp64, 2 * ns, kSmemMax);
    const int blocks = blocks_of(ns);
    // the kernel's shared-memory limit is state of the process: always the largest, so that
    // a thread with shorter signals does not lower it for another one
    cudaError_t e =
        cudaFuncSetAttribute(k_fft_strided<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax);
    if (e != cudaSuccess) return e;
    k_fft_strided<R><<<blocks, blocks > nsm ? 128 : 256, smem_of(ns), s>>>(
        reinterpret_cast<cx<R>*>(data), plan, reinterpret_cast<const cx<R>*>(tw),
        reinterpret_cast<const cx<R>*>(tw2), elem_stride, nsig_a, stride_a, stride_b, ns, rows ? 1 : 0,
        inverse ? 1 : 0);
    return cudaGetLastError();
}
template cudaError_t launch_fft_strided<float>(void*, const FftPlan&, const void*, const void*, long long, int, long long, int,
                                               long long, bool, cudaStream_t);
template cudaError_t launch_fft_strided<double>(void*, const FftPlan&, const void*, const void*, long long, int, long long, int,
                                                long long, bool, cudaStream_t);

#define CK(x)                                  \
    do {                                       \
        cudaError_t _e = (x);                  \
        if (_e != cudaSuccess) return _e;      \
    } while (0)

cudaError_t build_demag_kernel(int nx, int ny, double dx, double dy, double dz, bool fp64_out, void* khat_out,
                               double* k64_out_dev, cudaStream_t s, bool split_columns) {
    if (split_columns && (ny % 2) != 0) return cudaErrorInvalidValue;
    const int px = 2 * nx, py = 2 * ny;
    const long long np = (long long)px * py;
    double* quad = nullptr;
    cx<double>* planes = nullptr;
    cx<double>* twx = nullptr;
    cx<double>* twy = nullptr;
    cudaError_t err = cudaSuccess;
    auto cleanup = [&]() {
        if (quad) cudaFree(quad);
        if (planes) cudaFree(planes);
        if (twx) cudaFree(twx);
        if (twy) cudaFree(twy);
    };
    do {
        if ((err = cudaMalloc(&quad, sizeof(double) * 4 * (size_t)nx * ny)) != cudaSuccess) break;
        if ((err = cudaMalloc(&planes, sizeof(cx<double>) * 4 * (size_t)np)) != cudaSuccess) break;
        if ((err = cudaMalloc(&twx, sizeof(cx<double>) * 4 * (size_t)px)) != cudaSuccess) break;
        if ((err = cudaMalloc(&twy, sizeof(cx<double>) * 4 * (size_t)py)) != cudaSuccess) break;
        {
            long long warps = (long long)nx * ny;
            long long threads = warps * 32;
            int blocks = (int)((threads + 255) / 256);
            k_kernel_quadrant<<<blocks, 256, 0, s>>>(nx, ny, dx, dy, dz, 10.0 /* DEMAG_ACCURACY :432 */, quad);
            if ((err = cudaGetLastError()) != cudaSuccess) break;
        }
        k_kernel_expand<<<1184, 256, 0, s>>>(nx, ny, quad, planes);
        if ((err = cudaGetLastError()) != cudaSuccess) break;
        if ((err = launch_twiddles(twx, 2 * px, true, s)) != cudaSuccess) break;
        if ((err = launch_twiddles(twy, 2 * py, true, s)) != cudaSuccess) break;
        if ((err = launch_pass_tables(make_plan(px), twx + 2 * px, true, s)) != cudaSuccess) break;
        if ((err = launch_pass_tables(make_plan(py), twy + 2 * py, true, s)) != cudaSuccess) break;
        // rows: length px, contiguous; signals = py rows x 4 planes
        if ((err = launch_fft_strided<double>(planes, make_plan(px), twx + 2 * px, twx, 1, py, px, 4, np, false, s)) != cudaSuccess) break;
        // columns: length py, stride px; signals = px columns x 4 planes
        if ((err = launch_fft_strided<double>(planes, make_plan(py), twy + 2 * py, twy, px, px, 1, 4, np, false, s)) != cudaSuccess) break;
        const double scale = 1.0 / (double)np;
        int blocks = ((nx + 1) * (ny + 1) + 255) / 256;
        if (fp64_out)
            k_kernel_extract<double><<<blocks, 256, 0, s>>>(
                nx, ny, planes, scale, reinterpret_cast<r4<double>*>(khat_out), k64_out_dev, split_columns);
        else
            k_kernel_extract<float><<<blocks, 256, 0, s>>>(
                nx, ny, planes, scale, reinterpret_cast<r4<float>*>(khat_out), k64_out_dev, split_columns);
        if ((err = cudaGetLastError()) != cudaSuccess) break;
        err = cudaStreamSynchronize(s);
    } while (0);
    cleanup();
    return err;
}

// Unscaled k-space kernel planes (xx, xy, yy, zz; [c][iy][ix] complex) of Demag2D::new
// for pbc_x / pbc_y images (0 = open, padded to 2n), px = pbc_x ? nx : 2 nx.
cudaError_t build_demag_kernel_pbc(int nx, int ny, double dx, double dy, double dz, int pbc_x, int pbc_y,
                                   void* planes_out, cudaStream_t s) {
    const int px = pbc_x > 0 ? nx : 2 * nx, py = pbc_y > 0 ? ny : 2 * ny;
    const long long np = (long long)px * py;
    const int sx_max = pbc_x == 0 ? nx - 1 : nx * pbc_x - 1;
    const int sy_max = pbc_y == 0 ? ny - 1 : ny * pbc_y - 1;
    const long long ndisp = (2LL * sx_max + 1) * (2LL * sy_max + 1);
    cx<double>* planes = reinterpret_cast<cx<double>*>(planes_out);
    double* comp = nullptr;
    cx<double>* twx = nullptr;
    cx<double>* twy = nullptr;
    cudaError_t err = cudaSuccess;
    do {
        if ((err = cudaMalloc(&comp, sizeof(double) * 4 * (size_t)ndisp)) != cudaSuccess) break;
        if ((err = cudaMalloc(&twx, sizeof(cx<double>) * 4 * (size_t)px)) != cudaSuccess) break;
        if ((err = cudaMalloc(&twy, sizeof(cx<double>) * 4 * (size_t)py)) != cudaSuccess) break;
        const long long blocks = (ndisp * 32 + 255) / 256;
        k_kernel_displacements<<<(unsigned)blocks, 256, 0, s>>>(sx_max, sy_max, dx, dy, dz, 10.0, comp);
        if ((err = cudaGetLastError()) != cudaSuccess) break;
        k_kernel_wrap<<<1184, 256, 0, s>>>(sx_max, sy_max, px, py, comp, planes);
        if ((err = cudaGetLastError()) != cudaSuccess) break;
        if ((err = launch_twiddles(twx, 2 * px, true, s)) != cudaSuccess) break;
        if ((err = launch_twiddles(twy, 2 * py, true, s)) != cudaSuccess) break;
        if ((err = launch_pass_tables(make_plan(px), twx + 2 * px, true, s)) != cudaSuccess) break;
        if ((err = launch_pass_tables(make_plan(py), twy + 2 * py, true, s)) != cudaSuccess) break;
        if ((err = launch_fft_strided<double>(planes, make_plan(px), twx + 2 * px, twx, 1, py, px, 4, np, false, s)) != cudaSuccess) break;
        if ((err = launch_fft_strided<double>(planes, make_plan(py), twy + 2 * py, twy, px, px, 1, 4, np, false, s)) != cudaSuccess) break;
        err = cudaStreamSynchronize(s);
    } while (0);
    if (comp) cudaFree(comp);
    if (twx) cudaFree(twx);
    if (twy) cudaFree(twy);
    return err;
}

}  // namespace llg
