// demag_pbc.cu — demag field with periodic images, and the LLGDMAG v2 k-space
// kernel cache of the reference.
//
// Demag2D (demag_fft_uniform.rs:434-770) for pbc_x / pbc_y periodic images: no
// padding in a periodic direction (px = pbc_x ? nx : 2 nx, likewise py), the
// real-space kernel summed over the image ranges into wrapped bins
// (build_kernel_realspace_pbc, :941-1005), then the full complex px x py FFT
// convolution of add_field (:636-769).  Everything is FP64: this is the
// field-only entry compute_demag_field_pbc (demag.rs:146-156), which the
// reference's steppers do not call.  Transforms use the shared-memory FP64 FFT
// (one block per row or column), so px and py are limited to 4096.
//
// The k-space planes are stored unscaled exactly as write_kernel_kspace writes
// them (:279-319), so a cache file written here is read by the reference and
// one written by the reference is read here.
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <sys/stat.h>
#include <vector>

#include "../../include/llg_b200.h"
#include "build_api.h"
#include "field_kernels.cuh"

namespace llg {
int ctx_device(const llg_ctx* c);
}

struct llg_demag_op {
    int device = 0;
    int nx = 0, ny = 0, pbc_x = 0, pbc_y = 0, px = 0, py = 0;
    double dx = 0, dy = 0, dz = 0;
    llg::cx<double>* K = nullptr;    // [4][py][px] unscaled kernel spectrum
    llg::cx<double>* M = nullptr;    // [3][py][px] work planes
    double* stage = nullptr;         // [nx*ny*3] AoS staging
    llg::cx<double>* twx = nullptr;  // [2 px] exp(-2 pi i k / (2 px)), then [2 px] pass tables of planx
    llg::cx<double>* twy = nullptr;
    llg::FftPlan planx{}, plany{};
    // open boundaries in both directions: the folded real kernel of the pruned path
    // (nullptr: general path), and the plans / pass tables of lengths nx and ny
    llg::r4<double>* Kf = nullptr;   // [nx+1][ny+1] (xx, xy, yy, zz) / (px py)
    llg::FftPlan plan_nx{}, plan_ny{};
    int column_threads = 256;
    llg::cx<double>* tab_nx = nullptr;   // [2 nx] pass tables, then [2 nx] exp(-2 pi i k / (2 nx))
    llg::cx<double>* tab_ny = nullptr;
};

namespace {

using llg::cx;
using llg::mkc;

constexpr double kAccuracy = 10.0;   // DEMAG_ACCURACY, demag_fft_uniform.rs:432

int fail(int code, const char* fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    std::vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    llg_set_error_message(buf);
    return code;
}

#define PBC_TRY(x)                                                                                           \
    do {                                                                                                     \
        cudaError_t _e = (x);                                                                                \
        if (_e != cudaSuccess)                                                                               \
            return fail(_e == cudaErrorMemoryAllocation ? LLG_ERR_OOM : LLG_ERR_CUDA, "%s: %s", #x,          \
                        cudaGetErrorString(_e));                                                             \
    } while (0)

__global__ void k_pbc_pack(const double* __restrict__ m, int nx, int ny, int px, int py, double ms,
                           cx<double>* __restrict__ M) {
    const long long np = (long long)px * py;
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < np; e += (long long)gridDim.x * blockDim.x) {
        const int ix = (int)(e % px), iy = (int)(e / px);
        double v[3] = {0.0, 0.0, 0.0};
        if (ix < nx && iy < ny) {
            const double* mm = m + ((long long)iy * nx + ix) * 3;
            v[0] = ms * mm[0];
            v[1] = ms * mm[1];
            v[2] = ms * mm[2];
        }
        for (int c = 0; c < 3; ++c) M[c * np + e] = mkc(v[c], 0.0);
    }
}

// B = K M per bin with complex products, demag_fft_uniform.rs:700-742
__global__ void k_pbc_multiply(const cx<double>* __restrict__ K, long long np, cx<double>* __restrict__ M) {
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < np; e += (long long)gridDim.x * blockDim.x) {
        const cx<double> mx = M[e], my = M[np + e], mz = M[2 * np + e];
        const cx<double> kxx = K[e], kxy = K[np + e], kyy = K[2 * np + e], kzz = K[3 * np + e];
        M[e] = llg::cmul(kxx, mx) + llg::cmul(kxy, my);
        M[np + e] = llg::cmul(kxy, mx) + llg::cmul(kyy, my);
        M[2 * np + e] = llg::cmul(kzz, mz);
    }
}

__global__ void k_pbc_extract(const cx<double>* __restrict__ M, int nx, int ny, int px, int py, double scale,
                              double* __restrict__ b) {
    const long long np = (long long)px * py, n = (long long)nx * ny;
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
        const long long j = e / nx, i = e % nx, src = j * px + i;
        for (int c = 0; c < 3; ++c) b[e * 3 + c] = M[c * np + src].re * scale;
    }
}

// ---------------------------------------------------------------------------
// Open boundaries in both directions: the same convolution with its zeros and its
// symmetries left out.  A 2n-point transform whose upper half is zero is two
// n-point transforms (even and odd bins, the odd input multiplied by W_{2n}^i); two
// real signals share one complex transform, so only the nx+1 Hermitian bins of x
// are kept; the kernel spectrum of an open grid is real, even in kx and ky (Kxy odd
// in ky), so a quarter of it serves all bins; forward transform, kernel product and
// inverse of a column are one kernel.
//
// What bounds it: at 1536 x 1536 cells the general path moves about 5.8 GB through HBM
// (its padded planes are 453 MB and cross it twice in every pass) and takes 4.7 ms;
// this one about 0.8 GB (m in 56 MB, the spectrum [3][nx+1][ny] out and in twice, 113
// MB each way, the odd-bin half of the columns through scratch, mostly L2, the folded
// kernel 75 MB, the field out) in 0.59 ms.  What is left is latency: the FP64 buffers
// leave an SM 16 warps and little L1 for the pass tables (L1 at 50 to 58 % of its
// throughput, HBM at 11 to 13 %).
constexpr int kOpenThreads = 256;

// Component w of a row pair p (rows j0 = 2p, j0+1): row j0 + i row j0+1.  One signal
// per block: two transforms in 4 padded buffers, so that two blocks fit an SM at
// nx = 1536.  The two rows of a bin are neighbours in X: a lane pair takes them, so
// that every store is a whole 32-byte sector (at nx = ny = 1536 the forward rows went
// from 151 to 110 us, the inverse from 152 to 136).
__global__ void __launch_bounds__(kOpenThreads, 2) k_open_rows_forward(int nx, int ny, double ms,
                                                                    const double* __restrict__ m,
                                                                    cx<double>* __restrict__ X, llg::FftPlan plan,
                                                                    const cx<double>* __restrict__ tab,
                                                                    const cx<double>* __restrict__ tw) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int L = nx, LP = plan.stride(), K1 = nx + 1;
    cx<double>* A = reinterpret_cast<cx<double>*>(smem_raw);
    cx<double>* B = A + 2 * LP;
    const int p = blockIdx.x / 3, w = blockIdx.x - 3 * p, ja = 2 * p;
    const bool second = ja + 1 < ny;
    const double* ma = m + (long long)ja * nx * 3 + w;
    const double* mb = ma + (second ? (long long)nx * 3 : 0);
#pragma unroll 4
    for (int i = threadIdx.x; i < L; i += kOpenThreads) {
        const double a = ma[3 * (long long)i], b = mb[3 * (long long)i];
        const cx<double> v = mkc(ms * a, second ? ms * b : 0.0);
        A[plan.at(i)] = v;
        A[LP + plan.at(i)] = llg::cmul(v, tw[i]);
    }
    __syncthreads();
    const cx<double>* res = llg::fft_smem<double, false>(A, B, 2, plan, tab, tw);
    const int r = threadIdx.x & 1;
    if (r && !second) return;
    cx<double>* x = X + (long long)w * K1 * ny + ja + r;
    for (int k = threadIdx.x >> 1; k < K1; k += kOpenThreads / 2) {
        const int km = k ? 2 * L - k : 0;
        const cx<double> zk = res[(k & 1) * LP + plan.at(k >> 1)], zm = res[(km & 1) * LP + plan.at(km >> 1)];
        x[(long long)k * ny] = r ? mkc(0.5 * (zk.im + zm.im), 0.5 * (zm.re - zk.re))
                                 : mkc(0.5 * (zk.re + zm.re), 0.5 * (zk.im - zm.im));
    }
}

constexpr int kOpenColumnMax = 512;   // most threads of a column block (fft_block_threads)

// Two signals of a pair q of columns (kx = 2q, 2q + 1): w = 0, 1: x and y of column
// 2q + w, which the kernel couples; w = 2: z of both.  The odd and then the even ky
// bins (four padded buffers at a time), product with the folded kernel and inverse;
// the odd half waits in O, the even half adds it and replaces X.
//
// What bounds it: shared-memory passes, FP64 butterflies and the waits between them.
// Two signals per block let two blocks of 256 threads share an SM at ny = 1536, so
// that the passes of one fill the waits of the other; with all three components of a
// column per block (one block of 512 threads) the kernel took 412 us there, now 343 us.
__global__ void __launch_bounds__(kOpenColumnMax) k_open_column(int nx, int ny, const llg::r4<double>* __restrict__ Kf,
                                                              cx<double>* __restrict__ X, cx<double>* __restrict__ O,
                                                              llg::FftPlan plan, const cx<double>* __restrict__ tab,
                                                              const cx<double>* __restrict__ tw) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int L = ny, LP = plan.stride();
    const int q = blockIdx.x / 3, w = blockIdx.x - 3 * q;
    const int ka = w < 2 ? 2 * q + w : 2 * q;
    if (ka > nx) return;
    const bool second = w < 2 || ka + 1 <= nx;
    const long long plane = (long long)(nx + 1) * ny, other = w < 2 ? plane : ny;   // first to second signal
    cx<double>* A = reinterpret_cast<cx<double>*>(smem_raw);
    cx<double>* B = A + 2 * LP;
    cx<double>* xc = X + (w < 2 ? 0 : 2 * plane) + (long long)ka * ny;
    cx<double>* oc = O + (w < 2 ? 0 : 2 * plane) + (long long)ka * ny;
    const llg::r4<double>* kc = Kf + (long long)ka * (ny + 1);
    const llg::r4<double>* kd = w == 2 && second ? kc + (ny + 1) : kc;
    for (int par = 1; par >= 0; --par) {
#pragma unroll 2
        for (int y = threadIdx.x; y < L; y += blockDim.x) {
            const cx<double> x0 = xc[y], x1 = second ? xc[other + y] : mkc(0.0, 0.0), t = tw[y];
            const cx<double> t0 = llg::cmul(x0, t), t1 = llg::cmul(x1, t);
            const int at = plan.at(y);
            A[at] = mkc(par ? t0.re : x0.re, par ? t0.im : x0.im);
            A[LP + at] = mkc(par ? t1.re : x1.re, par ? t1.im : x1.im);
        }
        __syncthreads();
        cx<double>* res = llg::fft_smem<double, false>(A, B, 2, plan, tab, tw);
#pragma unroll 2
        for (int kk = threadIdx.x; kk < L; kk += blockDim.x) {
            const int ky = 2 * kk + par, kf = ky <= ny ? ky : 2 * ny - ky;
            cx<double>* s = res + plan.at(kk);
            const cx<double> Ma = s[0], Mb = s[LP];
            const llg::r4<double> K = kc[kf];
            if (w < 2) {
                const double kxy = ky <= ny ? K.y : -K.y;
                s[0] = mkc(K.x * Ma.re + kxy * Mb.re, K.x * Ma.im + kxy * Mb.im);
                s[LP] = mkc(kxy * Ma.re + K.z * Mb.re, kxy * Ma.im + K.z * Mb.im);
            } else {
                const double kb = kd[kf].w;
                s[0] = mkc(K.w * Ma.re, K.w * Ma.im);
                s[LP] = mkc(kb * Mb.re, kb * Mb.im);
            }
        }
        __syncthreads();
        const cx<double>* r2 = llg::fft_smem<double, true>(res, res == A ? B : A, 2, plan, tab, tw);
        // every y by the same thread in both rounds
        if (par) {
#pragma unroll 2
            for (int y = threadIdx.x; y < L; y += blockDim.x) {
                const cx<double> t = tw[y];
                const int at = plan.at(y);
                oc[y] = llg::cmulc(r2[at], t);
                if (second) oc[other + y] = llg::cmulc(r2[LP + at], t);
            }
        } else {
#pragma unroll 2
            for (int y = threadIdx.x; y < L; y += blockDim.x) {
                const cx<double> o0 = oc[y], o1 = second ? oc[other + y] : mkc(0.0, 0.0);
                const int at = plan.at(y);
                xc[y] = r2[at] + o0;
                if (second) xc[other + y] = r2[LP + at] + o1;
            }
        }
        __syncthreads();
    }
}

// Signals and lane pairs as in the forward pass; the field goes to the AoS output.
__global__ void __launch_bounds__(kOpenThreads, 2) k_open_rows_inverse(int nx, int ny, const cx<double>* __restrict__ X,
                                                                    llg::FftPlan plan,
                                                                    const cx<double>* __restrict__ tab,
                                                                    const cx<double>* __restrict__ tw,
                                                                    double* __restrict__ b) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int L = nx, LP = plan.stride(), K1 = nx + 1;
    cx<double>* A = reinterpret_cast<cx<double>*>(smem_raw);
    cx<double>* B = A + 2 * LP;
    const int p = blockIdx.x / 3, w = blockIdx.x - 3 * p, ja = 2 * p, r = threadIdx.x & 1;
    const bool second = ja + 1 < ny, reads = !r || second;
    const cx<double>* x = X + (long long)w * K1 * ny + ja + r;
#pragma unroll 4
    for (int k0 = 0; k0 < K1; k0 += kOpenThreads / 2) {
        const int k = k0 + (threadIdx.x >> 1), km = 2 * L - k;
        const cx<double> a = reads && k < K1 ? x[(long long)k * ny] : mkc(0.0, 0.0);
        // u of row ja and v of row ja + 1: bin k is u + i v, bin km conj(u) + i conj(v)
        const cx<double> o = mkc(__shfl_xor_sync(0xffffffffu, a.re, 1), __shfl_xor_sync(0xffffffffu, a.im, 1));
        if (!r && k < K1) A[(k & 1) * LP + plan.at(k >> 1)] = mkc(a.re - o.im, a.im + o.re);
        if (r && k > 0 && k < L) A[(km & 1) * LP + plan.at(km >> 1)] = mkc(o.re + a.im, a.re - o.im);
    }
    __syncthreads();
    const cx<double>* res = llg::fft_smem<double, true>(A, B, 2, plan, tab, tw);
    double* ba = b + (long long)ja * nx * 3 + w;
    for (int i = threadIdx.x; i < L; i += kOpenThreads) {
        const cx<double> z = res[plan.at(i)] + llg::cmulc(res[LP + plan.at(i)], tw[i]);
        ba[3 * (long long)i] = z.re;
        if (second) ba[3 * ((long long)nx + i)] = z.im;
    }
}

// Folded kernel of an open grid, scaled by 1/(px py), and in dev[0] the largest
// deviation of the planes from being real and even (Kxy odd in ky and in kx), in
// dev[1] the largest magnitude (bit patterns of non-negative doubles order like the
// values; a NaN ends up above every number).
__global__ void k_open_fold(const cx<double>* __restrict__ K, int nx, int ny, double scale,
                            llg::r4<double>* __restrict__ Kf, unsigned long long* __restrict__ dev) {
    const int px = 2 * nx, py = 2 * ny;
    const long long np = (long long)px * py;
    double worst = 0.0, big = 0.0;
    bool nan = false;
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < (long long)(nx + 1) * (ny + 1);
         e += (long long)gridDim.x * blockDim.x) {
        const int kx = (int)(e / (ny + 1)), ky = (int)(e % (ny + 1));
        const int mx = kx ? px - kx : 0, my = ky ? py - ky : 0;
        double v[4];
        for (int c = 0; c < 4; ++c) {
            const cx<double>* P = K + c * np;
            const double sg = c == 1 ? -1.0 : 1.0;
            const cx<double> a = P[(long long)ky * px + kx], q[3] = {P[(long long)ky * px + mx],
                                                                    P[(long long)my * px + kx],
                                                                    P[(long long)my * px + mx]};
            v[c] = a.re;
            const double d[7] = {a.im, q[0].re - sg * a.re, q[0].im, q[1].re - sg * a.re, q[1].im, q[2].re - a.re,
                                 q[2].im};
            for (int t = 0; t < 7; ++t) {
                nan |= d[t] != d[t];
                worst = fmax(worst, fabs(d[t]));
            }
            big = fmax(big, fabs(a.re));
        }
        llg::r4<double> o;
        o.x = v[0] * scale;
        o.y = v[1] * scale;
        o.z = v[2] * scale;
        o.w = v[3] * scale;
        Kf[e] = o;
    }
    // one atomic per warp that has entries: one per thread took 0.4 ms of every creation
    nan = __any_sync(0xffffffffu, nan);
    for (int o = 16; o > 0; o >>= 1) {
        worst = fmax(worst, __shfl_xor_sync(0xffffffffu, worst, o));
        big = fmax(big, __shfl_xor_sync(0xffffffffu, big, o));
    }
    if ((threadIdx.x & 31) == 0 && (nan || worst > 0.0 || big > 0.0)) {
        atomicMax(dev, nan ? 0x7ff8000000000000ull : (unsigned long long)__double_as_longlong(worst));
        atomicMax(dev + 1, (unsigned long long)__double_as_longlong(big));
    }
}

// Sets the pruned path of an open operator up.  The planes qualify when they are
// real and even to kOpenTol of their largest value: built kernels of cells about as thick
// as wide are to 1e-15 or so, and dropping what is below 1e-13 changes the field by no
// more than the rounding of the kernel sums themselves.  Sums over many points can
// exceed it (cells of 4 x 4 x 1 nm: 1.4e-13), and a cache file may hold any planes: such
// operators keep the general path, and so does one for which the extra buffers do not
// fit.
constexpr double kOpenTol = 1e-13;
void open_path_create(llg_demag_op* op) {
    const size_t nk = (size_t)(op->nx + 1) * (op->ny + 1);
    unsigned long long* dev = nullptr;
    unsigned long long h[2] = {~0ull, 0};
    bool ok = cudaMalloc(&op->Kf, nk * sizeof(llg::r4<double>)) == cudaSuccess &&
              cudaMalloc(&op->tab_nx, 4 * (size_t)op->nx * sizeof(cx<double>)) == cudaSuccess &&
              cudaMalloc(&op->tab_ny, 4 * (size_t)op->ny * sizeof(cx<double>)) == cudaSuccess &&
              cudaMalloc(&dev, sizeof(h)) == cudaSuccess && cudaMemset(dev, 0, sizeof(h)) == cudaSuccess;
    if (ok) {
        k_open_fold<<<1184, 256>>>(op->K, op->nx, op->ny, 1.0 / ((double)op->px * op->py), op->Kf, dev);
        ok = cudaGetLastError() == cudaSuccess && cudaMemcpy(h, dev, sizeof(h), cudaMemcpyDeviceToHost) == cudaSuccess;
    }
    if (ok) {
        double d[2];
        std::memcpy(d, h, sizeof(d));
        ok = d[0] <= kOpenTol * d[1];
    }
    constexpr size_t kMax = 227 * 1024;
    op->plan_nx = llg::padded_plan(llg::make_plan(op->nx), true, 4, kMax);
    op->plan_ny = llg::padded_plan(llg::make_plan(op->ny), true, 4, kMax);
    // 128 registers a thread: two blocks of 256 where their buffers fit an SM (1 KiB of
    // each is reserved), one of 512 where they do not
    const bool two = 2 * (4 * (size_t)op->plan_ny.stride() * sizeof(cx<double>) + 1024) <= kMax + 1024;
    op->column_threads = llg::fft_block_threads(op->plan_ny, 2, 8, two ? 256 : kOpenColumnMax);
    auto attr = [&](const void* f) {
        return cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMax) == cudaSuccess;
    };
    ok = ok && attr((const void*)k_open_rows_forward) && attr((const void*)k_open_column) &&
         attr((const void*)k_open_rows_inverse) &&
         llg::launch_pass_tables(op->plan_nx, op->tab_nx, true, 0) == cudaSuccess &&
         llg::launch_pass_tables(op->plan_ny, op->tab_ny, true, 0) == cudaSuccess &&
         llg::launch_twiddles(op->tab_nx + 2 * op->nx, 2 * op->nx, true, 0) == cudaSuccess &&
         llg::launch_twiddles(op->tab_ny + 2 * op->ny, 2 * op->ny, true, 0) == cudaSuccess;
    if (dev) cudaFree(dev);
    if (!ok) {
        cudaGetLastError();
        for (void* p : {(void*)op->Kf, (void*)op->tab_nx, (void*)op->tab_ny})
            if (p) cudaFree(p);
        op->Kf = nullptr;
        op->tab_nx = op->tab_ny = nullptr;
    }
}

}  // namespace

namespace llg {

int demag_op_apply_device(llg_demag_op* op, double ms, const double* d_m_aos, double* d_b_aos, cudaStream_t s) {
    const long long np = (long long)op->px * op->py;
    if (op->Kf) {
        cx<double>* X = op->M;
        cx<double>* O = op->M + 3 * (long long)(op->nx + 1) * op->ny;   // 6 (nx+1) ny <= 3 px py = 12 nx ny
        const cx<double>* twx = op->tab_nx + 2 * op->nx;
        const cx<double>* twy = op->tab_ny + 2 * op->ny;
        const size_t row = 4 * (size_t)op->plan_nx.stride() * sizeof(cx<double>);
        const size_t col = 4 * (size_t)op->plan_ny.stride() * sizeof(cx<double>);
        const int rows = 3 * ((op->ny + 1) / 2);
        k_open_rows_forward<<<rows, kOpenThreads, row, s>>>(op->nx, op->ny, ms, d_m_aos, X, op->plan_nx, op->tab_nx,
                                                            twx);
        k_open_column<<<3 * (op->nx / 2 + 1), op->column_threads, col, s>>>(op->nx, op->ny, op->Kf, X, O, op->plan_ny,
                                                                          op->tab_ny, twy);
        k_open_rows_inverse<<<rows, kOpenThreads, row, s>>>(op->nx, op->ny, X, op->plan_nx, op->tab_nx, twx, d_b_aos);
        PBC_TRY(cudaGetLastError());
        return LLG_OK;
    }
    k_pbc_pack<<<1184, 256, 0, s>>>(d_m_aos, op->nx, op->ny, op->px, op->py, ms, op->M);
    PBC_TRY(cudaGetLastError());
    PBC_TRY(llg::launch_fft_strided<double>(op->M, op->planx, op->twx + 2 * op->px, op->twx, 1, op->py, op->px, 3, np, false, s));
    PBC_TRY(llg::launch_fft_strided<double>(op->M, op->plany, op->twy + 2 * op->py, op->twy, op->px, op->px, 1, 3, np, false, s));
    k_pbc_multiply<<<1184, 256, 0, s>>>(op->K, np, op->M);
    PBC_TRY(cudaGetLastError());
    PBC_TRY(llg::launch_fft_strided<double>(op->M, op->planx, op->twx + 2 * op->px, op->twx, 1, op->py, op->px, 3, np, true, s));
    PBC_TRY(llg::launch_fft_strided<double>(op->M, op->plany, op->twy + 2 * op->py, op->twy, op->px, op->px, 1, 3, np, true, s));
    k_pbc_extract<<<1184, 256, 0, s>>>(op->M, op->nx, op->ny, op->px, op->py, 1.0 / (double)np, d_b_aos);
    PBC_TRY(cudaGetLastError());
    return LLG_OK;
}

void demag_op_info(const llg_demag_op* op, int* device, llg_grid* g, int* pbc_x, int* pbc_y) {
    *device = op->device;
    g->nx = op->nx;
    g->ny = op->ny;
    g->dx = op->dx;
    g->dy = op->dy;
    g->dz = op->dz;
    *pbc_x = op->pbc_x;
    *pbc_y = op->pbc_y;
}

}  // namespace llg

namespace {

// Rust's `{:.3e}`: mantissa with three decimals, exponent without sign padding.
std::string rust_exp3(double v) {
    char buf[64];
    std::snprintf(buf, sizeof(buf), "%.3e", v);
    std::string s(buf);
    const size_t p = s.find('e');
    if (p == std::string::npos) return s;
    const int ex = std::atoi(s.c_str() + p + 1);
    return s.substr(0, p) + "e" + std::to_string(ex);
}

std::string cache_name(int nx, int ny, int pbc_x, int pbc_y, int px, int py, double dx, double dy, double dz) {
    // demag_cache_path, demag_fft_uniform.rs:261-277
    char acc[32];
    std::snprintf(acc, sizeof(acc), "%.2f", kAccuracy);
    return "out/demag_cache/demag_kernel_nx" + std::to_string(nx) + "_ny" + std::to_string(ny) + "_pbcx" +
           std::to_string(pbc_x) + "_pbcy" + std::to_string(pbc_y) + "_px" + std::to_string(px) + "_py" +
           std::to_string(py) + "_dx" + rust_exp3(dx) + "_dy" + rust_exp3(dy) + "_dz" + rust_exp3(dz) + "_acc" + acc +
           ".bin";
}

#pragma pack(push, 1)
struct CacheHeader {          // KernelCacheHeader, demag_fft_uniform.rs:207-221 (little endian)
    char magic[8];
    uint32_t version, nx, ny, pbc_x, pbc_y, px, py;
    double dx, dy, dz, accuracy;
};
#pragma pack(pop)
static_assert(sizeof(CacheHeader) == 68, "LLGDMAG v2 header is 68 bytes");

CacheHeader make_header(const llg_demag_op* op) {
    CacheHeader h;
    std::memcpy(h.magic, "LLGDMAG\0", 8);
    h.version = 2;
    h.nx = (uint32_t)op->nx;
    h.ny = (uint32_t)op->ny;
    h.pbc_x = (uint32_t)op->pbc_x;
    h.pbc_y = (uint32_t)op->pbc_y;
    h.px = (uint32_t)op->px;
    h.py = (uint32_t)op->py;
    h.dx = op->dx;
    h.dy = op->dy;
    h.dz = op->dz;
    h.accuracy = kAccuracy;
    return h;
}

// try_load_kernel_kspace (:322-429): false (and nothing changed) on any mismatch or short file.
bool try_load(llg_demag_op* op, const char* path) {
    FILE* f = std::fopen(path, "rb");
    if (!f) return false;
    CacheHeader h;
    const CacheHeader want = make_header(op);
    bool ok = std::fread(&h, sizeof(h), 1, f) == 1 && std::memcmp(h.magic, want.magic, 8) == 0 && h.version == 2 &&
              h.nx == want.nx && h.ny == want.ny && h.pbc_x == want.pbc_x && h.pbc_y == want.pbc_y &&
              h.px == want.px && h.py == want.py && h.dx == want.dx && h.dy == want.dy && h.dz == want.dz &&
              h.accuracy == want.accuracy;
    const size_t np = (size_t)op->px * op->py;
    std::vector<cx<double>> host;
    if (ok) {
        host.resize(4 * np);
        ok = std::fread(host.data(), sizeof(cx<double>), host.size(), f) == host.size();
    }
    std::fclose(f);
    if (!ok) return false;
    return cudaMemcpy(op->K, host.data(), host.size() * sizeof(cx<double>), cudaMemcpyHostToDevice) == cudaSuccess;
}

// fs::create_dir_all of the file's parent directory, as write_kernel_kspace does
void make_parent_dirs(const char* path) {
    std::string p(path);
    for (size_t i = 1; i < p.size(); ++i)
        if (p[i] == '/') mkdir(p.substr(0, i).c_str(), 0777);
}

int save(const llg_demag_op* op, const char* path) {
    const size_t np = (size_t)op->px * op->py;
    make_parent_dirs(path);
    std::vector<cx<double>> host(4 * np);
    PBC_TRY(cudaMemcpy(host.data(), op->K, host.size() * sizeof(cx<double>), cudaMemcpyDeviceToHost));
    FILE* f = std::fopen(path, "wb");
    if (!f) return fail(LLG_ERR_INVALID, "cannot open %s for writing", path);
    const CacheHeader h = make_header(op);
    bool ok = std::fwrite(&h, sizeof(h), 1, f) == 1 &&
              std::fwrite(host.data(), sizeof(cx<double>), host.size(), f) == host.size();
    ok = (std::fclose(f) == 0) && ok;
    return ok ? LLG_OK : fail(LLG_ERR_INVALID, "short write to %s", path);
}

void destroy(llg_demag_op* op) {
    if (!op) return;
    cudaSetDevice(op->device);
    cudaFree(op->K);
    cudaFree(op->M);
    cudaFree(op->stage);
    cudaFree(op->twx);
    cudaFree(op->twy);
    cudaFree(op->Kf);
    cudaFree(op->tab_nx);
    cudaFree(op->tab_ny);
    delete op;
}

}  // namespace

extern "C" {

int llg_demag_cache_filename(const llg_grid* g, int64_t pbc_x, int64_t pbc_y, char* buf, int64_t len) {
    if (!g || !buf || len <= 0) return fail(LLG_ERR_INVALID, "null argument");
    const int px = pbc_x > 0 ? (int)g->nx : 2 * (int)g->nx, py = pbc_y > 0 ? (int)g->ny : 2 * (int)g->ny;
    const std::string s = cache_name((int)g->nx, (int)g->ny, (int)pbc_x, (int)pbc_y, px, py, g->dx, g->dy, g->dz);
    if ((int64_t)s.size() + 1 > len) return fail(LLG_ERR_INVALID, "buffer of %lld bytes too small", (long long)len);
    std::memcpy(buf, s.c_str(), s.size() + 1);
    return LLG_OK;
}

int llg_demag_op_create(llg_ctx* ctx, const llg_grid* g, int64_t pbc_x, int64_t pbc_y, const char* cache_path,
                        int32_t* loaded, llg_demag_op** out) {
    if (!ctx || !g || !out) return fail(LLG_ERR_INVALID, "null argument");
    if (g->nx < 1 || g->ny < 1 || pbc_x < 0 || pbc_y < 0 || pbc_x > 4096 || pbc_y > 4096 || !(g->dx > 0) ||
        !(g->dy > 0) || !(g->dz > 0))
        return fail(LLG_ERR_INVALID, "bad grid or image counts");
    const long long px = pbc_x > 0 ? g->nx : 2 * g->nx, py = pbc_y > 0 ? g->ny : 2 * g->ny;
    if (px > 4096 || py > 4096)
        return fail(LLG_ERR_INVALID, "padded size %lldx%lld exceeds 4096 (shared-memory FFT limit)", px, py);
    const long long sx = pbc_x == 0 ? g->nx - 1 : g->nx * pbc_x - 1, sy = pbc_y == 0 ? g->ny - 1 : g->ny * pbc_y - 1;
    if ((2 * sx + 1) * (2 * sy + 1) > (1LL << 26))
        return fail(LLG_ERR_INVALID, "%lld periodic-image displacements exceed 2^26",
                    (long long)((2 * sx + 1) * (2 * sy + 1)));
    llg_demag_op* op = new llg_demag_op();
    op->device = llg::ctx_device(ctx);
    op->nx = (int)g->nx;
    op->ny = (int)g->ny;
    op->pbc_x = (int)pbc_x;
    op->pbc_y = (int)pbc_y;
    op->px = (int)px;
    op->py = (int)py;
    op->dx = g->dx;
    op->dy = g->dy;
    op->dz = g->dz;
    op->planx = llg::make_plan(op->px);
    op->plany = llg::make_plan(op->py);
    const size_t np = (size_t)px * py;
    auto bail = [&](int rc) {
        destroy(op);
        return rc;
    };
    if (cudaSetDevice(op->device) != cudaSuccess) return bail(fail(LLG_ERR_CUDA, "cudaSetDevice failed"));
    if (cudaMalloc(&op->K, 4 * np * sizeof(cx<double>)) != cudaSuccess ||
        cudaMalloc(&op->M, 3 * np * sizeof(cx<double>)) != cudaSuccess ||
        cudaMalloc(&op->stage, 3 * (size_t)g->nx * g->ny * sizeof(double)) != cudaSuccess ||
        cudaMalloc(&op->twx, 4 * (size_t)px * sizeof(cx<double>)) != cudaSuccess ||
        cudaMalloc(&op->twy, 4 * (size_t)py * sizeof(cx<double>)) != cudaSuccess)
        return bail(fail(LLG_ERR_OOM, "cudaMalloc failed for a %lldx%lld demag operator", px, py));
    if (llg::launch_twiddles(op->twx, 2 * op->px, true, 0) != cudaSuccess ||
        llg::launch_twiddles(op->twy, 2 * op->py, true, 0) != cudaSuccess ||
        llg::launch_pass_tables(op->planx, op->twx + 2 * op->px, true, 0) != cudaSuccess ||
        llg::launch_pass_tables(op->plany, op->twy + 2 * op->py, true, 0) != cudaSuccess)
        return bail(fail(LLG_ERR_CUDA, "twiddle tables"));
    bool hit = cache_path && try_load(op, cache_path);
    if (!hit) {
        cudaError_t e = llg::build_demag_kernel_pbc(op->nx, op->ny, op->dx, op->dy, op->dz, op->pbc_x, op->pbc_y,
                                                    op->K, 0);
        if (e != cudaSuccess) return bail(fail(LLG_ERR_CUDA, "kernel build: %s", cudaGetErrorString(e)));
        if (cache_path && save(op, cache_path) != LLG_OK) {
            // like the reference, a cache that cannot be written is not an error
        }
    }
    if (pbc_x == 0 && pbc_y == 0) open_path_create(op);
    if (cudaDeviceSynchronize() != cudaSuccess) return bail(fail(LLG_ERR_CUDA, "demag operator set-up"));
    if (loaded) *loaded = hit ? 1 : 0;
    *out = op;
    return LLG_OK;
}

int llg_demag_op_destroy(llg_demag_op* op) {
    destroy(op);
    return LLG_OK;
}

int llg_demag_op_field(llg_demag_op* op, double ms, const double* m_aos, double* b_aos) {
    if (!op || !m_aos || !b_aos) return fail(LLG_ERR_INVALID, "null argument");
    PBC_TRY(cudaSetDevice(op->device));
    const long long n = (long long)op->nx * op->ny;
    PBC_TRY(cudaMemcpy(op->stage, m_aos, sizeof(double) * 3 * (size_t)n, cudaMemcpyHostToDevice));
    int rc = llg::demag_op_apply_device(op, ms, op->stage, op->stage, 0);
    if (rc) return rc;
    PBC_TRY(cudaMemcpy(b_aos, op->stage, sizeof(double) * 3 * (size_t)n, cudaMemcpyDeviceToHost));
    return LLG_OK;
}

int llg_demag_op_kspace(llg_demag_op* op, double* out) {
    if (!op || !out) return fail(LLG_ERR_INVALID, "null argument");
    PBC_TRY(cudaSetDevice(op->device));
    PBC_TRY(cudaMemcpy(out, op->K, 4 * (size_t)op->px * op->py * sizeof(cx<double>), cudaMemcpyDeviceToHost));
    return LLG_OK;
}

int llg_demag_op_save(llg_demag_op* op, const char* path) {
    if (!op || !path) return fail(LLG_ERR_INVALID, "null argument");
    PBC_TRY(cudaSetDevice(op->device));
    return save(op, path);
}

}  // extern "C"
