// noalloc.cu — demag field of one film without any device allocation.
//
// Some callers cannot allocate device memory when they need the field: a host
// framework that owns every device allocation through its own pool, a
// real-time loop that must not pay allocation latency, or code running where
// cudaMalloc is not permitted.  llg_demag_field_noalloc serves them: the
// caller passes device pointers for the magnetisation, the kernel planes and
// the output; the spectrum scratch and the twiddles live in one file-scope static
// device array of kScratchBytes (32 MiB), the pass tables of the two transforms in
// another of 64 KiB (every GPU that loads this library holds both until the process
// exits).  Every call rewrites both, so overlapping calls race on them.
//
// Same algorithm as the three evaluation passes of field_kernels.cuh (zero-
// padded FFT convolution, demag_fft_uniform.rs:636-769): pruned R2C rows ->
// per-column transform, multiply by the real kernel planes, inverse -> C2R rows.
#include <cstdio>
#include <mutex>

#include "../../include/llg_b200.h"
#include "build_api.h"
#include "fft_smem.cuh"

namespace llg {
namespace noalloc {

constexpr size_t kScratchBytes = size_t(32) << 20;  // 32 MiB
constexpr int kMaxDevices = 64;
constexpr int kMaxLen = 2048;  // largest nx, ny
constexpr int kT = 2;          // rows per block
constexpr int kThreads = 512;  // most threads per block (fft_block_threads)

// The shared scratch.  In host code this name is only a stand-in for the
// device array; kernels receive its device address from cudaGetSymbolAddress.
static __device__ __align__(256) unsigned char g_scratch[kScratchBytes];
// Pass tables of the two transforms (2 nx and 2 ny entries at most), beside it.
static __device__ __align__(256) cx<float> g_pass_tables[4 * kMaxLen];

std::mutex g_setup_mutex;
void* g_scratch_addr[kMaxDevices] = {nullptr};
void* g_tables_addr[kMaxDevices] = {nullptr};
int g_sm_count[kMaxDevices] = {0};

inline size_t align256(size_t b) { return (b + 255) & ~size_t(255); }

// exp(-2 pi i k / (2L)) of both lengths and the pass tables of both plans.  One sincospi,
// one plan index and a rolled loop over the passes keep the code short: its fetch is most
// of the kernel's 2 to 3 us.
struct Plans {
    FftPlan p[2];   // rows, columns
};
__global__ void k_na_twiddles(cx<float>* tw_row, int nx, cx<float>* tw_col, int ny,
                              const __grid_constant__ Plans plans, cx<float>* pass_row, cx<float>* pass_col) {
    const int total = 2 * nx + 2 * ny;
    // entries [0, total): twiddles, [total, 2 total): pass tables (one sincospi per thread)
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < 2 * total; q += gridDim.x * blockDim.x) {
        const bool tables = q >= total;
        const int e = tables ? q - total : q;
        const bool row = e < 2 * nx;
        const int k = row ? e : e - 2 * nx;
        int num = k, den = row ? 2 * nx : 2 * ny;
        if (tables && !pass_table_entry(plans.p[row ? 0 : 1], k, &num, &den)) continue;
        double s, c;
        sincospi(2.0 * (double)num / (double)den, &s, &c);
        cx<float>* out = tables ? (row ? pass_row : pass_col) : (row ? tw_row : tw_col);
        out[k] = mkc((float)c, (float)-s);
    }
}

// Rows j0..j0+kT-1: M = Ms*m, pruned R2C along x, Hermitian bins to X[c][kx][j].
__global__ void __launch_bounds__(kThreads) k_na_rows_forward(int nx, int ny, float ms, const float* __restrict__ m,
                                                              cx<float>* __restrict__ X,
                                                              const cx<float>* __restrict__ twp,
                                                              const cx<float>* __restrict__ tw, FftPlan plan) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int L = nx, G = kT + (kT + 1) / 2, n = nx * ny, K1 = nx + 1, L2 = 2 * nx, LP = plan.stride();
    cx<float>* A = reinterpret_cast<cx<float>*>(smem_raw);
    cx<float>* B = A + 2 * G * LP;
    const int j0 = blockIdx.x * kT;
    for (int e = threadIdx.x; e < kT * nx; e += blockDim.x) {
        const int r = e / nx, i = e - r * nx, j = j0 + r;
        float v0 = 0.f, v1 = 0.f, v2 = 0.f;
        if (j < ny) {
            const int idx = j * nx + i;
            v0 = m[idx]; v1 = m[n + idx]; v2 = m[2 * n + idx];
        }
        A[(2 * r) * LP + plan.at(i)] = mkc(ms * v0, ms * v1);
        cx<float>* zp = &A[(2 * (kT + r / 2)) * LP + plan.at(i)];
        if ((r & 1) == 0) zp->re = ms * v2;
        else zp->im = ms * v2;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < G * L; e += blockDim.x) {
        const int g = e / L, i = e - g * L;
        A[(2 * g + 1) * LP + plan.at(i)] = cmul(A[(2 * g) * LP + plan.at(i)], tw[i]);
    }
    __syncthreads();
    cx<float>* res = fft_smem<float, false>(A, B, 2 * G, plan, twp, tw);
    for (int e = threadIdx.x; e < 3 * K1 * kT; e += blockDim.x) {
        const int r = e % kT, rest = e / kT;
        const int k = rest % K1, c = rest / K1;
        const int j = j0 + r;
        if (j >= ny) continue;
        const int g = c < 2 ? r : kT + r / 2;
        const int half = c < 2 ? c : (r & 1);
        const int km = k ? L2 - k : 0;
        const cx<float> zk = res[(2 * g + (k & 1)) * LP + plan.at(k >> 1)];
        const cx<float> zm = res[(2 * g + (km & 1)) * LP + plan.at(km >> 1)];
        X[(c * K1 + k) * ny + j] = half == 0 ? mkc(0.5f * (zk.re + zm.re), 0.5f * (zk.im - zm.im))
                                             : mkc(0.5f * (zk.im + zm.im), 0.5f * (zm.re - zk.re));
    }
}

// One kx column: pruned y transform, kernel multiply, pruned inverse.
// kp: FP64 kernel planes [4][ny+1][nx+1] (xx, xy, yy, zz), unscaled.  A block reads 8 of
// every 32-byte sector of the planes (the L2 holds them for its neighbours): blocks of up
// to four columns, which read whole sectors, left SMs without a block on films up to 256
// cells wide and registers for one block per SM on wide ones (column pass at 64 x 256
// 20.5 us against 13, whole call at 1000 x 500 126 against 117).
__global__ void __launch_bounds__(kThreads) k_na_column(int nx, int ny, const double* __restrict__ kp, double scale,
                                                        cx<float>* __restrict__ X, const cx<float>* __restrict__ twp,
                                                        const cx<float>* __restrict__ tw, FftPlan plan) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int L = ny, K1 = nx + 1, kx = blockIdx.x, LP = plan.stride();
    const size_t plane = (size_t)(ny + 1) * (nx + 1);
    cx<float>* A = reinterpret_cast<cx<float>*>(smem_raw);
    cx<float>* B = A + 6 * LP;
    // signals: component c, parity p at 2 c + p
    for (int e = threadIdx.x; e < 3 * L; e += blockDim.x) {
        const int c = e / L, y = e - c * L;
        const cx<float> x = X[((size_t)c * K1 + kx) * ny + y];
        cx<float>* s = A + 2 * c * LP + plan.at(y);
        s[0] = x;
        s[LP] = cmul(x, tw[y]);
    }
    __syncthreads();
    cx<float>* res = fft_smem<float, false>(A, B, 6, plan, twp, tw);
    // one kernel entry serves both ky and 2 ny - ky (Kxy odd)
    for (int kyf = threadIdx.x; kyf <= ny; kyf += blockDim.x) {
        const int par = kyf & 1;
        const size_t o = (size_t)kyf * (nx + 1) + kx;
        const float kxx = (float)(kp[o] * scale), kyy = (float)(kp[2 * plane + o] * scale);
        const float kzz = (float)(kp[3 * plane + o] * scale);
        const float kxyf = (float)(kp[plane + o] * scale);
        for (int h = 0; h < 2; ++h) {
            const int ky = h ? 2 * ny - kyf : kyf;
            if (h && (kyf == 0 || kyf == ny)) break;
            const float kxy = kxyf * (h ? -1.f : 1.f);
            cx<float>* s = res + par * LP + plan.at(ky >> 1);
            const cx<float> Mx = s[0], My = s[2 * LP], Mz = s[4 * LP];
            s[0] = mkc(kxx * Mx.re + kxy * My.re, kxx * Mx.im + kxy * My.im);
            s[2 * LP] = mkc(kxy * Mx.re + kyy * My.re, kxy * Mx.im + kyy * My.im);
            s[4 * LP] = mkc(kzz * Mz.re, kzz * Mz.im);
        }
    }
    __syncthreads();
    cx<float>* other = res == A ? B : A;
    cx<float>* res2 = fft_smem<float, true>(res, other, 6, plan, twp, tw);
    for (int e = threadIdx.x; e < 3 * L; e += blockDim.x) {
        const int c = e / L, y = e - c * L;
        const cx<float>* s = res2 + 2 * c * LP + plan.at(y);
        X[((size_t)c * K1 + kx) * ny + y] = s[0] + cmulc(s[LP], tw[y]);
    }
}

// Most threads of a launch's blocks, transforms of length L.  Up to 64 cells 128 threads
// cover a pass in one round (1024 x 64: 52 us, 55 with 256).  Beyond, with at most one block
// per SM latency is all that counts: 512.  With more, registers (64 to 80 a thread) decide how many of the blocks that
// fit the shared memory are resident: 384 threads where a block's buffers exceed `wide`
// bytes, 256 otherwise (whole calls with rows of 512, 384 and 256 threads: 1000 x 400
// 110, 105, 107, 500 x 500 68, 65, 72; with columns: 1000 x 1000 247, 244, 254, 800 x 640 127, 125, 118 us).
int most_threads(int L, int blocks, int nsm, size_t smem, size_t wide) {
    return L <= 64 ? 128 : blocks <= nsm ? kThreads : smem > wide ? 384 : 256;
}

// Rows: C2R along x keeping nx cells, B_demag to b (SoA FP32).
__global__ void __launch_bounds__(kThreads) k_na_rows_inverse(int nx, int ny, const cx<float>* __restrict__ X,
                                                              const cx<float>* __restrict__ twp,
                                                              const cx<float>* __restrict__ tw, FftPlan plan,
                                                              float* __restrict__ b) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int L = nx, K1 = nx + 1, L2 = 2 * nx, G = kT + (kT + 1) / 2, P = (kT + 1) / 2, n = nx * ny;
    const int LP = plan.stride();
    cx<float>* A = reinterpret_cast<cx<float>*>(smem_raw);
    cx<float>* B = A + 2 * G * LP;
    const int j0 = blockIdx.x * kT;
    auto xval = [&](int c, int k, int j) -> cx<float> {
        if (k <= nx) return X[(c * K1 + k) * ny + j];
        return conjc(X[(c * K1 + (L2 - k)) * ny + j]);
    };
    for (int e = threadIdx.x; e < L2 * kT; e += blockDim.x) {
        const int r = e % kT, k = e / kT, j = j0 + r;
        cx<float> z = mkc(0.f, 0.f);
        if (j < ny) {
            const cx<float> bx = xval(0, k, j), by = xval(1, k, j);
            z = mkc(bx.re - by.im, bx.im + by.re);
        }
        A[(2 * r + (k & 1)) * LP + plan.at(k >> 1)] = z;
    }
    for (int e = threadIdx.x; e < L2 * P; e += blockDim.x) {
        const int p = e % P, k = e / P;
        const int ja = j0 + 2 * p, jb = ja + 1;
        const cx<float> za = ja < ny ? xval(2, k, ja) : mkc(0.f, 0.f);
        const cx<float> zb = (2 * p + 1 < kT && jb < ny) ? xval(2, k, jb) : mkc(0.f, 0.f);
        A[(2 * (kT + p) + (k & 1)) * LP + plan.at(k >> 1)] = mkc(za.re - zb.im, za.im + zb.re);
    }
    __syncthreads();
    cx<float>* res = fft_smem<float, true>(A, B, 2 * G, plan, twp, tw);
    for (int e = threadIdx.x; e < G * L; e += blockDim.x) {
        const int g = e / L, x = e - g * L;
        const cx<float> z = res[(2 * g) * LP + plan.at(x)] + cmulc(res[(2 * g + 1) * LP + plan.at(x)], tw[x]);
        if (g < kT) {
            const int j = j0 + g;
            if (j < ny) {
                b[j * nx + x] = z.re;
                b[n + j * nx + x] = z.im;
            }
        } else {
            const int ja = j0 + 2 * (g - kT), jb = ja + 1;
            if (ja < ny) b[2 * n + ja * nx + x] = z.re;
            if (2 * (g - kT) + 1 < kT && jb < ny) b[2 * n + jb * nx + x] = z.im;
        }
    }
}

// Per-device set-up: device address of the static scratch (with the device
// current) and the shared-memory opt-in of the three kernels.  It runs on the
// first call on a device, and again when the opt-in is gone (after
// cudaDeviceReset the device has a new context: the static array is reloaded,
// possibly at another address, and the kernels' attributes are back at their
// defaults), so a cached address never outlives the context it came from.
int setup(int dev, void** out, void** tables) {
    std::lock_guard<std::mutex> lock(g_setup_mutex);
    const int smax = 227 * 1024;
    if (g_scratch_addr[dev]) {
        cudaFuncAttributes fa;
        if (cudaFuncGetAttributes(&fa, k_na_rows_forward) == cudaSuccess && fa.maxDynamicSharedSizeBytes >= smax) {
            *out = g_scratch_addr[dev];
            *tables = g_tables_addr[dev];
            return LLG_OK;
        }
        cudaGetLastError();
        g_scratch_addr[dev] = nullptr;
    }
    void* ptr = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&ptr, g_scratch);
    if (e != cudaSuccess || !ptr) return LLG_ERR_CUDA;
    void* tab = nullptr;
    e = cudaGetSymbolAddress(&tab, g_pass_tables);
    if (e != cudaSuccess || !tab) return LLG_ERR_CUDA;
    if (cudaFuncSetAttribute(k_na_rows_forward, cudaFuncAttributeMaxDynamicSharedMemorySize, smax) != cudaSuccess ||
        cudaFuncSetAttribute(k_na_rows_inverse, cudaFuncAttributeMaxDynamicSharedMemorySize, smax) != cudaSuccess ||
        cudaFuncSetAttribute(k_na_column, cudaFuncAttributeMaxDynamicSharedMemorySize, smax) != cudaSuccess)
        return LLG_ERR_CUDA;
    int nsm = 148;
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    g_sm_count[dev] = nsm;
    g_scratch_addr[dev] = ptr;
    g_tables_addr[dev] = tab;
    *out = ptr;
    *tables = tab;
    return LLG_OK;
}

}  // namespace noalloc
}  // namespace llg

extern "C" int llg_demag_field_noalloc(int64_t nx, int64_t ny, double ms, const float* m, const double* kernel_planes,
                                       float* b_out, void* stream) {
    using namespace llg;
    using namespace llg::noalloc;
    char msg[256];
    auto fail = [&](int code, const char* text) {
        std::snprintf(msg, sizeof(msg), "llg_demag_field_noalloc: %s", text);
        llg_set_error_message(msg);
        return code;
    };
    if (!m || !kernel_planes || !b_out) return fail(LLG_ERR_INVALID, "null pointer");
    if (nx < 1 || ny < 1 || nx > 2048 || ny > 2048) return fail(LLG_ERR_INVALID, "nx and ny must lie in [1, 2048]");
    const size_t xbytes = align256(sizeof(cx<float>) * 3 * (size_t)(nx + 1) * (size_t)ny);
    const size_t twr = align256(sizeof(cx<float>) * 2 * (size_t)nx);
    const size_t twc = align256(sizeof(cx<float>) * 2 * (size_t)ny);
    if (xbytes + twr + twc > kScratchBytes)
        return fail(LLG_ERR_INVALID, "film too large for the 32 MiB static scratch (24*(nx+1)*ny + 16*(nx+ny) bytes)");
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices)
        return fail(LLG_ERR_CUDA, "no current CUDA device");
    void* base = nullptr;
    void* tables = nullptr;
    if (setup(dev, &base, &tables) != LLG_OK) return fail(LLG_ERR_CUDA, "static scratch set-up failed");
    unsigned char* b8 = static_cast<unsigned char*>(base);
    cx<float>* X = reinterpret_cast<cx<float>*>(b8);
    cx<float>* tw_row = reinterpret_cast<cx<float>*>(b8 + xbytes);
    cx<float>* tw_col = reinterpret_cast<cx<float>*>(b8 + xbytes + twr);
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const int inx = (int)nx, iny = (int)ny;
    const int G = kT + (kT + 1) / 2;
    const FftPlan prow = padded_plan(make_plan(inx), false, 4 * G, 227 * 1024);
    const FftPlan pcol = padded_plan(make_plan(iny), false, 12, 227 * 1024);
    cx<float>* pass_row = static_cast<cx<float>*>(tables);
    cx<float>* pass_col = pass_row + 2 * kMaxLen;
    const size_t smem_row = 4 * (size_t)G * prow.stride() * sizeof(cx<float>);
    const size_t smem_col = 12 * (size_t)pcol.stride() * sizeof(cx<float>);
    const int row_blocks = (iny + kT - 1) / kT;
    const int nsm = g_sm_count[dev];
    const int row_threads = fft_block_threads(prow, 2 * G, 6 * kT, most_threads(inx, row_blocks, nsm, smem_row, 45 * 1024));
    const int col_threads = fft_block_threads(pcol, 6, 8, most_threads(iny, inx + 1, nsm, smem_col, 75 * 1024));
    k_na_twiddles<<<(4 * inx + 4 * iny + 255) / 256, 256, 0, s>>>(tw_row, inx, tw_col, iny, Plans{{prow, pcol}},
                                                                 pass_row, pass_col);
    k_na_rows_forward<<<row_blocks, row_threads, smem_row, s>>>(inx, iny, (float)ms, m, X, pass_row, tw_row, prow);
    k_na_column<<<inx + 1, col_threads, smem_col, s>>>(inx, iny, kernel_planes, 1.0 / (4.0 * (double)nx * (double)ny),
                                                       X, pass_col, tw_col, pcol);
    k_na_rows_inverse<<<row_blocks, row_threads, smem_row, s>>>(inx, iny, X, pass_row, tw_row, prow, b_out);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        std::snprintf(msg, sizeof(msg), "llg_demag_field_noalloc: launch failed: %s", cudaGetErrorString(e));
        llg_set_error_message(msg);
        return LLG_ERR_CUDA;
    }
    return LLG_OK;
}
