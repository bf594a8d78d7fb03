// Streaming (online) covariance per instance with FP64 Welford updates, and
// its Pearson correlation.
//
// Restates the online co-moment of tvb_hpc/metric.py:87-108 (OnlineCov) and
// dsl/dsl_cuda/CUDAmodels/refs/covar.c:9-68 (update_cov), in FP64 and with
// the Welford form of the update: for the (n+1)-th sample x,
//   d_i    = x_i - mean_i
//   mean_i += d_i / (n + 1)
//   m2_ij  += d_i (x_j - mean_j')          (mean' the updated mean)
// so after n samples m2 is the co-moment sum_s (x_si - m_i)(x_sj - m_j) and
// corr_ij = m2_ij / sqrt(m2_ii m2_jj) (covar.c:73-109, whose 1/n
// normalisation cancels in the ratio).  The increments are symmetric
// (x_j - mean_j' = d_j n / (n + 1)), so the upper triangle is computed, in
// 32 x 32 tiles, and written to both.
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>

#include "tvbg_abi_internal.h"

namespace tvbg {

constexpr int kCovThreads = 256;
constexpr int kCovTile = 32;
// static shared memory of cov_update_kernel: its transposing tile
constexpr size_t kCovStaticBytes = sizeof(double) * kCovTile * (kCovTile + 1);
constexpr int kCovNodes = 3000;                     // largest network
constexpr int64_t kCovPassBytes = 192 * 1024;       // a pass's d and e, at least four samples
// the most dynamic shared memory of a launch: the limit that every launch asks
// for (another thread's smaller one may come between that and the launch)
constexpr size_t kCovSmemMax = sizeof(double) * kCovNodes + (kCovPassBytes > 64 * kCovNodes ? kCovPassBytes : 64 * kCovNodes);
static_assert(kCovSmemMax + kCovStaticBytes <= 227 * 1024, "shared memory of a CTA");

// Tile (ti <= tj) q of the upper triangle of nt x nt tiles, row-major.
__device__ __forceinline__ void cov_tile(int q, int nt, int& ti, int& tj) {
    ti = 0;
    while (q >= nt - ti) {
        q -= nt - ti;
        ++ti;
    }
    tj = ti + q;
}

// `rows` samples folded in order, RC at a time: the samples' d and x - mean'
// of every node in shared memory, then each entry of m2 takes the RC products
// between one read and one write.  CTA (blockIdx.x of gridDim.x, instance
// blockIdx.y) takes every gridDim.x-th tile; with one CTA per instance it also
// stores the means, else cov_mean_kernel does after it.
// FP64 products bound it (two per SM and clock): 8 samples of 256 x 84 nodes take
// 7.3 M of them, 12 us, where a launch per sample took 8 x 11.3.
__global__ void __launch_bounds__(kCovThreads)
    cov_update_kernel(const float* __restrict__ x, long long inst_stride, long long row_stride, int rows, int RC,
                      int N, long long n, double* __restrict__ mean, double* __restrict__ m2) {
    extern __shared__ double sh[];  // mean[N] | d[RC][N] | e[RC][N]
    __shared__ double tr[kCovTile][kCovTile + 1];
    double* m = sh;
    double* d = sh + N;
    double* e = d + static_cast<size_t>(RC) * N;
    const long long b = blockIdx.y;
    const float* xb = x + b * inst_stride;
    double* mb = mean + b * N;
    double* cb = m2 + b * static_cast<long long>(N) * N;
    const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
    const int nt = (N + kCovTile - 1) / kCovTile;
    for (int i = threadIdx.x; i < N; i += kCovThreads) m[i] = n == 0 ? 0.0 : mb[i];
    for (int r0 = 0; r0 < rows; r0 += RC) {
        const int rc = rows - r0 < RC ? rows - r0 : RC;
        for (int i = threadIdx.x; i < N; i += kCovThreads) {
            double mi = m[i];
            for (int r = 0; r < rc; ++r) {
                const double xi = static_cast<double>(__ldg(xb + (r0 + r) * row_stride + i));
                const double di = xi - mi;
                mi = mi + di * (1.0 / static_cast<double>(n + r0 + r + 1));
                d[r * N + i] = di;
                e[r * N + i] = xi - mi;
            }
            m[i] = mi;
        }
        __syncthreads();
        const bool start = n + r0 == 0;   // the first sample starts the co-moment
        for (int q = blockIdx.x; q < nt * (nt + 1) / 2; q += gridDim.x) {
            int ti, tj;
            cov_tile(q, nt, ti, tj);
            const int j = tj * kCovTile + lane;
#pragma unroll
            for (int u = 0; u < kCovTile / 8; ++u) {
                const int k = warp + 8 * u, i = ti * kCovTile + k;
                if (i < N && j < N && i <= j) {
                    double* p = cb + static_cast<long long>(i) * N + j;
                    double a = start ? 0.0 : *p;
                    for (int r = 0; r < rc; ++r) a = fma(d[r * N + i], e[r * N + j], a);
                    *p = a;
                    tr[k][lane] = a;
                }
            }
            __syncthreads();
#pragma unroll
            for (int u = 0; u < kCovTile / 8; ++u) {
                const int k = warp + 8 * u;
                const int i = ti * kCovTile + lane, jj = tj * kCovTile + k;   // entry (jj, i)
                if (i < jj && jj < N) cb[static_cast<long long>(jj) * N + i] = tr[lane][k];
            }
            __syncthreads();
        }
    }
    if (gridDim.x == 1)
        for (int i = threadIdx.x; i < N; i += kCovThreads) mb[i] = m[i];
}

// The means after the same samples, the same arithmetic.
__global__ void __launch_bounds__(kCovThreads)
    cov_mean_kernel(const float* __restrict__ x, long long inst_stride, long long row_stride, int rows, int N,
                    long long n, double* __restrict__ mean) {
    const long long b = blockIdx.y;
    const int i = blockIdx.x * kCovThreads + threadIdx.x;
    if (i >= N) return;
    double mi = n == 0 ? 0.0 : mean[b * N + i];
    for (int r = 0; r < rows; ++r) {
        const double di = static_cast<double>(__ldg(x + b * inst_stride + r * row_stride + i)) - mi;
        mi = mi + di * (1.0 / static_cast<double>(n + r + 1));
    }
    mean[b * N + i] = mi;
}

// One sample (updates of a running simulation): bound by the passes over m2,
// which are read and written row by row, without the mirror's transposed
// writes (300 instances of 84 nodes 17.4 -> 10.8 us, 4096 132 -> 82, 600 of 500 568 -> 398).  Entry (j, i) of the lower triangle takes the product of (i, j), so
// both kernels give the same bits.  CTA blockIdx.x of gridDim.x takes every
// gridDim.x-th run of 2048 entries; the means as in cov_update_kernel.
__global__ void __launch_bounds__(kCovThreads)
    cov_sample_kernel(const float* __restrict__ x, long long inst_stride, int N, long long n,
                      double* __restrict__ mean, double* __restrict__ m2) {
    extern __shared__ double sh[];  // d[N] | e[N]
    double* d = sh;
    double* e = sh + N;
    const long long b = blockIdx.y;
    double* mb = mean + b * N;
    double* cb = m2 + b * static_cast<long long>(N) * N;
    const double rn = 1.0 / static_cast<double>(n + 1);
    for (int i = threadIdx.x; i < N; i += kCovThreads) {
        const double mi = n == 0 ? 0.0 : mb[i];
        const double xi = static_cast<double>(__ldg(x + b * inst_stride + i));
        const double di = xi - mi;
        const double m_new = mi + di * rn;
        d[i] = di;
        e[i] = xi - m_new;
        if (gridDim.x == 1) mb[i] = m_new;
    }
    __syncthreads();
    // entries q, q + 256, ...: eight of them in flight
    constexpr int U = 8;
    const int NN = N * N, step_i = kCovThreads / N, step_j = kCovThreads % N;
    int q = blockIdx.x * (U * kCovThreads) + threadIdx.x;
    for (; q < NN; q += gridDim.x * (U * kCovThreads)) {
        double a[U];
#pragma unroll
        for (int u = 0; u < U; ++u) a[u] = n != 0 && q + u * kCovThreads < NN ? cb[q + u * kCovThreads] : 0.0;
        int i = q / N, j = q - i * N;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (q + u * kCovThreads < NN) cb[q + u * kCovThreads] = fma(d[min(i, j)], e[max(i, j)], a[u]);
            i += step_i;
            j += step_j;
            if (j >= N) {
                j -= N;
                ++i;
            }
        }
    }
}

// 32 x 32 tiles, a reciprocal square root per node of the tile and two
// products per pair (a root and a division per entry took 72 us for 256 x 84
// nodes).
__global__ void __launch_bounds__(kCovThreads)
    cov_corr_kernel(const double* __restrict__ m2, int N, float* __restrict__ corr) {
    __shared__ float tile[kCovTile][kCovTile + 1];
    __shared__ double ri[kCovTile], rj[kCovTile];
    const long long b = blockIdx.y;
    const double* cb = m2 + b * static_cast<long long>(N) * N;
    float* ob = corr + b * static_cast<long long>(N) * N;
    const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
    int ti, tj;
    cov_tile(blockIdx.x, (N + kCovTile - 1) / kCovTile, ti, tj);
    const int i0 = ti * kCovTile, j0 = tj * kCovTile;
    if (threadIdx.x < 2 * kCovTile) {
        const int k = threadIdx.x % kCovTile, v = (threadIdx.x < kCovTile ? i0 : j0) + k;
        (threadIdx.x < kCovTile ? ri : rj)[k] =
            v < N ? 1.0 / sqrt(cb[static_cast<long long>(v) * N + v]) : 0.0;
    }
    __syncthreads();
    for (int k = warp; k < kCovTile; k += 8) {
        const int i = i0 + k, j = j0 + lane;
        if (i <= j && j < N) {
            const float r = static_cast<float>(cb[static_cast<long long>(i) * N + j] * (ri[k] * rj[lane]));
            ob[static_cast<long long>(i) * N + j] = r;
            tile[k][lane] = r;
        }
    }
    __syncthreads();
    for (int k = warp; k < kCovTile; k += 8) {
        const int i = i0 + lane, j = j0 + k;   // entry (j, i)
        if (i < j && j < N) ob[static_cast<long long>(j) * N + i] = tile[lane][k];
    }
}

// Few nodes (N <= 32): a warp per instance, eight to a CTA; the arithmetic of
// cov_corr_kernel, whose CTA per instance is mostly start and synchronisation.
__global__ void __launch_bounds__(kCovThreads)
    cov_corr_small_kernel(const double* __restrict__ m2, int n_inst, int N, float* __restrict__ corr) {
    const long long b = blockIdx.x * static_cast<long long>(kCovThreads / 32) + threadIdx.x / 32;
    if (b >= n_inst) return;   // whole warps
    const int lane = threadIdx.x % 32, NN = N * N;
    const double* cb = m2 + b * NN;
    const double r = lane < N ? 1.0 / sqrt(cb[lane * N + lane]) : 0.0;
#pragma unroll 4
    for (int q0 = 0; q0 < NN; q0 += 32) {
        const int q = q0 + lane, i = q < NN ? q / N : 0, j = q < NN ? q % N : 0;
        const double ri = __shfl_sync(0xffffffffu, r, i), rj = __shfl_sync(0xffffffffu, r, j);
        if (q < NN)
            corr[b * NN + q] = static_cast<float>(cb[i <= j ? q : j * N + i] * (ri * rj));
    }
}

// Launch over all instances (gridDim.y at most 65535 at a time).
static int cov_rows(const float* x, int64_t inst_stride, int64_t row_stride, int rows, int n_inst, int N, int64_t n,
                    double* mean, double* m2, cudaStream_t st) {
    // (many instances of one tile: cov_update_kernel, 4096 of 5 nodes 15 us against 17)
    if (rows == 1 && !(N <= kCovTile && n_inst >= 600)) {
        // few instances of many nodes: about 1200 CTAs share the entries (and a
        // launch more sets the means)
        const int runs = (N * N + 8 * kCovThreads - 1) / (8 * kCovThreads);
        int parts = N <= 64 || n_inst >= 600 || (N <= 100 && n_inst >= 150) ? 1 : 1200 / n_inst;
        parts = parts > runs ? runs : parts;
        for (int b0 = 0; b0 < n_inst; b0 += 65535) {
            const unsigned nb = static_cast<unsigned>(n_inst - b0 < 65535 ? n_inst - b0 : 65535);
            const float* xb = x + b0 * inst_stride;
            double* mb = mean + static_cast<int64_t>(b0) * N;
            cov_sample_kernel<<<dim3(static_cast<unsigned>(parts), nb), kCovThreads, 2u * sizeof(double) * N, st>>>(
                xb, inst_stride, N, n, mb, m2 + static_cast<int64_t>(b0) * N * N);
            if (parts > 1)
                cov_mean_kernel<<<dim3(static_cast<unsigned>((N + kCovThreads - 1) / kCovThreads), nb), kCovThreads, 0,
                                  st>>>(xb, inst_stride, row_stride, 1, N, n, mb);
        }
        const cudaError_t e = cudaGetLastError();
        return e == cudaSuccess ? TVBG_OK : set_cuda_error(e, "tvbg_cov_update launch");
    }
    // samples per pass: as many as kCovPassBytes holds, 4 to 16
    int RC = static_cast<int>(kCovPassBytes / (16 * static_cast<int64_t>(N)));
    RC = RC > 16 ? 16 : (RC < 4 ? 4 : RC);
    if (RC > rows) RC = rows;
    const size_t smem = sizeof(double) * static_cast<size_t>(N) * (1 + 2 * RC);
    if (smem + kCovStaticBytes > 48u * 1024u) {   // the kernel's own tile counts too
        const cudaError_t e = cudaFuncSetAttribute(cov_update_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   static_cast<int>(kCovSmemMax));
        if (e != cudaSuccess) return set_cuda_error(e, "tvbg_cov_update: smem attribute");
    }
    const int nt = (N + kCovTile - 1) / kCovTile, tiles = nt * (nt + 1) / 2;
    // few instances: their tiles spread over about 1200 CTAs
    int parts = n_inst >= 600 ? 1 : 1200 / n_inst;
    parts = parts > tiles ? tiles : parts;
    for (int b0 = 0; b0 < n_inst; b0 += 65535) {
        const unsigned nb = static_cast<unsigned>(n_inst - b0 < 65535 ? n_inst - b0 : 65535);
        const float* xb = x + b0 * inst_stride;
        double* mb = mean + static_cast<int64_t>(b0) * N;
        cov_update_kernel<<<dim3(static_cast<unsigned>(parts), nb), kCovThreads, smem, st>>>(
            xb, inst_stride, row_stride, rows, RC, N, n, mb, m2 + static_cast<int64_t>(b0) * N * N);
        if (parts > 1)
            cov_mean_kernel<<<dim3(static_cast<unsigned>((N + kCovThreads - 1) / kCovThreads), nb), kCovThreads, 0,
                              st>>>(xb, inst_stride, row_stride, rows, N, n, mb);
    }
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? TVBG_OK : set_cuda_error(e, "tvbg_cov_update launch");
}

}  // namespace tvbg

using namespace tvbg;

extern "C" int tvbg_cov_update(const float* d_x, int64_t x_stride, int32_t n_inst, int32_t N,
                               int64_t n, double* d_mean, double* d_m2, void* stream) {
    return tvbg_cov_update_rows(d_x, x_stride, 0, 1, n_inst, N, n, d_mean, d_m2, stream);
}

extern "C" int tvbg_cov_update_rows(const float* d_x, int64_t x_stride, int64_t row_stride, int32_t rows,
                                    int32_t n_inst, int32_t N, int64_t n, double* d_mean, double* d_m2,
                                    void* stream) {
    if (n_inst < 0 || rows < 0 || N <= 0 || n < 0 || x_stride < N || (n_inst > 0 && (!d_x || !d_mean || !d_m2)))
        return set_error(TVBG_EINVAL, "tvbg_cov_update: bad arguments");
    if (N > kCovNodes) return set_error(TVBG_EINVAL, "tvbg_cov_update: N above 3000");
    if (n_inst == 0 || rows == 0) return TVBG_OK;
    return cov_rows(d_x, x_stride, row_stride, rows, n_inst, N, n, d_mean, d_m2,
                    static_cast<cudaStream_t>(stream));
}

extern "C" int tvbg_cov_corr(const double* d_m2, int32_t n_inst, int32_t N, float* d_corr,
                             void* stream) {
    if (n_inst < 0 || N <= 0 || (n_inst > 0 && (!d_m2 || !d_corr)))
        return set_error(TVBG_EINVAL, "tvbg_cov_corr: bad arguments");
    if (n_inst == 0) return TVBG_OK;
    // us, a warp / a tile of 32 x 32 per instance: N = 5, 600 instances 5.0 / 8.8, one 4.3 / 5.0;
    // N = 10, 64 instances 6.8 / 5.2, 600 6.8 / 8.9; N = 24, 600 instances 10.8 / 8.9, 1200 10.8 / 13.1;
    // N = 32, 4096 instances 37 / 34
    if (N <= 6 || (N <= 16 && n_inst >= 400) || (N <= 24 && n_inst >= 1000)) {
        constexpr int kPer = kCovThreads / 32;
        cov_corr_small_kernel<<<static_cast<unsigned>((static_cast<int64_t>(n_inst) + kPer - 1) / kPer), kCovThreads, 0,
                                static_cast<cudaStream_t>(stream)>>>(d_m2, n_inst, N, d_corr);
        const cudaError_t es = cudaGetLastError();
        return es == cudaSuccess ? TVBG_OK : set_cuda_error(es, "tvbg_cov_corr launch");
    }
    const long long nt = (static_cast<long long>(N) + kCovTile - 1) / kCovTile, tiles = nt * (nt + 1) / 2;
    if (tiles > 0x7fffffffLL) return set_error(TVBG_EINVAL, "tvbg_cov_corr: N too large");
    for (int b0 = 0; b0 < n_inst; b0 += 65535) {
        const unsigned nb = static_cast<unsigned>(n_inst - b0 < 65535 ? n_inst - b0 : 65535);
        const int64_t off = static_cast<int64_t>(b0) * N * N;
        cov_corr_kernel<<<dim3(static_cast<unsigned>(tiles), nb), kCovThreads, 0, static_cast<cudaStream_t>(stream)>>>(
            d_m2 + off, N, d_corr + off);
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return set_cuda_error(e, "tvbg_cov_corr launch");
    return TVBG_OK;
}
