// The FC-fit loss path of the adjoint (tvbg_fcfit_loss, below) and its
// product dL/dZ = Z A alone (tvbg_fcfit_zgrad).
//
// dL/dZ = Z A of the FC-fit loss, per instance: Z [T][N] (the normalised,
// centred series), A [N][N] (2 (FC - target) / P with a zero diagonal),
// FP32.  A batched tiled product on the CUDA cores: one CTA per 64 x 64
// output tile of one instance, 256 threads of 4 x 4 outputs each, the A and
// Z panels staged through shared memory 16 columns at a time.  It is a sum
// over the N nodes per sample (the loss's reductions over time, the FC
// itself, stay FP64 in the caller).
#include "tvbg_abi_internal.h"
#include "tvbg_gram.cuh"

namespace {

constexpr int kTM = 64, kTN = 64, kTK = 16;

__global__ void __launch_bounds__(256)
    fcgrad_kernel(const float* __restrict__ Z, const float* __restrict__ A, float* __restrict__ out,
                  int T, int N) {
    __shared__ float sZ[kTK][kTM + 4];  // [k][t]
    __shared__ float sA[kTK][kTN];      // [k][j]
    const int b = blockIdx.z;
    const int t0 = blockIdx.y * kTM, j0 = blockIdx.x * kTN;
    const float* Zb = Z + static_cast<size_t>(b) * T * N;
    const float* Ab = A + static_cast<size_t>(b) * N * N;
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;  // 16 x 16 threads, 4 x 4 outputs each
    float acc[4][4] = {};
    for (int k0 = 0; k0 < N; k0 += kTK) {
        // Z panel: 64 rows (t) x 16 columns (k); A panel: 16 rows (k) x 64 columns (j)
        for (int i = threadIdx.x; i < kTM * kTK; i += 256) {
            const int r = i / kTK, c = i % kTK;
            const int t = t0 + r, k = k0 + c;
            sZ[c][r] = (t < T && k < N) ? __ldg(Zb + static_cast<size_t>(t) * N + k) : 0.0f;
        }
        for (int i = threadIdx.x; i < kTK * kTN; i += 256) {
            const int r = i / kTN, c = i % kTN;
            const int k = k0 + r, j = j0 + c;
            sA[r][c] = (k < N && j < N) ? __ldg(Ab + static_cast<size_t>(k) * N + j) : 0.0f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kTK; ++k) {
            float z[4], a[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                z[u] = sZ[k][ty * 4 + u];
                a[u] = sA[k][tx * 4 + u];
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int v = 0; v < 4; ++v) acc[u][v] = fmaf(z[u], a[v], acc[u][v]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int t = t0 + ty * 4 + u;
        if (t >= T) continue;
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            const int j = j0 + tx * 4 + v;
            if (j < N) out[static_cast<size_t>(b) * T * N + static_cast<size_t>(t) * N + j] = acc[u][v];
        }
    }
}

}  // namespace

extern "C" int tvbg_fcfit_zgrad(const float* d_z, const float* d_a, float* d_out, int32_t n_inst,
                               int32_t T, int32_t N, void* stream) {
    if (n_inst < 0 || T < 0 || N < 0 || n_inst > 65535 ||
        (static_cast<long long>(n_inst) * T * N > 0 && (!d_z || !d_a || !d_out)))
        return tvbg::set_error(TVBG_EINVAL, "tvbg_fcfit_zgrad: bad arguments");
    if (n_inst == 0 || T == 0 || N == 0) return TVBG_OK;
    const dim3 grid((N + kTN - 1) / kTN, (T + kTM - 1) / kTM, n_inst);
    if (grid.y > 65535u) return tvbg::set_error(TVBG_EINVAL, "tvbg_fcfit_zgrad: T too large");
    fcgrad_kernel<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(d_z, d_a, d_out, T, N);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? TVBG_OK : tvbg::set_cuda_error(e, "tvbg_fcfit_zgrad launch");
}

// ---------------------------------------------------------------------------
// The whole FC-fit loss path (tvbg_fcfit_loss): for instance b, the series
// X_b [T][N] (rows 0..T-2 from x, row T-1 from `last` when given), its
// Pearson FC in FP64, the loss mean_{i<j} (FC_ij - F*_ij)^2 and
// dL/dX = (Z A - Z diag(FC A)) / nrm, Z = (X - mean) / nrm, A = 2 (FC - F*) / P
// with a zero diagonal (P = N (N - 1) / 2).  Kernels: means and the centred
// Gram to FP64 accuracy (tvbg_gram.cuh); per instance the norms from the Gram's
// diagonal, FC, loss, A and diag(FC A) (the chain rule's time reduction
// sum_t Z_ti (Z A)_ti, taken from FC in FP64); dL/dX in FP32 (Z A is a sum
// over N nodes per sample, the precision of the backward).  The Pearson FC
// restates refs/covar.c:70-109 / metric.py:111-139 as a two-pass sum
// (centred Gram of the centred series) accurate to FP64 level.
// ---------------------------------------------------------------------------

namespace {

using tvbg::SeriesView;

// FP64 means and the centred Gram (tvbg_gram.cuh), both triangles written.
// Pass per adjoint at N = 84, 256 instances, 2000 samples: 1.54 ms with FP32
// error-free products on the FP32 pipe and 0.31 for the means before.
struct GramOut {
    double* g;       // the instance's [N][N]
    double* mean;    // the instance's [N]
    int N;
    __device__ __forceinline__ void put(int i, int j, double x, bool first) const {
        double* p = g + static_cast<int64_t>(i) * N + j;
        const double s = first ? x : *p + x;
        *p = s;
        g[static_cast<int64_t>(j) * N + i] = s;
    }
};

// N <= ROWS: one CTA per instance.
template <int ROWS>
__global__ void __launch_bounds__(tvbg::kGramThreads) fcfit_gram_kernel(SeriesView v, double* mean, double* G) {
    extern __shared__ __align__(16) unsigned char gram_smem[];
    __shared__ tvbg::GramNode nodes[ROWS];
    __shared__ double scale[ROWS];
    const int b = blockIdx.x;
    const GramOut out{G + static_cast<int64_t>(b) * v.N * v.N, mean + static_cast<int64_t>(b) * v.N, v.N};
    tvbg::gram_whole<ROWS>(
        v, b, [=](int i, double m) { out.mean[i] = m; },
        [=](int i, int j, double g, bool first) { out.put(i, j, g, first); },
        reinterpret_cast<__nv_bfloat16*>(gram_smem), nodes, scale);
}

// Larger N: one CTA per 64 x 64 tile of the upper triangle (blockIdx.y).
__global__ void __launch_bounds__(tvbg::kGramThreads) fcfit_gram_tiles_kernel(SeriesView v, double* mean, double* G) {
    extern __shared__ __align__(16) unsigned char gram_smem[];
    __shared__ tvbg::GramNode nodes[128];
    __shared__ double scale[128];
    const int b = blockIdx.x;
    const GramOut out{G + static_cast<int64_t>(b) * v.N * v.N, mean + static_cast<int64_t>(b) * v.N, v.N};
    tvbg::gram_pair(
        v, b, blockIdx.y, [=](int i, double m) { out.mean[i] = m; },
        [=](int i, int j, double g, bool first) { out.put(i, j, g, first); },
        reinterpret_cast<__nv_bfloat16*>(gram_smem), nodes, scale);
}

// Per instance (one CTA): nrm_i = sqrt(G_ii) (the centred sum of squares);
// FC_ij = G_ij / (nrm_i nrm_j) in place; loss_b = sum_{i<j} (FC - F*)^2 / P;
// A = 2 (FC - F*) / P with a zero diagonal (FP32 copy for Z A);
// zg_i = sum_j FC_ij A_ij (FP64); and the FP32 factors of the dL/dX
// epilogue per node: mean, 1 / nrm, zg / nrm (rounded once from FP64).
__global__ void __launch_bounds__(256) fcfit_loss_kernel(double* fc, const double* __restrict__ target,
                                                         int N, const double* __restrict__ mean,
                                                         double* nrm, double* loss, float* a32,
                                                         double* zg, float* fs) {
    __shared__ double red[256];
    const int b = blockIdx.x;
    const double P = 0.5 * static_cast<double>(N) * (N - 1);
    double* fb = fc + static_cast<int64_t>(b) * N * N;
    double* nb = nrm + static_cast<int64_t>(b) * N;
    float* ab = a32 + static_cast<int64_t>(b) * N * N;
    for (int i = threadIdx.x; i < N; i += blockDim.x) nb[i] = sqrt(fb[static_cast<int64_t>(i) * N + i]);
    __syncthreads();
    double part = 0.0;
    for (int64_t k = threadIdx.x; k < static_cast<int64_t>(N) * N; k += blockDim.x) {
        const int i = static_cast<int>(k / N), j = static_cast<int>(k % N);
        const double r = fb[k] / (nb[i] * nb[j]);
        fb[k] = r;
        const double d = r - target[k];
        if (j > i) part = fma(d, d, part);
        ab[k] = i == j ? 0.0f : static_cast<float>(2.0 * d / P);
    }
    red[threadIdx.x] = part;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if (static_cast<int>(threadIdx.x) < s) red[threadIdx.x] += red[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0) loss[b] = red[0] / P;
    for (int i = threadIdx.x; i < N; i += blockDim.x) {
        double s = 0.0;
        for (int j = 0; j < N; ++j) {
            if (j == i) continue;
            const double d = fb[static_cast<int64_t>(i) * N + j] - target[static_cast<int64_t>(i) * N + j];
            s = fma(fb[static_cast<int64_t>(i) * N + j], 2.0 * d / P, s);
        }
        const int64_t bi = static_cast<int64_t>(b) * N + i;
        zg[bi] = s;
        fs[3 * bi] = static_cast<float>(mean[bi]);
        fs[3 * bi + 1] = static_cast<float>(1.0 / nb[i]);
        fs[3 * bi + 2] = static_cast<float>(s / nb[i]);
    }
}

// dL/dX_tj = ((Z A)_tj - Z_tj zg_j) / nrm_j with Z = (x - mean) / nrm formed
// on the fly in FP32 (the backward's precision); the tiled FP32 product of
// fcgrad_kernel with that epilogue.
// Grid (instance, sample tile, node tile), instances fastest.
__global__ void __launch_bounds__(256)
    fcfit_dx_kernel(SeriesView v, const float* __restrict__ fs, const float* __restrict__ A,
                    float* __restrict__ dx, int64_t dxs) {
    __shared__ float sZ[kTK][kTM + 4];  // [k][t]
    __shared__ float sA[kTK][kTN];      // [k][j]
    const int b = blockIdx.x;
    const int T = v.T, N = v.N;
    const int t0 = blockIdx.y * kTM, j0 = blockIdx.z * kTN;
    const float* fb = fs + static_cast<int64_t>(b) * N * 3;   // [N][mean, 1/nrm, zg/nrm]
    const float* Ab = A + static_cast<size_t>(b) * N * N;
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
    float acc[4][4] = {};
    for (int k0 = 0; k0 < N; k0 += kTK) {
        for (int i = threadIdx.x; i < kTM * kTK; i += 256) {
            const int r = i / kTK, c = i % kTK;
            const int t = t0 + r, k = k0 + c;
            sZ[c][r] = (t < T && k < N) ? (v.at(b, t, k) - fb[3 * k]) * fb[3 * k + 1] : 0.0f;
        }
        for (int i = threadIdx.x; i < kTK * kTN; i += 256) {
            const int r = i / kTN, c = i % kTN;
            const int k = k0 + r, j = j0 + c;
            sA[r][c] = (k < N && j < N) ? __ldg(Ab + static_cast<size_t>(k) * N + j) : 0.0f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kTK; ++k) {
            float z[4], a[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                z[u] = sZ[k][ty * 4 + u];
                a[u] = sA[k][tx * 4 + u];
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int w = 0; w < 4; ++w) acc[u][w] = fmaf(z[u], a[w], acc[u][w]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int t = t0 + ty * 4 + u;
        if (t >= T) continue;
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            const int j = j0 + tx * 4 + w;
            if (j >= N) continue;
            const float z = (v.at(b, t, j) - fb[3 * j]) * fb[3 * j + 1];
            dx[b * dxs + static_cast<int64_t>(t) * N + j] =
                fmaf(-z, fb[3 * j + 2], acc[u][w] * fb[3 * j + 1]);
        }
    }
}

// The same product for N <= 16 WN, whole rows: CTA = (instance blockIdx.x,
// 64 samples blockIdx.y), A_b [N][16 WN] and the Z tile [64][N + 1] staged
// in shared memory once; thread (tx, ty) of 16 x 16 owns samples 4 ty .. +3
// and nodes tx + 16 w.  Sums over k in order, as fcfit_dx_kernel: the same
// results.
template <int WN>
__global__ void __launch_bounds__(256)
    fcfit_dx_rows_kernel(SeriesView v, const float* __restrict__ fs, const float* __restrict__ A,
                         float* __restrict__ dx, int64_t dxs) {
    extern __shared__ float sm[];
    constexpr int NP = 16 * WN;
    const int b = blockIdx.x;
    const int T = v.T, N = v.N;
    const int t0 = blockIdx.y * 64;
    float* sA = sm;             // [N][NP]
    float* sZ = sm + N * NP;    // [64][N + 1]
    const int zs = N + 1;
    const float* fb = fs + static_cast<int64_t>(b) * N * 3;
    const float* Ab = A + static_cast<size_t>(b) * N * N;
    for (int e = threadIdx.x; e < N * NP; e += 256) {
        const int k = e / NP, j = e % NP;
        sA[e] = j < N ? __ldg(Ab + static_cast<size_t>(k) * N + j) : 0.0f;
    }
    for (int e = threadIdx.x; e < 64 * N; e += 256) {
        const int r = e / N, k = e % N;
        const int t = t0 + r;
        sZ[r * zs + k] = t < T ? (v.at(b, t, k) - fb[3 * k]) * fb[3 * k + 1] : 0.0f;
    }
    __syncthreads();
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
    float acc[4][WN] = {};
    for (int k = 0; k < N; ++k) {
        float z[4], a[WN];
#pragma unroll
        for (int u = 0; u < 4; ++u) z[u] = sZ[(ty * 4 + u) * zs + k];
#pragma unroll
        for (int w = 0; w < WN; ++w) a[w] = sA[k * NP + tx + 16 * w];
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int w = 0; w < WN; ++w) acc[u][w] = fmaf(z[u], a[w], acc[u][w]);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int t = t0 + ty * 4 + u;
        if (t >= T) continue;
#pragma unroll
        for (int w = 0; w < WN; ++w) {
            const int j = tx + 16 * w;
            if (j >= N) continue;
            const float z = sZ[(ty * 4 + u) * zs + j];
            dx[b * dxs + static_cast<int64_t>(t) * N + j] =
                fmaf(-z, fb[3 * j + 2], acc[u][w] * fb[3 * j + 1]);
        }
    }
}

template <int WN>
int launch_dx_rows(SeriesView v, const float* fs, const float* A, float* dx, int64_t dxs, int n_inst,
                   cudaStream_t st) {
    const size_t smem = 4u * (static_cast<size_t>(v.N) * 16 * WN + 64u * (v.N + 1));
    if (smem > 48u * 1024u) {
        const cudaError_t e = cudaFuncSetAttribute(reinterpret_cast<const void*>(fcfit_dx_rows_kernel<WN>),
                                                   cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   static_cast<int>(smem));
        if (e != cudaSuccess) return tvbg::set_cuda_error(e, "tvbg_fcfit_loss: smem attribute");
    }
    const dim3 grid(static_cast<unsigned>(n_inst), static_cast<unsigned>((v.T + 63) / 64));
    fcfit_dx_rows_kernel<WN><<<grid, 256, smem, st>>>(v, fs, A, dx, dxs);
    return TVBG_OK;
}

}  // namespace

extern "C" int tvbg_fcfit_scratch_bytes(int32_t n_inst, int32_t N, int64_t* bytes) {
    if (!bytes || n_inst <= 0 || N <= 0) return tvbg::set_error(TVBG_EINVAL, "tvbg_fcfit_scratch_bytes: bad args");
    const int64_t nn = static_cast<int64_t>(N) * N, in = static_cast<int64_t>(n_inst);
    // mean, nrm, zg [I][N] FP64; FC [I][N][N] FP64; A [I][N][N] FP32; the
    // epilogue factors [I][N][3] FP32 (each 256-byte aligned)
    auto al = [](int64_t x) { return (x + 255) & ~static_cast<int64_t>(255); };
    *bytes = 3 * al(in * N * 8) + al(in * nn * 8) + al(in * nn * 4) + al(in * N * 12);
    return TVBG_OK;
}

extern "C" int tvbg_fcfit_loss(const float* d_x, int64_t x_inst_stride, const float* d_last,
                               int64_t last_inst_stride, int64_t last_node_stride, int32_t lanes,
                               int32_t n_inst, int32_t T, int32_t N, const double* d_target,
                               double* d_loss, float* d_dx, int64_t dx_inst_stride, double* d_fc,
                               void* d_scratch, void* stream) {
    return tvbg_fcfit_loss_ex(d_x, x_inst_stride, 1, d_last, last_inst_stride, last_node_stride, lanes, n_inst, T,
                              N, d_target, d_loss, d_dx, dx_inst_stride, d_fc, d_scratch, stream);
}

extern "C" int tvbg_fcfit_loss_ex(const float* d_x, int64_t x_inst_stride, int32_t x_cols, const float* d_last,
                                  int64_t last_inst_stride, int64_t last_node_stride, int32_t lanes,
                                  int32_t n_inst, int32_t T, int32_t N, const double* d_target,
                                  double* d_loss, float* d_dx, int64_t dx_inst_stride, double* d_fc,
                                  void* d_scratch, void* stream) {
    if (!d_x || !d_target || !d_loss || !d_scratch || n_inst <= 0 || n_inst > 65535 || T < 2 ||
        N < 2 || x_inst_stride < 0 || x_cols < 1 || x_cols > 1024 || lanes < 1 || lanes > 8 ||
        (d_dx && dx_inst_stride < static_cast<int64_t>(T) * N))
        return tvbg::set_error(TVBG_EINVAL, "tvbg_fcfit_loss: bad arguments (need T >= 2, N >= 2)");
    const int64_t nn = static_cast<int64_t>(N) * N, in = static_cast<int64_t>(n_inst);
    auto al = [](int64_t x) { return (x + 255) & ~static_cast<int64_t>(255); };
    char* s = static_cast<char*>(d_scratch);
    double* mean = reinterpret_cast<double*>(s);
    double* nrm = reinterpret_cast<double*>(s + al(in * N * 8));
    double* zg = reinterpret_cast<double*>(s + 2 * al(in * N * 8));
    double* fc = d_fc ? d_fc : reinterpret_cast<double*>(s + 3 * al(in * N * 8));
    float* a32 = reinterpret_cast<float*>(s + 3 * al(in * N * 8) + al(in * nn * 8));
    float* fsc = reinterpret_cast<float*>(s + 3 * al(in * N * 8) + al(in * nn * 8) + al(in * nn * 4));
    SeriesView v{d_x, x_inst_stride, d_last, last_inst_stride, last_node_stride, T, N, lanes, x_cols};
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if ((T + 63) / 64 > 65535) return tvbg::set_error(TVBG_EINVAL, "tvbg_fcfit_loss: T too large");
    const int64_t nt = (N + 63) / 64;
    if (N > 128 && nt * (nt + 1) / 2 > 65535)
        return tvbg::set_error(TVBG_EINVAL, "tvbg_fcfit_loss: N too large");
    {
        const bool whole = N <= 128, half = N <= 96;
        auto kfn = half ? fcfit_gram_kernel<96> : whole ? fcfit_gram_kernel<128> : fcfit_gram_tiles_kernel;
        const size_t smem = tvbg::gram_plane_bytes(half ? 96 : 128);
        const cudaError_t e = cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   static_cast<int>(smem));
        if (e != cudaSuccess) return tvbg::set_cuda_error(e, "tvbg_fcfit_loss: smem attribute");
        kfn<<<dim3(n_inst, whole ? 1 : static_cast<unsigned>(nt * (nt + 1) / 2)), tvbg::kGramThreads, smem, st>>>(
            v, mean, fc);
    }
    fcfit_loss_kernel<<<n_inst, 256, 0, st>>>(fc, d_target, N, mean, nrm, d_loss, a32, zg, fsc);
    if (d_dx) {
        int rc = TVBG_OK;
        if (N <= 32) rc = launch_dx_rows<2>(v, fsc, a32, d_dx, dx_inst_stride, n_inst, st);
        else if (N <= 64) rc = launch_dx_rows<4>(v, fsc, a32, d_dx, dx_inst_stride, n_inst, st);
        else if (N <= 96) rc = launch_dx_rows<6>(v, fsc, a32, d_dx, dx_inst_stride, n_inst, st);
        else if (N <= 128) rc = launch_dx_rows<8>(v, fsc, a32, d_dx, dx_inst_stride, n_inst, st);
        else {
            const dim3 grid(n_inst, (T + kTM - 1) / kTM, (N + kTN - 1) / kTN);
            if (grid.z > 65535u) return tvbg::set_error(TVBG_EINVAL, "tvbg_fcfit_loss: N too large");
            fcfit_dx_kernel<<<grid, 256, 0, st>>>(v, fsc, a32, d_dx, dx_inst_stride);
        }
        if (rc != TVBG_OK) return rc;
    }
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? TVBG_OK : tvbg::set_cuda_error(e, "tvbg_fcfit_loss launch");
}
