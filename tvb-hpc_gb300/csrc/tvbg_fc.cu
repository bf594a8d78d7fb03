// Pearson functional connectivity per instance with an FP64-accurate
// reduction, and the FC-fit error against a target matrix.
//
// Restates tvb_hpc/metric.py:18-139 (Covar one-pass co-moment + CovToCorr)
// and dsl/dsl_cuda/CUDAmodels/refs/covar.c:9-109 as a two-pass method:
// means, then the centred Gram  C_ij = sum_t (x_ti - m_i)(x_tj - m_j) (exact
// products of fixed-point digits, tvbg_gram.cuh), corr_ij = C_ij / sqrt(C_ii C_jj)
// in FP64.  (The 1/n normalisation of covar.c:155-159 cancels in the ratio.)
#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>

#include "tvbg_abi_internal.h"
#include "tvbg_gram.cuh"

namespace tvbg {

constexpr int kFcSmallMax = 127;   // largest N of the one-CTA path

// Index of (i, j), i <= j, in a packed upper triangle of N rows.
__device__ __forceinline__ int packed(int i, int j, int N) { return i * N - i * (i - 1) / 2 + j - i; }

// N <= 127: one CTA per instance, the Gram in shared memory; FP64 units do
// only the normalisation, five operations a pair (a reciprocal square root
// per node, where a root and a division per pair took half of the old
// kernel's time).  4096 instances of 40 x 84 samples: 1.90 ms before.
template <int ROWS>
__global__ void __launch_bounds__(kGramThreads)
    fc_small_kernel(SeriesView v, float* __restrict__ fc, const float* __restrict__ target,
                    double* __restrict__ err) {
    extern __shared__ __align__(16) unsigned char fc_smem[];   // planes | packed Gram
    __shared__ GramNode nodes[ROWS];
    __shared__ double scale[ROWS];
    __shared__ double rn[ROWS];
    __shared__ double part[kGramThreads / 32];
    auto* planes = reinterpret_cast<__nv_bfloat16*>(fc_smem);
    auto* gram = reinterpret_cast<double*>(fc_smem + gram_plane_bytes(ROWS));
    const int N = v.N, b = blockIdx.x;
    gram_whole<ROWS>(
        v, b, [](int, double) {},
        [=](int i, int j, double g, bool first) {
            double* p = gram + packed(i, j, N);
            *p = first ? g : *p + g;
        },
        planes, nodes, scale);
    for (int i = threadIdx.x; i < N; i += kGramThreads) rn[i] = 1.0 / sqrt(gram[packed(i, i, N)]);
    __syncthreads();
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    double e_local = 0.0;
    for (int i = warp; i < N; i += kGramThreads / 32) {
        const double ri = rn[i];
        for (int j = i + lane; j < N; j += 32) {
            double* p = gram + packed(i, j, N);
            const double r = *p * (ri * rn[j]);
            if (target && i < j) {
                const double dd = r - static_cast<double>(__ldg(target + i * N + j));
                e_local = fma(dd, dd, e_local);
            }
            *reinterpret_cast<float*>(p) = static_cast<float>(r);   // read back below
        }
    }
    __syncthreads();
    float* fcb = fc + static_cast<long long>(b) * N * N;
    for (int i = warp; i < N; i += kGramThreads / 32)
        for (int j = lane; j < N; j += 32)
            fcb[i * N + j] = *reinterpret_cast<const float*>(gram + (i <= j ? packed(i, j, N) : packed(j, i, N)));
    if (err) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) e_local += __shfl_down_sync(0xffffffffu, e_local, o);
        if (lane == 0) part[warp] = e_local;
        __syncthreads();
        if (threadIdx.x == 0) {
            double e = 0.0;
            for (int k = 0; k < kGramThreads / 32; ++k) e += part[k];
            err[b] = e;
        }
    }
}

// Few nodes and short series: one CTA per instance, FP64 sums of the centred
// samples, three pairs of the upper triangle per thread.  The digit path works
// through whole tiles of 96 rows and 64 samples and costs 75 ns an instance before its first
// sample, this one 12 (us for 4096 instances, digits / FP64 sums: 10 nodes x 20 samples 384 / 72, 50 x 8 525 / 284).
constexpr int kDirectThreads = 512;
constexpr int kDirectTile = 32;
constexpr int kDirectNodes = 50;
constexpr int kDirectPairs = (kDirectNodes * (kDirectNodes + 1) / 2 + kDirectThreads - 1) / kDirectThreads;
__global__ void __launch_bounds__(kDirectThreads)
    fc_direct_kernel(const float* __restrict__ x, int T, int N, long long inst_stride, float* __restrict__ fc,
                     const float* __restrict__ target, double* __restrict__ err) {
    __shared__ double mean[kDirectNodes], rn[kDirectNodes];
    __shared__ double tile[kDirectTile][kDirectNodes];
    __shared__ double part[kDirectThreads / 32];
    const float* xb = x + blockIdx.x * inst_stride;
    const int tid = threadIdx.x, lane = tid % 32, warp = tid / 32;
    if (tid < N) {
        double s = 0.0;
#pragma unroll 8
        for (int t = 0; t < T; ++t) s += static_cast<double>(__ldg(xb + static_cast<long long>(t) * N + tid));
        mean[tid] = s / static_cast<double>(T);
    }
    const int npairs = N * (N + 1) / 2;
    double acc[kDirectPairs];
    int pi[kDirectPairs], pj[kDirectPairs];   // row-major upper triangle
#pragma unroll
    for (int q = 0; q < kDirectPairs; ++q) {
        acc[q] = 0.0;
        int i = 0, rem = tid + q * kDirectThreads;
        if (rem < npairs) {
            while (rem >= N - i) {
                rem -= N - i;
                ++i;
            }
        } else {
            rem = 0;
        }
        pi[q] = i;
        pj[q] = i + rem;
    }
    for (int t0 = 0; t0 < T; t0 += kDirectTile) {
        const int nt = T - t0 < kDirectTile ? T - t0 : kDirectTile;
        __syncthreads();
        for (int e = tid; e < nt * N; e += kDirectThreads) {
            const int tt = e / N, i = e - tt * N;
            tile[tt][i] = static_cast<double>(__ldg(xb + static_cast<long long>(t0 + tt) * N + i)) - mean[i];
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < kDirectPairs; ++q)
            if (tid + q * kDirectThreads < npairs)
                for (int tt = 0; tt < nt; ++tt) acc[q] = fma(tile[tt][pi[q]], tile[tt][pj[q]], acc[q]);
    }
#pragma unroll
    for (int q = 0; q < kDirectPairs; ++q)
        if (tid + q * kDirectThreads < npairs && pi[q] == pj[q]) rn[pi[q]] = 1.0 / sqrt(acc[q]);
    __syncthreads();
    double e_local = 0.0;
    float* fcb = fc + static_cast<long long>(blockIdx.x) * N * N;
#pragma unroll
    for (int q = 0; q < kDirectPairs; ++q)
        if (tid + q * kDirectThreads < npairs) {
            const int i = pi[q], j = pj[q];
            const double r = acc[q] * (rn[i] * rn[j]);
            fcb[i * N + j] = static_cast<float>(r);
            fcb[j * N + i] = static_cast<float>(r);
            if (target && i < j) {
                const double dd = r - static_cast<double>(__ldg(target + i * N + j));
                e_local = fma(dd, dd, e_local);
            }
        }
    if (err) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) e_local += __shfl_down_sync(0xffffffffu, e_local, o);
        if (lane == 0) part[warp] = e_local;
        __syncthreads();
        if (tid == 0) {
            double e = 0.0;
            for (int k = 0; k < kDirectThreads / 32; ++k) e += part[k];
            err[blockIdx.x] = e;
        }
    }
}

// Larger N: the upper triangle of the Gram, one CTA per 64 x 64 tile.
__global__ void __launch_bounds__(kGramThreads) fc_gram_kernel(SeriesView v, double* __restrict__ gram) {
    extern __shared__ __align__(16) unsigned char fc_smem[];
    __shared__ GramNode nodes[128];
    __shared__ double scale[128];
    const int N = v.N, b = blockIdx.y;
    double* gb = gram + static_cast<long long>(b) * N * N;
    gram_pair(
        v, b, blockIdx.x, [](int, double) {},
        [=](int i, int j, double g, bool first) {
            double* p = gb + static_cast<long long>(i) * N + j;
            *p = first ? g : *p + g;
        },
        reinterpret_cast<__nv_bfloat16*>(fc_smem), nodes, scale);
}

// Correlations from the Gram's upper triangle: tiles of 32 x 32 entries (q =
// blockIdx.x, then every gridDim.x-th), written to both triangles through
// shared memory; the CTA's error sum goes to parts[blockIdx.x].
constexpr int kNormTile = 32;
__global__ void __launch_bounds__(256)
    fc_norm_kernel(const double* __restrict__ gram, int N, int tiles, float* __restrict__ fc,
                   const float* __restrict__ target, double* __restrict__ parts, long long parts_stride) {
    __shared__ float tile[kNormTile][kNormTile + 1];
    __shared__ double ri[kNormTile], rj[kNormTile];
    __shared__ double red[8];
    const int b = blockIdx.y;
    const double* g = gram + static_cast<long long>(b) * N * N;
    float* fb = fc + static_cast<long long>(b) * N * N;
    const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
    double e = 0.0;
    for (int q = blockIdx.x; q < tiles; q += gridDim.x) {
        int it, jt;
        gram_triangle(q, (N + kNormTile - 1) / kNormTile, it, jt);
        const int i0 = it * kNormTile, j0 = jt * kNormTile;
        __syncthreads();
        if (threadIdx.x < 2 * kNormTile) {
            const int k = threadIdx.x % kNormTile;
            const int n = (threadIdx.x < kNormTile ? i0 : j0) + k;
            const double r = n < N ? 1.0 / sqrt(g[static_cast<long long>(n) * N + n]) : 0.0;
            (threadIdx.x < kNormTile ? ri : rj)[k] = r;
        }
        __syncthreads();
        for (int k = warp; k < kNormTile; k += 8) {
            const int i = i0 + k, j = j0 + lane;
            float rf = 0.0f;
            if (i <= j && j < N) {
                const double r = g[static_cast<long long>(i) * N + j] * (ri[k] * rj[lane]);
                rf = static_cast<float>(r);
                fb[static_cast<long long>(i) * N + j] = rf;
                if (target && i < j) {
                    const double dd = r - static_cast<double>(__ldg(target + static_cast<long long>(i) * N + j));
                    e = fma(dd, dd, e);
                }
            }
            tile[k][lane] = rf;
        }
        __syncthreads();
        for (int k = warp; k < kNormTile; k += 8) {
            const int i = i0 + lane, j = j0 + k;   // entry (j, i)
            if (i < j && j < N) fb[static_cast<long long>(j) * N + i] = tile[lane][k];
        }
    }
    if (parts) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) e += __shfl_down_sync(0xffffffffu, e, o);
        if (lane == 0) red[warp] = e;
        __syncthreads();
        if (threadIdx.x == 0) {
            double s = 0.0;
            for (int k = 0; k < 8; ++k) s += red[k];
            parts[b * parts_stride + blockIdx.x] = s;
        }
    }
}

// err[b] = sum of its n parts, in a fixed order.
__global__ void __launch_bounds__(256) fc_err_kernel(const double* __restrict__ parts, long long stride, int n,
                                                     double* __restrict__ err) {
    __shared__ double red[8];
    const int b = blockIdx.x, lane = threadIdx.x % 32, warp = threadIdx.x / 32;
    double e = 0.0;
    for (int k = threadIdx.x; k < n; k += 256) e += parts[b * stride + k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) e += __shfl_down_sync(0xffffffffu, e, o);
    if (lane == 0) red[warp] = e;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int k = 0; k < 8; ++k) s += red[k];
        err[b] = s;
    }
}

}  // namespace tvbg

using namespace tvbg;

namespace {
// Whether N nodes take the one-CTA small path (no scratch).
bool fc_small_path(int32_t N) { return N <= kFcSmallMax; }
// Whether the call takes FP64 sums: up to the line where an FP64 kernel had taken as
// long as the digits.  On it this one wins (us for 4096 instances, FP64 / digits:
// N = 10, T = 150 231 / 739; N = 16, T = 100 247 / 606; N = 50, T = 20 405 / 571); 64 nodes were equal
// at T = 3 already.
bool direct_is_faster(int32_t T, int32_t N) {
    return N <= kDirectNodes && static_cast<int64_t>(T) * (N * N + 300) <= 70000;
}
}  // namespace

extern "C" int tvbg_fc_scratch_bytes(int32_t n_inst, int32_t N, int64_t* bytes) {
    if (!bytes || n_inst <= 0 || N <= 0) return set_error(TVBG_EINVAL, "tvbg_fc_scratch_bytes: bad args");
    if (fc_small_path(N)) {
        *bytes = 0;
    } else {
        *bytes = static_cast<int64_t>(n_inst) * N * (static_cast<int64_t>(N) + 1) *
                 static_cast<int64_t>(sizeof(double));
    }
    return TVBG_OK;
}

// Large-N FC needs caller scratch of tvbg_fc_scratch_bytes() (FP64: an error part per
// node, and the Gram).
extern "C" int tvbg_fc_ex(const float* d_x, int32_t n_inst, int32_t T, int32_t N,
                          int64_t inst_stride, float* d_fc, const float* d_target, double* d_err,
                          double* d_scratch, void* stream) {
    if (!d_x || !d_fc || n_inst <= 0 || T < 2 || N <= 0 || inst_stride < static_cast<int64_t>(T) * N)
        return set_error(TVBG_EINVAL, "tvbg_fc: bad arguments (need T >= 2, inst_stride >= T*N)");
    if ((d_target == nullptr) != (d_err == nullptr))
        return set_error(TVBG_EINVAL, "tvbg_fc: d_target and d_err go together");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const SeriesView v{d_x, inst_stride, nullptr, 0, 0, T, N, 1, 1};
    if (direct_is_faster(T, N)) {
        fc_direct_kernel<<<n_inst, kDirectThreads, 0, st>>>(d_x, T, N, inst_stride, d_fc, d_target, d_err);
    } else if (fc_small_path(N)) {
        const bool half = N <= 96;
        const size_t smem = gram_plane_bytes(half ? 96 : 128) + sizeof(double) * (static_cast<size_t>(N) * (N + 1) / 2);
        auto kfn = half ? fc_small_kernel<96> : fc_small_kernel<128>;
        // the limit of the kernel's largest N: another thread's smaller call may
        // come between this and the launch
        const int top = half ? 96 : kFcSmallMax;
        const size_t most = gram_plane_bytes(half ? 96 : 128) + sizeof(double) * (static_cast<size_t>(top) * (top + 1) / 2);
        cudaError_t e = cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(most));
        if (e != cudaSuccess) return set_cuda_error(e, "tvbg_fc: smem attribute");
        kfn<<<n_inst, kGramThreads, smem, st>>>(v, d_fc, d_target, d_err);
    } else {
        if (!d_scratch) return set_error(TVBG_EINVAL, "tvbg_fc: N > 127 needs d_scratch (tvbg_fc_scratch_bytes)");
        // scratch: N error parts per instance, then the Gram
        double* gram = d_scratch + static_cast<long long>(n_inst) * N;
        const size_t smem = gram_plane_bytes(128);
        cudaError_t e = cudaFuncSetAttribute(fc_gram_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             static_cast<int>(smem));
        if (e != cudaSuccess) return set_cuda_error(e, "tvbg_fc: smem attribute");
        const long long nt = (N + 63) / 64, nn = (N + kNormTile - 1) / kNormTile;
        const long long tiles = nt * (nt + 1) / 2, norms = nn * (nn + 1) / 2;
        if (norms > 0x7fffffffLL) return set_error(TVBG_EINVAL, "tvbg_fc: N too large");
        const int ncta = static_cast<int>(norms < N ? norms : N);   // one error part each
        for (int b0 = 0; b0 < n_inst; b0 += 65535) {   // gridDim.y
            const int nb = n_inst - b0 < 65535 ? n_inst - b0 : 65535;
            const SeriesView vb{d_x + b0 * inst_stride, inst_stride, nullptr, 0, 0, T, N, 1, 1};
            double* gb = gram + static_cast<long long>(b0) * N * N;
            fc_gram_kernel<<<dim3(static_cast<unsigned>(tiles), nb), kGramThreads, smem, st>>>(vb, gb);
            double* parts = d_err ? d_scratch + static_cast<long long>(b0) * N : nullptr;
            fc_norm_kernel<<<dim3(ncta, nb), 256, 0, st>>>(gb, N, static_cast<int>(norms),
                                                           d_fc + static_cast<long long>(b0) * N * N, d_target,
                                                           parts, N);
            if (d_err) fc_err_kernel<<<nb, 256, 0, st>>>(parts, N, ncta, d_err + b0);
        }
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return set_cuda_error(e, "tvbg_fc launch");
    return TVBG_OK;
}

extern "C" int tvbg_fc(const float* d_x, int32_t n_inst, int32_t T, int32_t N, int64_t inst_stride,
                       float* d_fc, const float* d_target, double* d_err, void* stream) {
    return tvbg_fc_ex(d_x, n_inst, T, N, inst_stride, d_fc, d_target, d_err, nullptr, stream);
}

// ---- allocation-free variant (tvbg_fc_noalloc) ------------------------------
// Scratch for callers that cannot allocate device memory: a file-scope device
// array, one instance per device that loads this library.  Host code must not
// pass `g_fc_noalloc_scratch` itself to a kernel (in host code the name is a
// host-side stand-in); its device address comes from cudaGetSymbolAddress.
static __device__ __align__(256) double g_fc_noalloc_scratch[TVBG_FC_NOALLOC_MAX_DOUBLES];

namespace {
constexpr int kMaxDevices = 64;
std::mutex g_noalloc_mutex;
double* g_noalloc_addr[kMaxDevices] = {};

// Device address of the scratch array on `dev` (the current device), looked
// up once per device on first use.
int noalloc_scratch(int dev, double** out) {
    if (dev < 0 || dev >= kMaxDevices) return set_error(TVBG_EINVAL, "tvbg_fc_noalloc: device index out of range");
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_addr[dev]) {
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_fc_noalloc_scratch);
        if (e != cudaSuccess) return set_cuda_error(e, "tvbg_fc_noalloc: cudaGetSymbolAddress");
        g_noalloc_addr[dev] = static_cast<double*>(p);
    }
    *out = g_noalloc_addr[dev];
    return TVBG_OK;
}
}  // namespace

extern "C" int tvbg_fc_noalloc(const float* d_x, int32_t n_inst, int32_t T, int32_t N,
                               int64_t inst_stride, float* d_fc, const float* d_target,
                               double* d_err, void* stream) {
    if (n_inst <= 0 || N <= 0) return set_error(TVBG_EINVAL, "tvbg_fc_noalloc: bad arguments");
    int64_t need = 0;
    int rc = tvbg_fc_scratch_bytes(n_inst, N, &need);
    if (rc) return rc;
    need /= static_cast<int64_t>(sizeof(double));
    if (need > TVBG_FC_NOALLOC_MAX_DOUBLES)
        return set_error(TVBG_EINVAL,
                         "tvbg_fc_noalloc: n_inst * N * (N + 1) exceeds TVBG_FC_NOALLOC_MAX_DOUBLES; "
                         "split the instances over several calls or use tvbg_fc_ex");
    double* scratch = nullptr;
    if (need > 0) {
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e != cudaSuccess) return set_cuda_error(e, "tvbg_fc_noalloc: cudaGetDevice");
        rc = noalloc_scratch(dev, &scratch);
        if (rc) return rc;
    }
    // the Gram and norm kernels write every scratch entry that is read later,
    // so the previous call's contents need no clearing
    return tvbg_fc_ex(d_x, n_inst, T, N, inst_stride, d_fc, d_target, d_err, scratch, stream);
}
