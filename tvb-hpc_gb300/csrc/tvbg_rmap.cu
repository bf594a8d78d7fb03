// Region mapping between node and region (roi) arrays, tvb_hpc/network.py:
// RMapToAvg (179-191): roi[i, j] = sum over k with rmap[k] == i of node[k, j]
// (the reference zeroes roi and accumulates, so it is a sum);
// RMapFromAvg (194-202): node[k, j] = roi[rmap[k], j].
//
// to_avg: few nodes are scanned by one CTA per region (rmap_scan_kernel).  Else
// one cluster of CTAs reads every node once where nroi * nvar <= 1600
// (kBins) and nvar <= 32 (kVars); beyond, one cluster for each part of the regions and
// variables, and each scans the whole rmap.  A cluster's CTAs take the nodes in
// consecutive parts, warp by warp; each warp adds its nodes, 32 at a time and
// in order, to bins of its own in shared memory; the warps' bins meet in warp
// order and the CTAs' in rank order, in FP64.  Every sum has a fixed order, so
// the result is deterministic (it differs from the reference's sequential one
// by rounding only).  Bound by latency: 515 056 nodes, 68 regions, 2 variables
// take 20 us on 16 CTAs (6.2 MB), 499 us before (one CTA per region, each scanning the
// whole map).  Entries of rmap outside [0, nroi) contribute to no region, and
// from_avg leaves their node rows unchanged.
#include <algorithm>
#include <cstring>

#include "tvbg_abi_internal.h"
#include "tvbg_lanes.cuh"

namespace {

constexpr int kThreads = 1024;
constexpr int kWarps = kThreads / 32;
constexpr int kClusterMax = 16;
constexpr int kBins = 1600;   // bins per warp: 32 x 1600 floats, 205 KB of shared memory
constexpr int kVars = 32;     // variables per cluster

// NJ: the variables of the cluster where they are few enough to be read ahead
// into registers (1 to 4), 0 for any number up to kVars.
// Regions [i0, i0 + ni) (from `first` on) and variables [j0, j0 + nj) (from
// `first_var` on) of one
// cluster (blockIdx.y, blockIdx.z), ni nj <= kBins; nj <= kVars.  Shared memory: [kWarps][ni nj]
// floats, whose start becomes the CTA's [ni nj] sums in FP64.
template <int NJ>
__global__ void __launch_bounds__(kThreads, 1)
    rmap_to_avg_kernel(int nroi, int nvar, int nnode, int roi_step, int first, int first_var,
                       const int32_t* __restrict__ rmap, const float* __restrict__ node, float* __restrict__ roi) {
    extern __shared__ __align__(16) float rmap_bins[];
    const int i0 = first + blockIdx.y * roi_step, j0 = first_var + blockIdx.z * kVars;
    const int ni = min(roi_step, nroi - i0), nj = NJ ? NJ : min(kVars, nvar - j0);
    const int bins = ni * nj;
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const int C = static_cast<int>(tvbg::cluster_nranks()), rank = static_cast<int>(tvbg::cluster_rank());
    for (int q = threadIdx.x; q < kWarps * bins; q += kThreads) rmap_bins[q] = 0.0f;
    __syncthreads();
    float* mine = rmap_bins + warp * bins;
    // this warp's nodes: whole groups of 32, consecutive
    const long long groups = (static_cast<long long>(nnode) + 31) / 32, parts = static_cast<long long>(C) * kWarps;
    const long long part = static_cast<long long>(rank) * kWarps + warp;
    const int g0 = static_cast<int>(groups * part / parts), g1 = static_cast<int>(groups * (part + 1) / parts);
    constexpr int U = NJ >= 3 ? 4 : 8;   // groups of 32 nodes read ahead
    constexpr int NX = NJ ? NJ : 1;
    for (int gb = g0; gb < g1; gb += U) {
        int reg[U];
        float xa[U][NX];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const long long k = (static_cast<long long>(gb) + u) * 32 + lane;
            const bool in = gb + u < g1 && k < nnode;
            reg[u] = in ? __ldg(rmap + k) - i0 : -1;
#pragma unroll
            for (int j = 0; j < NX; ++j) xa[u][j] = in ? __ldg(node + k * nvar + j0 + j) : 0.0f;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const long long k = (static_cast<long long>(gb) + u) * 32 + lane;
            const bool valid = reg[u] >= 0 && reg[u] < ni;
            const int i = valid ? reg[u] : -1;
            const unsigned peers = __match_any_sync(0xffffffffu, i);
            if (__all_sync(0xffffffffu, i < 0)) continue;
            if (peers == 0xffffffffu) {          // one region: a tree over the lanes
                auto add = [&](int j, float x) {
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
                    if (lane == 0) mine[i * nj + j] += x;
                };
#pragma unroll
                for (int j = 0; j < NX; ++j) add(j, xa[u][j]);
                for (int j = NX; j < nj; ++j) add(j, __ldg(node + k * nvar + j0 + j));
            } else {                             // each region's nodes one after another, in lane order
                const int turn = __popc(peers & ((1u << lane) - 1u));
                const int turns = __reduce_max_sync(0xffffffffu, valid ? __popc(peers) : 0);
                for (int r = 0; r < turns; ++r) {
                    if (valid && turn == r) {
#pragma unroll
                        for (int j = 0; j < NX; ++j) mine[i * nj + j] += xa[u][j];
                        for (int j = NX; j < nj; ++j) mine[i * nj + j] += __ldg(node + k * nvar + j0 + j);
                    }
                    __syncwarp();
                }
            }
            __syncwarp();
        }
    }
    __syncthreads();
    // the warps' bins in warp order, the CTAs' in rank order
    constexpr int kPer = (kBins + kThreads - 1) / kThreads;
    double s[kPer];
#pragma unroll
    for (int p = 0; p < kPer; ++p) {
        const int q = threadIdx.x + p * kThreads;
        s[p] = 0.0;
        if (q < bins)
#pragma unroll
            for (int w = 0; w < kWarps; ++w) s[p] += static_cast<double>(rmap_bins[w * bins + q]);
    }
    __syncthreads();
    double* sums = reinterpret_cast<double*>(rmap_bins);
#pragma unroll
    for (int p = 0; p < kPer; ++p) {
        const int q = threadIdx.x + p * kThreads;
        if (q < bins) sums[q] = s[p];
    }
    tvbg::group_barrier(C > 1);
    for (int q = rank * kThreads + threadIdx.x; q < bins; q += C * kThreads) {
        double v[kClusterMax];   // the CTAs' sums, read together
#pragma unroll
        for (int c = 0; c < kClusterMax; ++c) {
            uint32_t remote;     // past the last CTA: its sum again, not added
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                         : "=r"(remote)
                         : "r"(tvbg::smem_addr(sums + q)), "r"(min(c, C - 1)));
            asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v[c]) : "r"(remote) : "memory");
        }
        double t = 0.0;
#pragma unroll
        for (int c = 0; c < kClusterMax; ++c)
            if (c < C) t += v[c];
        roi[static_cast<size_t>(i0 + q / nj) * nvar + j0 + q % nj] = static_cast<float>(t);
    }
    tvbg::group_barrier(C > 1);   // no CTA leaves while its sums may be read
}

// Few nodes: one CTA per region and NJ variables scans the whole map; the
// threads add their strided nodes, and meet in a fixed tree, in pairs of FP32
// words (TwoSum; FP64 adds, two per SM and clock, made the scan twice as slow).
constexpr int kScanThreads = 256;
constexpr int kScanVars = 4;

struct SumPair {
    float s = 0.0f, c = 0.0f;
    __device__ __forceinline__ void add(float x, float xc) {
        const float t = __fadd_rn(s, x), b = __fsub_rn(t, s);
        const float e = __fadd_rn(__fsub_rn(s, __fsub_rn(t, b)), __fsub_rn(x, b));
        s = t;
        c = __fadd_rn(c, __fadd_rn(e, xc));
    }
    // an infinite or NaN sum has a NaN error word
    __device__ __forceinline__ float value() const { return isfinite(s) ? __fadd_rn(s, c) : s; }
};

template <int NJ>
__global__ void __launch_bounds__(kScanThreads)
    rmap_scan_kernel(int nvar, int nnode, const int32_t* __restrict__ rmap, const float* __restrict__ node,
                     float* __restrict__ roi) {
    __shared__ float2 part[kScanThreads / 32][NJ];
    const int i = blockIdx.x, warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    for (int j0 = blockIdx.y * NJ; j0 < nvar; j0 += gridDim.y * NJ) {
        SumPair s[NJ];
        constexpr int U = 8;   // map entries read ahead
        for (int k0 = threadIdx.x; k0 < nnode; k0 += U * kScanThreads) {
            int r[U];
#pragma unroll
            for (int u = 0; u < U; ++u) r[u] = k0 + u * kScanThreads < nnode ? __ldg(rmap + k0 + u * kScanThreads) : -1;
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (r[u] == i) {
                    const float* p = node + static_cast<size_t>(k0 + u * kScanThreads) * nvar + j0;
#pragma unroll
                    for (int j = 0; j < NJ; ++j)
                        if (j0 + j < nvar) s[j].add(__ldg(p + j), 0.0f);
                }
        }
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const float x = __shfl_down_sync(0xffffffffu, s[j].s, o), c = __shfl_down_sync(0xffffffffu, s[j].c, o);
                s[j].add(x, c);
            }
            if (lane == 0) part[warp][j] = make_float2(s[j].s, s[j].c);
        }
        __syncthreads();
        if (threadIdx.x < NJ && j0 + static_cast<int>(threadIdx.x) < nvar) {
            SumPair t;
#pragma unroll
            for (int w = 0; w < kScanThreads / 32; ++w) t.add(part[w][threadIdx.x].x, part[w][threadIdx.x].y);
            roi[static_cast<size_t>(i) * nvar + j0 + threadIdx.x] = t.value();
        }
        __syncthreads();
    }
}

__global__ void rmap_from_avg_kernel(int nroi, int nvar, long long n, const int32_t* __restrict__ rmap,
                                     const float* __restrict__ roi, float* __restrict__ node) {
    for (long long e = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; e < n;
         e += static_cast<long long>(gridDim.x) * blockDim.x) {
        const long long k = e / nvar;
        const int j = static_cast<int>(e - k * nvar);
        const int i = __ldg(rmap + k);
        if (i >= 0 && i < nroi) node[e] = __ldg(roi + static_cast<size_t>(i) * nvar + j);
    }
}

// Which kernel: their times in ns.  The scan takes 5 us and 0.06 us for every 256
// nodes (0.12 with few regions, whose warps add at every trip), and all its CTAs
// together 3 ns each and 0.2 ps per map entry; the cluster takes 9 us and 22 ns
// for every bin, which 32 warps clear and add up.  us, scan / cluster, random maps:
// 4000 nodes of 400 regions, 4 variables 6.8 / 47, 16 000 9.3 / 46; 8000 of 2
// regions, one variable 7.4 / 13, 16 000 of 2, two variables about 18 / 13.
bool scan_is_faster(int nroi, int nvar, int nnode) {
    const double ctas = static_cast<double>(nroi) * ((nvar + kScanVars - 1) / kScanVars);
    const double scan = 5000.0 + nnode / (nroi < 128 ? 2.2 : 4.0) + ctas * (3.0 + nnode / 5000.0);
    const int nj = std::min(nvar, kVars);
    const double bins = static_cast<double>(std::min(nroi, kBins / nj)) * nj;   // of one cluster
    return scan < 9000.0 + 22.0 * bins;
}

}  // namespace

extern "C" {

int tvbg_rmap_to_avg(int32_t nroi, int32_t nvar, int32_t nnode, const int32_t* d_rmap,
                     const float* d_node, float* d_roi, void* stream) {
    if (nroi < 0 || nvar < 0 || nnode < 0 || (nnode > 0 && (!d_rmap || !d_node)) ||
        (nroi > 0 && nvar > 0 && !d_roi))
        return tvbg::set_error(TVBG_EINVAL, "tvbg_rmap_to_avg: bad arguments");
    if (nroi == 0 || nvar == 0) return TVBG_OK;
    if (scan_is_faster(nroi, nvar, nnode)) {
        const int gv = (nvar + kScanVars - 1) / kScanVars;
        const auto scan = nvar <= 2 ? rmap_scan_kernel<2> : rmap_scan_kernel<kScanVars>;
        scan<<<dim3(static_cast<unsigned>(nroi), static_cast<unsigned>(std::min(gv, 65535))), kScanThreads, 0,
                           static_cast<cudaStream_t>(stream)>>>(nvar, nnode, d_rmap, d_node, d_roi);
        const cudaError_t es = cudaGetLastError();
        return es == cudaSuccess ? TVBG_OK : tvbg::set_cuda_error(es, "tvbg_rmap_to_avg launch");
    }
    const int nj = std::min(nvar, kVars);
    const int roi_step = std::min(nroi, kBins / nj);
    const long long gy = (static_cast<long long>(nroi) + roi_step - 1) / roi_step;
    const long long gz = (static_cast<long long>(nvar) + kVars - 1) / kVars;
    // a cluster's CTAs: at least 4096 nodes each, as many as the device launches
    int cluster = 1;
    while (cluster < kClusterMax && static_cast<long long>(cluster) * 4096 < nnode) cluster *= 2;
    const size_t smem = sizeof(float) * kWarps * static_cast<size_t>(roi_step) * nj;
    const auto kernel = nvar == 1   ? rmap_to_avg_kernel<1>
                        : nvar == 2 ? rmap_to_avg_kernel<2>
                        : nvar == 3 ? rmap_to_avg_kernel<3>
                        : nvar == 4 ? rmap_to_avg_kernel<4>
                                    : rmap_to_avg_kernel<0>;
    const void* kfn = reinterpret_cast<const void*>(kernel);
    // the limit of the largest call: another thread's smaller one may come between this and the launch
    cudaError_t e = cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(sizeof(float) * kWarps * kBins));
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kfn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return tvbg::set_cuda_error(e, "tvbg_rmap_to_avg: kernel attributes");
    cudaLaunchConfig_t lc;
    std::memset(&lc, 0, sizeof(lc));
    lc.blockDim = dim3(kThreads, 1, 1);
    lc.dynamicSmemBytes = smem;
    lc.stream = static_cast<cudaStream_t>(stream);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    lc.attrs = attr;
    lc.numAttrs = 1;
    for (;; cluster /= 2) {
        attr[0].val.clusterDim.x = static_cast<unsigned>(cluster);
        lc.gridDim = dim3(static_cast<unsigned>(cluster), 1, 1);
        int n = 0;
        if (cluster <= 8) break;
        if (cudaOccupancyMaxActiveClusters(&n, kfn, &lc) == cudaSuccess && n > 0) break;
        cudaGetLastError();
    }
    constexpr long long kGrid = 65535;
    for (long long z0 = 0; z0 < gz && e == cudaSuccess; z0 += kGrid)
        for (long long y0 = 0; y0 < gy && e == cudaSuccess; y0 += kGrid) {
            lc.gridDim = dim3(static_cast<unsigned>(cluster), static_cast<unsigned>(std::min(kGrid, gy - y0)),
                              static_cast<unsigned>(std::min(kGrid, gz - z0)));
            e = cudaLaunchKernelEx(&lc, kernel, nroi, nvar, nnode, roi_step,
                                   static_cast<int>(y0 * roi_step), static_cast<int>(z0 * kVars), d_rmap, d_node,
                                   d_roi);
        }
    return e == cudaSuccess ? TVBG_OK : tvbg::set_cuda_error(e, "tvbg_rmap_to_avg launch");
}

int tvbg_rmap_from_avg(int32_t nroi, int32_t nvar, int32_t nnode, const int32_t* d_rmap,
                       const float* d_roi, float* d_node, void* stream) {
    if (nroi < 0 || nvar < 0 || nnode < 0 || (nnode > 0 && nvar > 0 && (!d_rmap || !d_node)) ||
        (nroi > 0 && nvar > 0 && !d_roi))
        return tvbg::set_error(TVBG_EINVAL, "tvbg_rmap_from_avg: bad arguments");
    const long long n = static_cast<long long>(nnode) * nvar;
    if (n == 0) return TVBG_OK;
    const long long blocks = std::min<long long>((n + 255) / 256, 65536);
    rmap_from_avg_kernel<<<static_cast<unsigned>(blocks), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        nroi, nvar, n, d_rmap, d_roi, d_node);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? TVBG_OK : tvbg::set_cuda_error(e, "tvbg_rmap_from_avg launch");
}

}  // extern "C"
