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
#include "tvbg_step_launch.cuh"

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
// with a zero diagonal (P = N (N - 1) / 2).  Kernels: FP64 means and the
// centred Gram (FP32 error-free transformations for N <= 192, digit products
// above); per instance the norms from the Gram's
// diagonal, FC, loss, A and diag(FC A) (the chain rule's time reduction
// sum_t Z_ti (Z A)_ti, taken from FC in FP64); dL/dX in FP32 (Z A is a sum
// over N nodes per sample, the precision of the backward).  The Pearson FC
// restates refs/covar.c:70-109 / metric.py:111-139 as a two-pass sum
// (centred Gram of the centred series) accurate to FP64 level.
// ---------------------------------------------------------------------------

namespace {

using tvbg::SeriesView;

// FP64 mean of every (instance, node): the samples split into kMS slices
// of consecutive samples, one thread each, the slices' sums added in slice
// order.  CTA = 32 (node, lane) pairs x kMS slices of one block of instances
// (blockIdx.y), lanes fastest: a warp reads whole sectors of a
// lane-interleaved series (256 x 84 series of 2000 samples: 187 us; 223 with one
// lane per CTA).
constexpr int kMS = 8;
__global__ void __launch_bounds__(256) fcfit_mean_kernel(SeriesView v, int n_inst, double* mean) {
    __shared__ double part[kMS][32];
    const int q = blockIdx.x * 32 + static_cast<int>(threadIdx.x);
    const int i = q / v.lanes;
    const int b = static_cast<int>(blockIdx.y) * v.lanes + q % v.lanes;
    const bool own = i < v.N && b < n_inst;
    const int per = (v.T + kMS - 1) / kMS;
    const int t0 = static_cast<int>(threadIdx.y) * per;
    const int t1 = t0 + per < v.T ? t0 + per : v.T;
    double s = 0.0;
    if (own) {
        const tvbg::SeriesRow row(v, b, i);
#pragma unroll 8
        for (int t = t0; t < t1; ++t) s += static_cast<double>(row.at(t));
    }
    part[threadIdx.y][threadIdx.x] = s;
    __syncthreads();
    if (threadIdx.y == 0 && own) {
        double m = 0.0;
#pragma unroll
        for (int k = 0; k < kMS; ++k) m += part[k][threadIdx.x];
        mean[static_cast<int64_t>(b) * v.N + i] = m / static_cast<double>(v.T);
    }
}

// Centred Gram G_ij = sum_t c_ti c_tj, c = x - mean, for N <= kSplitMaxN,
// all in FP32 arithmetic with error-free transformations: Knuth's TwoSum and
// TwoProduct by FMA, as in Ogita, Rump and Oishi, "Accurate sum and dot
// product", SIAM J. Sci. Comput. 26(6), 2005.  Every operation is an
// explicitly rounded intrinsic: nothing is contracted or reordered.
//
// A, 1 / nrm and zg / nrm are rounded to FP32 from this Gram, and the backward
// carries those roundings into dL/deta: two Grams that differ by 1e-14 give
// gradients that differ by up to 5e-8.  So these sums keep one arithmetic
// (the digit products of tvbg_gram.cuh are as accurate, but not the same bits).
//
// Work split: tiles of RB x 4 pairs of the upper triangle, one per thread,
// CTA = (instance blockIdx.x, part blockIdx.y of the tiles), instances
// fastest so that the lanes of a lane-interleaved group read the same
// sectors together.
//
// Centring: each mean (FP64) is split once into mh + ml (FP32 words); a
// sample x becomes c = (x - mh) - ml as (hi, lo) with hi + lo = c up to
// about 2^-48 (|c| + 2 |mean|): TwoSum(x, -mh) = (d, de), then
// TwoSum(d, de - ml).  kSplitL samples of every node staged per pass.
//
// Products: per pair and sample hi_i hi_j = p + e exactly (TwoProduct);
// p is summed by TwoSum (rounding errors collected in a second word),
// e + hi_i lo_j + lo_i hi_j (2^-24 of the product) in a third word; lo_i lo_j
// (2^-48) is dropped.  Every kSplitL samples the three words are added into
// the pair's double-FP32 sum (TwoSum, then the small words, then TwoSum
// again), converted to FP64 at the end.  The error is bounded by about
// kSplitL^2 2^-48 sum_t |c_ti c_tj| (the collected rounding errors of a pass
// summed in FP32), below 4e-12 of ||c_i|| ||c_j||; typical errors are near
// 1e-14.  Both triangles of G written.
//
// What bounds it: 12 FP32 operations per pair and sample, 256 x 84 nodes x 2000
// samples 1.28 ms (1.52 with 2 x 2 blocks of pairs and a division per staged
// sample; scalar operations 1.34).  They run two pairs at a time on the packed instructions; a subtraction is an FMA by -1 (the
// same rounding), and the third word is kept negated, which lets
// e = hi_i hi_j - p come from -hi_i.
constexpr int kSplitL = 32;
constexpr int kSplitMaxN = 192;   // staging (kSplitL + 1) x N pairs of words <= 50.7 KB
constexpr int kSplitThreads = 128;
constexpr int kSplitWarps = kSplitThreads / 32;

// Tiles of row block bi: column blocks from its first pair on or above the
// diagonal.
template <int RB>
__host__ __device__ __forceinline__ int split_tiles(int N) {
    int n = 0;
    for (int i = 0; i < N; i += RB) n += (N + 3) / 4 - i / 4;
    return n;
}

template <int RB>
__global__ void __launch_bounds__(kSplitThreads, 4) fcfit_gram_split_kernel(SeriesView v, const double* __restrict__ mean,
                                                                         int per_part, double* G) {
    extern __shared__ __align__(16) float sh[];  // [kSplitL][Np] hi, [kSplitL][Np] lo, [Np] mh, [Np] ml
    const int b = blockIdx.x;
    const int N = v.N;
    const int nc = (N + 3) / 4;
    const int Np = 4 * nc;
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    float* const shi = sh;
    float* const slo = sh + kSplitL * Np;
    float* const smh = sh + 2 * kSplitL * Np;
    float* const sml = smh + Np;
    const int first = static_cast<int>(blockIdx.y) * per_part;
    int i0 = 0, j0 = 0;
    bool act = false;
    if (static_cast<int>(threadIdx.x) < per_part) {
        int rem = first + static_cast<int>(threadIdx.x);
        while (i0 < N && rem >= nc - i0 / 4) {
            rem -= nc - i0 / 4;
            i0 += RB;
        }
        act = i0 < N;
        j0 = act ? 4 * (i0 / 4 + rem) : 0;
        if (!act) i0 = 0;
    }
    const double* mb = mean + static_cast<int64_t>(b) * N;
    for (int c = threadIdx.x; c < Np; c += kSplitThreads) {
        const double m = c < N ? mb[c] : 0.0;
        const float mh = __double2float_rn(m);
        smh[c] = mh;
        sml[c] = __double2float_rn(m - static_cast<double>(mh));
    }
    float2 ah[RB][2], al[RB][2];  // double-FP32 sums
#pragma unroll
    for (int u = 0; u < RB; ++u)
#pragma unroll
        for (int w = 0; w < 2; ++w) ah[u][w] = al[u][w] = make_float2(0.0f, 0.0f);
    __syncthreads();
    for (int t0 = 0; t0 < v.T; t0 += kSplitL) {
        // a warp takes whole rows of samples, its lanes the nodes
        for (int c = lane; c < Np; c += 32) {
            const tvbg::SeriesRow row(v, b, c < N ? c : 0);
            const float mh = smh[c], ml = sml[c];
            float x[kSplitL / kSplitWarps];
#pragma unroll
            for (int k = 0; k < kSplitL / kSplitWarps; ++k) {
                const int t = t0 + warp + k * kSplitWarps;
                x[k] = c < N && t < v.T ? row.at(t) : 0.0f;
            }
#pragma unroll
            for (int k = 0; k < kSplitL / kSplitWarps; ++k) {
                const int r = warp + k * kSplitWarps;
                float hi = 0.0f, lo = 0.0f;
                if (c < N && t0 + r < v.T) {
                    float d, de;
                    tvbg::gram_two_sum(x[k], -mh, d, de);
                    tvbg::gram_two_sum(d, __fsub_rn(de, ml), hi, lo);
                }
                shi[r * Np + c] = hi;
                slo[r * Np + c] = lo;
            }
        }
        __syncthreads();
        if (act) {
            float2 s[RB][2], cp[RB][2], nm[RB][2];  // nm: the small words, negated
#pragma unroll
            for (int u = 0; u < RB; ++u)
#pragma unroll
                for (int w = 0; w < 2; ++w) s[u][w] = cp[u][w] = nm[u][w] = make_float2(0.0f, 0.0f);
#pragma unroll 1
            for (int r = 0; r < kSplitL; ++r) {
                const float* const xh = shi + r * Np + i0;
                const float* const xl = slo + r * Np + i0;
                const float4 yh4 = *reinterpret_cast<const float4*>(shi + r * Np + j0);
                const float4 yl4 = *reinterpret_cast<const float4*>(slo + r * Np + j0);
                const float2 yh[2] = {make_float2(yh4.x, yh4.y), make_float2(yh4.z, yh4.w)};
                const float2 yl[2] = {make_float2(yl4.x, yl4.y), make_float2(yl4.z, yl4.w)};
                float h[RB], q[RB];
                if constexpr (RB == 4) {
                    *reinterpret_cast<float4*>(h) = *reinterpret_cast<const float4*>(xh);
                    *reinterpret_cast<float4*>(q) = *reinterpret_cast<const float4*>(xl);
                } else if constexpr (RB == 2) {
                    *reinterpret_cast<float2*>(h) = *reinterpret_cast<const float2*>(xh);
                    *reinterpret_cast<float2*>(q) = *reinterpret_cast<const float2*>(xl);
                } else {
                    h[0] = *xh;
                    q[0] = *xl;
                }
#pragma unroll
                for (int u = 0; u < RB; ++u) {
                    const float2 hh = make_float2(h[u], h[u]), nh = make_float2(-h[u], -h[u]);
                    const float2 nq = make_float2(-q[u], -q[u]);
#pragma unroll
                    for (int w = 0; w < 2; ++w) {
                        const float2 p = __fmul2_rn(hh, yh[w]);
                        const float2 ne = __ffma2_rn(nh, yh[w], p);  // p - hi hi, exact
                        nm[u][w] = __fadd2_rn(nm[u][w], __ffma2_rn(nh, yl[w], __ffma2_rn(nq, yh[w], ne)));
                        float2 t, err;
                        tvbg::gram_two_sum2(s[u][w], p, t, err);
                        s[u][w] = t;
                        cp[u][w] = __fadd2_rn(cp[u][w], err);
                    }
                }
            }
#pragma unroll
            for (int u = 0; u < RB; ++u)
#pragma unroll
                for (int w = 0; w < 2; ++w) {  // (ah, al) += s + (cp + small words)
                    float2 hi, lo;
                    tvbg::gram_two_sum2(ah[u][w], s[u][w], hi, lo);
                    lo = __fadd2_rn(lo, __fadd2_rn(al[u][w], tvbg::gram_sub2(cp[u][w], nm[u][w])));
                    tvbg::gram_two_sum2(hi, lo, ah[u][w], al[u][w]);
                }
        }
        __syncthreads();
    }
    if (!act) return;
    double* gb = G + static_cast<int64_t>(b) * N * N;
#pragma unroll
    for (int u = 0; u < RB; ++u)
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            const int i = i0 + u, j = j0 + w;
            if (i < N && j < N && j >= i) {
                const double g = w % 2 ? static_cast<double>(ah[u][w / 2].y) + static_cast<double>(al[u][w / 2].y)
                                       : static_cast<double>(ah[u][w / 2].x) + static_cast<double>(al[u][w / 2].x);
                gb[static_cast<int64_t>(i) * N + j] = g;
                gb[static_cast<int64_t>(j) * N + i] = g;
            }
        }
}

template <int RB>
int launch_gram_split(SeriesView v, const double* mean, double* G, int n_inst, cudaStream_t st) {
    const int tiles = split_tiles<RB>(v.N);
    const int parts = (tiles + kSplitThreads - 1) / kSplitThreads;
    const size_t smem = 8u * (kSplitL + 1) * 4u * static_cast<size_t>((v.N + 3) / 4);
    if (smem > 48u * 1024u) {
        // the limit of the largest N: another thread's smaller call may come
        // between this and the launch
        const cudaError_t e = cudaFuncSetAttribute(fcfit_gram_split_kernel<RB>,
                                                   cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   static_cast<int>(8u * (kSplitL + 1) * kSplitMaxN));
        if (e != cudaSuccess) return tvbg::set_cuda_error(e, "tvbg_fcfit_loss: smem attribute");
    }
    fcfit_gram_split_kernel<RB><<<dim3(n_inst, parts), kSplitThreads, smem, st>>>(v, mean, (tiles + parts - 1) / parts, G);
    return TVBG_OK;
}

// The tallest tiles that put a warp on every scheduler: 4 x 4 read the least
// from shared memory, 1 x 4 are four times as many.  Whole loss path, us, with
// 4 x 4 and 2 x 4 tiles: 256 x 84 nodes x 2000 samples 2070 and 2100, 64 x 84 x 1500
// 668 and 632, 4 x 84 x 2000 756 and 629, 200 x 31 x 700 328 and 244.
template <int RB>
bool split_fills(int n_inst, int N) {
    return static_cast<int64_t>(n_inst) * split_tiles<RB>(N) >=
           static_cast<int64_t>(tvbg::device_sms()) * kSplitThreads;
}

// N > kSplitMaxN: FP64 means and Gram by digit products (tvbg_gram.cuh), both
// triangles written.
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

// N > kSplitMaxN: one CTA per 64 x 64 tile of the upper triangle (blockIdx.y).
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
// 8 TY samples blockIdx.y), A_b [N][16 WN] and the Z tile, transposed, staged
// in shared memory once; thread (tx, ty) of 16 x TY owns samples 8 ty .. + 7
// and nodes 2 tx + 32 w, + 1.  Sums over k in order, as fcfit_dx_kernel: the
// same results.  Bound by shared memory and the FP32 pipe: 2 + WN / 2 loads for
// 4 WN packed FMAs per k; with 4 samples per thread and a load for each operand
// (10 for 24 FMAs) it took 460 us for 256 x 84 series of 2000 samples, 268 now.
template <int WN, int TY>
__global__ void __launch_bounds__(16 * TY)
    fcfit_dx_rows_kernel(SeriesView v, const float* __restrict__ fs, const float* __restrict__ A,
                         float* __restrict__ dx, int64_t dxs) {
    extern __shared__ __align__(16) float sm[];
    constexpr int NP = 16 * WN, TS = 8 * TY, ZS = TS + 4;
    const int b = blockIdx.x;
    const int T = v.T, N = v.N;
    const int t0 = blockIdx.y * TS;
    float* sA = sm;             // [N][NP]
    float* sZ = sm + N * NP;    // [N][ZS]
    const float* fb = fs + static_cast<int64_t>(b) * N * 3;
    const float* Ab = A + static_cast<size_t>(b) * N * N;
    const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
    constexpr int kWarps = TY / 2;
    for (int k = warp; k < N; k += kWarps)
#pragma unroll
        for (int j = lane; j < NP; j += 32) sA[k * NP + j] = j < N ? __ldg(Ab + static_cast<size_t>(k) * N + j) : 0.0f;
    for (int k = lane; k < N; k += 32) {   // a warp takes whole samples, its lanes the nodes
        const tvbg::SeriesRow row(v, b, k);
        const float mean = fb[3 * k], inv = fb[3 * k + 1];
#pragma unroll
        for (int r0 = 0; r0 < TS; r0 += 8 * kWarps) {
            float x[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int t = t0 + r0 + u * kWarps + warp;
                x[u] = t < T ? row.at(t) : mean;
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) sZ[k * ZS + r0 + u * kWarps + warp] = (x[u] - mean) * inv;
        }
    }
    __syncthreads();
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
    float2 acc[8][WN / 2];
#pragma unroll
    for (int u = 0; u < 8; ++u)
#pragma unroll
        for (int w = 0; w < WN / 2; ++w) acc[u][w] = make_float2(0.0f, 0.0f);
#pragma unroll 2
    for (int k = 0; k < N; ++k) {
        float z[8];
        *reinterpret_cast<float4*>(z) = *reinterpret_cast<const float4*>(sZ + k * ZS + 8 * ty);
        *reinterpret_cast<float4*>(z + 4) = *reinterpret_cast<const float4*>(sZ + k * ZS + 8 * ty + 4);
        float2 a[WN / 2];
#pragma unroll
        for (int w = 0; w < WN / 2; ++w) a[w] = *reinterpret_cast<const float2*>(sA + k * NP + 2 * tx + 32 * w);
#pragma unroll
        for (int u = 0; u < 8; ++u)
#pragma unroll
            for (int w = 0; w < WN / 2; ++w) acc[u][w] = __ffma2_rn(make_float2(z[u], z[u]), a[w], acc[u][w]);
    }
#pragma unroll
    for (int w = 0; w < WN / 2; ++w)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const int j = 2 * tx + 32 * w + c;
            if (j >= N) continue;
            const float inv = fb[3 * j + 1], zg = fb[3 * j + 2];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int t = t0 + ty * 8 + u;
                if (t < T)
                    dx[b * dxs + static_cast<int64_t>(t) * N + j] =
                        fmaf(-sZ[j * ZS + ty * 8 + u], zg, (c ? acc[u][w].y : acc[u][w].x) * inv);
            }
        }
}

template <int WN>
int launch_dx_rows(SeriesView v, const float* fs, const float* A, float* dx, int64_t dxs, int n_inst,
                   cudaStream_t st) {
    constexpr int TY = WN < 8 ? 16 : 8;   // two CTAs per SM at the largest N
    const size_t smem = 4u * static_cast<size_t>(v.N) * (16 * WN + 8 * TY + 4);
    if (smem > 48u * 1024u) {
        const cudaError_t e = cudaFuncSetAttribute(reinterpret_cast<const void*>(fcfit_dx_rows_kernel<WN, TY>),
                                                   cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   static_cast<int>(4u * 16 * WN * (16 * WN + 8 * TY + 4)));
        if (e != cudaSuccess) return tvbg::set_cuda_error(e, "tvbg_fcfit_loss: smem attribute");
    }
    const dim3 grid(static_cast<unsigned>(n_inst), static_cast<unsigned>((v.T + 8 * TY - 1) / (8 * TY)));
    fcfit_dx_rows_kernel<WN, TY><<<grid, 16 * TY, smem, st>>>(v, fs, A, dx, dxs);
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
    if (N > kSplitMaxN && nt * (nt + 1) / 2 > 65535)
        return tvbg::set_error(TVBG_EINVAL, "tvbg_fcfit_loss: N too large");
    if (N <= kSplitMaxN) {
        fcfit_mean_kernel<<<dim3((N * lanes + 31) / 32, (n_inst + lanes - 1) / lanes), dim3(32, kMS), 0, st>>>(
            v, n_inst, mean);
        const int rc = split_fills<4>(n_inst, N)   ? launch_gram_split<4>(v, mean, fc, n_inst, st)
                       : split_fills<2>(n_inst, N) ? launch_gram_split<2>(v, mean, fc, n_inst, st)
                                                   : launch_gram_split<1>(v, mean, fc, n_inst, st);
        if (rc != TVBG_OK) return rc;
    } else {
        const size_t smem = tvbg::gram_plane_bytes(128);
        const cudaError_t e = cudaFuncSetAttribute(fcfit_gram_tiles_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   static_cast<int>(smem));
        if (e != cudaSuccess) return tvbg::set_cuda_error(e, "tvbg_fcfit_loss: smem attribute");
        fcfit_gram_tiles_kernel<<<dim3(n_inst, static_cast<unsigned>(nt * (nt + 1) / 2)), tvbg::kGramThreads, smem,
                                  st>>>(v, mean, fc);
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
