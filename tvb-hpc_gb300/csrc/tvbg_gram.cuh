// Centred Gram matrices of many time series, to FP64 accuracy on the tensor
// cores:  G_ij = sum_t (x_ti - m_i)(x_tj - m_j)  (the co-moment of
// tvb_hpc/metric.py:18-139 and dsl/dsl_cuda/CUDAmodels/refs/covar.c:9-109).
//
// GB300 executes two FP64 operations per SM and clock, so an FP64 Gram is
// bound by its products (one DFMA each: 16 x 1200 x 400 series took 6.4 ms).
// Here every centred sample is written as a fixed-point number of its node,
// split into seven signed 8-bit digits, and the products of digits are summed
// exactly: splitting a product into exact slices on faster units is the
// scheme of Ozaki, Ogita, Oishi and Rump, "Error-free transformations of
// matrix multiplication" (Numer. Algorithms 59, 2012).
//
// Fixed point.  Node i has s = float(m_i) and an exponent e with
// |x - m| < 2^e for all samples.  x - s = d + de exactly (TwoSum), and
//   Q = (x - m) 2^(54-e) = digits D_0 .. D_6 in [-128, 127], Q = sum D_a 2^(48-8a),
// |D_0| <= 64, rounded to 1.5 units: about 2^-53 of the node's largest deviation,
// where an FP64 difference has 2^-53 of the sample.  D_a is exact in bf16.
//
// Products.  L_s = sum_t sum_{a+b=s} D_a D_b for s = 0..6 (28 bf16 mma per
// 16 x 8 x 16 block of the product; the levels above 6, below 2^-53 of it, are
// dropped).  |L_s| < 7 * 2^14 * 64 < 2^23 over a chunk of 64 samples, so the FP32
// accumulators hold exact integers; each chunk is added to two 64-bit integers,
//   hi = sum_{s<=3} L_s 2^(24-8s),  lo = sum_{s=4..6} L_s 2^(48-8s),
//   G_ij = (hi + lo 2^-24) 2^(e_i + e_j - 36).
// A node whose mean is not finite gives NaN; a constant one gives exact zeros.
//
// mma.sync rather than tcgen05: 28 products per chunk accumulate into seven
// separate levels that leave the unit after every 64 samples, and the
// conversion to digits takes about as long as the products.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

namespace tvbg {

// Instance b of a series lives in block b / lanes at lane b % lanes:
// lanes = 1 for per-instance arrays, 8 for lane-interleaved groups.
struct SeriesView {
    const float* x;      // row s (s < T - 1, or every row without `last`):
    int64_t xs;          //   x + (b / lanes) xs + b % lanes + (s N + i) cols lanes
    const float* last;   // row T - 1: last + (b / lanes) ls + b % lanes + i lns, or NULL
    int64_t ls, lns;
    int T, N, lanes;
    int cols;            // values of a node and sample in x; the series is the first
    __device__ __forceinline__ float at(int b, int s, int i) const {
        const int g = b / lanes, l = b % lanes;
        if (last && s == T - 1) return __ldg(last + g * ls + l + static_cast<int64_t>(i) * lns);
        return __ldg(x + g * xs + l + (static_cast<int64_t>(s) * N + i) * (lanes * cols));
    }
};

// One node's series: sample t at p[t * stride], sample `end` at *last.
struct SeriesRow {
    const float* p;
    const float* last;
    int64_t stride;
    int end;
    __device__ __forceinline__ SeriesRow(const SeriesView& v, int b, int i) {
        const int g = b / v.lanes, l = b % v.lanes;
        p = v.x + g * v.xs + l + static_cast<int64_t>(i) * (v.lanes * v.cols);
        stride = static_cast<int64_t>(v.N) * (v.lanes * v.cols);
        last = v.last ? v.last + g * v.ls + l + static_cast<int64_t>(i) * v.lns : nullptr;
        end = v.last ? v.T - 1 : v.T;
    }
    __device__ __forceinline__ float at(int t) const { return __ldg(t == end ? last : p + t * stride); }
};

constexpr int kGramThreads = 256;   // 8 warps, up to 255 registers a thread
constexpr int kGramChunk = 64;      // samples per chunk
constexpr int kGramStride = 72;     // bf16 per staged row: 16-byte rows that ldmatrix reads without conflicts
constexpr int kGramDigits = 7;
constexpr int kGramTiles = 3;       // 16 x 16 tiles per warp and pass
constexpr int kGramSegment = 1 << 20;  // samples summed in the 64-bit integers
// Samples of a node and thread summed in three FP32 words (TwoSum twice) before
// they go to FP64.  Of at most 256 floats of one magnitude the words hold the exact sum,
// so the mean of a constant node is that constant, at any length; against 80-bit
// means of 40 to 20 000 normal and lognormal samples the error is that of an
// FP64 sum.  (Two words over the whole series lost the constant from 17 000
// samples on, and up to 1e4 times an FP64 sum's error on lognormal samples.)
constexpr int kMeanRun = 256;

__host__ __device__ constexpr size_t gram_plane_bytes(int rows) {
    return static_cast<size_t>(2) * kGramDigits * rows * kGramStride;
}

// Knuth's TwoSum: a + b = s + e exactly, every operation rounded as written.
__device__ __forceinline__ void gram_two_sum(float a, float b, float& s, float& e) {
    const float t = __fadd_rn(a, b);
    const float bb = __fsub_rn(t, a);
    e = __fadd_rn(__fsub_rn(a, __fsub_rn(t, bb)), __fsub_rn(b, bb));
    s = t;
}

// The same for two pairs; a subtraction is an FMA by -1 (the same rounding).
__device__ __forceinline__ float2 gram_sub2(float2 a, float2 b) {
    return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a);
}
__device__ __forceinline__ void gram_two_sum2(float2 a, float2 b, float2& s, float2& e) {
    const float2 t = __fadd2_rn(a, b);
    const float2 bb = gram_sub2(t, a);
    e = __fadd2_rn(gram_sub2(a, gram_sub2(t, bb)), gram_sub2(b, bb));
    s = t;
}

// What the conversion of a node's samples needs.
struct GramNode {
    float f0;          // 1, or 1/4 where x - s may exceed the FP32 range
    float s;           // f0 float(mean)
    float f1, f2;      // f0 f1 f2 = 2^(30-e), in factors that are in range
    int mh, ml;        // (mean - s) 2^(54-e) = mh 2^24 + ml
};

// Mean, deviation bound and conversion of every staged row, by all threads.
// node(r) is the node of row r, or -1.  mean_out(r, m) is called once per row
// with a node.  scale[r] = 2^(e-18) (0 without a node, NaN where the mean is
// not finite).  red: 2 doubles per thread.
template <int ROWS, class NodeOf, class MeanOut>
__device__ __forceinline__ void gram_stats(const SeriesView& v, int b, NodeOf node, MeanOut mean_out,
                                           GramNode* nodes, double* scale, double* red) {
    constexpr int SL = kGramThreads / ROWS;  // time slices per row
    const int r = threadIdx.x % ROWS, sl = threadIdx.x / ROWS;
    const int n = sl < SL ? node(r) : -1;
    double sum_t = 0.0;
    float lo = INFINITY, hi = -INFINITY;
    if (n >= 0) {
        const SeriesRow row(v, b, n);
        for (int t0 = sl; t0 < v.T; t0 += SL * kMeanRun) {
            // two samples a step, in the halves of the packed instructions
            float2 s = make_float2(0.0f, 0.0f), c = s, cc = s;
            const int t1 = v.T - t0 < SL * kMeanRun ? v.T : t0 + SL * kMeanRun;
            int t = t0;
            for (; t + 7 * SL < t1; t += 8 * SL) {
                float x[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) x[u] = row.at(t + u * SL);
#pragma unroll
                for (int u = 0; u < 8; u += 2) {
                    float2 e, e2;
                    gram_two_sum2(s, make_float2(x[u], x[u + 1]), s, e);
                    gram_two_sum2(c, e, c, e2);
                    cc = __fadd2_rn(cc, e2);
                    lo = fminf(lo, fminf(x[u], x[u + 1]));
                    hi = fmaxf(hi, fmaxf(x[u], x[u + 1]));
                }
            }
            for (; t < t1; t += SL) {
                const float x = row.at(t);
                float e, e2;
                gram_two_sum(s.x, x, s.x, e);
                gram_two_sum(c.x, e, c.x, e2);
                cc.x = __fadd_rn(cc.x, e2);
                lo = fminf(lo, x);
                hi = fmaxf(hi, x);
            }
            sum_t += static_cast<double>(s.x) + (static_cast<double>(c.x) + static_cast<double>(cc.x));
            sum_t += static_cast<double>(s.y) + (static_cast<double>(c.y) + static_cast<double>(cc.y));
        }
    }
    float* rng = reinterpret_cast<float*>(red + kGramThreads);
    red[threadIdx.x] = sum_t;
    rng[2 * threadIdx.x] = lo;
    rng[2 * threadIdx.x + 1] = hi;
    __syncthreads();
    if (threadIdx.x < ROWS) {
        GramNode g = {0.0f, 0.0f, 0.0f, 0.0f, 0, 0};
        double sc = 0.0;
        if (n >= 0) {
            double sum = 0.0;
#pragma unroll
            for (int k = 0; k < SL; ++k) {
                sum += red[r + k * ROWS];
                lo = fminf(lo, rng[2 * (r + k * ROWS)]);
                hi = fmaxf(hi, rng[2 * (r + k * ROWS) + 1]);
            }
            double m = sum / static_cast<double>(v.T);
            if (!isfinite(m) && isfinite(lo) && isfinite(hi)) {  // the FP32 sum overflowed, or a NaN
                const SeriesRow row(v, b, n);
                sum = 0.0;
                for (int t = 0; t < v.T; ++t) sum += static_cast<double>(row.at(t));
                m = sum / static_cast<double>(v.T);
            }
            mean_out(r, m);
            if (isfinite(m) && isfinite(lo) && isfinite(hi)) {
                // the largest deviation from s, or of m from s
                const double sd = static_cast<double>(static_cast<float>(m));
                const double a = fmax(fmax(static_cast<double>(hi) - sd, sd - static_cast<double>(lo)),
                                      fabs(m - sd));
                int e = 0;
                if (a > 0.0) {
                    frexp(a, &e);
                    e += 1;
                }
                g.f0 = a > 4.0e37 ? 0.25f : 1.0f;
                g.s = static_cast<float>(m) * g.f0;
                const int k0 = 30 - e, k = a > 4.0e37 ? k0 + 2 : k0, k1 = k > 100 ? 100 : k;
                g.f1 = ldexpf(1.0f, k1);
                g.f2 = ldexpf(1.0f, k - k1);
                const double y = ldexp(m - sd, k0);
                const double yh = rint(y);
                g.mh = static_cast<int>(yh);
                g.ml = static_cast<int>(rint((y - yh) * 16777216.0));
                sc = ldexp(1.0, e - 18);
            } else {
                sc = static_cast<double>(NAN);
            }
        }
        nodes[r] = g;
        scale[r] = sc;
    }
    __syncthreads();
}

// The digits of one sample, packed as bf16 bits into `out[a]`.
__device__ __forceinline__ void gram_digits(float x, const GramNode& g, uint32_t out[kGramDigits]) {
    float d, de;
    gram_two_sum(x * g.f0, -g.s, d, de);
    const float y = d * g.f1 * g.f2, ye = de * g.f1 * g.f2;
    const float yr = rintf(y), yer = rintf(ye);
    int h = __float2int_rn(yr) + __float2int_rn(yer) - g.mh;
    int l = __float2int_rn((y - yr) * 16777216.0f) + __float2int_rn((ye - yer) * 16777216.0f) - g.ml;
#pragma unroll
    for (int a = kGramDigits - 1; a >= 0; --a) {
        int dg;
        if (a >= 4) {            // three digits from the low word, its carry into the high one
            dg = ((l + 128) & 255) - 128;
            l = (l - dg) >> 8;
            if (a == 4) h += l;
        } else if (a > 0) {
            dg = ((h + 128) & 255) - 128;
            h = (h - dg) >> 8;
        } else {
            dg = h;
        }
        // |dg| <= 128: the float's upper half is the bf16
        out[a] = __float_as_uint(__int_as_float(0x4B400000 + dg) - 12582912.0f) >> 16;
    }
}

// Digits of samples [t0, t0 + 64) of every staged row into the planes
// [digit][row][72]; 8 samples per thread and item, one 16-byte store per digit.
template <int ROWS, class NodeOf>
__device__ __forceinline__ void gram_convert(const SeriesView& v, int b, int t0, int nt, NodeOf node,
                                             const GramNode* nodes, __nv_bfloat16* planes) {
    for (int it = threadIdx.x; it < ROWS * (kGramChunk / 8); it += kGramThreads) {
        const int r = it % ROWS, k = it / ROWS * 8;
        if (k >= ((nt + 15) & ~15)) break;   // k grows with it
        const int n = node(r);
        const GramNode g = nodes[r];
        const SeriesRow row(v, b, n < 0 ? 0 : n);
        uint32_t w[kGramDigits][4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            uint32_t p[kGramDigits], q[kGramDigits];
            const int t = k + 2 * u;
            const bool ok0 = n >= 0 && t < nt, ok1 = n >= 0 && t + 1 < nt;
            const float x0 = ok0 ? row.at(t0 + t) : 0.0f, x1 = ok1 ? row.at(t0 + t + 1) : 0.0f;
            gram_digits(x0, g, p);
            gram_digits(x1, g, q);
#pragma unroll
            for (int a = 0; a < kGramDigits; ++a) w[a][u] = (ok0 ? p[a] : 0u) | ((ok1 ? q[a] : 0u) << 16);
        }
#pragma unroll
        for (int a = 0; a < kGramDigits; ++a)
            *reinterpret_cast<uint4*>(planes + (a * ROWS + r) * kGramStride + k) =
                make_uint4(w[a][0], w[a][1], w[a][2], w[a][3]);
    }
}

__device__ __forceinline__ void gram_ldmatrix(uint32_t addr, uint32_t r[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr)
                 : "memory");
}

__device__ __forceinline__ void gram_mma(float c[4], const uint32_t a[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
        "{%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// One warp, one 16 x 16 tile (row blocks bi, bj of the planes), one chunk:
// its levels added to the tile's integers.  Output q of a lane: rows
// lane / 4 + 8 (q / 2 % 2), columns 8 (q / 4) + 2 (lane % 4) + q % 2.
template <int ROWS>
__device__ __forceinline__ void gram_tile(uint32_t planes, int bi, int bj, int ksteps, long long hi[8],
                                          long long lo[8]) {
    const int lane = threadIdx.x & 31;
    const uint32_t ra = planes + 2u * ((bi * 16 + lane % 16) * kGramStride + (lane / 16) * 8);
    const uint32_t rb = planes + 2u * ((bj * 16 + lane % 8 + (lane / 16) * 8) * kGramStride + ((lane / 8) % 2) * 8);
    constexpr uint32_t kPlane = 2u * ROWS * kGramStride;
    float acc[kGramDigits][8];
#pragma unroll
    for (int s = 0; s < kGramDigits; ++s)
#pragma unroll
        for (int q = 0; q < 8; ++q) acc[s][q] = 0.0f;
#pragma unroll 1
    for (int k = 0; k < ksteps; ++k) {
        uint32_t bf[kGramDigits][4];
#pragma unroll
        for (int d = 0; d < kGramDigits; ++d) gram_ldmatrix(rb + d * kPlane + 32u * k, bf[d]);
#pragma unroll
        for (int a = 0; a < kGramDigits; ++a) {
            uint32_t af[4];
            gram_ldmatrix(ra + a * kPlane + 32u * k, af);
#pragma unroll
            for (int d = 0; a + d < kGramDigits; ++d) {
                gram_mma(acc[a + d], af, bf[d][0], bf[d][1]);
                gram_mma(acc[a + d] + 4, af, bf[d][2], bf[d][3]);
            }
        }
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        int L[kGramDigits];
#pragma unroll
        for (int s = 0; s < kGramDigits; ++s) L[s] = __float2int_rn(acc[s][q]);
        // |L_0| < 2^18, |L_s| < 2^23: the pairs fit 32 bits
        hi[q] += static_cast<long long>(L[0] * 256 + L[1]) * 65536 + (L[2] * 256 + L[3]);
        lo[q] += static_cast<long long>(L[4] * 256 + L[5]) * 256 + L[6];
    }
}

// The Gram of one CTA's staged rows.  tile(q, bi, bj): row blocks of tile q
// (q < ntiles); put(ri, rj, g, first): g() is the value of rows ri, rj, added to
// what earlier segments of samples left there unless `first`.
template <int ROWS, class NodeOf, class MeanOut, class TileOf, class Put>
__device__ __forceinline__ void gram_cta(const SeriesView& v, int b, NodeOf node, MeanOut mean_out, int ntiles,
                                         TileOf tile, Put put, __nv_bfloat16* planes, GramNode* nodes,
                                         double* scale) {
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    constexpr int kWarps = kGramThreads / 32;
    gram_stats<ROWS>(v, b, node, mean_out, nodes, scale, reinterpret_cast<double*>(planes));
    const uint32_t pl = static_cast<uint32_t>(__cvta_generic_to_shared(planes));
    for (int q0 = 0; q0 < ntiles; q0 += kWarps * kGramTiles) {
        for (int s0 = 0; s0 < v.T; s0 += kGramSegment) {
            const int s1 = v.T - s0 < kGramSegment ? v.T : s0 + kGramSegment;
            long long hi[kGramTiles][8], lo[kGramTiles][8];
#pragma unroll
            for (int j = 0; j < kGramTiles; ++j)
#pragma unroll
                for (int q = 0; q < 8; ++q) hi[j][q] = lo[j][q] = 0;
            for (int t0 = s0; t0 < s1; t0 += kGramChunk) {
                const int nt = s1 - t0 < kGramChunk ? s1 - t0 : kGramChunk;
                __syncthreads();
                gram_convert<ROWS>(v, b, t0, nt, node, nodes, planes);
                __syncthreads();
#pragma unroll
                for (int j = 0; j < kGramTiles; ++j) {
                    const int q = q0 + warp + kWarps * j;
                    if (q < ntiles) {
                        int bi, bj;
                        tile(q, bi, bj);
                        gram_tile<ROWS>(pl, bi, bj, (nt + 15) / 16, hi[j], lo[j]);
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < kGramTiles; ++j) {
                const int q = q0 + warp + kWarps * j;
                if (q < ntiles) {
                    int bi, bj;
                    tile(q, bi, bj);
#pragma unroll
                    for (int o = 0; o < 8; ++o) {
                        const int ri = bi * 16 + lane / 4 + 8 * ((o / 2) % 2);
                        const int rj = bj * 16 + 8 * (o / 4) + 2 * (lane % 4) + o % 2;
                        put(ri, rj,
                            [&] {
                                return (static_cast<double>(hi[j][o]) +
                                        static_cast<double>(lo[j][o]) * (1.0 / 16777216.0)) *
                                       (scale[ri] * scale[rj]);
                            },
                            s0 == 0);
                    }
                }
            }
        }
    }
    __syncthreads();
}

// Row blocks (bi <= bj) of tile q of the upper triangle, row-major.
__device__ __forceinline__ void gram_triangle(int q, int nb, int& bi, int& bj) {
    bi = 0;
    while (q >= nb - bi) {
        q -= nb - bi;
        ++bi;
    }
    bj = bi + q;
}

// N <= ROWS: one CTA holds the instance.  put(i, j, g, first) for i <= j < N.
template <int ROWS, class MeanOut, class Put>
__device__ __forceinline__ void gram_whole(const SeriesView& v, int b, MeanOut mean_out, Put put,
                                           __nv_bfloat16* planes, GramNode* nodes, double* scale) {
    const int N = v.N, nb = (N + 15) / 16;
    gram_cta<ROWS>(
        v, b, [N](int r) { return r < N ? r : -1; }, mean_out, nb * (nb + 1) / 2,
        [nb](int q, int& bi, int& bj) { gram_triangle(q, nb, bi, bj); },
        [N, &put](int i, int j, auto g, bool first) {
            if (i <= j && j < N) put(i, j, g(), first);
        },
        planes, nodes, scale);
}

// Any N: CTA `pair` of nt (nt + 1) / 2 (nt = ceil(N / 64)) takes one 64 x 64 tile of
// the upper triangle, its 64 + 64 rows staged together.
template <class MeanOut, class Put>
__device__ __forceinline__ void gram_pair(const SeriesView& v, int b, int pair, MeanOut mean_out, Put put,
                                          __nv_bfloat16* planes, GramNode* nodes, double* scale) {
    const int N = v.N;
    int it, jt;
    gram_triangle(pair, (N + 63) / 64, it, jt);
    const int i0 = it * 64, j0 = jt * 64;
    const bool diag = it == jt;
    gram_cta<128>(
        v, b,
        [=](int r) {
            const int n = r < 64 ? i0 + r : (diag ? N : j0 + r - 64);
            return n < N ? n : -1;
        },
        [=](int r, double m) {
            if (diag) mean_out(i0 + r, m);
        },
        diag ? 10 : 16,
        [=](int q, int& bi, int& bj) {
            if (diag) {
                gram_triangle(q, 4, bi, bj);
            } else {
                bi = q / 4;
                bj = 4 + q % 4;
            }
        },
        [=, &put](int ri, int rj, auto g, bool first) {
            const int i = i0 + ri, j = diag ? i0 + rj : j0 + rj - 64;
            if (i <= j && j < N) put(i, j, g(), first);
        },
        planes, nodes, scale);
}

}  // namespace tvbg
