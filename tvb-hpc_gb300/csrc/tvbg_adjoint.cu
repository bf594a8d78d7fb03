// Reverse-time adjoint of the delayed Euler scheme (Montbrio-Pazo-Roxin,
// linear coupling): one CTA per instance and one thread per node
// (adjoint_mpr_kernel), or lane-interleaved groups of 8 instances,
// time-blocked (adjoint_group_kernel).  The recursion and its terms are
// documented at tvbg_adjoint_mpr in tvbg.h.
#include <cuda_runtime.h>

#include <cstring>

#include "tvbg_abi_internal.h"
#include "tvbg_device.cuh"
#include "tvbg_lanes.cuh"

namespace tvbg {

// One reverse step of one node, shared by both kernels so that they compute
// the same numbers.  adj_mu_r: mu_r(t+1) = lambda_r(t+1), masked where the
// rate update of step t was clamped at 0 (rpre as MPR::drift computes it).
struct AdjMpr {
    float J, tau, dt;
    float f0, itau, c2;   // Delta / (pi tau), 1 / tau, 2 pi^2 tau^2
    double c;             // dt / tau

    __device__ __forceinline__ AdjMpr(const float* consts, float dt_) : J(consts[1]), tau(consts[2]), dt(dt_) {
        const float pi = 3.14159265358979323846f;
        f0 = consts[0] / (pi * tau);
        itau = 1.0f / tau;
        c2 = __fmul_rn(__fmul_rn(__fmul_rn(__fmul_rn(2.0f, pi), pi), tau), tau);
        c = static_cast<double>(__fdiv_rn(dt, tau));
    }

    __device__ __forceinline__ float mu_r(float r, float V, float lr) const {
        const float fr = __fmul_rn(__fmaf_rn(__fmul_rn(2.0f, r), V, f0), itau);  // as MPR::drift
        const float rpre = __fmaf_rn(dt, fr, r);
        return rpre >= 0.0f ? lr : 0.0f;
    }

    // lambda(t) from mu(t+1) = (mr, mv), the coupling gather and dL/dr(t).
    // Every rounding is spelled out (no contraction left to the compiler), so
    // both kernels produce the same bits.  UNIT: tau = 1 (the model's
    // default), where x / tau is x and the three divisions of a step, each a
    // reciprocal with its correction, go.
    template <bool UNIT>
    __device__ __forceinline__ void update(float r, float V, float mr, float mv, float coup,
                                           float cG, float drt, float& lr, float& lv) const {
        const auto over_tau = [&](float x) { return UNIT ? x : __fdiv_rn(x, tau); };
        const float dfr_dr = over_tau(__fmul_rn(2.0f, V));  // = dfV_dV
        const float dfr_dV = over_tau(__fmul_rn(2.0f, r));
        const float dfV_dr = over_tau(__fsub_rn(__fmul_rn(J, tau), __fmul_rn(c2, r)));
        float nlr = __fmaf_rn(dt, __fmaf_rn(mv, dfV_dr, __fmul_rn(mr, dfr_dr)), mr);
        nlr = __fmaf_rn(cG, coup, nlr);
        const float nlv = __fmaf_rn(dt, __fmaf_rn(mv, dfr_dr, __fmul_rn(mr, dfr_dV)), mv);
        lr = __fadd_rn(nlr, drt);
        lv = nlv;
    }
};

// Partial sums of dL/deta and dL/dG over steps, without their common factor
// dt / tau, which add() applies in one FMA: two FP64 operations a step (the
// FP64 pipe does two a cycle and SM, 100 cycles for each operation of 21
// nodes; with the factor in every step the group kernel took 987 us where it
// takes 880, 84 nodes, 256 instances, 2000 steps).
struct AdjSums {
    double m = 0.0, mS = 0.0;

    __device__ __forceinline__ void step(float mv, float S) {
        const double d = static_cast<double>(mv);
        m = __dadd_rn(m, d);
        mS = __fma_rn(d, static_cast<double>(S), mS);
    }
    __device__ __forceinline__ void add(double c, double* deta, double* dG) {
        *deta = __fma_rn(c, m, *deta);
        *dG = __fma_rn(c, mS, *dG);
        m = mS = 0.0;
    }
};

// The adjoint ring of mu_V: global memory, or staged in shared memory for
// the kernel's run (loaded at the start, stored at the end: it carries mu_V
// across segments).
template <bool SMEM>
struct AdjRing;
template <>
struct AdjRing<false> {
    float* p;
    __device__ __forceinline__ float ld(uint32_t i) const { return p[i]; }
    __device__ __forceinline__ void st(uint32_t i, float v) const { p[i] = v; }
};
template <>
struct AdjRing<true> {
    float* p;  // shared
    __device__ __forceinline__ float ld(uint32_t i) const { return p[i]; }
    __device__ __forceinline__ void st(uint32_t i, float v) const { p[i] = v; }
};

template <bool SMEM>
__device__ __forceinline__ void adjoint_segment(const tvbg_adjoint& a, AdjRing<SMEM> ring) {
    const int j = threadIdx.x;
    const int N = a.N;
    const bool own = j < N;
    const uint32_t lognh = static_cast<uint32_t>(a.lognh);
    const uint32_t mask = (1u << lognh) - 1u;
    const AdjMpr m(a.consts, a.dt);
    const float cG = a.dt * a.G / a.consts[2];
    float lr = 0.f, lv = 0.f;
    AdjSums sums;
    int lo = 0, hi = 0;
    if (own) {
        lr = a.lam[2 * j];
        lv = a.lam[2 * j + 1];
        lo = __ldg(a.row_t + j);
        hi = __ldg(a.row_t + j + 1);
    }
    const uint32_t my_row = static_cast<uint32_t>(j) << lognh;
    const uint2* __restrict__ edges = reinterpret_cast<const uint2*>(a.edges_t);
    for (int k = a.len - 1; k >= 0; --k) {
        const long long t = a.t0 + k;
        const uint32_t tm = static_cast<uint32_t>(t) & mask;
        float r = 0.f, V = 0.f, S = 0.f, mr = 0.f, mv = 0.f;
        if (own) {
            const long long sl = a.seg_lanes > 1 ? a.seg_lanes : 1;
            const float* x = a.seg + (static_cast<long long>(k) * N + j) * 3 * sl;
            r = x[0];
            V = x[sl];
            S = x[2 * sl];
            mr = m.mu_r(r, V, lr);
            mv = lv;
            ring.st(my_row | ((tm + 1u + static_cast<uint32_t>(j)) & mask), mv);
        }
        __syncthreads();
        if (own) {
            // out-edges in order, four loads in flight
            float coup = 0.0f;
            int e = lo;
            for (; e + 4 <= hi; e += 4) {
                float v[4], w[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const uint2 ew = __ldg(edges + e + u);
                    v[u] = ring.ld(((tm + ew.x) & mask) | (ew.x & ~mask));
                    w[u] = __uint_as_float(ew.y);
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) coup = fmaf(w[u], v[u], coup);
            }
            for (; e < hi; ++e) {
                const uint2 ew = __ldg(edges + e);
                coup = fmaf(__uint_as_float(ew.y), ring.ld(((tm + ew.x) & mask) | (ew.x & ~mask)), coup);
            }
            m.update<false>(r, V, mr, mv, coup, cG, a.dr[static_cast<long long>(k) * N + j], lr, lv);
            sums.step(mv, S);
        }
        __syncthreads();
    }
    if (own) {
        a.lam[2 * j] = lr;
        a.lam[2 * j + 1] = lv;
        sums.add(m.c, a.deta + j, a.dG + j);
    }
}

// smem_ring: bytes of shared memory for the ring (0 = global); an instance
// whose ring does not fit uses the global ring.
__global__ void __launch_bounds__(1024, 1)
    adjoint_mpr_kernel(const tvbg_adjoint* __restrict__ adj, int32_t n_inst, uint32_t smem_ring) {
    extern __shared__ __align__(16) float s_ring[];
    if (static_cast<int>(blockIdx.x) >= n_inst) return;
    const tvbg_adjoint a = adj[blockIdx.x];
    const uint32_t floats = static_cast<uint32_t>(a.N) << a.lognh;
    if (smem_ring >= 4u * floats && a.N > 0) {
        for (uint32_t i = threadIdx.x; i < floats; i += blockDim.x) s_ring[i] = a.ring[i];
        __syncthreads();
        adjoint_segment<true>(a, AdjRing<true>{s_ring});
        for (uint32_t i = threadIdx.x; i < floats; i += blockDim.x) a.ring[i] = s_ring[i];
    } else {
        adjoint_segment<false>(a, AdjRing<false>{a.ring});
    }
}

// ---------------------------------------------------------------------------
// Lane-interleaved groups, time-blocked
// ---------------------------------------------------------------------------

// One group per CTA (or cluster of C CTAs): thread t of CTA r is lane
// l = t % 8 of node slot q = (t / 8) C + r.  Per block of K reverse steps
// (tb, tb - 1, ..., tb - K + 1): the gather of all K steps (reads slots
// t + 1 + d >= tb + 2, written by earlier blocks since d >= K), then the K
// updates from registers, each writing mu_V(t + 1) to slot t + 1, then one
// barrier.  A slot written in a block aliases slot + nh, which no read of
// the block reaches (nh >= d_max + K).  The gather is the forward group
// kernel's (gather_run over records staged in shared memory): the out-edge
// records of a node are the in-edge records of the transposed network.
//
// PIPE: two thread teams of blockDim / 2 on the same (node slot, lane)
// pairs; the update team runs block b from one coupling-sum buffer while
// the gather team sums block b + 1 into the other.  Block b + 1 reads slots
// >= tb - 2K + 2 + d_min, all written before block b started when
// d_min >= 2K; the slots block b writes ([tb - K + 2, tb + 1]) alias none of
// them (nh > d_max - 1).  The CTAs of a cluster meet by ClusterPhases.  With
// d_min >= 3K (lag) the gather of phase b reads nothing newer than block
// b - 2, so a phase is published by one warp during the next one and awaited
// at that one's end.  A CTA may then be one phase ahead, writing slots down
// to tb - 2K + 2 while another reads up to tb - K + 1 + d_max: nh >= d_max + K
// keeps them apart.  Same per-step code and gather order: the same results.
//
// What bounds it: the steps of the update team, their serial chain and FP64
// sums (without the coupling gather the kernel takes the same time).  The
// trace and dL/dr of a step come from DRAM; each step reads those of the
// same step of the next block into the registers it has just used, so that
// they have a block's time to arrive.
template <int K, bool PIPE>
__global__ void __launch_bounds__(512, 1)
    adjoint_group_kernel(const tvbg_adjoint_group* __restrict__ adj, int32_t n_groups,
                         int32_t* __restrict__ status) {
    __shared__ __align__(16) tvbg_adjoint_group s;
    __shared__ EdgeStage stage;
    __shared__ ClusterPhases phases;
    extern __shared__ __align__(16) float csum[];  // [(PIPE ? 2 : 1)][K][team threads]: out-edge sums; records
    const int cid = static_cast<int>(cluster_id_x());
    if (cid >= n_groups) return;  // uniform over the cluster
    {
        static_assert(sizeof(tvbg_adjoint_group) % 4 == 0, "record size");
        const uint32_t* src = reinterpret_cast<const uint32_t*>(adj + cid);
        uint32_t* dst = reinterpret_cast<uint32_t*>(&s);
        for (int i = threadIdx.x; i < static_cast<int>(sizeof(tvbg_adjoint_group) / 4); i += blockDim.x)
            dst[i] = __ldg(src + i);
        __syncthreads();
    }
    const uint32_t C = cluster_nranks();
    const uint32_t rank = cluster_rank();
    const bool cluster = C > 1;
    const int N = s.N;
    const int H = PIPE ? static_cast<int>(blockDim.x) / 2 : static_cast<int>(blockDim.x);
    const int P = H / kLanes;
    if (N < 1 || N > 65535 || static_cast<int>(C) * P < N || s.lognh < 1 || s.lognh > 16 ||
        (1 << s.lognh) < K || s.dmin < (PIPE ? 2 * K : K) || (H & 31) || s.len < 0 || s.lanes < 1 ||
        s.lanes > kLanes || !s.ring || !s.seg || !s.edges_t || !s.row_t ||
        (reinterpret_cast<uintptr_t>(s.ring) & 15u) != 0) {
        if (threadIdx.x == 0) report(status, TVBG_EINVAL);
        return;  // uniform over the cluster: same record, same launch shape
    }
    const bool lag = s.dmin >= 3 * K;
    const bool gather_team = PIPE && static_cast<int>(threadIdx.x) >= H;
    const int tid = static_cast<int>(threadIdx.x) - (gather_team ? H : 0);
    const int l = tid % kLanes;
    const int q = (tid / kLanes) * static_cast<int>(C) + static_cast<int>(rank);
    const bool valid = q < N;
    const int n = valid ? (s.nodes ? __ldg(s.nodes + q) : q) : 0;
    const bool live = valid && l < s.lanes;
    const uint32_t nh = 1u << s.lognh;
    const uint32_t mask = nh - 1u;
    const uint32_t R = nh + K;
    float* const ring = s.ring;
    float* cs = csum + (tid - l);
    const int bufsz = K * H;
    const long long t0 = s.t0;
    const int len = s.len;
    const long long top = t0 + len - 1;
    const int lo = valid ? __ldg(s.row_t + n) : 0;
    const int deg = valid ? __ldg(s.row_t + n + 1) - lo : 0;
    if (PIPE && threadIdx.x == 0) phases.init(C);
    // the gathering threads carry the slots (their tid is the scan's)
    const uint2* edges = stage_edges(reinterpret_cast<const uint2*>(s.edges_t), stage,
                                     reinterpret_cast<uint2*>(csum + (PIPE ? 2 : 1) * bufsz), P,
                                     PIPE && !gather_team ? H + tid : tid, lo, deg);
    const bool vec = run_vec<K, 1>(ring, N, R);
    // out-edge sums of the K steps tb - K + 1 .. tb of this thread's slot
    const auto gather = [&](long long tb, float* dst) {
        const uint32_t tm = static_cast<uint32_t>(tb - K + 2) & mask;
        if (vec)
            gather_run<TVBG_CFUN_LINEAR, K, 1, true, PIPE ? 64 : 32>(ring, nullptr, edges, deg, tm, mask, R, l, dst, H);
        else
            gather_run_any<TVBG_CFUN_LINEAR, K, 1>(ring, nullptr, edges, deg, tm, mask, R, l, dst, H);
    };
    if (PIPE) group_barrier(cluster);  // the phases are initialised
    if (gather_team) {
        // the last gather warp, whose nodes have the fewest edges, keeps the phases
        const bool keeper = cluster && tid >= H - 32;
        if (len > 0) gather(top, cs);
        __syncthreads();
        uint32_t ph = 0;  // phases ended
        for (long long tb = top; tb >= t0; tb -= K) {
            if (keeper && lag && ph > 0) phases.publish(C);
            if (tb - K >= t0) gather(tb - K, cs + ((ph + 1) & 1u) * bufsz);
            if (keeper && lag && ph > 0) phases.await(ph - 1, ph);
            __syncthreads();
            if (cluster && !lag) {
                if (keeper) {
                    phases.publish(C);
                    phases.await(ph, ph);
                }
                __syncthreads();
            }
            if (cluster && phases.failed(ph)) break;
            ++ph;
        }
    } else {
        const AdjMpr m(s.consts, s.dt);
        const float cG = s.dt * s.G[l] / s.consts[2];
        float lr = 0.0f, lv = 0.0f;
        if (live) {
            lr = s.lam[2LL * N * l + 2 * n];
            lv = s.lam[2LL * N * l + 2 * n + 1];
        }
        AdjSums sums;
        double* const deta_n = s.deta + static_cast<long long>(N) * l + n;
        double* const dG_n = s.dG + static_cast<long long>(N) * l + n;
        float* __restrict__ ring_n = ring + static_cast<size_t>(n) * R * kLanes + l;
        // step t0 + k of this thread: r, V and S at seg_k, dL/dr at dr_k;
        // read in the order of the steps, a block ahead of their use
        const long long seg_row = 3LL * kLanes * N;
        int kload = len - 1;
        const float* __restrict__ seg_k = s.seg + (static_cast<size_t>(n) * 3 * kLanes + l) + kload * seg_row;
        const float* __restrict__ dr_k = s.dr + s.dr_stride * l + n + static_cast<long long>(kload) * N;
        float r[K], V[K], S[K], drt[K];
        const auto load = [&](int i) {
            if (kload >= 0) {
                r[i] = __ldg(seg_k);
                V[i] = __ldg(seg_k + kLanes);
                S[i] = __ldg(seg_k + 2 * kLanes);
                if (live) drt[i] = __ldg(dr_k);
            }
            seg_k -= seg_row;
            dr_k -= N;
            --kload;
        };
#pragma unroll
        for (int i = 0; i < K; ++i) {
            r[i] = V[i] = S[i] = drt[i] = 0.0f;
            load(i);
        }
        if (PIPE) __syncthreads();  // block 0's sums
        // partial sums go to memory after each step t with
        // t % flush_every == 0 (the grouping of one launch per segment):
        // after `until` more steps
        const int fe = s.flush_every > 0 ? s.flush_every : 0;
        int until = fe ? static_cast<int>(top % fe) : -1;
        bool pending = false;
        const auto block = [&](auto unit, auto whole, long long tb, int cnt, const float* csb) {
#pragma unroll
            for (int i = 0; i < K; ++i) {
                if (!whole.value && i >= cnt) break;
                const float mr = m.mu_r(r[i], V[i], lr);
                const float mv = lv;
                if (valid) {
                    const uint32_t pos = static_cast<uint32_t>(tb - i + 1) & mask;
                    ring_n[pos * kLanes] = mv;
                    if (pos < static_cast<uint32_t>(K)) ring_n[(pos + nh) * kLanes] = mv;
                }
                m.update<decltype(unit)::value>(r[i], V[i], mr, mv, csb[(K - 1 - i) * H + l], cG, drt[i], lr, lv);
                sums.step(mv, S[i]);
                load(i);
                pending = true;
                if (until-- == 0) {
                    if (live) sums.add(m.c, deta_n, dG_n);
                    sums = AdjSums();
                    pending = false;
                    until = fe - 1;
                }
            }
        };
        const auto run = [&](auto unit) {
            uint32_t ph = 0;
            for (long long tb = top; tb >= t0; tb -= K) {
                const int cnt = (tb - t0 + 1) < K ? static_cast<int>(tb - t0 + 1) : K;
                if (!PIPE) {
                    gather(tb, cs);
                    __syncwarp();
                }
                const float* csb = PIPE ? cs + (ph & 1u) * bufsz : cs;
                if (cnt == K)
                    block(unit, Flag<true>{}, tb, K, csb);
                else
                    block(unit, Flag<false>{}, tb, cnt, csb);
                if (PIPE) {
                    __syncthreads();
                    if (cluster && !lag) __syncthreads();
                    if (cluster && phases.failed(ph)) break;
                } else {
                    group_barrier(cluster);
                }
                ++ph;
            }
        };
        if (m.tau == 1.0f)
            run(Flag<true>{});
        else
            run(Flag<false>{});
        if (live) {
            s.lam[2LL * N * l + 2 * n] = lr;
            s.lam[2LL * N * l + 2 * n + 1] = lv;
            if (pending) sums.add(m.c, deta_n, dG_n);
        }
    }
    if (PIPE && cluster) {
        if (threadIdx.x == 0 && phases.fail) report(status, TVBG_ETIMEOUT);
        group_barrier(true);  // no CTA leaves while another may still arrive on its phases
    }
}

}  // namespace tvbg

using namespace tvbg;

extern "C" size_t tvbg_adjoint_group_size(void) { return sizeof(tvbg_adjoint_group); }

extern "C" int tvbg_adjoint_mpr_groups(const tvbg_adjoint_group* d_adj, int32_t n_groups,
                                       int32_t threads, int32_t cluster, int32_t block_k,
                                       int32_t pipelined, int32_t* d_status, void* stream) {
    if (n_groups < 0 || (n_groups > 0 && !d_adj) || threads < 32 || threads > 512 || (threads & 31) ||
        cluster < 1 || cluster > 16 || (block_k != 4 && block_k != 8) || pipelined < 0 ||
        pipelined > 1 || (pipelined && (threads & 63)))
        return set_error(TVBG_EINVAL, "tvbg_adjoint_mpr_groups: bad arguments");
    if (n_groups == 0) return TVBG_OK;
    using Fn = void (*)(const tvbg_adjoint_group*, int32_t, int32_t*);
    const Fn kfn = pipelined ? (block_k == 8 ? adjoint_group_kernel<8, true> : adjoint_group_kernel<4, true>)
                             : (block_k == 8 ? adjoint_group_kernel<8, false> : adjoint_group_kernel<4, false>);
    const size_t smem = 4u * static_cast<size_t>(block_k) * static_cast<size_t>(threads) +
                        static_cast<size_t>(stage_bytes(pipelined ? threads / 2 : threads));
    cudaError_t e = cudaSuccess;
    if (cluster > 8) {
        e = cudaFuncSetAttribute(reinterpret_cast<const void*>(kfn),
                                 cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        if (e != cudaSuccess) return set_cuda_error(e, "tvbg_adjoint_mpr_groups: cluster attribute");
    }
    cudaLaunchConfig_t lc;
    std::memset(&lc, 0, sizeof(lc));
    lc.gridDim = dim3(static_cast<unsigned>(n_groups) * static_cast<unsigned>(cluster), 1, 1);
    lc.blockDim = dim3(static_cast<unsigned>(threads), 1, 1);
    lc.dynamicSmemBytes = smem;
    lc.stream = static_cast<cudaStream_t>(stream);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = static_cast<unsigned>(cluster);
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    lc.attrs = attr;
    lc.numAttrs = cluster > 1 ? 1 : 0;
    e = cudaLaunchKernelEx(&lc, kfn, d_adj, n_groups, d_status);
    if (e != cudaSuccess) return set_cuda_error(e, "tvbg_adjoint_mpr_groups launch");
    return TVBG_OK;
}

static int adjoint_launch(const tvbg_adjoint* d_adj, int32_t n_inst, int32_t threads,
                          int32_t smem_ring, void* stream) {
    if (!d_adj || n_inst < 0 || threads < 32 || threads > 1024 || (threads & 31) || smem_ring < 0)
        return set_error(TVBG_EINVAL, "tvbg_adjoint_mpr: bad arguments");
    if (n_inst == 0) return TVBG_OK;
    const size_t smem = static_cast<size_t>(smem_ring);
    if (smem > 48u * 1024u) {
        int dev = 0, optin = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e == cudaSuccess)
            e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
        if (e != cudaSuccess) return set_cuda_error(e, "tvbg_adjoint_mpr: device attributes");
        if (smem > static_cast<size_t>(optin))
            return set_error(TVBG_EINVAL, "tvbg_adjoint_mpr: ring exceeds the shared memory of one CTA");
        e = cudaFuncSetAttribute(reinterpret_cast<const void*>(adjoint_mpr_kernel),
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
        if (e != cudaSuccess) return set_cuda_error(e, "tvbg_adjoint_mpr: smem attribute");
    }
    adjoint_mpr_kernel<<<n_inst, threads, smem, static_cast<cudaStream_t>(stream)>>>(
        d_adj, n_inst, static_cast<uint32_t>(smem_ring));
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return set_cuda_error(e, "tvbg_adjoint_mpr launch");
    return TVBG_OK;
}

extern "C" int tvbg_adjoint_mpr(const tvbg_adjoint* d_adj, int32_t n_inst, int32_t threads,
                                void* stream) {
    return adjoint_launch(d_adj, n_inst, threads, 0, stream);
}

extern "C" int tvbg_adjoint_mpr_ex(const tvbg_adjoint* d_adj, int32_t n_inst, int32_t threads,
                                   int32_t smem_ring, void* stream) {
    return adjoint_launch(d_adj, n_inst, threads, smem_ring, stream);
}
