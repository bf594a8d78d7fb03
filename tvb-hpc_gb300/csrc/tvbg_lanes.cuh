// Lane-interleaved group kernel: TVBG_GROUP_LANES (8) instances that share a
// connectome, a delay table, the model constants and t0 run together, one
// instance per lane of an 8-lane slice of a warp.
//
// Canonical step (CUDA order, the same as tvbg_step.cuh and
// tvbg_step_blocked.cuh; tvb_hpc/network.py:115-143, coupling.py:103-116,
// model.py:131-155, scheme.py:88-107, ring addressing of
// dsl/dsl_cuda/CUDAmodels/kuramoto.c:92,108,128):
//   S     = sum_e w_e pre(ring[t - d_e][col_e])          (CSR order)
//   c     = post(S, obs0(x_i), sum_e w_e)
//   x'    = limit(x + dt f(x, c, p) + sqrt(dt) sigma z)   z: Philox(seed_lo, inst; node, t/SPC, seed_hi)
//           (Box-Muller with CUDA's fast intrinsics, box_muller_fast)
//   ring[t+1][i] = obs0(x')
//
// Layout.  Every per-node quantity is interleaved over the 8 instances of
// the group, so a lane slice reading "node j, slot s" reads 32 contiguous
// bytes -- one DRAM/L2 sector -- and the edge record (column, delay,
// weight) is the same for the 8 lanes:
//   ring   [N][R][8], R = nh + 8: slot s of node j at (j R + (s & (nh-1))) 8 + l,
//          positions < 8 mirrored at +nh so a run of K <= 8 slots never wraps;
//          with the Kuramoto coupling [N][R][2][8]: sin and cos of the observable
//   state  [N][NS][8], nparam [N][NP][8], bold [4][N][8],
//   bold_out [bold_len][N][8], trace [trace_len][N][trace_nobs][8].
//
// Thread mapping.  Thread t of CTA r (cluster of C CTAs) is lane l = t % 8
// of node slot q = t / 8; node slot q of CTA r serves the node positions
// q C + r, q C + r + C P, ... (P = blockDim / 8) of the group's node order
// (the host sorts nodes by in-degree, so the slots of a warp see similar
// edge counts and the C CTAs of a cluster the same work).
//
// Time blocking.  A value written at step t is first read at t + 1 + d_min,
// so the K <= d_min + 1 steps of a block read only slots that exist when the
// block starts; with nh >= d_max + 1 + K no slot written in a block aliases
// one read in it.  The cluster meets at one barrier per block.
//
// Gather.  The 8 lanes of a node slot sum its in-edges for the K steps of the
// block: the K slots of an edge are one run of consecutive floats, split over
// the lanes in 32-byte loads (gather_run), and the sums cross to their owners
// through shared memory.  L2 serves such runs to one CTA of 512 threads per
// SM at 21.6 TB/s from a 48 MB working set, 17.0 TB/s from 96 MB and 9.1 TB/s
// from 192 MB, in 32-byte loads or in two 16-byte loads that are contiguous
// over the lanes (21.4, 16.2, 9.2); one float per lane and load reached 10.0, 9.2
// and 7.2, two 16-byte loads of a lane's own 32 bytes 10.7, 10.6 and 8.6.
// (Staging the runs in shared memory with cp.async.bulk was measured slower;
// a rolling window of loads or predicated loads inside the batch spill at
// these register counts and were slower too.)
//
// What bounds it.  Per block of 8 steps, N = 84 on clusters of 2 CTAs (128
// groups of MPR with noise): gather 8300-9000 cycles, update 4400, the CTA
// barrier and phase handling under 700; before, two waits of 2300 cycles at
// cluster barriers that also dropped the L1 lines of the edge records.
// 128 groups x 84 nodes x 800 steps: 1.62 ms before, 0.89 now; 32 groups
// on 6 CTAs each 0.674 -> 0.320; N = 192 (32 groups) 1.065 -> 0.55; N = 998
// (2 groups) 1.284 -> 0.67.
#pragma once

#include "tvbg_step_blocked.cuh"

namespace tvbg {

constexpr int kLanes = TVBG_GROUP_LANES;

// Steps of a whole block unrolled together (update_node).  Per block of 8 MPR
// steps without noise (N = 84, 256 instances): rolled 3000 cycles, 2 at a
// time 1440, 4 at a time 1290; 8 at a time spills and was slower.
constexpr int kStepUnroll = 4;

// Floats in flight per gather thread in a kernel built for CTAs of at most
// `bound` threads: 128, 80 or 64 registers a thread for 512, 768 or 1024.
__host__ __device__ constexpr int gather_floats(int bound) { return bound <= 512 ? 64 : 32; }


__device__ __forceinline__ uint32_t cluster_nranks() {
    uint32_t n;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(n));
    return n;
}
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t cluster_id_x() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%clusterid.x;" : "=r"(r));
    return r;
}

// Block barrier of the group: the CTA, or every CTA of the cluster.
__device__ __forceinline__ void group_barrier(bool cluster) {
    if (cluster) {
        asm volatile("barrier.cluster.arrive.release.aligned;\n\t"
                     "barrier.cluster.wait.acquire.aligned;" ::: "memory");
    } else {
        __syncthreads();
    }
}

// Copy a group descriptor into shared memory (word-parallel).
__device__ __forceinline__ void stage_group(const tvbg_group* src, tvbg_group* dst) {
    static_assert(sizeof(tvbg_group) % 4 == 0, "descriptor size");
    const uint32_t* s = reinterpret_cast<const uint32_t*>(src);
    uint32_t* d = reinterpret_cast<uint32_t*>(dst);
    for (int i = threadIdx.x; i < static_cast<int>(sizeof(tvbg_group) / 4); i += blockDim.x)
        d[i] = __ldg(s + i);
    __syncthreads();
}

// Normal number r (0..3) of one Philox call, without dynamic indexing.
__device__ __forceinline__ float pick4(const float z[4], int r) {
    const float a = (r & 1) ? z[1] : z[0];
    const float b = (r & 1) ? z[3] : z[2];
    return (r & 2) ? b : a;
}

template <int CF>
__device__ __forceinline__ float lane_pre(float xj, const float* cf_p) {
    if constexpr (CF == TVBG_CFUN_SIGMOIDAL) {
        return cf_p[0] / (1.0f + expf(cf_p[2] * (cf_p[1] - xj)));
    } else {
        return xj;
    }
}

template <int CF>
__device__ __forceinline__ float lane_post(float S, float xi, float wsum, float a, float b) {
    if constexpr (CF == TVBG_CFUN_DIFF) {
        return a * (S - xi * wsum) + b;
    } else if constexpr (CF == TVBG_CFUN_SIGMOIDAL) {
        return a * S;
    } else {
        return a * S + b;
    }
}

// W consecutive floats at p (W * 4-byte aligned) in one load, cached in L2
// only: with a cluster the values come from other SMs.
template <int W>
__device__ __forceinline__ void ldcg_run(const float* p, float v[W]) {
    if constexpr (W == 8) {
        asm volatile("ld.global.cg.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]),
                       "=f"(v[6]), "=f"(v[7])
                     : "l"(p));
    } else if constexpr (W == 4) {
        const float4 q = __ldcg(reinterpret_cast<const float4*>(p));
        v[0] = q.x;
        v[1] = q.y;
        v[2] = q.z;
        v[3] = q.w;
    } else if constexpr (W == 2) {
        const float2 q = __ldcg(reinterpret_cast<const float2*>(p));
        v[0] = q.x;
        v[1] = q.y;
    } else {
        v[0] = __ldcg(p);
    }
}

// Coupling sums of one node slot (deg in-edges at edges, shared or global
// memory) for the K steps of the block at ring position tm.  The K slots an edge reads are one run of
// 8 K NC consecutive floats (step-major, then channel, then instance), and
// the 8 lanes of the slot split that run instead of each taking its own
// instance: load j of lane l covers floats j 64 + l W .. + W - 1, so a warp
// instruction moves whole 32-byte sectors, W floats per lane (W = 8: one
// 32-byte load per edge and lane).  acc sums w_e pre(v_e) of its (step,
// channel, instance) in CSR order, pairs of them in one packed FP32 FMA
// (__ffma2_rn: each half rounded as fmaf).  The sums cross to their
// owners through shared memory: cs_slot[(ch K + k) stride + m] holds step k
// of instance m (the caller orders the reads after the writes).
// VEC: run_vec holds (every ring of the Python layer); otherwise W scalar
// loads and 64-bit indices.
template <int CF, int K, int NC, bool VEC, int FLOATS>
__device__ __forceinline__ void gather_run(const float* __restrict__ ring_g, const float* cf_p, const uint2* edges,
                                           int deg, uint32_t tm, uint32_t mask, uint32_t R, int l, float* cs_slot,
                                           int stride) {
    constexpr int F = K * NC;               // floats of a run per lane
    constexpr int W = F < 8 ? F : 8;        // floats per load
    constexpr int NJ = F / W;               // loads per edge and lane
    constexpr int U = !VEC ? 1 : (FLOATS / F < 8 ? FLOATS / F : 8);  // edges in flight
    const float* __restrict__ ring = ring_g + l * W;
    float2 acc[NJ][(W + 1) / 2];
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
        for (int i = 0; i < (W + 1) / 2; ++i) acc[j][i] = make_float2(0.0f, 0.0f);
    // No branch inside a batch: the loads past the last edge repeat it and
    // their products are dropped, so U ring loads leave back to back.
    for (int e = 0; e < deg; e += U) {
        float v[U][NJ][W];
        float w[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint2 ed = edges[min(e + u, deg - 1)];
            w[u] = __uint_as_float(ed.y);
            // the ring mask is below 2^16; N R < 2^32 where VEC (run_vec)
            const uint32_t pos = (tm + ed.x) & mask;
            const size_t row = VEC ? static_cast<size_t>((ed.x >> 16) * R + pos)
                                   : static_cast<size_t>(ed.x >> 16) * R + pos;
            const float* p = ring + row * (kLanes * NC);
#pragma unroll
            for (int j = 0; j < NJ; ++j) {
                if constexpr (VEC) {
                    ldcg_run<W>(p + 64 * j, v[u][j]);
                } else {
#pragma unroll
                    for (int i = 0; i < W; ++i) ldcg_run<1>(p + 64 * j + i, &v[u][j][i]);
                }
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (e + u < deg) {
                const float2 ww = make_float2(w[u], w[u]);
#pragma unroll
                for (int j = 0; j < NJ; ++j) {
                    if constexpr (W == 1) {
                        acc[j][0].x = fmaf(w[u], lane_pre<CF>(v[u][j][0], cf_p), acc[j][0].x);
                    } else {
#pragma unroll
                        for (int i = 0; i < W / 2; ++i)
                            acc[j][i] = __ffma2_rn(ww,
                                                   make_float2(lane_pre<CF>(v[u][j][2 * i], cf_p),
                                                               lane_pre<CF>(v[u][j][2 * i + 1], cf_p)),
                                                   acc[j][i]);
                    }
                }
            }
        }
    }
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
        const int o = 64 * j + l * W;   // first float of this lane's part of the run
        float* dst = cs_slot + (((o / kLanes) % NC) * K + o / (kLanes * NC)) * stride + o % kLanes;
        if constexpr (W >= 4) {
#pragma unroll
            for (int i = 0; i < W / 4; ++i)
                reinterpret_cast<float4*>(dst)[i] = make_float4(acc[j][2 * i].x, acc[j][2 * i].y,
                                                                acc[j][2 * i + 1].x, acc[j][2 * i + 1].y);
        } else if constexpr (W == 2) {
            *reinterpret_cast<float2*>(dst) = acc[j][0];
        } else {
            dst[0] = acc[j][0].x;
        }
    }
}

// gather_run for a ring of any alignment, out of line: its registers stay
// out of the callers' loops.
template <int CF, int K, int NC>
__device__ __noinline__ void gather_run_any(const float* ring, const float* cf_p, const uint2* edges, int deg,
                                            uint32_t tm, uint32_t mask, uint32_t R, int l, float* cs_slot,
                                            int stride) {
    gather_run<CF, K, NC, false, 16>(ring, cf_p, edges, deg, tm, mask, R, l, cs_slot, stride);
}

// Whether a ring takes gather_run's vector loads and 32-bit row indices.
template <int K, int NC>
__device__ __forceinline__ bool run_vec(const float* ring, int N, uint32_t R) {
    constexpr uint32_t align = K * NC < 8 ? 4u * K * NC : 32u;
    return (reinterpret_cast<uintptr_t>(ring) & (align - 1u)) == 0 &&
           static_cast<unsigned long long>(N) * R <= 0xffffffffull;
}

// Ring channels per (node, slot): 2 (sin, cos) for the Kuramoto coupling and
// the LEMS sine coupling, 2 for a LEMS model's two couplings, else 1.
template <int CF>
__host__ __device__ constexpr int ring_channels() {
    return (CF == TVBG_CFUN_KURAMOTO || CF == TVBG_CFUN_LEMS_SC || CF == TVBG_CFUN_LEMS_2) ? 2 : 1;
}

// Value a one-channel ring slot holds for observable o: o itself, or for a
// LEMS model its separable pre-synaptic term pre(o), so the gather sums
// w_e * pre(x_j) without evaluating pre per edge.
template <class M, int CF>
__device__ __forceinline__ float ring_val(float o, const float* p) {
    if constexpr (CF == TVBG_CFUN_LEMS) {
        return M::ring_value(o, p);
    } else {
        return o;
    }
}

// Static shared memory of a group CTA, at most (the descriptor, the edge
// offsets and the cluster phases).
constexpr size_t kGroupStaticBytes = sizeof(tvbg_group) + 640;

// Bytes of staged edge records for node slots of `threads` lanes.
constexpr int kStageEdges = 48;
__host__ __device__ constexpr int stage_bytes(int threads) { return threads / kLanes * kStageEdges * 8; }

// Dynamic shared memory of a group CTA: the K coupling sums (per ring
// channel) of every thread, and the staged edge records.
__host__ __device__ constexpr uint32_t group_smem_bytes(int K, int threads, int nc) {
    return static_cast<uint32_t>(4 * K * threads * nc + stage_bytes(threads));
}

// Per-thread constants of a group run (lane l of one node slot).
struct GroupLane {
    int l;                  // lane = instance of the group
    uint32_t nh, mask, R;   // ring length, mask, row length (nh + ghost slots)
    uint32_t flags;
    bool noise, bold, trace;
    bool vec;               // ring aligned for gather_run's vector loads
    float cf_a;
    long long t0, t_end;    // this lane updates while t < t_end
    uint32_t inst_id;
};

// allow_csum: the pipelined kernel's one-channel couplings can write the
// raw coupling sum into the trace (TVBG_F_TRACE_CSUM).
template <class M, int CF>
__device__ __forceinline__ bool group_descriptor_ok(const tvbg_group& g, bool allow_csum = false) {
    const int N = g.N;
    const uint32_t bad = TVBG_F_TRACKA | TVBG_F_MIDSYNC |
                         ((allow_csum && ring_channels<CF>() == 1) ? 0u : TVBG_F_TRACE_CSUM);
    return !(N <= 0 || N > 65535 || g.lognh < 3 || g.lognh > 16 || g.model != M::ID || g.cfun != CF ||
             g.nsteps < 0 || (g.flags & bad) ||
             (!Noise<M>::kOK && !WideNoise<M>::value && (g.flags & TVBG_F_NOISE)));
}

template <class M, int CF, int K>
__device__ __forceinline__ GroupLane make_lane(const tvbg_group& g, int l) {
    GroupLane c;
    c.l = l;
    c.nh = 1u << g.lognh;
    c.mask = c.nh - 1u;
    c.R = c.nh + kGhost;
    c.flags = g.flags;
    c.noise = (g.flags & TVBG_F_NOISE) != 0;
    c.bold = (g.flags & TVBG_F_BOLD) != 0 && g.bold != nullptr && g.bold_out != nullptr;
    c.trace = (g.flags & TVBG_F_TRACE) != 0 && g.trace != nullptr;
    c.vec = run_vec<K, ring_channels<CF>()>(g.ring, g.N, c.R);
    c.cf_a = g.lanes[l].cf_a;
    const int my_steps = g.lanes[l].nsteps < g.nsteps ? g.lanes[l].nsteps : g.nsteps;
    c.inst_id = g.lanes[l].inst_id;
    c.t0 = g.t0;
    c.t_end = g.t0 + my_steps;
    return c;
}

// Seed: ring slot t0 of node n holds obs0 (or the ring channels) of the
// state at t0.
template <class M, int CF>
__device__ __forceinline__ void seed_node(const tvbg_group& g, const GroupLane& c, int n) {
    constexpr int NS = M::NS;
    constexpr int NP = M::NP;
    constexpr int NC = ring_channels<CF>();
    constexpr int RL = kLanes * NC;
    const int l = c.l;
    const uint32_t pos = static_cast<uint32_t>(c.t0) & c.mask;
    float x[NS];
#pragma unroll
    for (int v = 0; v < NS; ++v) x[v] = g.state[(n * NS + v) * kLanes + l];
    const size_t idx = (static_cast<size_t>(n) * c.R + pos) * RL + l;
    const float o = M::obs(x, 0);
    float p[NP];
#pragma unroll
    for (int v = 0; v < NP; ++v) p[v] = __ldg(g.nparam + (n * NP + v) * kLanes + l);
    float* __restrict__ ring = g.ring;
    if constexpr (NC == 2) {
        float sn, cs;
        if constexpr (CF == TVBG_CFUN_LEMS_2) {
            sn = M::ring_value(o, p);
            cs = M::ring_value2(x[M::CVAR2], p);
        } else {
            sincosf(o, &sn, &cs);
        }
        ring[idx] = sn;
        ring[idx + kLanes] = cs;
        if (pos < kGhost) {
            ring[idx + static_cast<size_t>(c.nh) * RL] = sn;
            ring[idx + static_cast<size_t>(c.nh) * RL + kLanes] = cs;
        }
    } else {
        const float rv = ring_val<M, CF>(o, p);
        ring[idx] = rv;
        if (pos < kGhost) ring[idx + static_cast<size_t>(c.nh) * kLanes] = rv;
    }
}

// Coupling sums of a node slot's node (degree 0: none) for the K steps of
// the block at ring position tm; edges, cs_slot and stride as gather_run's.
template <class M, int CF, int K, int BOUND>
__device__ __forceinline__ void gather_node(const tvbg_group& g, const GroupLane& c, const uint2* edges, int deg,
                                            uint32_t tm, float* cs_slot, int stride) {
    constexpr int NC = ring_channels<CF>();
    if (c.vec)
        gather_run<CF, K, NC, true, gather_floats(BOUND)>(g.ring, g.cf_p, edges, deg, tm, c.mask, c.R, c.l, cs_slot,
                                                          stride);
    else
        gather_run_any<CF, K, NC>(g.ring, g.cf_p, edges, deg, tm, c.mask, c.R, c.l, cs_slot, stride);
}

// In-edge records of the CTA's node slots, staged in shared memory for the
// whole run.  The acquire side of each block's barrier drops the L1 cache,
// so records read from global memory would come from L2 again in every
// block, in front of the ring reads that need them (measured per block at
// N = 84: 1090 cycles for each four edges, L2's own latency being 290-440).
// `records` holds kStageEdges per slot on average; a CTA with more edges
// than that reads them from global memory.
struct EdgeStage {
    int off[129];   // first record of each node slot (at most 128 slots)
};

// All threads of the CTA; threads [0, 8 P) are the lanes of the P slots,
// with the degree deg of their slot's node and its first edge lo.  Returns
// the slot's records (valid for threads < 8 P).  Ends with a barrier.
__device__ __forceinline__ const uint2* stage_edges(const uint2* edges, EdgeStage& st, uint2* records,
                                                    int P, int tid, int lo, int deg) {
    const int slot = tid / kLanes, l = tid % kLanes;
    if (slot < P && l == 0) st.off[slot + 1] = deg;
    __syncthreads();
    if (tid < 32) {  // exclusive scan of at most 128 degrees by one warp
        int base = 0;
        for (int i = 0; i < P; i += 32) {
            int v = i + tid < P ? st.off[i + tid + 1] : 0;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int o = __shfl_up_sync(kFullMask, v, d);
                if (tid >= d) v += o;
            }
            __syncwarp();
            if (i + tid < P) st.off[i + tid + 1] = base + v;
            base += __shfl_sync(kFullMask, v, 31);
        }
        if (tid == 0) st.off[0] = 0;
    }
    __syncthreads();
    const uint2* src = edges + lo;
    const uint2* out = src;
    if (st.off[P] <= P * kStageEdges) {
        if (slot < P) {
            uint2* dst = records + st.off[slot];
            for (int e = l; e < deg; e += kLanes) dst[e] = __ldg(src + e);
            out = dst;
        }
        __syncthreads();
    }
    return out;
}

// Monitor schedule as 32-bit counters carried across blocks (the 64-bit
// divisions run once per kernel): BOLD sample after step t when
// (t + 1) % bold_period == 0, trace row before step t when
// t % trace_every == 0.
struct MonitorClock {
    int bper, tev;
    int b_until, b_row, tr_until, tr_row;

    __device__ __forceinline__ void init(const tvbg_group& g, const GroupLane& c) {
        bper = g.bold_period > 0 ? g.bold_period : 1;
        tev = g.trace_every > 0 ? g.trace_every : 1;
        const long long t0 = c.t0;
        b_until = c.bold ? static_cast<int>((bper - 1) - t0 % bper) : 0;  // steps to the next sample
        b_row = c.bold ? static_cast<int>((t0 + b_until + 1) / bper - 1) : 0;
        tr_until = c.trace ? static_cast<int>((tev - t0 % tev) % tev) : 0;
        tr_row = c.trace ? static_cast<int>(((t0 + tr_until) / tev) % g.trace_len) : 0;
    }
    // advance the counters past a block of cnt steps
    __device__ __forceinline__ void advance(const tvbg_group& g, const GroupLane& c, int cnt) {
        if (c.bold) {
            while (b_until < cnt) {
                b_until += bper;
                b_row += 1;
            }
            b_until -= cnt;
        }
        if (c.trace) {
            while (tr_until < cnt) {
                tr_until += tev;
                tr_row = tr_row + 1 == g.trace_len ? 0 : tr_row + 1;
            }
            tr_until -= cnt;
        }
    }
};

template <bool B>
struct Flag {
    static constexpr bool value = B;
};

// State, parameters and monitor state of one (node, instance), in registers.
template <class M, int CF>
struct NodeRegs {
    static constexpr int NS = M::NS;
    static constexpr int NP = M::NP;
    float x[NS], p[NP];
    float wsum;
    float bs, bF, bV, bQ;    // balloon (with BOLD)

    __device__ __forceinline__ void load(const tvbg_group& g, const GroupLane& c, int n) {
        const int l = c.l, N = g.N;
#pragma unroll
        for (int v = 0; v < NS; ++v) x[v] = g.state[(n * NS + v) * kLanes + l];
#pragma unroll
        for (int v = 0; v < NP; ++v) p[v] = __ldg(g.nparam + (n * NP + v) * kLanes + l);
        wsum = (CF == TVBG_CFUN_DIFF && g.wsum) ? __ldg(g.wsum + n) : 0.0f;
        bs = bF = bV = bQ = 0.0f;
        if (c.bold) {
            bs = g.bold[(0 * N + n) * kLanes + l];
            bF = g.bold[(1 * N + n) * kLanes + l];
            bV = g.bold[(2 * N + n) * kLanes + l];
            bQ = g.bold[(3 * N + n) * kLanes + l];
        }
    }
    __device__ __forceinline__ void store(const tvbg_group& g, const GroupLane& c, int n) const {
        const int l = c.l, N = g.N;
#pragma unroll
        for (int v = 0; v < NS; ++v) g.state[(n * NS + v) * kLanes + l] = x[v];
        if (c.bold) {
            g.bold[(0 * N + n) * kLanes + l] = bs;
            g.bold[(1 * N + n) * kLanes + l] = bF;
            g.bold[(2 * N + n) * kLanes + l] = bV;
            g.bold[(3 * N + n) * kLanes + l] = bQ;
        }
    }
};

// The cnt (<= K) updates of node n for the block starting at step tb, from
// the coupling sums cs[k * stride] (second channel cs[(K + k) * stride]):
// drift, Euler-Maruyama, limit, ring write, balloon/BOLD and trace.
template <class M, int CF, int K>
__device__ __forceinline__ void update_node(const tvbg_group& g, const GroupLane& c, NodeRegs<M, CF>& r, int n,
                                            long long tb, int cnt, const float* cs, int stride,
                                            const MonitorClock& mc) {
    constexpr int NS = M::NS;
    constexpr int SPC = Noise<M>::SPC;
    constexpr int NC = ring_channels<CF>();
    constexpr int RL = kLanes * NC;  // floats per (node, slot)
    const int N = g.N;
    const int l = c.l;
    const uint32_t mask = c.mask, nh = c.nh;
    const bool noise = c.noise, bold = c.bold, trace = c.trace;
    const float dt = g.dt, sqrt_dt = g.sqrt_dt;
    float* __restrict__ ring = g.ring + static_cast<size_t>(n) * c.R * RL + l;  // this node's row
    // the record lives in shared memory, which the compiler must take to be
    // written by the ring stores: what every step reads is copied here, so
    // expressions of the constants are evaluated once per block
    float Kc[16];
#pragma unroll
    for (int v = 0; v < 16; ++v) Kc[v] = g.consts[v];
    float sig[4];
#pragma unroll
    for (int v = 0; v < 4; ++v) sig[v] = g.sigma[v];
    const float cf_b = g.cf_b, dt_bold = g.dt_bold;
    const int bold_obs = g.bold_obs;
    const uint32_t seed_lo = g.seed_lo, seed_hi = g.seed_hi;
    float obs0 = M::obs(r.x, 0);
    float sn0 = 0.0f, cs0 = 0.0f;  // sin, cos of obs0 (Kuramoto coupling)
    if constexpr (NC == 2 && CF != TVBG_CFUN_LEMS_2) sincosf(obs0, &sn0, &cs0);
    float zz[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    int b_next = mc.b_until, tr_next = mc.tr_until;
    int brow = mc.b_row, trow = mc.tr_row;
    const int kend = c.t_end - tb < cnt ? static_cast<int>(c.t_end - tb) : cnt;  // this lane's steps
    // one step; MON: trace and BOLD may be on; ALIGNED: tb % SPC == 0, so the
    // step's place in its Philox call is k % SPC
    auto step = [&](int k, auto mon, auto aligned) {
        constexpr bool MON = decltype(mon)::value, ALIGNED = decltype(aligned)::value;

        const long long t = tb + k;
        if (MON && trace && k == tr_next) {
            // a trace row holds the observables, then with TVBG_F_TRACE_CSUM
            // the raw coupling sum of the step (one-channel couplings)
            const bool csum = (c.flags & TVBG_F_TRACE_CSUM) != 0;
            const int tw = g.trace_nobs + (csum ? 1 : 0);
            float* dst = g.trace + ((static_cast<size_t>(trow) * N + n) * tw) * kLanes + l;
            for (int o = 0; o < g.trace_nobs; ++o) dst[o * kLanes] = M::obs(r.x, o);
            if constexpr (NC == 1) {
                if (csum) dst[g.trace_nobs * kLanes] = cs[k * stride];
            }
            tr_next += mc.tev;
            trow = trow + 1 == g.trace_len ? 0 : trow + 1;
        }
        const float xbold = (MON && bold) ? M::obs(r.x, bold_obs) : 0.0f;
        float cc, c2 = 0.0f;
        if constexpr (CF == TVBG_CFUN_LEMS_2) {
            cc = M::coupling(cs[k * stride], r.x, r.p);
            c2 = M::coupling2(cs[(K + k) * stride], r.x, r.p);
        } else if constexpr (NC == 2) {
            // sum_e w sin(x_j - x_i); Kuramoto: post = a * mean (coupling.py:119-121)
            const float S = cs0 * cs[k * stride] - sn0 * cs[(K + k) * stride];
            if constexpr (CF == TVBG_CFUN_LEMS_SC) {
                cc = M::coupling(S, r.x, r.p);
            } else {
                cc = c.cf_a * (S / static_cast<float>(N));
            }
        } else if constexpr (CF == TVBG_CFUN_LEMS) {
            cc = M::coupling(cs[k * stride], r.x, r.p);
        } else {
            cc = lane_post<CF>(cs[k * stride], obs0, r.wsum, c.cf_a, cf_b);
        }
        float f[NS];
        if constexpr (CF == TVBG_CFUN_LEMS_2) {
            M::drift2(r.x, cc, c2, r.p, Kc, f);
        } else {
            M::drift(r.x, cc, r.p, Kc, f);
        }
#pragma unroll
        for (int v = 0; v < NS; ++v) r.x[v] = fmaf(dt, f[v], r.x[v]);
        if constexpr (Noise<M>::kOK) {
            if (noise) {
                const int r0 = ALIGNED ? k % SPC : static_cast<int>(t & (SPC - 1));
                if (ALIGNED ? r0 == 0 : (k == 0 || r0 == 0)) {
                    const u32x4 w = philox4x32_10(static_cast<uint32_t>(n), static_cast<uint32_t>(t / SPC),
                                                  seed_hi, 0u, seed_lo, c.inst_id);
                    box_muller_fast(w.v[0], w.v[1], zz[0], zz[1]);
                    box_muller_fast(w.v[2], w.v[3], zz[2], zz[3]);
                }
#pragma unroll
                for (int v = 0; v < NS; ++v) r.x[v] = fmaf(sqrt_dt * pick4(zz, r0 * NS + v), sig[v], r.x[v]);
            }
        } else if constexpr (WideNoise<M>::value) {
            if (noise) {
                float z8[8];
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    const u32x4 w = philox4x32_10(static_cast<uint32_t>(n), static_cast<uint32_t>(t), seed_hi,
                                                  static_cast<uint32_t>(b), seed_lo, c.inst_id);
                    box_muller_fast(w.v[0], w.v[1], z8[4 * b], z8[4 * b + 1]);
                    box_muller_fast(w.v[2], w.v[3], z8[4 * b + 2], z8[4 * b + 3]);
                }
#pragma unroll
                for (int v = 0; v < NS; ++v)
                    r.x[v] = fmaf(sqrt_dt * z8[v], sig[0] * NoiseScale<M>::at(v), r.x[v]);
            }
        }
        M::limit(r.x, c.flags);
        obs0 = M::obs(r.x, 0);
        const uint32_t pos = (static_cast<uint32_t>(t) + 1u) & mask;
        const uint32_t idx = pos * RL;
        if constexpr (NC == 2) {
            if constexpr (CF == TVBG_CFUN_LEMS_2) {
                sn0 = M::ring_value(obs0, r.p);
                cs0 = M::ring_value2(r.x[M::CVAR2], r.p);
            } else {
                sincosf(obs0, &sn0, &cs0);
            }
            ring[idx] = sn0;
            ring[idx + kLanes] = cs0;
            if (pos < kGhost) {
                ring[idx + nh * RL] = sn0;
                ring[idx + nh * RL + kLanes] = cs0;
            }
        } else {
            const float rv = ring_val<M, CF>(obs0, r.p);
            ring[idx] = rv;
            if (pos < kGhost) ring[idx + nh * RL] = rv;
        }
        if (MON && bold) {
            Balloon::step(r.bs, r.bF, r.bV, r.bQ, xbold, dt_bold);
            if (k == b_next) {
                if (brow >= 0 && brow < g.bold_len)
                    g.bold_out[(static_cast<size_t>(brow) * N + n) * kLanes + l] = Balloon::signal(r.bV, r.bQ);
                b_next += mc.bper;
                brow += 1;
            }
        }
    };
    // Whole blocks are unrolled: the generator and the addresses of later
    // steps do not depend on the state, so they fill the waits of the earlier
    // ones.  (The models with long drifts, or sincosf per step, stay rolled.)
    if constexpr (NS <= 2 && NC == 1 && CF != TVBG_CFUN_LEMS) {
        if (kend == K && (tb & (SPC - 1)) == 0) {
            if (bold || trace) {
#pragma unroll 1
                for (int k0 = 0; k0 < K; k0 += kStepUnroll)
#pragma unroll
                    for (int k = 0; k < kStepUnroll; ++k) step(k0 + k, Flag<true>{}, Flag<true>{});
            } else {
#pragma unroll 1
                for (int k0 = 0; k0 < K; k0 += kStepUnroll)
#pragma unroll
                    for (int k = 0; k < kStepUnroll; ++k) step(k0 + k, Flag<false>{}, Flag<true>{});
            }
            return;
        }
    }
#pragma unroll 1
    for (int k = 0; k < kend; ++k) step(k, Flag<true>{}, Flag<false>{});
}

// Plain group run: per block, every thread gathers its node's sums and then
// runs its updates; a slot takes several nodes in turn (rounds) where the
// CTAs hold fewer slots than nodes.
template <class M, int CF, int K, int BOUND>
__device__ __forceinline__ void run_group(const tvbg_group& g, float* csum, EdgeStage& stage, int32_t* status) {
    uint2* records = reinterpret_cast<uint2*>(csum + ring_channels<CF>() * K * blockDim.x);
    const int N = g.N;
    const uint32_t C = cluster_nranks();
    const uint32_t rank = cluster_rank();
    const bool cluster = C > 1;
    if (!group_descriptor_ok<M, CF>(g)) {
        if (threadIdx.x == 0) report(status, TVBG_EINVAL);
        return;  // every CTA of the cluster reads the same descriptor and leaves here
    }
    const int l = threadIdx.x % kLanes;
    const int P = blockDim.x / kLanes;
    const int stride = static_cast<int>(C) * P;
    const int rounds = (N + stride - 1) / stride;       // warp-uniform node loop
    const int q0 = (threadIdx.x / kLanes) * static_cast<int>(C) + static_cast<int>(rank);
    const GroupLane c = make_lane<M, CF, K>(g, l);
    // with one node per slot the edge records are staged
    const int n0 = q0 < N ? (g.nodes ? __ldg(g.nodes + q0) : q0) : 0;
    const int lo0 = q0 < N ? __ldg(g.row + n0) : 0;
    const int deg0 = q0 < N ? __ldg(g.row + n0 + 1) - lo0 : 0;
    const uint2* edges0 = reinterpret_cast<const uint2*>(g.edges) + lo0;
    if (rounds == 1) edges0 = stage_edges(reinterpret_cast<const uint2*>(g.edges), stage, records, P, threadIdx.x, lo0, deg0);
    for (int q = q0; q < N; q += stride) seed_node<M, CF>(g, c, g.nodes ? __ldg(g.nodes + q) : q);
    group_barrier(cluster);
    MonitorClock mc;
    mc.init(g, c);
    const long long t_stop = c.t0 + g.nsteps;
    for (long long tb = c.t0; tb < t_stop; tb += K) {
        const int cnt = (t_stop - tb) < K ? static_cast<int>(t_stop - tb) : K;
        for (int r = 0; r < rounds; ++r) {
            const int q = q0 + r * stride;
            const bool valid = q < N;
            int n = n0, deg = deg0;
            const uint2* edges = edges0;
            if (r > 0) {
                n = valid ? (g.nodes ? __ldg(g.nodes + q) : q) : 0;
                const int lo = valid ? __ldg(g.row + n) : 0;
                deg = valid ? __ldg(g.row + n + 1) - lo : 0;
                edges = reinterpret_cast<const uint2*>(g.edges) + lo;
                __syncwarp();  // the last round's sums have been read
            }
            gather_node<M, CF, K, BOUND>(g, c, edges, deg, static_cast<uint32_t>(tb) & c.mask, csum + threadIdx.x - l,
                                  blockDim.x);
            __syncwarp();             // the slot's lanes read each other's sums
            if (!valid) continue;
            NodeRegs<M, CF> x;
            x.load(g, c, n);
            update_node<M, CF, K>(g, c, x, n, tb, cnt, csum + threadIdx.x, blockDim.x, mc);
            x.store(g, c, n);
        }
        mc.advance(g, c, cnt);
        group_barrier(cluster);
    }
}

// Phase counter of a cluster (pipelined kernel): every CTA's mbarrier takes
// one arrival from each CTA of the cluster per phase.  One warp publishes a
// phase (fence, then a remote arrive per CTA) and awaits it, in place of a
// barrier.cluster with release and acquire by every thread, which cost
// about 2300 cycles per block of 8 steps with nothing else to do.
struct ClusterPhases {
    unsigned long long bar;
    int fail;             // a wait ran out in phase fail - 1: every thread leaves after that phase

    __device__ __forceinline__ void init(uint32_t C) {  // one thread; cluster barrier before use
        fail = 0;
        mbar_init(smem_addr(&bar), C);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // One warp, after a CTA barrier: what the CTA wrote before that barrier
    // is visible to the cluster once this phase is awaited (the fence and the
    // release are cumulative over the CTA barrier).
    __device__ __forceinline__ void publish(uint32_t C) {
        const uint32_t lane = threadIdx.x & 31u;
        if (lane < C) {
            asm volatile("fence.acq_rel.cluster;" ::: "memory");
            uint32_t remote;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_addr(&bar)), "r"(lane));
            asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(remote) : "memory");
        }
        __syncwarp();
    }
    // One warp, in phase `now`: wait (bounded) for phase `ph` of every CTA.
    __device__ __forceinline__ void await(uint32_t ph, uint32_t now) {
        const uint32_t a = smem_addr(&bar);
        uint32_t ok = 0;
        for (int it = 0; it < (1 << 20) && !ok; ++it)
            asm volatile(
                "{\n\t.reg .pred p;\n\t"
                "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
                "selp.u32 %0, 1, 0, p;\n\t}"
                : "=r"(ok)
                : "r"(a), "r"(ph & 1u)
                : "memory");
        if (!ok) fail = static_cast<int>(now + 1);
        __syncwarp();
    }
    // After the CTA barrier of phase `now`: the same answer in every thread.
    __device__ __forceinline__ bool failed(uint32_t now) const {
        const int f = *const_cast<const volatile int*>(&fail);
        return f != 0 && static_cast<uint32_t>(f) <= now + 1;
    }
};

// Pipelined group run: the CTA's warps form two teams of H = blockDim / 2
// threads, both mapped onto the same (node, lane) pairs.  In phase b the
// update team runs the K steps of block b from the coupling sums in one
// shared buffer while the gather team sums block b + 1 into the other; a CTA
// barrier ends the phase.  Block b + 1 reads ring slots up to
// tb + 2K - 1 - d_min, so with d_min >= 2K - 1 every slot it reads was
// written before block b started, and the newest slot written in block b
// (tb + K) is at most d_max < nh slots ahead of the oldest read, so no read
// aliases a write.  Same arithmetic in the same order as run_group, so the
// results are identical.  Needs one node per slot (C * H / 8 >= N), K in
// {4, 8} and a 16-byte aligned ring.
//
// Across the CTAs of a cluster a phase must not start before the writes it
// reads have been published.  With d_min >= 3K - 1 (lag) the gather of phase
// b reads nothing newer than block b - 2, so the phase that ends is
// published by one warp during the next phase and awaited at that one's
// end: no thread stands at a cluster-wide barrier.  A CTA may then be one
// phase ahead of another, writing up to slot tb + 2K while tb + K - d_max is
// read: K + d_max < nh, which nh >= d_max + 1 + K covers.  With shorter
// delays the phase is awaited before the next one starts.
template <class M, int CF, int K, int BOUND>
__device__ __forceinline__ void run_group_pipelined(const tvbg_group& g, float* csum, EdgeStage& stage,
                                                    ClusterPhases& phases, int32_t* status) {
    constexpr int NC = ring_channels<CF>();
    const int N = g.N;
    const uint32_t C = cluster_nranks();
    const uint32_t rank = cluster_rank();
    const bool cluster = C > 1;
    const int H = static_cast<int>(blockDim.x) / 2;
    const int P = H / kLanes;
    if (!group_descriptor_ok<M, CF>(g, true) || g.dmin < 2 * K - 1 || (H & 31) ||
        static_cast<int>(C) * P < N || (reinterpret_cast<uintptr_t>(g.ring) & 15u) != 0) {
        if (threadIdx.x == 0) report(status, TVBG_EINVAL);
        return;  // uniform over the cluster: same descriptor, same launch shape
    }
    const bool lag = g.dmin >= 3 * K - 1;
    const bool gather_team = static_cast<int>(threadIdx.x) >= H;
    const int tid = static_cast<int>(threadIdx.x) - (gather_team ? H : 0);
    const int l = tid % kLanes;
    const int q = (tid / kLanes) * static_cast<int>(C) + static_cast<int>(rank);
    const bool valid = q < N;
    const int n = valid ? (g.nodes ? __ldg(g.nodes + q) : q) : 0;
    const int lo = valid ? __ldg(g.row + n) : 0;
    const int deg = valid ? __ldg(g.row + n + 1) - lo : 0;
    const GroupLane c = make_lane<M, CF, K>(g, l);
    const int bufsz = NC * K * H;  // floats per coupling-sum buffer
    if (threadIdx.x == 0) phases.init(C);
    // the gather team's threads carry the slots (their tid is the scan's)
    const int st_tid = gather_team ? tid : H + tid;
    const uint2* edges = stage_edges(reinterpret_cast<const uint2*>(g.edges), stage,
                                     reinterpret_cast<uint2*>(csum + 2 * bufsz), P, st_tid, lo, deg);

    if (!gather_team && valid) seed_node<M, CF>(g, c, n);
    group_barrier(cluster);
    // each team runs its own loop (disjoint live ranges); both meet at the
    // same barriers
    const long long t_stop = c.t0 + g.nsteps;
    if (gather_team) {
        // the last gather warp, whose nodes have the fewest edges, keeps the phases
        const bool keeper = cluster && tid >= H - 32;
        if (g.nsteps > 0)
            gather_node<M, CF, K, BOUND>(g, c, edges, deg, static_cast<uint32_t>(c.t0) & c.mask, csum + tid - l, H);
        __syncthreads();
        uint32_t ph = 0;  // phases ended
        for (long long tb = c.t0; tb < t_stop; tb += K) {
            if (keeper && lag && ph > 0) phases.publish(C);
            if (tb + K < t_stop)
                gather_node<M, CF, K, BOUND>(g, c, edges, deg, static_cast<uint32_t>(tb + K) & c.mask,
                                      csum + ((ph + 1) & 1u) * bufsz + tid - l, H);
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
        __syncthreads();
        MonitorClock mc;
        mc.init(g, c);
        NodeRegs<M, CF> r;       // one node per thread: its state stays in registers
        if (valid) r.load(g, c, n);
        uint32_t ph = 0;
        for (long long tb = c.t0; tb < t_stop; tb += K) {
            const int cnt = (t_stop - tb) < K ? static_cast<int>(t_stop - tb) : K;
            if (valid) update_node<M, CF, K>(g, c, r, n, tb, cnt, csum + (ph & 1u) * bufsz + tid, H, mc);
            mc.advance(g, c, cnt);
            __syncthreads();
            if (cluster && !lag) __syncthreads();
            if (cluster && phases.failed(ph)) break;
            ++ph;
        }
        if (valid) r.store(g, c, n);
    }
    if (cluster) {
        if (threadIdx.x == 0 && phases.fail) report(status, TVBG_ETIMEOUT);
        group_barrier(true);  // no CTA leaves while another may still arrive on its phases
    }
}

// Dynamic shared memory of a pipelined group CTA: two coupling-sum buffers
// of half the CTA each, and the staged edge records.
__host__ __device__ constexpr uint32_t group_pipelined_smem_bytes(int K, int threads, int nc) {
    return static_cast<uint32_t>(4 * 2 * K * (threads / 2) * nc + stage_bytes(threads / 2));
}

// One group per CTA (or per cluster of CTAs): group index = order[cluster id].
// BOUND: the largest CTA the instance is built for (its registers a thread).
template <class M, int CF, int K, int BOUND = 1024>
__global__ void __launch_bounds__(BOUND, 1)
    group_kernel(const tvbg_group* __restrict__ groups, int32_t n_groups,
                 const int32_t* __restrict__ order, int32_t* __restrict__ status) {
    __shared__ __align__(16) tvbg_group s_grp;
    __shared__ EdgeStage s_stage;
    extern __shared__ __align__(16) float csum[];  // [channels][K][blockDim]: the block's sums; edge records
    const int cid = static_cast<int>(cluster_id_x());
    if (cid >= n_groups) return;  // uniform over the cluster
    const int idx = order ? __ldg(order + cid) : cid;
    stage_group(groups + idx, &s_grp);
    run_group<M, CF, K, BOUND>(s_grp, csum, s_stage, status);
}

// The most dynamic shared memory that a group CTA takes (8 steps, 1024 threads,
// two channels).  A kernel whose CTAs need the opt-in is given this limit at
// every launch, not its CTAs' own size: the limit belongs to the kernel, and
// another thread's launch of a smaller CTA would lower it between the two calls.
constexpr size_t kGroupSmemMax = group_smem_bytes(8, 1024, 2) > group_pipelined_smem_bytes(8, 1024, 2)
                                     ? group_smem_bytes(8, 1024, 2)
                                     : group_pipelined_smem_bytes(8, 1024, 2);

// Pipelined variant (run_group_pipelined): blockDim = 2 teams x 8 lanes x
// node slots; same tables and results as group_kernel.
template <class M, int CF, int K, int BOUND = 1024>
__global__ void __launch_bounds__(BOUND, 1)
    group_kernel_pipelined(const tvbg_group* __restrict__ groups, int32_t n_groups,
                           const int32_t* __restrict__ order, int32_t* __restrict__ status) {
    __shared__ __align__(16) tvbg_group s_grp;
    __shared__ EdgeStage s_stage;
    __shared__ ClusterPhases s_phases;
    static_assert(sizeof(EdgeStage) + sizeof(ClusterPhases) + 64 <= 640, "kGroupStaticBytes");
    extern __shared__ __align__(16) float csum[];  // [2][channels][K][blockDim / 2]; edge records
    const int cid = static_cast<int>(cluster_id_x());
    if (cid >= n_groups) return;  // uniform over the cluster
    const int idx = order ? __ldg(order + cid) : cid;
    stage_group(groups + idx, &s_grp);
    run_group_pipelined<M, CF, K, BOUND>(s_grp, csum, s_stage, s_phases, status);
}

}  // namespace tvbg
