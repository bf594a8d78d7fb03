// C ABI of the lane-interleaved group kernels (tvbg_group_run and helpers).
#include <cstring>

#include "tvbg_abi_internal.h"
#include "tvbg_group_launch.cuh"

using namespace tvbg;

namespace {

GroupKernel lookup_group(int model, int cfun, int k, GroupForm form) {
    switch (model) {
        case TVBG_MODEL_KURAMOTO: return group_kernel_kuramoto(cfun, k, form);
        case TVBG_MODEL_G2DO: return group_kernel_g2do(cfun, k, form);
        case TVBG_MODEL_MPR: return group_kernel_mpr(cfun, k, form);
        case TVBG_MODEL_LINEAR: return group_kernel_linear(cfun, k, form);
        case TVBG_MODEL_G2DOSC: return group_kernel_g2dosc(cfun, k, form);
        case TVBG_MODEL_RWW: return group_kernel_rww(cfun, k, form);
        case TVBG_MODEL_JANSENRIT: return group_kernel_jansenrit(cfun, k, form);
        default: return nullptr;
    }
}

const ErrSink kSink{set_error, set_cuda_error};

// Validate a group launch; its dynamic shared memory holds the K coupling
// sums of every thread and the staged edge records.
int check_group_launch(const tvbg_launch* cfg, int* cluster, size_t* smem) {
    int rc = check_group_cfg(cfg, kSink, cluster, (1u << 4) | (1u << 8), true);
    if (rc) return rc;
    *smem = cfg->tpn == TVBG_GROUP_PIPELINED
                ? group_pipelined_smem_bytes(cfg->block_k, cfg->threads, group_channels(cfg->cfun))
                : group_smem_bytes(cfg->block_k, cfg->threads, group_channels(cfg->cfun));
    return TVBG_OK;
}

int find_kernel(const tvbg_launch* cfg, GroupForm form, GroupKernel* kfn) {
    *kfn = lookup_group(cfg->model, cfg->cfun, cfg->block_k, form);
    return *kfn ? TVBG_OK
                : set_error(TVBG_EUNSUPPORTED, "group kernel not built for this model/coupling/block_k");
}

int opt_in(GroupKernel kfn, int cluster, size_t smem) {
    cudaError_t e = cudaSuccess;
    if (smem + kGroupStaticBytes > 48u * 1024u)  // beyond the default
        e = cudaFuncSetAttribute(reinterpret_cast<const void*>(kfn), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(kGroupSmemMax));
    if (e == cudaSuccess && cluster > 8)
        e = cudaFuncSetAttribute(reinterpret_cast<const void*>(kfn), cudaFuncAttributeNonPortableClusterSizeAllowed,
                                 1);
    return e == cudaSuccess ? TVBG_OK : set_cuda_error(e, "group kernel attributes");
}

// The builds that launches of cfg's shape take, by their number of CTAs
// (group_form): returns their count.
int shape_forms(const tvbg_launch* cfg, GroupForm forms[2]) {
    const bool pipe = cfg->tpn == TVBG_GROUP_PIPELINED;
    if (pipe && cfg->threads <= 512) {
        forms[0] = kPipe512;
        forms[1] = kPipe768;
        return 2;
    }
    forms[0] = group_form(cfg->threads, 1, pipe);
    return 1;
}

// Clusters of one build that are resident at once.
int resident_clusters(const tvbg_launch* cfg, GroupForm form, int cluster, size_t smem, int32_t* clusters) {
    GroupKernel kfn = nullptr;
    int rc = find_kernel(cfg, form, &kfn);
    if (!rc) rc = opt_in(kfn, cluster, smem);
    if (rc) return rc;
    cudaLaunchConfig_t lc;
    std::memset(&lc, 0, sizeof(lc));
    lc.gridDim = dim3(static_cast<unsigned>(cluster), 1, 1);
    lc.blockDim = dim3(static_cast<unsigned>(cfg->threads), 1, 1);
    lc.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = static_cast<unsigned>(cluster);
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    lc.attrs = attr;
    lc.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, reinterpret_cast<const void*>(kfn), &lc) != cudaSuccess) {
        cudaGetLastError();  // an unschedulable shape is reported here, before any launch
        n = 0;
    }
    *clusters = n;
    return TVBG_OK;
}

}  // namespace

GroupKernel tvbg::lookup_group_kernel(int model, int cfun, int k, GroupForm form) {
    return lookup_group(model, cfun, k, form);
}

// More registers a thread put more ring loads in flight, so each CTA runs
// faster, but fewer CTAs are resident: the 512-thread build is taken unless
// the 768-thread one needs fewer waves of CTAs.  Measured (ms, 800 steps,
// MPR; 512 / 768 build): N = 84, 32 groups, 256 x 6 threads 0.320 / 0.369; N = 84,
// 128 groups, 448 x 3 0.97 / 1.10 (one CTA per SM in both); N = 192, 32
// groups, 256 x 12 0.75 / 0.55 (two waves against one).
GroupForm tvbg::group_form(int threads, long long ctas, bool pipe) {
    if (!pipe) return threads > 768 ? kPlain1024 : kPlain768;
    if (threads > 768) return kPipe1024;
    if (threads > 512) return kPipe768;
    const int sms = device_sms();
    if (sms <= 0) return kPipe768;
    const long long wide = static_cast<long long>(512 / threads) * sms;       // resident CTAs, 128 registers
    const long long mid = static_cast<long long>(65536 / (80 * threads)) * sms;  // 80 registers
    return (ctas + wide - 1) / wide > (ctas + mid - 1) / mid ? kPipe768 : kPipe512;
}

extern "C" {

size_t tvbg_group_size(void) { return sizeof(tvbg_group); }

int tvbg_pack_edges_group(int32_t N, int32_t nnz, const int32_t* row, const int32_t* col,
                          const float* weights, const int32_t* delays, int32_t lognh,
                          tvbg_edge* out) {
    if (N < 0 || nnz < 0 || !row || (nnz > 0 && (!col || !weights || !delays || !out)))
        return set_error(TVBG_EINVAL, "tvbg_pack_edges_group: bad arguments");
    if (lognh < 3 || lognh > 16 || N > 65536)
        return set_error(TVBG_EINVAL, "tvbg_pack_edges_group: needs lognh in [3, 16], N <= 65536");
    if (row[0] != 0 || row[N] != nnz)
        return set_error(TVBG_EINVAL, "tvbg_pack_edges_group: row must run from 0 to nnz");
    const uint32_t nh = 1u << lognh;
    const uint32_t mask = nh - 1u;
    for (int32_t i = 0; i < N; ++i) {
        if (row[i + 1] < row[i]) return set_error(TVBG_EINVAL, "tvbg_pack_edges_group: row not monotone");
        for (int32_t e = row[i]; e < row[i + 1]; ++e) {
            const int32_t c = col[e], d = delays[e];
            if (c < 0 || c >= N) return set_error(TVBG_EINVAL, "tvbg_pack_edges_group: col out of range");
            if (d < 0 || static_cast<uint32_t>(d) >= nh)
                return set_error(TVBG_EINVAL, "tvbg_pack_edges_group: delay outside [0, nh)");
            out[e].pk = (static_cast<uint32_t>(c) << 16) | ((nh - static_cast<uint32_t>(d)) & mask);
            out[e].w = weights[e];
        }
    }
    return TVBG_OK;
}

int tvbg_group_run(const tvbg_group* d_groups, int32_t n_groups, const tvbg_launch* cfg,
                   void* stream) {
    GroupKernel kfn = nullptr;
    int cluster = 1;
    size_t smem = 0;
    int rc = check_group_launch(cfg, &cluster, &smem);
    if (!rc)
        rc = find_kernel(cfg, group_form(cfg->threads, static_cast<long long>(n_groups) * cluster,
                                         cfg->tpn == TVBG_GROUP_PIPELINED), &kfn);
    if (rc) return rc;
    return launch_group_kernel(kfn, d_groups, n_groups, cfg, cluster, smem, stream, kSink);
}

int tvbg_group_occupancy(const tvbg_launch* cfg, int32_t* ctas_per_sm, int32_t* sms) {
    if (!ctas_per_sm || !sms) return set_error(TVBG_EINVAL, "tvbg_group_occupancy: null");
    int cluster = 1;
    size_t smem = 0;
    int rc = check_group_launch(cfg, &cluster, &smem);
    if (rc) return rc;
    GroupForm forms[2];
    const int nf = shape_forms(cfg, forms);
    int most = 0;
    for (int i = 0; i < nf; ++i) {
        GroupKernel kfn = nullptr;
        rc = find_kernel(cfg, forms[i], &kfn);
        if (!rc) rc = opt_in(kfn, 1, smem);
        if (rc) return rc;
        int n = 0;
        const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, reinterpret_cast<const void*>(kfn),
                                                                            cfg->threads, smem);
        if (e != cudaSuccess) return set_cuda_error(e, "cudaOccupancyMaxActiveBlocksPerMultiprocessor");
        most = n > most ? n : most;
    }
    const int nsm = device_sms();
    if (nsm <= 0) return set_error(TVBG_ECUDA, "tvbg_group_occupancy: SM count");
    *ctas_per_sm = most;
    *sms = nsm;
    return TVBG_OK;
}

int tvbg_group_max_clusters_for(const tvbg_launch* cfg, int32_t n_groups, int32_t* max_clusters) {
    if (!max_clusters || n_groups < 0) return set_error(TVBG_EINVAL, "tvbg_group_max_clusters: bad arguments");
    int cluster = 1;
    size_t smem = 0;
    int rc = check_group_launch(cfg, &cluster, &smem);
    if (rc) return rc;
    if (n_groups > 0)
        return resident_clusters(cfg, group_form(cfg->threads, static_cast<long long>(n_groups) * cluster,
                                                 cfg->tpn == TVBG_GROUP_PIPELINED),
                                 cluster, smem, max_clusters);
    GroupForm forms[2];
    const int nf = shape_forms(cfg, forms);
    int32_t most = 0;
    for (int i = 0; i < nf; ++i) {
        int32_t n = 0;
        rc = resident_clusters(cfg, forms[i], cluster, smem, &n);
        if (rc) return rc;
        most = n > most ? n : most;
    }
    *max_clusters = most;
    return TVBG_OK;
}

int tvbg_group_max_clusters(const tvbg_launch* cfg, int32_t* max_clusters) {
    return tvbg_group_max_clusters_for(cfg, 0, max_clusters);
}

}  // extern "C"
