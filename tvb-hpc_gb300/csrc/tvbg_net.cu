// C ABI of the node-parallel kernel for one very large network (tvbg_net_run).
#include "tvbg_abi_internal.h"
#include "tvbg_net.cuh"

using namespace tvbg;

namespace {

using NetKernel = void (*)(const tvbg_net, long long, int, int32_t*);
using SeedKernel = void (*)(const tvbg_net, long long);
using WideKernel = void (*)(const tvbg_net, long long, int, float*);

template <class M, int CF>
WideKernel pick_j(int j) {
    return j == 2 ? net_kernel_wide<M, CF, 2> : net_kernel_wide<M, CF, 3>;
}

template <class M>
WideKernel wide_cf(int cfun, int j) {
    switch (cfun) {
        case TVBG_CFUN_LINEAR: return pick_j<M, TVBG_CFUN_LINEAR>(j);
        case TVBG_CFUN_DIFF: return pick_j<M, TVBG_CFUN_DIFF>(j);
        case TVBG_CFUN_SIGMOIDAL: return pick_j<M, TVBG_CFUN_SIGMOIDAL>(j);
        default: return nullptr;
    }
}

WideKernel lookup_wide(int model, int cfun, int j) {
    switch (model) {
        case TVBG_MODEL_G2DO: return wide_cf<G2DO>(cfun, j);
        case TVBG_MODEL_G2DOSC: return wide_cf<G2DOsc>(cfun, j);
        case TVBG_MODEL_MPR: return wide_cf<MPR>(cfun, j);
        case TVBG_MODEL_LINEAR: return wide_cf<Linear>(cfun, j);
        default: return nullptr;
    }
}

// lanes == 1: one thread per node; lanes == K: K lanes per node.
template <class M, int CF>
NetKernel pick_k(int k, bool lanes) {
    switch (k) {
        case 4: return lanes ? net_kernel_lanes<M, CF, 4> : net_kernel<M, CF, 4>;
        case 8: return lanes ? net_kernel_lanes<M, CF, 8> : net_kernel<M, CF, 8>;
        default: return nullptr;
    }
}

template <class M>
NetKernel pick_cf(int cfun, int k, bool lanes) {
    switch (cfun) {
        case TVBG_CFUN_LINEAR: return pick_k<M, TVBG_CFUN_LINEAR>(k, lanes);
        case TVBG_CFUN_DIFF: return pick_k<M, TVBG_CFUN_DIFF>(k, lanes);
        case TVBG_CFUN_SIGMOIDAL: return pick_k<M, TVBG_CFUN_SIGMOIDAL>(k, lanes);
        default: return nullptr;
    }
}

int lookup(int model, int cfun, int k, bool lanes, NetKernel* kfn, SeedKernel* sfn) {
    switch (model) {
        case TVBG_MODEL_G2DO: *kfn = pick_cf<G2DO>(cfun, k, lanes); *sfn = net_seed_kernel<G2DO>; break;
        case TVBG_MODEL_G2DOSC:
            *kfn = pick_cf<G2DOsc>(cfun, k, lanes);
            *sfn = net_seed_kernel<G2DOsc>;
            break;
        case TVBG_MODEL_MPR: *kfn = pick_cf<MPR>(cfun, k, lanes); *sfn = net_seed_kernel<MPR>; break;
        case TVBG_MODEL_LINEAR:
            *kfn = pick_cf<Linear>(cfun, k, lanes);
            *sfn = net_seed_kernel<Linear>;
            break;
        default: *kfn = nullptr;
    }
    return *kfn ? TVBG_OK : set_error(TVBG_EUNSUPPORTED, "tvbg_net_run: model/coupling/block_k not built");
}

}  // namespace

extern "C" size_t tvbg_net_size(void) { return sizeof(tvbg_net); }

extern "C" int tvbg_net_run(const tvbg_net* net, int64_t t0, int32_t nsteps, const tvbg_launch* cfg,
                            void* stream) {
    return tvbg_net_run_ex(net, t0, nsteps, cfg, 0, nullptr, 0, stream);
}

// `dmin`: the smallest delay (0 = not known); d_stage: floats for the new
// slots of blocks launched together, [N][8 J].  J = 3 or 2 blocks of 8 steps
// share a launch where dmin >= 8 J - 1 and the buffer holds them (lanes mapping,
// block_k = 8); so does a tail of more than 8 steps, and one of at most 8
// takes the single-block kernel.
extern "C" int tvbg_net_run_ex(const tvbg_net* net, int64_t t0, int32_t nsteps, const tvbg_launch* cfg,
                               int32_t dmin, float* d_stage, int64_t stage_floats, void* stream) {
    if (!net || !cfg || nsteps < 0 || t0 < 0 || dmin < 0 || stage_floats < 0)
        return set_error(TVBG_EINVAL, "tvbg_net_run: bad arguments");
    if (net->N <= 0 || net->lognh < 3 || net->lognh > 16 || !net->row || !net->ring ||
        !net->state || !net->nparam || (net->flags & (TVBG_F_TRACKA | TVBG_F_MIDSYNC)))
        return set_error(TVBG_EINVAL, "tvbg_net_run: bad network descriptor");
    if (cfg->block_k != 4 && cfg->block_k != 8)
        return set_error(TVBG_EINVAL, "tvbg_net_run: block_k must be 4 or 8");
    if (cfg->threads < 32 || cfg->threads > 1024 || (cfg->threads & 31))
        return set_error(TVBG_EINVAL, "threads must be a multiple of 32 in [32, 1024]");
    if (net->model != cfg->model || net->cfun != cfg->cfun)
        return set_error(TVBG_EINVAL, "tvbg_net_run: descriptor and launch disagree on model/coupling");
    const int lanes = cfg->tpn > 1 ? cfg->tpn : 1;
    if (lanes != 1 && lanes != cfg->block_k)
        return set_error(TVBG_EINVAL, "tvbg_net_run: tpn must be 0, 1 or block_k");
    NetKernel kfn = nullptr;
    SeedKernel sfn = nullptr;
    int rc = lookup(net->model, net->cfun, cfg->block_k, lanes > 1, &kfn, &sfn);
    if (rc) return rc;
    const long long seed_blocks = (net->N + cfg->threads - 1) / cfg->threads;
    const long long blocks = (net->N * lanes + cfg->threads - 1) / cfg->threads;
    if (blocks > 0x7fffffffLL || net->N > 0x7fffffffLL * 8) return set_error(TVBG_EINVAL, "tvbg_net_run: N too large");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    sfn<<<static_cast<unsigned>(seed_blocks), cfg->threads, 0, st>>>(*net, t0);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return set_cuda_error(e, "tvbg_net_run: seed launch");
    int J = 1;
    if (d_stage && lanes == 8 && cfg->threads <= 256)
        for (int j = 3; j >= 2 && J == 1; --j)
            if (dmin >= 8 * j - 1 && stage_floats >= net->N * static_cast<int64_t>(8 * j)) J = j;
    const WideKernel wfn = J > 1 ? lookup_wide(net->model, net->cfun, J) : nullptr;
    long long first = t0;
    if (wfn) {
        const int W = 8 * J;
        const long long copy_blocks = (net->N * W + 255) / 256;
        // a remainder of more than one block still takes a whole launch
        for (; t0 + nsteps - first > 8; first += W) {
            const int cnt = static_cast<int>(t0 + nsteps - first < W ? t0 + nsteps - first : W);
            wfn<<<static_cast<unsigned>(blocks), cfg->threads, 0, st>>>(*net, first, cnt, d_stage);
            net_copy_kernel<<<static_cast<unsigned>(copy_blocks), 256, 0, st>>>(*net, first, cnt, W, d_stage);
            e = cudaGetLastError();
            if (e != cudaSuccess) return set_cuda_error(e, "tvbg_net_run: step launch");
        }
    }
    for (long long tb = first; tb < t0 + nsteps; tb += cfg->block_k) {
        const int cnt = static_cast<int>((t0 + nsteps - tb) < cfg->block_k ? (t0 + nsteps - tb)
                                                                            : cfg->block_k);
        kfn<<<static_cast<unsigned>(blocks), cfg->threads, 0, st>>>(*net, tb, cnt, cfg->d_status);
        e = cudaGetLastError();
        if (e != cudaSuccess) return set_cuda_error(e, "tvbg_net_run: step launch");
    }
    return TVBG_OK;
}
