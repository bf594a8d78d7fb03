// Lane-interleaved group kernels for the G2DOsc model: separable couplings
// (LINEAR, DIFF, SIGMOIDAL) x block length 4, 8, plain and
// pipelined (group_kernel_pipelined).
#include "tvbg_abi_internal.h"
#include "tvbg_lanes.cuh"

namespace tvbg {

template <int CF, int K>
static GroupKernel pick_form(GroupForm form) {
    switch (form) {
        case kPlain1024: return group_kernel<G2DOsc, CF, K, 1024>;
        case kPlain768: return group_kernel<G2DOsc, CF, K, 768>;
        case kPipe1024: return group_kernel_pipelined<G2DOsc, CF, K, 1024>;
        case kPipe768: return group_kernel_pipelined<G2DOsc, CF, K, 768>;
        case kPipe512: return group_kernel_pipelined<G2DOsc, CF, K, 512>;
    }
    return nullptr;
}

template <int CF>
static GroupKernel pick_k(int k, GroupForm form) {
    switch (k) {
        case 4: return pick_form<CF, 4>(form);
        case 8: return pick_form<CF, 8>(form);
        default: return nullptr;
    }
}

GroupKernel group_kernel_g2dosc(int cfun, int k, GroupForm form) {
    switch (cfun) {
        case TVBG_CFUN_LINEAR: return pick_k<TVBG_CFUN_LINEAR>(k, form);
        case TVBG_CFUN_DIFF: return pick_k<TVBG_CFUN_DIFF>(k, form);
        case TVBG_CFUN_SIGMOIDAL: return pick_k<TVBG_CFUN_SIGMOIDAL>(k, form);
        default: return nullptr;
    }
}

}  // namespace tvbg
