// Time-blocked step-kernel instances for the G2DOsc model: separable couplings
// (LINEAR, DIFF, SIGMOIDAL) x gather width 2, 4, 8 x block length 4, 8.
#include "tvbg_abi_internal.h"
#include "tvbg_step_blocked.cuh"

namespace tvbg {

template <int CF, int K, int BOUND>
static BlockedKernel pick_tpn_b(int tpn) {
    switch (tpn) {
        case 2: return blocked_kernel<G2DOsc, CF, 2, K, BOUND>;
        case 4: return blocked_kernel<G2DOsc, CF, 4, K, BOUND>;
        case 8: return blocked_kernel<G2DOsc, CF, 8, K, BOUND>;
        default: return nullptr;
    }
}

template <int CF>
static BlockedKernel pick_k(int tpn, int k, bool wide) {
    switch (k) {
        case 4: return wide ? pick_tpn_b<CF, 4, 512>(tpn) : pick_tpn_b<CF, 4, 1024>(tpn);
        case 8: return wide ? pick_tpn_b<CF, 8, 512>(tpn) : pick_tpn_b<CF, 8, 1024>(tpn);
        default: return nullptr;
    }
}

BlockedKernel blocked_kernel_g2dosc(int cfun, int tpn, int k, bool wide) {
    switch (cfun) {
        case TVBG_CFUN_LINEAR: return pick_k<TVBG_CFUN_LINEAR>(tpn, k, wide);
        case TVBG_CFUN_DIFF: return pick_k<TVBG_CFUN_DIFF>(tpn, k, wide);
        case TVBG_CFUN_SIGMOIDAL: return pick_k<TVBG_CFUN_SIGMOIDAL>(tpn, k, wide);
        default: return nullptr;
    }
}

}  // namespace tvbg
