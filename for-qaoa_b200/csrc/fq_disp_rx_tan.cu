// fq_disp_rx_tan.cu -- strided RX passes of the fused engine with the
// reduced gate [[1,-it],[-it,1]], t = tan(beta/2), for a circuit's last
// pass writing both halves of the state and optionally accumulating <C>.
#include "fq_launch.cuh"

namespace fq {

int dispatch_rx_tan(fq_ctx* ctx, bool integer, bool energy, const PassArgs& A) {
    if (!A.full) {
        FQ_CHECK(!energy, FQ_ERR_INVALID, "<C> belongs to a circuit's last pass");
        return launch_pass<int, PH_NONE, GM_TAN, EX_NONE, 1>(ctx, A);
    }
    if (!energy) return launch_pass<int, PH_NONE, GM_TAN, EX_NONE, 2>(ctx, A);
    if (integer) return launch_pass<int, PH_NONE, GM_TAN, EX_ENERGY, 2>(ctx, A);
    return launch_pass<double, PH_NONE, GM_TAN, EX_ENERGY, 2>(ctx, A);
}

}  // namespace fq
