// fq_disp_fused.cuh -- launch of the fused two-layer pass (k_pass with
// GM2): RX of one layer, the next layer's cost phase and its RX, in one sweep.
#pragma once

#include "fq_launch.cuh"
#include "fq_pass_col.cuh"

namespace fq {

// Strided tiles with rows of 8 to 128 amplitudes (targets among tile bits
// 3..11, some of them below bit 8) with the engine's tables, and eight tiles
// per SM or more, so that the ring is filled and its set-up (four sincos per
// thread) is spread: faster there at every size measured (fq_pass_col.cuh).
inline bool col_ok(fq_ctx* ctx, const PassArgs& A) {
    return !A.mir && A.l >= 3 && A.l <= 7 && !(A.tmask & 7u) && A.img && A.tcut &&
           A.ntiles >= 8ll * ctx->num_sms;
}

template <typename WT, int GM1, int GM2>
inline int launch_col(fq_ctx* ctx, const PassArgs& A, const CUtensorMap& map, TmaGeom G) {
    auto fn = k_pass_col<WT, GM1, GM2>;
    FQ_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)col_smem_bytes<WT>()));
    const i64 grid = std::min<i64>(A.ntiles / 2, (i64)ctx->num_sms);
    const int tok = prof_begin(ctx);
    fn<<<(unsigned)grid, kColThreads, col_smem_bytes<WT>(), ctx->stream>>>(A, map, G);
    FQ_CUDA(cudaGetLastError());
    ctx->last_grid = (int)grid;
    prof_end(ctx, tok, pass_kind<PH_MUL, GM1, EX_NONE, 1>(), pass_bytes<PH_MUL, EX_NONE, 1>(A));
    ctx->launches++;
    return FQ_OK;
}

template <typename WT, int GM1, int GM2>
inline int fused_launch(fq_ctx* ctx, const PassArgs& A) {
    if (col_ok(ctx, A)) {
        alignas(64) CUtensorMap map;
        TmaGeom G;
        if (make_pass_tmap(A, &map, &G) && G.kind != TG_CONTIG)
            return launch_col<WT, GM1, GM2>(ctx, A, map, G);
    }
    switch (schedule_for(A.tmask)) {
        case SC_L021: return launch_ldg<WT, PH_MUL, GM1, EX_NONE, true, SC_L021, GM2>(ctx, A);
        case SC_L01: return launch_ldg<WT, PH_MUL, GM1, EX_NONE, true, SC_L01, GM2>(ctx, A);
        default: return launch_ldg<WT, PH_MUL, GM1, EX_NONE, true, SC_L0, GM2>(ctx, A);
    }
}

template <typename WT>
inline int fused_dispatch(fq_ctx* ctx, int gm1, int gm2, const PassArgs& A) {
    FQ_CHECK((gm1 == GM_TAN || gm1 == GM_COT) && (gm2 == GM_TAN || gm2 == GM_COT),
             FQ_ERR_INVALID, "fused pass needs reduced gates (%d, %d)", gm1, gm2);
    if (gm1 == GM_TAN)
        return gm2 == GM_TAN ? fused_launch<WT, GM_TAN, GM_TAN>(ctx, A)
                             : fused_launch<WT, GM_TAN, GM_COT>(ctx, A);
    return gm2 == GM_TAN ? fused_launch<WT, GM_COT, GM_TAN>(ctx, A)
                         : fused_launch<WT, GM_COT, GM_COT>(ctx, A);
}

}  // namespace fq
