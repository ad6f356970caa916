// fq_mid.cu -- host side of the instances of 16..19 qubits in one cooperative
// launch (fq_mid.cuh).
#include <algorithm>

#include "fq_ctx.h"
#include "fq_engine.h"
#include "fq_mid.cuh"

namespace fq {

// Amplitude bits per CTA: 128 CTAs (64 at N=16), as small as two warps.  On
// B200, gradient p=6, integer weights, with 9, 10, 11, 12 bits: N=16 107, 117,
// 141, 189 us; N=18 124 with 10, 150, 202; N=19 148 with 11, 206 with 12.
static int mid_bits(int N) { return std::max(kMidMinBits, N - 8); }

bool mid_ok(const fq_ctx* ctx, int N, int P) {
    return N >= kMidMinQubits && N <= kMidMaxQubits && P <= kMidMaxLayers &&
           1 << (N - 1 - mid_bits(N)) <= std::min(ctx->num_sms, kMidMaxCtas) && ctx->cooperative;
}

int run_mid(fq_ctx* ctx, const GraphPrep& g, int P, const double* gammas, const double* betas,
            int flags, double2* state, double2* lam, double* out) {
    const int N = g.N, nb = mid_bits(N), grid = 1 << (N - 1 - nb), threads = 1 << (nb - kSmallBits);
    const bool grad = flags & SJ_GRAD;
    MidArgs a;
    a.nb = nb;
    small_job(g, P, gammas, betas, flags, kMidTable, 16 * threads, a.job, a.data);
    a.job.out = out;
    a.job.state = state;
    a.lam = lam;
    a.partial = ctx->d_partial;
    a.counter = ctx->d_counter;
    a.err = ctx->err;
    a.polls = ctx->polls < 0 ? kMidPolls : std::min(ctx->polls, kMidPolls);
    const void* fn = grad ? (const void*)k_mid<true> : (const void*)k_mid<false>;
    // Only the tables the job has: instances of other lanes fit beside it.
    const size_t smem = mid_smem_bytes(nb, grad, a.job.ntab * (a.job.keep ? P : 1));
    // The largest size for every N: contexts on other threads set it too.
    FQ_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)mid_smem_bytes(kMidMaxBits, grad, kMidTable)));
    void* args[1] = {&a};
    const int tok = prof_begin(ctx);
    const cudaError_t e = cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(threads), args, smem,
                                                      ctx->stream);
    prof_end(ctx, tok, FQ_KIND_OTHER, 0.0);
    if (e == cudaErrorCooperativeLaunchTooLarge) {
        // The stream has fewer SMs than the device: the passes from now on.
        cudaGetLastError();
        ctx->cooperative = false;
        return FQ_OK;
    }
    FQ_CUDA(e);
    ctx->launches++;
    return FQ_OK;
}

}  // namespace fq
