// fq_small.cu -- host side of the small-instance kernels (fq_small.cuh): one
// instance with its data in the kernel parameters, or batches of one size
// class.  The clusters (fq_small_cluster.cu) and the cooperative grid (fq_mid.cu)
// are translation units of their own: a process loads a unit whole when it first
// uses one of its kernels.  All in one took 3.4 ms with the first call on B200.
#include <math.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "fq_ctx.h"
#include "fq_engine.h"
#include "fq_small.cuh"

namespace fq {

void small_job(const GraphPrep& g, int P, const double* gammas, const double* betas, int flags,
               int cap, long long most, SmallJob& J, double* data) {
    const int N = g.N;
    memset(&J, 0, sizeof(J));
    J.N = N;
    J.P = P;
    J.flags = flags;
    const long long range = g.cmax - g.cmin + 1;
    J.ntab = g.integer && range <= cap && range <= most ? (int)range : 0;
    J.keep = J.ntab > 0 && (long long)P * range <= cap;
    J.cmin = (int)g.cmin;
    J.W = g.W;
    for (int i = 0; i < N; i++)
        for (int j = i + 1; j < N; j++) *data++ = g.wd[i * N + j];
    int cot = 0;
    for (int p = 0; p < P; p++) {
        int gm;
        double gx, f;
        gate_params(betas[p], gm, gx, f);
        cot += gm != GM_TAN;
        *data++ = gammas[p];
        *data++ = gm == GM_TAN ? gx : -gx;
        *data++ = pow(f, N) * (p == 0 ? fq_init_amp(N) : 1.0);
        *data++ = f * f;
    }
    J.rot = (int)((long long)N * cot & 3);
}

namespace {

// The largest of the one-CTA classes, which share their kernels.
size_t small_smem_max(bool grad) {
    size_t m = 0;
    for (int c = 0; c <= 3; c++) m = std::max(m, small_smem_bytes(c, grad, true));
    return m;
}

// One size class c: a single instance (one != null) or njobs descriptors on the
// device.
template <bool GRAD>
int launch_any(int c, const SmallArgs* one, const SmallJob* jobs, int njobs, cudaStream_t st) {
    if (c > 3) return launch_small_cluster(c, GRAD, one, jobs, njobs, st);
    void* args[1] = {one ? (void*)one : (void*)&jobs};
    const size_t smem = small_smem_bytes(c, GRAD, one != nullptr);
    const void* fn = one ? (const void*)k_small_one<GRAD> : (const void*)k_small_batch<GRAD>;
    // Every class shares the function, and threads set this concurrently:
    // always the largest class's size.
    FQ_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)small_smem_max(GRAD)));
    // A warp at least; one instance alone also gets warps that only help
    // to fill the phase tables.
    const int threads = std::max(32 << c, one ? 256 : 32);
    FQ_CUDA(cudaLaunchKernel(fn, dim3((unsigned)njobs), dim3(threads), args, smem, st));
    return FQ_OK;
}

}  // namespace

int launch_small_batch(const SmallJob* jobs, int njobs, int c, cudaStream_t st) {
    return launch_any<true>(c, nullptr, jobs, njobs, st);
}

// Room for `words` in ctx->d_job (forward circuits of more than 2048 layers
// outgrow it), also during a capture.
static int job_buffer(fq_ctx* ctx, size_t words) {
    if (words <= ctx->job_words) return FQ_OK;
    words = std::max(words, 2 * ctx->job_words);  // so the outgrown ones stay below the last
    void* d = nullptr;
    FQ_CUDA(alloc_any_time(&d, words * sizeof(double)));
    ctx->retired.push_back(ctx->d_job);
    ctx->d_job = (double*)d;
    ctx->job_words = words;
    return FQ_OK;
}

int run_small(fq_ctx* ctx, const GraphPrep& g, int P, const double* gammas, const double* betas,
              int flags, double2* state, double* out) {
    const int c = small_class(g.N), words = small_words(g.N, P);
    const bool grad = flags & SJ_GRAD;
    const int tok = prof_begin(ctx);
    if (words <= kSmallArgWords) {
        SmallArgs a;
        small_job(g, P, gammas, betas, flags, small_table_cap(c, true), small_table_most(g.N), a.job,
                  a.data);
        a.job.out = out;
        a.job.state = state;
        FQ_TRY(grad ? launch_any<true>(c, &a, nullptr, 1, ctx->stream)
                    : launch_any<false>(c, &a, nullptr, 1, ctx->stream));
    } else {
        // Deep circuits: descriptor and data through the context's buffer.
        std::vector<double> h(job_words(g.N, P));
        FQ_TRY(job_buffer(ctx, h.size()));
        const size_t at = h.size() - words;
        SmallJob J;
        small_job(g, P, gammas, betas, flags, small_table_cap(c, false), small_table_most(g.N), J,
                  h.data() + at);
        J.w = ctx->d_job + at;
        J.lay = J.w + g.N * (g.N - 1) / 2;
        J.out = out;
        J.state = state;
        memcpy(h.data(), &J, sizeof(J));
        FQ_TRY(put_words(ctx, ctx->d_job, h.data(), h.size()));
        const SmallJob* const d = (const SmallJob*)ctx->d_job;
        FQ_TRY(grad ? launch_any<true>(c, nullptr, d, 1, ctx->stream)
                    : launch_any<false>(c, nullptr, d, 1, ctx->stream));
    }
    prof_end(ctx, tok, FQ_KIND_OTHER, 0.0);
    ctx->launches++;
    return FQ_OK;
}

}  // namespace fq
