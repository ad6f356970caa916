// fq_small.cu -- host side of the small-instance kernels (fq_small.cuh): one
// instance with its data in the kernel parameters, or batches of one size
// class.
#include <math.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "fq_ctx.h"
#include "fq_engine.h"
#include "fq_mid.cuh"

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

template <typename Fn>
int launch_cluster(Fn fn, int cb, int njobs, size_t smem, cudaStream_t st, void** args) {
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3((unsigned)njobs << cb);
    cfg.blockDim = dim3(kSmallThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = 1u << cb;
    at.val.clusterDim.y = 1;
    at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    FQ_CUDA(cudaLaunchKernelExC(&cfg, (const void*)fn, args));
    return FQ_OK;
}

// One size class C (small_class): a single instance (one != null) or njobs
// descriptors on the device.
template <int C, bool GRAD>
int launch_class(const SmallArgs* one, const SmallJob* jobs, int njobs, cudaStream_t st) {
    void* args[1] = {one ? (void*)one : (void*)&jobs};
    if constexpr (C <= 3) {
        const size_t smem = small_smem_bytes(C, GRAD, one != nullptr);
        const void* fn = one ? (const void*)k_small_one<GRAD> : (const void*)k_small_batch<GRAD>;
        // Every class shares the function, and threads set this concurrently:
        // always the largest class's size.
        FQ_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)small_smem_max(GRAD)));
        // A warp at least; one instance alone also gets warps that only help
        // to fill the phase tables.
        const int threads = std::max(32 << C, one ? 256 : 32);
        FQ_CUDA(cudaLaunchKernel(fn, dim3((unsigned)njobs), dim3(threads), args, smem, st));
        return FQ_OK;
    } else {
        constexpr int CB = C - 3;
        const size_t smem = small_cluster_smem_bytes(GRAD);
        const void* fn = one ? (const void*)k_small_cluster_one<CB, GRAD>
                             : (const void*)k_small_cluster_batch<CB, GRAD>;
        FQ_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        return launch_cluster(fn, CB, njobs, smem, st, args);
    }
}

template <bool GRAD>
int launch_any(int c, const SmallArgs* one, const SmallJob* jobs, int njobs, cudaStream_t st) {
    switch (c) {
        case 0: return launch_class<0, GRAD>(one, jobs, njobs, st);
        case 1: return launch_class<1, GRAD>(one, jobs, njobs, st);
        case 2: return launch_class<2, GRAD>(one, jobs, njobs, st);
        case 3: return launch_class<3, GRAD>(one, jobs, njobs, st);
        case 4: return launch_class<4, GRAD>(one, jobs, njobs, st);
        case 5: return launch_class<5, GRAD>(one, jobs, njobs, st);
        default: return launch_class<6, GRAD>(one, jobs, njobs, st);
    }
}

}  // namespace

int launch_small_batch(const SmallJob* jobs, int njobs, int c, cudaStream_t st) {
    return launch_any<true>(c, nullptr, jobs, njobs, st);
}

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
