// fq_small_cluster.cu -- launches of the small instances of 13..15 qubits, a
// cluster of CTAs each (fq_small.cuh).
#include <string.h>

#include "fq_engine.h"
#include "fq_small.cuh"

namespace fq {

namespace {

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

template <int CB, bool GRAD>
int launch_class(const SmallArgs* one, const SmallJob* jobs, int njobs, cudaStream_t st) {
    void* args[1] = {one ? (void*)one : (void*)&jobs};
    const size_t smem = small_cluster_smem_bytes(GRAD);
    const void* fn = one ? (const void*)k_small_cluster_one<CB, GRAD>
                         : (const void*)k_small_cluster_batch<CB, GRAD>;
    FQ_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    return launch_cluster(fn, CB, njobs, smem, st, args);
}

template <bool GRAD>
int launch_any(int c, const SmallArgs* one, const SmallJob* jobs, int njobs, cudaStream_t st) {
    switch (c) {
        case 4: return launch_class<1, GRAD>(one, jobs, njobs, st);
        case 5: return launch_class<2, GRAD>(one, jobs, njobs, st);
        default: return launch_class<3, GRAD>(one, jobs, njobs, st);
    }
}

}  // namespace

int launch_small_cluster(int c, bool grad, const SmallArgs* one, const SmallJob* jobs, int njobs,
                         cudaStream_t st) {
    return grad ? launch_any<true>(c, one, jobs, njobs, st)
                : launch_any<false>(c, one, jobs, njobs, st);
}

}  // namespace fq
