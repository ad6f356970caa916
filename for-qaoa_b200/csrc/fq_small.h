// fq_small.h -- job descriptor of the small-instance kernels (fq_small.cuh):
// one whole QAOA instance per CTA (N <= 12) or per cluster of 2^(N-12) CTAs
// (N = 13..15).
#pragma once

#include <vector>

#include "fq_common.cuh"

namespace fq {

constexpr int kSmallMaxQubits = 12;     // qubits of a one-CTA instance
constexpr int kSmallJobMaxQubits = 15;  // of a cluster's, and of a request that needs no
                                        // buffers (FQ_SMALL_MAX_QUBITS)

enum { SJ_GRAD = 1, SJ_STATE = 2 };

struct SmallJob {
    int N, P, flags;
    int ntab;           // integer weights: cut values cmin..cmin+ntab-1 get a phase table; 0: sincos
    int keep;           // every layer's table is kept (P * ntab entries), else one at a time
    int cmin;
    int rot;            // the final state is (-i)^rot times what the layers give (see small_job)
    double W;           // total weight
    const double* w;    // upper triangle, row by row: N(N-1)/2
    const double* lay;  // 4 per layer: gamma, t, the phase's scale, f^2
    double* out;        // [0] <C>, then with SJ_GRAD dE/dgamma[P], dE/dbeta[P]
    double2* state;     // final state (SJ_STATE), 2^N
};

// Data words of a job behind its descriptor.
__host__ __device__ inline int small_words(int N, int P) { return N * (N - 1) / 2 + 4 * P; }

// Words of a job in device memory: descriptor, then data.
__host__ __device__ inline size_t job_words(int N, int P) {
    return (sizeof(SmallJob) + 7) / 8 + (size_t)small_words(N, P);
}
// Room every context has: any gradient's (1 + 2P results of kResultWords).
constexpr size_t kJobWords = (sizeof(SmallJob) + 7) / 8 +
                             kSmallJobMaxQubits * (kSmallJobMaxQubits - 1) / 2 + 4 * 2048;

// Size class of an N-qubit instance: 0..3 for one CTA of 2^(8..11)
// amplitudes (a half state from N = 9 on), 4..6 for clusters of 2, 4, 8.
constexpr int kSmallClasses = 7;
__host__ __device__ inline int small_class(int N) { return N <= 9 ? 0 : N - 9; }
// Phase-table entries of a job of size class c: what is left of the shared
// memory at the residency its registers allow in a batch (two CTAs per SM of
// class 3, more below), and more for an instance alone.  Clusters use the
// room integer cut values leave free.
__host__ __device__ inline int small_table_cap(int c, bool alone) {
    return c > 3 ? 1088 : alone ? 4096 : 128 << c;
}

// A table is worth its sincos (half its entries) up to the 2^(N-1) amplitudes.
inline long long small_table_most(int N) { return 1ll << N; }

}  // namespace fq
