// fq_small.cuh -- whole QAOA instances on chip: up to 12 qubits in one CTA,
// 13..15 qubits in a cluster of 2, 4 or 8 CTAs.
//
// An instance keeps psi and, for the gradient, lambda in registers (8
// amplitudes of each per thread) for the whole circuit; shared memory only
// carries the changes of layout, and HBM only inputs and results.  From 9
// qubits on it keeps the half with the top qubit = 0 (fq_pass.cuh): 2^(N-1)
// amplitudes.  A launch takes one instance (its data in the kernel
// parameters, no upload) or a batch of one size class.
//
// One CTA: 2^nb amplitudes on 2^(nb-3) threads, in layouts whose 3 register
// bits lie at nb-3, nb-6, ... and 0.  A layer is phase, then rotations and
// layout changes from the top layout to the bottom one or, in every other
// layer, back up.  On the half state RX on the top qubit pairs x with ~x, so
// the layer's last exchange reads both and combines them.
//
// Cluster: CTA `rank` holds a tile of 2^11, alternately the mirror tile
// (qubits 0..9 and N-1) and the strided tile (qubits 10..N-2, the tile's top
// bits), as in the engine's passes.  As in the engine's fused schedule a
// layer ends on the tile the next one starts on, so each layer takes one
// exchange through distributed shared memory.
//
// Eight amplitudes per thread and one rolled copy of the rounds.  On B200,
// kernel times in microseconds with tiles of 2^12 per CTA in clusters: N=12
// p=4 gradient (integer weights) 42.6, N=15 p=6 (FP64 weights) 156; sixteen
// per thread 41.8 and 163 (one warp per scheduler waits for its own results
// where eight pay a third exchange); sixteen with every round unrolled 46 and
// 143, but 92 and 223 with a cold instruction cache, which is a batch's or a
// first call's case.  Tiles of 2^11 (twice the CTAs) took the N=15 call from
// 178 to 133.
//
// Only the tangent form of the reduced RX is needed: the cotangent gate
// [[u,-i],[-i,u]] is -i X [[1,iu],[iu,1]], and X on every qubit leaves these
// states as they are, so such a layer runs with t = -u and the final state
// takes a factor (-i)^N (SmallJob::rot).
//
// Phases are one sincos of the reference's own argument (2C - W) gamma / 2
// per cut value (a table, integer weights) or per amplitude.  Sums are fixed
// trees: an instance gives the same bits alone and in a batch.
//
// What bounds it: one SM's shared-memory traffic and dependent rounds.  Of
// the 80 k cycles of the N=12 gradient above 32 k are layout changes (each
// near its 512 to 1536 cycles of shared-memory wavefronts), 23 k rotations
// (FP64 pipe half busy), 12 k phases, 6 k set-up; in a cluster the exchange
// between CTAs adds 4.8 k cycles per layer and direction.  Against the
// shared-memory butterflies this replaces (whole calls, A/B in one call):
// gradient N=12 p=4 64 against 260 us, N=15 p=6 133 against 627 us; forward
// N=9 p=2 31 against 72 us.
#pragma once

#include <cooperative_groups.h>

#include "fq_pass.cuh"
#include "fq_small.h"

namespace fq {

// Slots of one vector's exchange buffer (padded: pslot).
__host__ __device__ constexpr size_t small_slots(int nb) {
    return ((size_t)1 << nb) + ((size_t)1 << (nb - 4));
}
// Shared memory: the exchange buffer (one or two vectors), the cut values of
// one tile (a cluster: two), the phase table, the weights and sums.  FP64
// weights keep a phase per amplitude in the first vector's buffer instead.
constexpr int kSmallBits = 3;   // register bits
constexpr int kSmallRegs = 8;
constexpr int kSmallThreads = 256;  // of the largest CTA
constexpr int kSmallWarps = kSmallThreads / 32;
constexpr int kWsStride = 17;   // row stride of the weights (kSmallJobMaxQubits rows)
constexpr int kSumLayers = 32;  // layers whose sums are kept before they are written out
// Doubles of the weights and the sums, an even number (16-byte pieces follow).
constexpr size_t kSmallFixed =
    sizeof(double) * ((kSmallJobMaxQubits * kWsStride + (2 * kSumLayers + 1) * kSmallWarps +
                       2 * kSumLayers + 2) / 2 * 2 + 2);
static_assert(kSmallFixed % sizeof(double2) == 0 && small_slots(8) % 2 == 0, "aligned tables");
// One-CTA classes 0..3 (nb = 8..11).
__host__ __device__ inline size_t small_smem_bytes(int c, bool grad, bool alone) {
    const size_t s = small_slots(8 + c);
    return (grad ? 2 : 1) * s * sizeof(double2) + s * sizeof(double) + kSmallFixed +
           (size_t)small_table_cap(c, alone) * sizeof(double2);
}
// Clusters: integer weights keep 4-byte cut values and the phase table in
// the second half of the cut values' room.
__host__ __device__ inline size_t small_cluster_smem_bytes(bool grad) {
    const size_t s = small_slots(11);
    return (grad ? 2 : 1) * s * sizeof(double2) + 2 * s * sizeof(double) + kSmallFixed;
}

// Weights into shared memory (symmetric, zero-padded rows), all threads.
__device__ __forceinline__ void small_weights(const SmallJob& J, double* ws, int nthreads) {
    for (int i = threadIdx.x; i < kSmallJobMaxQubits * kWsStride; i += nthreads) ws[i] = 0;
    __syncthreads();
    const int N = J.N;
    for (int e = threadIdx.x; e < N * N; e += nthreads) {
        const int i = e / N, j = e - i * N;
        if (j > i) {
            const double x = J.w[i * (2 * N - i - 1) / 2 + (j - i - 1)];
            ws[i * kWsStride + j] = x;
            ws[j * kWsStride + i] = x;
        }
    }
    __syncthreads();
}

// Cut values of a thread's 8 registers, whose bits are the qubits q0..q2
// (all clear in z, which has the thread's other bits), over the first NQ
// qubits.
template <int NQ>
__device__ __forceinline__ void small_cuts(const double* ws, int z, int q0, int q1, int q2,
                                           double (&c)[kSmallRegs]) {
    const int q[3] = {q0, q1, q2};
    double cb = 0, g[3];
#pragma unroll 1
    for (int i = 0; i < NQ; i++) {
        const double* row = ws + i * kWsStride;
        const int m = z ^ -((z >> i) & 1);  // bit j set: edge (i, j) is cut
        double s = 0;
#pragma unroll
        for (int j = 0; j < NQ; j++)
            if (j > i && ((m >> j) & 1)) s += row[j];
        cb += s;
    }
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const double* row = ws + q[k] * kWsStride;
        // Setting register bit k cuts its edges to clear bits (the other
        // register bits among them) and uncuts those to set bits.
        double s = 0;
#pragma unroll
        for (int j = 0; j < NQ; j++) s += ((z >> j) & 1) ? -row[j] : row[j];
        g[k] = s;
    }
#pragma unroll
    for (int r = 0; r < kSmallRegs; r++) {
        double s = cb;
#pragma unroll
        for (int k = 0; k < 3; k++)
            if ((r >> k) & 1) {
                s += g[k];
#pragma unroll
                for (int k2 = 0; k2 < k; k2++)  // no cut between two set bits: counted twice
                    if ((r >> k2) & 1) s -= 2 * ws[q[k] * kWsStride + q[k2]];
            }
        c[r] = s;
    }
}

// (-i)^rot * a.
__device__ __forceinline__ double2 small_turned(double2 a, int rot) {
    if (rot & 2) a = make_double2(-a.x, -a.y);
    if (rot & 1) a = make_double2(a.y, -a.x);
    return a;
}

__device__ __forceinline__ double small_warp_sum(double x) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

// A thread's slots in the layout whose register bits start at bit p:
// register r at b + at(r), the amplitude of ~x at c + at(7 - r).
struct SmallLay {
    int b, c, p;
    __device__ __forceinline__ int at(int r) const { return pslot(r << p); }
};

// One instance on one CTA (CB = 0, run-time nb) or on a cluster of 2^CB
// CTAs (nb = 11).  blockDim.x may exceed the 2^(nb-3) threads that hold
// amplitudes: the others help to fill the phase tables.
template <bool GRAD, int CB>
struct SmallRun {
    const SmallJob& J;
    int nb, nt;      // amplitude bits, threads that hold amplitudes
    int nq;          // qubits among the amplitude bits
    int S;           // slots per vector
    bool on;         // this thread holds amplitudes
    double2* buf;
    double* cz;      // cut values: double, or int with a phase table
    double2* tab0;   // phase tables (integer weights), and the current layer's
    double2* tab;
    double* red;     // [2 * kSumLayers + 1][kSmallWarps]
    double2 v[kSmallRegs], w[GRAD ? kSmallRegs : 1];
    double sc, gb;   // scale of the vectors and dE/dbeta in the reverse sweep

    __device__ __forceinline__ SmallRun(const SmallJob& j) : J(j) {}

    // First register bit of layout k, and the layout.
    __device__ __forceinline__ int pos(int k) const { return max(nb - kSmallBits * (k + 1), 0); }
    __device__ __forceinline__ SmallLay lay(int k) const {
        const int p = pos(k), t = threadIdx.x, u = nt - 1 - t, lo = (1 << p) - 1;
        return {pslot((t & lo) | ((t & ~lo) << kSmallBits)),
                pslot((u & lo) | ((u & ~lo) << kSmallBits)), p};
    }
    // Layouts that cover every bit from nb down to `first`.
    __device__ __forceinline__ int rounds_from(int first) const {
        return (nb - first + kSmallBits - 1) / kSmallBits;
    }
    // Targets of layout k: its bits not covered by the layout above, from
    // `first` on, and below nq.
    __device__ __forceinline__ unsigned targets(int k, int first) const {
        const int p = pos(k);
        const int hi = min(k == 0 ? nb : pos(k - 1), nq), lo = max(p, first);
        return hi > lo ? ((1u << (hi - p)) - 1u) & ~((1u << (lo - p)) - 1u) : 0u;
    }

    __device__ __forceinline__ double cut(const double* c, int slot) const {
        return J.ntab ? (double)(reinterpret_cast<const int*>(c)[slot] + J.cmin) : c[slot];
    }

    // Cut values of a tile, registers in the top layout.
    template <int NQ>
    __device__ __forceinline__ void put_cuts(const double* ws, double* c, int z, int q0, int q1,
                                             int q2) {
        if (!on) return;
        double x[kSmallRegs];
        small_cuts<NQ>(ws, z, q0, q1, q2, x);
        const SmallLay L = lay(0);
#pragma unroll
        for (int r = 0; r < kSmallRegs; r++) {
            if (J.ntab)
                reinterpret_cast<int*>(c)[L.b + L.at(r)] = (int)x[r] - J.cmin;
            else
                c[L.b + L.at(r)] = x[r];
        }
    }

    // Phase tables of `layers` layers from layer k on, all threads.  The cut
    // values lie symmetrically around W/2, so one sincos gives the entries of
    // c and W - c (conjugates, S odd around the middle).
    __device__ __forceinline__ void tables(int k, int layers) {
        const int h = (J.ntab + 1) / 2;
#pragma unroll 1
        for (int i = threadIdx.x; i < layers * h; i += blockDim.x) {
            const int p = i / h, e = i - p * h;
            const double gamma = J.lay[4 * (k + p)], scale = J.lay[4 * (k + p) + 2];
            double sn, cs;
            sincos((2.0 * (double)(J.cmin + e) - J.W) * gamma / 2, &sn, &cs);
            double2* const t = tab0 + p * J.ntab;
            t[e] = make_double2(cs * scale, sn * scale);
            t[J.ntab - 1 - e] = make_double2(cs * scale, -sn * scale);
        }
    }
    // Makes scale * exp(i*gamma*S/2) of layer k ready for phase_at: by cut
    // value (tab), or by amplitude of the tile whose cut values are c, each
    // thread its own slots L of buf (nothing in buf is live here).
    __device__ __forceinline__ void fill(const double* c, const SmallLay& L, int k) {
        if (J.keep) {
            tab = tab0 + k * J.ntab;
        } else if (J.ntab) {
            __syncthreads();
            tables(k, 1);
            __syncthreads();
        } else if (on) {
            const double gamma = J.lay[4 * k], scale = J.lay[4 * k + 2];
#pragma unroll 1
            for (int q = 0; q < kSmallRegs; q += 4) {
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    const int o = L.b + L.at(q + r);
                    double sn, cs;
                    sincos((2.0 * c[o] - J.W) * gamma / 2, &sn, &cs);
                    buf[o] = make_double2(cs * scale, sn * scale);
                }
            }
        }
    }
    __device__ __forceinline__ double2 phase_at(const double* c, int slot) const {
        return J.ntab ? tab[reinterpret_cast<const int*>(c)[slot]] : buf[slot];
    }
    // Writes layer 0's phase (init) or multiplies layer k's in.
    __device__ __forceinline__ void phase(const double* c, const SmallLay& L, bool init) {
        if (!on) return;
#pragma unroll
        for (int r = 0; r < kSmallRegs; r++) {
            const double2 ph = phase_at(c, L.b + L.at(r));
            v[r] = init ? ph : cmul(v[r], ph);
        }
    }

    // RX on the register bits of m (with DUAL on both vectors, adding each
    // qubit's Im<w|X_q|v> times sc to gb first, see rx_regs_dual).
    template <bool DUAL>
    __device__ __forceinline__ void rot(unsigned m, double t, double f2) {
#pragma unroll
        for (int k = 0; k < kSmallBits; k++) {
            if (!((m >> k) & 1u)) continue;
            double ta = 0, tb = 0;
#pragma unroll
            for (int r = 0; r < kSmallRegs; r++) {
                const int q = r | (1 << k);
                if (q == r) continue;
                if constexpr (DUAL) {
                    ta = fma(w[r].x, v[q].y, ta);
                    ta = fma(-w[r].y, v[q].x, ta);
                    tb = fma(w[q].x, v[r].y, tb);
                    tb = fma(-w[q].y, v[r].x, tb);
                    rx_pair<GM_TAN>(w[r], w[q], t, 0.0, 0.0);
                }
                rx_pair<GM_TAN>(v[r], v[q], t, 0.0, 0.0);
            }
            if constexpr (DUAL) {
                gb = fma(sc, ta + tb, gb);
                sc *= f2;
            }
        }
    }

    // Layout change through buf; flip also rotates the top qubit of a half
    // state, the pair of x and ~x.  Every reader of buf is past a barrier
    // when it ends, so the next writes (own slots) need none before them and
    // run alongside other warps' rotations.
    template <bool DUAL>
    __device__ __forceinline__ void exchange(const SmallLay& f, const SmallLay& g, bool flip,
                                             double t, double f2) {
        if (on) {
#pragma unroll
            for (int r = 0; r < kSmallRegs; r++) {
                buf[f.b + f.at(r)] = v[r];
                if (DUAL) buf[S + f.b + f.at(r)] = w[DUAL ? r : 0];
            }
        }
        __syncthreads();
        if (on && !flip) {
#pragma unroll
            for (int r = 0; r < kSmallRegs; r++) {
                v[r] = buf[g.b + g.at(r)];
                if (DUAL) w[DUAL ? r : 0] = buf[S + g.b + g.at(r)];
            }
        } else if (on) {
            double ta = 0;
#pragma unroll
            for (int r = 0; r < kSmallRegs; r++) {
                const int o = g.b + g.at(r), oc = g.c + g.at(kSmallRegs - 1 - r);
                const double2 q = buf[oc];
                v[r] = rx_self<GM_TAN>(buf[o], q, t, 0.0, 0.0);
                if (DUAL) {
                    const double2 m = buf[S + o];
                    ta = fma(m.x, q.y, ta);
                    ta = fma(-m.y, q.x, ta);
                    w[DUAL ? r : 0] = rx_self<GM_TAN>(m, buf[S + oc], t, 0.0, 0.0);
                }
            }
            if (DUAL) {
                gb = fma(sc, ta, gb);
                sc *= f2;
            }
        }
        __syncthreads();
    }

    // The n rounds of a tile on its bits from `first` on, down (top layout
    // first) or up.  A cluster's CTAs have all read their tile once the first
    // round is past `wait`.
    template <bool DUAL>
    __device__ __forceinline__ void rounds(int n, int first, bool down, bool flip, bool wait,
                                           double t, double f2) {
#pragma unroll 1
        for (int i = 0; i < n; i++) {
            const int k = down ? i : n - 1 - i;
            if (on) rot<DUAL>(targets(k, first), t, f2);
            if constexpr (CB > 0)
                if (i == 0 && wait) cooperative_groups::this_cluster().barrier_wait();
            if (i + 1 < n) exchange<DUAL>(lay(k), lay(down ? k + 1 : k - 1), flip && i == n - 2, t, f2);
        }
    }

    // <C>'s partial sum, and lambda = C psi.
    __device__ __forceinline__ void energy(const double* c, const SmallLay& L) {
        double e = 0;
        if (on) {
#pragma unroll
            for (int r = 0; r < kSmallRegs; r++) {
                const double x = cut(c, L.b + L.at(r));
                e = fma(fma(v[r].x, v[r].x, v[r].y * v[r].y), x, e);
                if constexpr (GRAD) w[r] = make_double2(x * v[r].x, x * v[r].y);
            }
        }
        e = small_warp_sum(e);
        if ((threadIdx.x & 31) == 0 && on) red[2 * kSumLayers * kSmallWarps + (threadIdx.x >> 5)] = e;
    }

    // dE/dgamma_k's sum and the inverse phase of layer k (k > 0).
    __device__ __forceinline__ double unphase(const double* c, const SmallLay& L, int k) {
        double s = 0;
        if constexpr (GRAD) {
            if (on) {
#pragma unroll
                for (int r = 0; r < kSmallRegs; r++)
                    s = fma(w[r].x * v[r].y - w[r].y * v[r].x,
                            2.0 * cut(c, L.b + L.at(r)) - J.W, s);
            }
            if (k > 0) {
                fill(c, L, k);
                if (on) {
#pragma unroll
                    for (int r = 0; r < kSmallRegs; r++) {
                        double2 ph = phase_at(c, L.b + L.at(r));
                        ph.y = -ph.y;
                        v[r] = cmul(v[r], ph);
                        w[r] = cmul(w[r], ph);
                    }
                }
            }
        }
        return sc * s;
    }

    // Keeps layer k's sums; true when a group of layers k .. k + kSumLayers - 1
    // is complete (after a barrier).
    __device__ __forceinline__ bool keep(int k, double gg) {
        const double b = small_warp_sum(on ? gb : 0.0);
        gg = small_warp_sum(on ? gg : 0.0);
        const int j = k % kSumLayers;
        if ((threadIdx.x & 31) == 0 && on) {
            red[(2 * j) * kSmallWarps + (threadIdx.x >> 5)] = gg;
            red[(2 * j + 1) * kSmallWarps + (threadIdx.x >> 5)] = b;
        }
        if (j == 0) __syncthreads();
        return j == 0;
    }
    __device__ __forceinline__ double row_sum(int i) const {
        const int nw = (nt + 31) / 32;
        double s = 0;
        for (int x = 0; x < nw; x++) s += red[i * kSmallWarps + x];
        return s;
    }
};

// ---------------------------------------------------------------- one CTA --

template <bool GRAD>
__device__ __forceinline__ void small_run(const SmallJob& J, unsigned char* sm) {
    SmallRun<GRAD, 0> R(J);
    const int c = small_class(J.N), nb = 8 + c;
    R.nb = nb;
    R.nt = 1 << (nb - kSmallBits);
    R.nq = min(J.N, nb);
    R.S = (int)small_slots(nb);
    R.on = (int)threadIdx.x < R.nt;
    R.buf = reinterpret_cast<double2*>(sm);
    R.cz = reinterpret_cast<double*>(R.buf + (GRAD ? 2 : 1) * R.S);
    double* ws = R.cz + R.S;
    R.red = ws + kSmallJobMaxQubits * kWsStride;
    R.tab = R.tab0 = reinterpret_cast<double2*>(ws + kSmallFixed / sizeof(double));
    const int tid = threadIdx.x, N = J.N, P = J.P;
    const bool half = N > nb;
    const double mul = half ? 2.0 : 1.0;  // a half state's sums
    const int n = R.rounds_from(0);
    small_weights(J, ws, blockDim.x);
    R.template put_cuts<kSmallMaxQubits>(ws, R.cz, tid, nb - 3, nb - 2, nb - 1);
    if (J.keep) R.tables(0, P);
    __syncthreads();
#pragma unroll 1
    for (int p = 0; p < P; p++) {
        const bool down = !(p & 1);
        const SmallLay L = R.lay(down ? 0 : n - 1);
        R.fill(R.cz, L, p);
        R.phase(R.cz, L, p == 0);
        if (p == 0 && N < 8) {  // the amplitudes beyond 2^N stay zero
#pragma unroll
            for (int r = 0; r < kSmallRegs; r++)
                if ((tid | (r << (nb - kSmallBits))) >> N) R.v[r] = make_double2(0.0, 0.0);
        }
        R.template rounds<false>(n, 0, down, half, false, J.lay[4 * p + 1], 0.0);
    }
    const int end = P & 1 ? n - 1 : 0;  // the layout the circuit ended in
    if ((J.flags & SJ_STATE) && R.on) {
        const int step = end ? 1 : 1 << (nb - kSmallBits), base = end ? tid << kSmallBits : tid;
#pragma unroll
        for (int r = 0; r < kSmallRegs; r++) {
            const int x = base + r * step;
            const double2 a = small_turned(R.v[r], J.rot);
            if (x < (1 << N)) J.state[x] = a;
            if (half) J.state[(1 << N) - 1 - x] = a;
        }
    }
    R.energy(R.cz, R.lay(end));
    if constexpr (GRAD) {
#pragma unroll 1
        for (int k = P - 1; k >= 0; k--) {
            R.sc = 1;
            R.gb = 0;
            // Layer k went down for even k: back up, to where its phase was.
            const bool down = k & 1;
            R.template rounds<true>(n, 0, down, half, false, -J.lay[4 * k + 1],
                                    J.lay[4 * k + 3]);
            const double gg = R.unphase(R.cz, R.lay(down ? n - 1 : 0), k);
            if (R.keep(k, gg)) {
                for (int i = tid; i < 2 * kSumLayers && k + (i >> 1) < P; i += blockDim.x)
                    J.out[1 + ((i & 1) ? P : 0) + k + (i >> 1)] =
                        ((i & 1) ? mul : -mul) * R.row_sum(i);
                __syncthreads();
            }
        }
    }
    __syncthreads();
    if (tid == 0) J.out[0] = mul * R.row_sum(2 * kSumLayers);
}

// One instance, its data behind the descriptor in the kernel parameters.
constexpr int kSmallArgWords = 105 + 4 * 32;
struct SmallArgs {
    SmallJob job;
    double data[kSmallArgWords];
};

__device__ __forceinline__ SmallJob small_arg_job(const SmallArgs& a) {
    SmallJob J = a.job;
    J.w = a.data;
    J.lay = a.data + J.N * (J.N - 1) / 2;
    return J;
}

template <bool GRAD>
__global__ void __launch_bounds__(kSmallThreads, 2) k_small_one(const __grid_constant__ SmallArgs a) {
    extern __shared__ __align__(16) unsigned char smraw[];
    const SmallJob J = small_arg_job(a);
    small_run<GRAD>(J, smraw);
}

template <bool GRAD>
__global__ void __launch_bounds__(kSmallThreads, 2) k_small_batch(const SmallJob* jobs) {
    extern __shared__ __align__(16) unsigned char smraw[];
    const SmallJob J = jobs[blockIdx.x];
    small_run<GRAD>(J, smraw);
}

// ---------------------------------------------------------------- cluster --

// The tile changes hands through distributed shared memory.  Register r of
// a tile in the top layout (index tid | r << 8) comes from the CTA and slot
// that held it as the other kind of tile; which CTA depends on r and, with 8
// CTAs, on the thread's top bit (the same across a warp, which reads 512
// contiguous bytes).  The upper half of either tile is the mirror image of
// the other's addresses: hi is the slot of register 4.
template <int CB>
__device__ __forceinline__ void small_fetch(double2 (&v)[kSmallRegs],
                                            double2* const (&peer)[1 << CB], int lo, int hi) {
    const bool b = threadIdx.x >> 7;
#pragma unroll
    for (int r = 0; r < kSmallRegs; r++) {
        const int u = r < 4 ? r : 7 - r;  // bits 8, 9 of the unmirrored index
        // Row bits among the registers (one with 2 CTAs): slots of 2^8.
        const int row = CB == 1 ? (r & 1) * 272 : 0;
        const double2* p;
        if (CB == 3)
            p = (r < 4) == b ? peer[(2 * u + 1) & ((1 << CB) - 1)] : peer[(2 * u) & ((1 << CB) - 1)];
        else
            p = peer[CB == 2 ? u : u >> 1];
        v[r] = r < 4 ? p[lo + row] : p[hi - row];
    }
}

template <int CB, bool GRAD>
__device__ __forceinline__ void small_cluster_run(const SmallJob& J, unsigned char* sm) {
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    constexpr int N = 12 + CB, S = (int)small_slots(11), l = 10 - CB;
    SmallRun<GRAD, CB> R(J);
    R.nb = 11;
    R.nt = kSmallThreads;
    R.nq = 11;
    R.S = S;
    R.on = true;
    R.buf = reinterpret_cast<double2*>(sm);
    double* const cA = reinterpret_cast<double*>(R.buf + (GRAD ? 2 : 1) * S);
    double* const ws = cA + 2 * S;
    R.red = ws + kSmallJobMaxQubits * kWsStride;
    double* const part = R.red + (2 * kSumLayers + 1) * kSmallWarps;  // read by rank 0
    double* const cB = J.ntab ? cA + S / 2 : cA + S;
    R.tab = R.tab0 = reinterpret_cast<double2*>(cA + S);
    const int tid = threadIdx.x, rank = (int)cl.block_rank(), P = J.P;
    // Rounds and first target bit of the mirror and the strided tile.
    constexpr int nA = 4, nB = CB == 3 ? 2 : 1;
    double2* peer[1 << CB];
#pragma unroll
    for (int r = 0; r < (1 << CB); r++) peer[r] = cl.map_shared_rank(R.buf, r);
    small_weights(J, ws, kSmallThreads);
    // Mirror tile: registers = qubits 8, 9, N-1, the rank's bits from 10;
    // strided tile: registers = tile bits 8..10 (and tile bit 7 of the thread
    // is qubit 10 with 8 CTAs), the rank's bits from l.
    auto q = [](int j) { return j < l ? j : j + 10 - l; };
    const int zB = CB == 3 ? (tid & 127) | ((tid >> 7) << q(7)) : tid;
    R.template put_cuts<N>(ws, cA, tid | (rank << 10), 8, 9, N - 1);
    R.template put_cuts<N>(ws, cB, zB | (rank << l), q(8), q(9), q(10));
    const int row = tid & ((1 << l) - 1);  // the row bits (all of tid but with 8 CTAs)
    const int lo = pslot(row | (rank << l));
    const int hiB = pslot(1024 | (1023 - (row | (rank << l))));
    const int hiA = pslot(((1 << l) - 1 - row) | (((2 << CB) - 1 - rank) << l));
    // The tile leaves from layout L; the other kind of tile arrives in H.  The
    // barrier_wait that matches the arrive comes before buf is written again.
    auto change = [&](const SmallLay& L, bool to_strided, auto dual) {
        [[maybe_unused]] constexpr bool D = decltype(dual)::value;
#pragma unroll
        for (int r = 0; r < kSmallRegs; r++) {
            R.buf[L.b + L.at(r)] = R.v[r];
            if constexpr (GRAD)
                if (D) R.buf[S + L.b + L.at(r)] = R.w[r];
        }
        cl.sync();
        const int hi = to_strided ? hiB : hiA;
        small_fetch<CB>(R.v, peer, lo, hi);
        if constexpr (GRAD)
            if (D) small_fetch<CB>(R.w, peer, S + lo, S + hi);
        cl.barrier_arrive();
    };
    if (J.keep) R.tables(0, P);
    __syncthreads();
    // Pass s: the rest of layer s-1's mixer on this tile, then (s < P) layer
    // s's phase and its mixer's first part; odd passes on the strided tile.
    R.fill(cA, R.lay(0), 0);
    R.phase(cA, R.lay(0), true);
    R.template rounds<false>(nA, 0, true, false, false, J.lay[1], 0.0);
#pragma unroll 1
    for (int s = 1; s <= P; s++) {
        const bool str = s & 1;
        const int n = str ? nB : nA, first = str ? l : 0;
        const double* const c = str ? cB : cA;
        change(R.lay(s == 1 ? nA - 1 : 0), str, std::false_type());
        R.template rounds<false>(n, first, true, false, true, J.lay[4 * s - 3], 0.0);
        if (s < P) {
            const SmallLay L = R.lay(n - 1);
            R.fill(c, L, s);
            R.phase(c, L, false);
            R.template rounds<false>(n, first, false, false, false, J.lay[4 * s + 1], 0.0);
        }
    }
    // The circuit ended in the bottom layout of the strided (odd P) or mirror tile.
    const bool strided = P & 1;
    const int end = strided ? nB - 1 : nA - 1;
    if (J.flags & SJ_STATE) {
        constexpr int M = (1 << (N - 1)) - 1, full = (1 << N) - 1;
        const int p = R.pos(end), lom = (1 << p) - 1;
#pragma unroll
        for (int r = 0; r < kSmallRegs; r++) {
            const int i = (tid & lom) | ((tid & ~lom) << kSmallBits) | (r << p);
            int x;
            if (strided) {
                x = (i & ((1 << l) - 1)) | (rank << l) | ((i >> l) << 10);
            } else {
                x = (i & 1023) | (rank << 10);
                if (i >> 10) x = M - x;
            }
            const double2 a = small_turned(R.v[r], J.rot);
            J.state[x] = a;
            J.state[full - x] = a;
        }
    }
    R.energy(strided ? cB : cA, R.lay(end));
    if constexpr (GRAD) {
        R.sc = 1;
        R.gb = 0;
        R.template rounds<true>(end + 1, strided ? l : 0, false, false, false, -J.lay[4 * P - 3],
                                J.lay[4 * P - 1]);
#pragma unroll 1
        for (int k = P - 1; k >= 0; k--) {
            // Pass k back: completes layer k's mixer, then layer k-1's part.
            const bool str = k & 1;
            const int n = str ? nB : nA, first = str ? l : 0;
            const double* const c = str ? cB : cA;
            change(R.lay(0), str, std::true_type());
            R.template rounds<true>(n, first, true, false, true, -J.lay[4 * k + 1],
                                    J.lay[4 * k + 3]);
            const double gg = R.unphase(c, R.lay(n - 1), k);
            if (R.keep(k, gg)) {
                if (tid < 2 * kSumLayers) part[tid] = R.row_sum(tid);
                cl.sync();
                const int kk = k + (tid >> 1);
                if (rank == 0 && tid < 2 * kSumLayers && kk < P) {
                    double s = 0;
                    for (int x = 0; x < (1 << CB); x++) s += cl.map_shared_rank(part, x)[tid];
                    J.out[1 + ((tid & 1) ? P : 0) + kk] = (tid & 1) ? 2.0 * s : -2.0 * s;
                }
                cl.sync();
            }
            if (k > 0) {
                R.sc = 1;
                R.gb = 0;
                R.template rounds<true>(n, first, false, false, false, -J.lay[4 * k - 3],
                                        J.lay[4 * k - 1]);
            }
        }
    }
    __syncthreads();
    if (tid == 0) part[2 * kSumLayers] = R.row_sum(2 * kSumLayers);
    cl.sync();
    if (rank == 0 && tid == 0) {
        double s = 0;
        for (int x = 0; x < (1 << CB); x++) s += cl.map_shared_rank(part, x)[2 * kSumLayers];
        J.out[0] = 2.0 * s;
    }
    cl.sync();  // no CTA leaves while a peer may still read its memory
}

template <int CB, bool GRAD>
__global__ void __launch_bounds__(kSmallThreads, 2)
    k_small_cluster_one(const __grid_constant__ SmallArgs a) {
    extern __shared__ __align__(16) unsigned char smraw[];
    const SmallJob J = small_arg_job(a);
    small_cluster_run<CB, GRAD>(J, smraw);
}

template <int CB, bool GRAD>
__global__ void __launch_bounds__(kSmallThreads, 2) k_small_cluster_batch(const SmallJob* jobs) {
    extern __shared__ __align__(16) unsigned char smraw[];
    const SmallJob J = jobs[blockIdx.x >> CB];
    small_cluster_run<CB, GRAD>(J, smraw);
}

}  // namespace fq
