// fq_mid.cuh -- whole circuits and gradients of 16..19 qubits in one
// cooperative launch.
//
// As passes over HBM (k_pass) these sizes are one tile per CTA and pass:
// every pass is a launch, its tables and the latency of a tile.  Here every
// CTA keeps its tile of 2^nb amplitudes of a half state (fq_pass.cuh) in
// registers and shared memory for the whole circuit, alternately as mirror
// (qubits 0..nb-2 and N-1) and as strided tile (qubits nb-1..N-2), like a
// cluster of fq_small.cuh, and its tables too.  nb is chosen to spread the
// amplitudes over most of the SMs (mid_bits).  The tiles change hands through the state buffers, which stay in L2: every CTA
// writes its tile, a grid barrier, every CTA reads its tile of the other kind
// (only the CTA itself touches a tile's addresses between two barriers).
// The cooperative launch keeps all CTAs resident; the barrier's wait is
// bounded.  Phases take one sincos of the reference's argument per cut value
// or amplitude, as in fq_small.cuh.
//
// Measured on B200 (whole calls, p=6, in one run; as passes / here): forward
// N=16 101 / 71 us, N=18 87 / 71, N=19 88 / 79, N=20 93 / 101; gradient N=16
// 197 / 105, N=18 204 / 120, N=19 206 / 148, N=20 218 / 212: the line lies at
// N = 19 (the passes launched one by one; chained, N=20 forward, p=5, takes
// 12 us less).  What bounds it: per pass a grid barrier of 2.7 k cycles, 1.5 k of
// loads and stores, and the rounds (as in fq_small.cuh).
#pragma once

#include "fq_small.cuh"

namespace fq {

constexpr int kMidMinQubits = 16;
constexpr int kMidMaxQubits = 19;
constexpr int kMidMinBits = 9;   // amplitude bits per CTA: two warps
constexpr int kMidMaxBits = 11;
constexpr int kMidMaxLayers = 64;
constexpr int kMidStride = kMidMaxQubits + 1;  // row stride of the weights
constexpr int kMidWords = kMidMaxQubits * (kMidMaxQubits - 1) / 2 + 4 * kMidMaxLayers;

struct MidArgs {
    SmallJob job;      // state = psi's buffer (a whole state with SJ_STATE)
    double2* lam;      // lambda's buffer (SJ_GRAD)
    double* partial;   // (2P + 1) x CTAs
    unsigned* counter; // grid barrier: arrivals, a multiple of kMidMaxCtas between launches
    int nb;
    int polls;         // the barrier's limit (kMidPolls)
    int* err;
    double data[kMidWords];
};
static_assert(sizeof(MidArgs) <= 4096, "kernel parameters");

constexpr int kMidMaxCtas = 128;
constexpr int kMidPolls = 1 << 21;  // of some 0.7 us each
constexpr int kMidTable = 4096;  // phase-table entries at most
// `table`: entries of the job's phase tables.
__host__ __device__ constexpr size_t mid_smem_bytes(int nb, bool grad, int table) {
    return (grad ? 2 : 1) * small_slots(nb) * sizeof(double2) +
           2 * small_slots(nb) * sizeof(double) +
           sizeof(double) * ((kMidMaxQubits * kMidStride + 1) / 2 * 2 + 12 * 13 + 16 +
                             (2 * kSumLayers + 1) * kSmallWarps) +
           table * sizeof(double2);
}
static_assert(mid_smem_bytes(kMidMaxBits, true, kMidTable) <= 227 * 1024, "one CTA per SM");
static_assert((12 * 13 + 16 + (2 * kSumLayers + 1) * kSmallWarps) % 2 == 0, "aligned tables");

// All CTAs of the grid (all resident: cooperative launch).  False if the
// bounded wait gave up.
__device__ __forceinline__ bool mid_barrier(const MidArgs& a, unsigned target) {
    __shared__ int ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        ok = 0;
        __threadfence();
        atomicAdd(a.counter, 1u);
        for (int i = 0; i < a.polls; i++) {
            unsigned c;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(c) : "l"(a.counter) : "memory");
            if ((int)(c - target) >= 0) {
                ok = 1;
                break;
            }
        }
        if (!ok) *(volatile int*)a.err = 1;
    }
    __syncthreads();
    return ok;
}

// Cut values of a tile into R's array c: tile bit j is qubit q(j), the other
// qubits have the bits of zfix.  K and e_u as in k_pass's cut tables.
template <typename Run, typename Q>
__device__ __forceinline__ void mid_cuts(Run& R, const double* ws, double* tw, double* te, double* c,
                                         int N, int zfix, Q q) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nb = R.nb;
    int tile = 0;
    for (int u = 0; u < nb; u++) tile |= 1 << q(u);
    __syncthreads();
    for (int e = tid; e < nb * nb; e += R.nt) {
        const int u = e / nb, v = e - nb * u;
        tw[u * 13 + v] = ws[q(u) * kMidStride + q(v)];
    }
    if (warp == 1 && lane < nb) {
        double s = 0;
        for (int m = 0; m < N; m++)
            if (!((tile >> m) & 1)) {
                const double w = ws[q(lane) * kMidStride + m];
                s += ((zfix >> m) & 1) ? -w : w;
            }
        te[lane] = s;
    } else if (warp == 0) {
        // Lane m: its cut edges to later fixed qubits and, when set, all its
        // edges into the tile (e_u takes them back where the tile bit is set).
        double h = 0;
        const int zm = (zfix >> lane) & 1;
        if (lane < N && !((tile >> lane) & 1))
            for (int m = 0; m < N; m++) {
                const double w = ws[lane * kMidStride + m];
                if ((tile >> m) & 1)
                    h += zm ? w : 0.0;
                else if (m > lane)
                    h += (((zfix >> m) & 1) ^ zm) ? w : 0.0;
            }
        h = small_warp_sum(h);
        if (lane == 0) te[12] = h;
    }
    __syncthreads();
    double cb = te[12], g[3];
#pragma unroll
    for (int u = 0; u < kMidMaxBits - 3; u++) {
        if (u >= nb - 3) break;
        const int zu = (tid >> u) & 1;
        double s = zu ? te[u] : 0.0;
#pragma unroll
        for (int v = u + 1; v < kMidMaxBits; v++)  // the register bits nb-3..nb-1 are clear in tid
            if (v < nb && (((tid >> v) & 1) ^ zu)) s += tw[u * 13 + v];
        cb += s;
    }
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const int u = nb - 3 + k;
        double s = te[u];
#pragma unroll
        for (int v = 0; v < kMidMaxBits; v++) {
            if (v == u || v >= nb) continue;
            const double w = tw[u * 13 + v];
            s += ((tid >> v) & 1) ? -w : w;
        }
        g[k] = s;
    }
    const SmallLay L = R.lay(0);
#pragma unroll
    for (int r = 0; r < kSmallRegs; r++) {
        double s = cb;
#pragma unroll
        for (int k = 0; k < 3; k++)
            if ((r >> k) & 1) {
                s += g[k];
#pragma unroll
                for (int k2 = 0; k2 < k; k2++)
                    if ((r >> k2) & 1) s -= 2 * tw[(nb - 3 + k) * 13 + nb - 3 + k2];
            }
        if (R.J.ntab)
            reinterpret_cast<int*>(c)[L.b + L.at(r)] = (int)s - R.J.cmin;
        else
            c[L.b + L.at(r)] = s;
    }
}

template <bool GRAD>
__global__ void __launch_bounds__(1 << (kMidMaxBits - kSmallBits)) k_mid(const __grid_constant__ MidArgs a) {
    extern __shared__ __align__(16) unsigned char smraw[];
    SmallJob J = a.job;
    const int N = J.N, P = J.P, nb = a.nb, l = 2 * nb - N;  // row bits of a strided tile
    J.w = a.data;
    J.lay = a.data + N * (N - 1) / 2;
    const int S = (int)small_slots(nb);
    SmallRun<GRAD, 0> R(J);
    R.nb = R.nq = nb;
    R.nt = blockDim.x;
    R.S = S;
    const int nA = R.rounds_from(0);
    R.on = true;
    R.buf = reinterpret_cast<double2*>(smraw);
    double* const cA = reinterpret_cast<double*>(R.buf + (GRAD ? 2 : 1) * S);
    double* const ws = cA + 2 * S;
    double* const tw = ws + (kMidMaxQubits * kMidStride + 1) / 2 * 2;
    double* const te = tw + 12 * 13;
    R.red = te + 16;
    double* const cB = cA + S;
    R.tab = R.tab0 = reinterpret_cast<double2*>(R.red + (2 * kSumLayers + 1) * kSmallWarps);
    const int tid = threadIdx.x, rank = (int)blockIdx.x, grid = (int)gridDim.x;
    const int nB = R.rounds_from(l);
    for (int e = tid; e < N * N; e += R.nt) {
        const int i = e / N, j = e - i * N, lo = min(i, j), hi = max(i, j);
        ws[i * kMidStride + j] =
            i == j ? 0.0 : J.w[lo * (2 * N - lo - 1) / 2 + (hi - lo - 1)];
    }
    // Mirror tile: tile bits 0..nb-2 = qubits 0..nb-2, bit nb-1 = qubit N-1,
    // the rank's bits from qubit nb-1.  Strided tile: tile bits l..nb-1 =
    // qubits nb-1..N-2, the rank's bits from qubit l.
    const int h = nb - 1, lowm = (1 << h) - 1, top = nb - kSmallBits;
    mid_cuts(R, ws, tw, te, cA, N, rank << h, [&](int j) { return j < h ? j : N - 1; });
    mid_cuts(R, ws, tw, te, cB, N, rank << l, [&](int j) { return j < l ? j : j + h - l; });
    if (J.keep) R.tables(0, P);
    __syncthreads();
    const int M = (1 << (N - 1)) - 1;
    // Storage index of a tile's index i.
    auto index = [&](bool strided, int i) {
        if (strided) return (i & ((1 << l) - 1)) | (rank << l) | ((i >> l) << h);
        const int x = (rank << h) | (i & lowm);
        return i >> h ? M - x : x;
    };
    // The barrier counts up without a reset, so that a captured launch can be
    // replayed: every launch finds and leaves a multiple of kMidMaxCtas, and
    // fewer than that many CTAs can have arrived before this one has.
    unsigned target = 0;
    if (tid == 0) target = *(volatile unsigned*)a.counter & ~(unsigned)(kMidMaxCtas - 1);
    // The tile (in the top layout) for this CTA's tile of the other kind.
    auto change = [&](bool strided, bool dual) -> bool {
#pragma unroll
        for (int r = 0; r < kSmallRegs; r++) {
            const int x = index(!strided, tid | (r << top));
            __stcg(J.state + x, R.v[r]);
            if constexpr (GRAD)
                if (dual) __stcg(a.lam + x, R.w[r]);
        }
        if (!mid_barrier(a, target += grid)) return false;
#pragma unroll
        for (int r = 0; r < kSmallRegs; r++) {
            const int x = index(strided, tid | (r << top));
            R.v[r] = __ldcg(J.state + x);
            if constexpr (GRAD)
                if (dual) R.w[r] = __ldcg(a.lam + x);
        }
        return true;
    };
    // Pass s: the rest of layer s-1's mixer on this tile, then (s < P) layer
    // s's phase and its mixer's first part; odd passes on the strided tile.
    R.fill(cA, R.lay(nA - 1), 0);
    R.phase(cA, R.lay(nA - 1), true);
    R.template rounds<false>(nA, 0, false, false, false, J.lay[1], 0.0);
#pragma unroll 1
    for (int s = 1; s <= P; s++) {
        const bool str = s & 1;
        const int n = str ? nB : nA, first = str ? l : 0;
        const double* const c = str ? cB : cA;
        if (!change(str, false)) return;
        R.template rounds<false>(n, first, true, false, false, J.lay[4 * s - 3], 0.0);
        if (s < P) {
            const SmallLay L = R.lay(n - 1);
            R.fill(c, L, s);
            R.phase(c, L, false);
            R.template rounds<false>(n, first, false, false, false, J.lay[4 * s + 1], 0.0);
        }
    }
    const bool strided = P & 1;
    const int end = strided ? nB - 1 : nA - 1;
    R.energy(strided ? cB : cA, R.lay(end));
    if (J.flags & SJ_STATE) {
        if (end) R.template exchange<false>(R.lay(end), R.lay(0), false, 0.0, 0.0);
        const int full = (1 << N) - 1;
#pragma unroll
        for (int r = 0; r < kSmallRegs; r++) {
            const int x = index(strided, tid | (r << top));
            const double2 v = small_turned(R.v[r], J.rot);
            J.state[x] = v;
            J.state[full - x] = v;
        }
    }
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
            if (!change(str, true)) return;
            R.template rounds<true>(n, first, true, false, false, -J.lay[4 * k + 1],
                                    J.lay[4 * k + 3]);
            const double gg = R.unphase(c, R.lay(n - 1), k);
            if (R.keep(k, gg)) {
                if (tid < 2 * kSumLayers && k + (tid >> 1) < P)  // 64 threads or more
                    a.partial[(2 * k + tid) * grid + rank] = R.row_sum(tid);
                __syncthreads();
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
    const int nv = GRAD ? 2 * P : 0;
    if (tid == 0) a.partial[nv * grid + rank] = R.row_sum(2 * kSumLayers);
    if (!mid_barrier(a, target += grid)) return;
    if (rank == 0 && tid == 0) {
        const unsigned pad = (0u - target) & (kMidMaxCtas - 1);
        if (pad) atomicAdd(a.counter, pad);
    }
    // Value v's partial sums, in a fixed order, on a warp of CTA v % grid.
    for (int i = rank; i <= nv; i += grid) {
        if ((i / grid) % (R.nt / 32) != tid >> 5) continue;
        double s = 0;
        for (int x = tid & 31; x < grid; x += 32) s += __ldcg(a.partial + i * grid + x);
        s = small_warp_sum(s);
        if ((tid & 31) == 0) {
            if (i == nv)
                J.out[0] = 2.0 * s;
            else
                J.out[1 + ((i & 1) ? P : 0) + (i >> 1)] = (i & 1) ? 2.0 * s : -2.0 * s;
        }
    }
}

}  // namespace fq
