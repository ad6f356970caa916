// fq_swap.cu -- qubit permutations in HBM: the block exchange that replaces
// swap_gate_conti's single-device path (src/swap.cu:104-202, kernel :76-102)
// and the general permutation of fq_permute_qubits.
//
// Exchanging bit blocks [o, o+k) and [i, i+k) of every index is, for each
// value of the other bits, a transpose of a 2^k x 2^k matrix of "elements"
// (runs of 2^o contiguous amplitudes) whose rows are 2^i apart.  The
// reference walks a host-built table of all (s1, s2) block-value pairs and
// swaps one 16-byte amplitude per thread, so one side of every access is
// strided.  Here each CTA owns a PAIR of 2^a x 2^a sub-tiles, (I, J) and its
// mirror (J, I) (I, J = high k-a bits of each block), loads both with rows
// of >= 2^(a + eb) contiguous amplitudes, and writes each one transposed
// into the other's place through a padded shared tile, so reads and writes
// are both row-contiguous.  Diagonal sub-tiles (I == J) transpose in place.
//
// Both kernels are bound by HBM.  A thread's offsets within a tile are the
// same for every tile: they are computed once, and a tile's loads (four per
// thread and sub-tile) all go out before the first is stored to shared
// memory.  On B200 at N=26 (copy: 328 us): permutation 331 us (1177 with one
// amplitude per thread and scattered writes), swap of 12-qubit blocks 353 us
// (439 with the index arithmetic and one load at a time in the tile loop),
// of 2-qubit blocks 379 us (478).
#include <math.h>
#include <string.h>

#include <algorithm>

#include "fq_ctx.h"
#include "fq_engine.h"

namespace fq {

struct SwapArgs {
    double2* sv;
    int N, o, i, k;
    int eb;      // element bits kept inside a tile row (<= o)
    int a;       // sub-tile bits taken from each block
    int m;       // bits [o+k, o+k+m) also kept inside a row (only when a == k)
    int nob;     // "other" bits: [eb,o), [o+k+m,i), [i+k,N)
    i64 npairs;  // sub-tile pairs (I <= J)
    i64 nitems;
};

// Amplitudes of a sub-tile at most, and of a permutation's tile.
constexpr int kSwapTile = 1024;
constexpr int kSwapThreads = 256;
constexpr int kSwapPer = kSwapTile / kSwapThreads;

__global__ void __launch_bounds__(kSwapThreads) k_swap_blocks(const SwapArgs S) {
    extern __shared__ __align__(16) double2 sm[];
    // A row holds the element bits e (eb), the out-block low bits x (a) and
    // the free bits f above the out block (m): 2^(eb+a+m) amplitudes,
    // contiguous when o <= 6 and a == k.
    const int rowlen = 1 << (S.a + S.eb + S.m);
    const int rows = 1 << S.a;
    const int stride = rowlen + 1;  // padding keeps the transposed read conflict-free
    const int tsize = rows * rowlen;
    double2* t0 = sm;
    double2* t1 = sm + rows * stride;
    const int n1 = S.o - S.eb, n2 = S.i - S.o - S.k - S.m;
    const int xeb = S.a + S.eb;  // bits of (e, x) in a row index
    // Load: row y of a sub-tile = in-block low bits y; a row holds the
    // out-block low bits x and the element bits e (contiguous when o <= 6,
    // runs of 2^eb = 64 amplitudes otherwise).  Element (x, y) of (I, J)
    // lands at (y, x) of (J, I), and vice versa: the same offset, read from
    // the transposed place of the tile.
    i64 off[kSwapPer];
    int in[kSwapPer], out[kSwapPer];
#pragma unroll
    for (int r = 0; r < kSwapPer; r++) {
        const int idx = threadIdx.x + r * kSwapThreads;
        const int y = idx >> (xeb + S.m), xe = idx & (rowlen - 1);
        const int f = xe >> xeb, x = (xe >> S.eb) & ((1 << S.a) - 1);
        const int e = xe & ((1 << S.eb) - 1);
        off[r] = e + ((i64)x << S.o) + ((i64)f << (S.o + S.k)) + ((i64)y << S.i);
        in[r] = y * stride + xe;
        out[r] = x * stride + (f << xeb) + (y << S.eb) + e;
    }
    for (i64 item = blockIdx.x; item < S.nitems; item += gridDim.x) {
        const i64 oi = item & ((1ll << S.nob) - 1);
        const i64 p = item >> S.nob;
        i64 J = (i64)((sqrt(8.0 * (double)p + 1.0) - 1.0) * 0.5);
        while (J * (J + 1) / 2 > p) J--;
        while ((J + 1) * (J + 2) / 2 <= p) J++;
        const i64 I = p - J * (J + 1) / 2;
        const i64 base = ((oi & ((1ll << n1) - 1)) << S.eb) |
                         (((oi >> n1) & ((1ll << n2) - 1)) << (S.o + S.k + S.m)) |
                         ((oi >> (n1 + n2)) << (S.i + S.k));
        double2* const pIJ = S.sv + (base | (I << (S.o + S.a)) | (J << (S.i + S.a)));
        double2* const pJI = S.sv + (base | (J << (S.o + S.a)) | (I << (S.i + S.a)));
        const bool diag = (I == J);
        double2 u[kSwapPer], v[kSwapPer];
#pragma unroll
        for (int r = 0; r < kSwapPer; r++)
            if ((int)threadIdx.x + r * kSwapThreads < tsize) {
                u[r] = __ldcs(pIJ + off[r]);
                if (!diag) v[r] = __ldcs(pJI + off[r]);
            }
#pragma unroll
        for (int r = 0; r < kSwapPer; r++)
            if ((int)threadIdx.x + r * kSwapThreads < tsize) {
                t0[in[r]] = u[r];
                if (!diag) t1[in[r]] = v[r];
            }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kSwapPer; r++)
            if ((int)threadIdx.x + r * kSwapThreads < tsize) {
                __stcs(pJI + off[r], t0[out[r]]);
                if (!diag) __stcs(pIJ + off[r], t1[out[r]]);
            }
        __syncthreads();
    }
}

// dst[y] = src[x], bit perm[b] of y = bit b of x, as tiles of 2^t amplitudes
// whose t index bits hold the lowest bits of both x and y: rows of 2^kPermRow
// contiguous amplitudes are read and written (a thread per amplitude writing
// single 16-byte words took 3.6 times the copy's time).
constexpr int kPermRow = 5;
struct PermArgs {
    const double2* src;
    double2* dst;
    int N, t;
    i64 ntiles;
    int s[10];            // source bits of the tile, ascending
    int d[10];            // destination bits of the tile, ascending
    int q[10];            // source bit s[j] is the tile's destination bit q[j]
    int so[kMaxQubits];   // the other source bits, ascending, and where they go
    int to[kMaxQubits];
};

// Slot of tile index i: its 3-bit groups folded onto the lowest, so that
// eight lanes that differ in three bits of neighbouring (or any, modulo 3)
// positions fall in distinct banks.
__device__ __forceinline__ int perm_slot(int i) { return i ^ ((i >> 3 ^ i >> 6 ^ i >> 9) & 7); }

__global__ void __launch_bounds__(kSwapThreads) k_permute(const __grid_constant__ PermArgs A) {
    __shared__ __align__(16) double2 sm[kSwapTile];
    const int n = 1 << A.t;
    i64 from[kSwapPer], to[kSwapPer];
    int in[kSwapPer], out[kSwapPer];
#pragma unroll
    for (int r = 0; r < kSwapPer; r++) {
        const int i = threadIdx.x + r * kSwapThreads;
        from[r] = to[r] = 0;
        int m = 0;
        for (int j = 0; j < A.t; j++) {
            from[r] |= (i64)((i >> j) & 1) << A.s[j];
            to[r] |= (i64)((i >> j) & 1) << A.d[j];
            m |= ((i >> j) & 1) << A.q[j];
        }
        in[r] = perm_slot(m & (kSwapTile - 1));
        out[r] = perm_slot(i);
    }
    for (i64 T = blockIdx.x; T < A.ntiles; T += gridDim.x) {
        i64 bs = 0, bd = 0;
        for (int b = 0; b < A.N - A.t; b++) {
            bs |= ((T >> b) & 1) << A.so[b];
            bd |= ((T >> b) & 1) << A.to[b];
        }
        double2 u[kSwapPer];
#pragma unroll
        for (int r = 0; r < kSwapPer; r++)
            if ((int)threadIdx.x + r * kSwapThreads < n) u[r] = __ldcs(A.src + bs + from[r]);
#pragma unroll
        for (int r = 0; r < kSwapPer; r++)
            if ((int)threadIdx.x + r * kSwapThreads < n) sm[in[r]] = u[r];
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kSwapPer; r++)
            if ((int)threadIdx.x + r * kSwapThreads < n) __stcs(A.dst + bd + to[r], sm[out[r]]);
        __syncthreads();
    }
}

}  // namespace fq

using namespace fq;

extern "C" int fq_swap_blocks(fq_ctx* ctx, void* sv, int N, int swap_out, int swap_in,
                              int num_swap) {
    FQ_TRY(validate_ctx(ctx));
    FQ_CHECK(sv != nullptr && ((uintptr_t)sv & 15) == 0, FQ_ERR_INVALID, "bad state pointer");
    FQ_CHECK(N >= 1 && N <= kMaxQubits, FQ_ERR_INVALID, "N=%d out of range", N);
    FQ_CHECK(num_swap >= 0 && swap_out >= 0 && swap_out + num_swap <= swap_in &&
                 swap_in + num_swap <= N,
             FQ_ERR_INVALID,
             "block swap needs out + k <= in and in + k <= N (out=%d in=%d k=%d N=%d)", swap_out,
             swap_in, num_swap, N);
    if (num_swap == 0) return FQ_OK;
    SwapArgs S;
    S.sv = (double2*)sv;
    S.N = N;
    S.o = swap_out;
    S.i = swap_in;
    S.k = num_swap;
    S.eb = std::min(swap_out, 6);
    S.a = std::min(num_swap, std::max(0, (10 - S.eb) / 2));
    // A small block (the whole block in one sub-tile) leaves rows short;
    // the free bits right above the out block fill them up to 2^10
    // amplitudes per sub-tile (a swap of 2-qubit blocks at bit 0 took 7.9 ms
    // at N=26 with 4-amplitude rows).
    S.m = S.a == num_swap ? std::max(0, std::min(swap_in - swap_out - num_swap,
                                                  10 - 2 * S.a - S.eb))
                          : 0;
    S.nob = (swap_out - S.eb) + (swap_in - swap_out - num_swap - S.m) +
            (N - swap_in - num_swap);
    const i64 M = 1ll << (num_swap - S.a);
    S.npairs = M * (M + 1) / 2;
    S.nitems = S.npairs << S.nob;
    const size_t smem = sizeof(double2) * 2 * (1 << S.a) * ((1 << (S.a + S.eb + S.m)) + 1);
    const i64 grid = std::min<i64>(S.nitems, (i64)ctx->num_sms * 8);
    const int tok = prof_begin(ctx);
    k_swap_blocks<<<(unsigned)grid, kSwapThreads, smem, ctx->stream>>>(S);
    FQ_CUDA(cudaGetLastError());
    // Amplitudes whose two blocks hold equal values stay put.
    prof_end(ctx, tok, FQ_KIND_SWAP, 32.0 * (double)(1ull << N) * (1.0 - 1.0 / (1ull << num_swap)));
    ctx->launches++;
    return FQ_OK;
}

extern "C" int fq_permute_qubits(fq_ctx* ctx, const void* src, void* dst, int N,
                                 const int* perm) {
    FQ_TRY(validate_ctx(ctx));
    FQ_TRY(check_state((void*)src, N));
    FQ_TRY(check_state(dst, N));
    FQ_CHECK(src != dst, FQ_ERR_INVALID, "permutation must be out of place");
    FQ_CHECK(perm != nullptr, FQ_ERR_INVALID, "null permutation");
    PermArgs A;
    memset(&A, 0, sizeof(A));
    int inv[kMaxQubits];
    unsigned long long seen = 0;
    for (int b = 0; b < N; b++) {
        FQ_CHECK(perm[b] >= 0 && perm[b] < N && !((seen >> perm[b]) & 1ull), FQ_ERR_INVALID,
                 "perm is not a permutation of 0..N-1");
        seen |= 1ull << perm[b];
        inv[perm[b]] = b;
    }
    // The tile: the low bits of both sides, filled up with the next source bits.
    A.t = std::min(N, 10);
    unsigned long long tile = 0;
    for (int b = 0; b < std::min(N, kPermRow); b++) tile |= 1ull << b | 1ull << inv[b];
    for (int b = 0; b < N && __builtin_popcountll(tile) < A.t; b++) tile |= 1ull << b;
    unsigned long long dtile = 0;
    for (int b = 0; b < N; b++)
        if ((tile >> b) & 1) dtile |= 1ull << perm[b];
    int j = 0, o = 0, k = 0;
    for (int b = 0; b < N; b++) {
        if ((tile >> b) & 1) {
            A.s[j] = b;
            A.q[j++] = __builtin_popcountll(dtile & ((1ull << perm[b]) - 1));
        } else {
            A.so[o] = b;
            A.to[o++] = perm[b];
        }
        if ((dtile >> b) & 1) A.d[k++] = b;
    }
    A.src = (const double2*)src;
    A.dst = (double2*)dst;
    A.N = N;
    A.ntiles = 1ll << (N - A.t);
    const i64 grid = std::min<i64>(A.ntiles, (i64)ctx->num_sms * 8);
    const int tok = prof_begin(ctx);
    k_permute<<<(unsigned)grid, kSwapThreads, 0, ctx->stream>>>(A);
    FQ_CUDA(cudaGetLastError());
    prof_end(ctx, tok, FQ_KIND_OTHER, 32.0 * (double)(1ull << N));
    ctx->launches++;
    return FQ_OK;
}
