// fq_pass_col.cuh -- the fused two-layer pass over strided tiles as a
// pipeline of independent warps.
//
// k_pass's fused pass is bound by its load/store instructions and by moving
// in step: every warp copies its part of the next tile by 16-byte cp.async,
// reads it back, exchanges through shared memory twice under barriers of 256
// threads and stores each amplitude itself.  Here the TMA moves whole tiles,
// both ways, and a tile is split so that no warp needs another's data: a
// tile of rows of 2^l >= 8 amplitudes lands as 512 lines of 128 bytes, and
// warp c of a group of 8 takes chunk c (16 bytes) of every line.  The 128-byte
// swizzle of the landed tile puts those chunks in distinct banks, the warp's
// 512 amplitudes hold all of the tile's targets (tile bits 3..11), and its
// 512 chunks of the tile are its own buffer for its two layout changes.  Warps
// meet only at a stage's "landed" mbarrier and at its count of finished warps:
// the last of the eight stores the tile and loads the stage's next one.
//
// Two groups of 8 warps work on tiles 2U and 2U+1 (adjacent 128-byte rows,
// so DRAM sees 256-byte rows as with k_pass's paired CTAs); a ring of three
// stages lets one tile load or store while two are computed.
//
// Layouts, with i = tile bits 3..11 (the line): A: registers = i bits 5..8
// (tile bits 8..11), lane = i bits 0..4.  B: registers = i bits 1..4 (tile
// bits 4..7), lane = i bit 0, then bits 5..8.  Their thread and register bits
// are those of k_pass's L0 and L1, so the cut tables serve both kernels.
//
// Measured on B200 (A/B in one call, passes of a p=5 circuit): 4.27 against
// 4.47 ms at N=30 (8-amplitude rows), 0.91 against 1.00 at N=28 and 0.23
// against 0.24 at N=26 (16-amplitude rows).  What bounds it now: a group
// spends 12 k cycles on a tile (shared-memory data path 70% busy) and waits
// 4 k more for its next one; three 64 KB stages are all an SM holds.
#pragma once

#include "fq_pass_tma.cuh"

namespace fq {

constexpr int kColThreads = 2 * kPassThreads;  // two groups
constexpr int kColStages = 3;
// A landed barrier per stage and group (stages are odd, so tile j and tile
// j + 3 of a stage belong to different groups): tile j's is j % 6.  With one
// per stage a group two tiles ahead would wait for tile j + 3 while tile j is
// still landing, and the parity of that earlier phase would let it through.
constexpr int kColBars = 2 * kColStages;

// Shared memory behind the ring.  The phase needs five constants per thread
// and tile, z^g_k of its four register bits and phase(cbase).  g_k is a part
// f_k of the thread alone plus e_u of the tile: z^f_k is kept per thread
// (zf), z^e_u is the same for the whole warp, so four of the five lookups of
// the phase table are broadcasts, not gathers with bank conflicts (FP64
// weights: two sincos per thread and tile instead of five).
template <typename WT>
struct ColSmem {
    static constexpr size_t bar = (size_t)kColStages * kTileBytes;      // mbarriers, counts
    static constexpr size_t kp = bar + 128;                             // K, e_u of six tiles
    static constexpr size_t creg = kp + kColBars * kTcutStride * sizeof(WT);  // 16, layout L1
    static constexpr size_t cthr = creg + 16 * sizeof(WT);              // 256: the thread's cut
    static constexpr size_t qtab = cthr + kPassThreads * sizeof(WT);    // 16: z^creg[r]
    static constexpr size_t zf = qtab + 16 * sizeof(double2);           // 4 x 256
    static constexpr size_t smtab = zf + 4 * kPassThreads * sizeof(double2);
    static constexpr size_t bytes =
        smtab + (sizeof(WT) == sizeof(int) ? sizeof(double2) * (kPhaseLo + kPhaseHiMax) : 0);
    static_assert(kp % 16 == 0 && qtab % 16 == 0 && smtab % 16 == 0, "16-byte pieces");
    static_assert(bytes + 1024 <= 227 * 1024, "ring + tables fit one SM");
};
// 1 KB of slack aligns the ring.
template <typename WT>
__host__ __device__ constexpr size_t col_smem_bytes() {
    return 1024 + ColSmem<WT>::bytes;
}

__device__ __forceinline__ void tma_store_5d(const CUtensorMap* map, const void* src, int c0, int c1,
                                             int c2, int c3, int c4) {
    asm volatile(
        "cp.async.bulk.tensor.5d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4, %5, %6}], "
        "[%1];" ::"l"((unsigned long long)map),
        "r"(smem_addr(src)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4)
        : "memory");
}

// `bytes` (a multiple of 16) from global to shared memory, counted on bar.
__device__ __forceinline__ void bulk_load(void* dst, const void* src, unsigned bytes,
                                          unsigned long long* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, "
        "[%3];" ::"r"(smem_addr(dst)),
        "l"(src), "r"(bytes), "r"(smem_addr(bar))
        : "memory");
}

// Slots of a warp's amplitudes during a layout change: line i goes to line
// i ^ (i bits 5, 6 at bits 1, 2), which keeps eight lanes in distinct banks
// in both layouts.  A register's slot is one of four bases (by its two low
// bits) plus a constant.
struct ColSlots {
    int b[4];
};
__device__ __forceinline__ ColSlots col_slots_a(int lane, int c) {
    ColSlots s;
#pragma unroll
    for (int u = 0; u < 4; u++) {
        const int r = lane ^ (u << 1);
        s.b[u] = r * 8 + (c ^ (r & 7));
    }
    return s;
}
__device__ __forceinline__ ColSlots col_slots_b(int lane, int c) {
    ColSlots s;
    const int b0 = lane & 1, h = lane >> 1;
#pragma unroll
    for (int u = 0; u < 4; u++) {
        const int r = b0 | ((u ^ (h & 3)) << 1);
        s.b[u] = h * 256 + r * 8 + (c ^ r);
    }
    return s;
}
// Register r: layout A at b[r & 3] + 256 r, layout B at b[r & 3] + 64 (r >> 2).
template <bool FROM_A>
__device__ __forceinline__ int col_off(int r) {
    return FROM_A ? r * 256 : (r >> 2) * 64;
}

// Layout change A -> B or B -> A within a warp; lane_rx: preceded by RX on
// tile bit 3, lane bit 0 of both layouts, as in exchange_lanet (fq_pass.cuh).
template <bool FROM_A, int GM>
__device__ __forceinline__ void col_exchange(double2 (&v)[kRegs], double2* st, int lane, int c,
                                             bool lane_rx, double g) {
    int x = lane;
    asm volatile("" : "+r"(x));  // slots recomputed here, not held across the tile loop
    const ColSlots f = FROM_A ? col_slots_a(x, c) : col_slots_b(x, c);
    if (lane_rx) {
        const bool hi = x & 1;
#pragma unroll
        for (int r = 0; r < kRegs; r += 2) {
            const double2 keep = hi ? v[r | 1] : v[r], send = hi ? v[r] : v[r | 1];
            double2 q;
            q.x = __shfl_xor_sync(0xffffffffu, send.x, 1);
            q.y = __shfl_xor_sync(0xffffffffu, send.y, 1);
            v[r] = rx_self<GM>(keep, q, g, 0.0, 0.0);
            v[r | 1] = rx_self<GM>(q, keep, g, 0.0, 0.0);
        }
        __syncwarp();  // earlier reads of the warp's chunks are done
        const ColSlots p = FROM_A ? col_slots_a(x ^ 1, c) : col_slots_b(x ^ 1, c);
        // Registers r | hi of this lane and of its partner.
        const int d = hi ? col_off<FROM_A>(1) : 0;
        const int k0 = (hi ? f.b[1] : f.b[0]) + d, k2 = (hi ? f.b[3] : f.b[2]) + d;
        const int p0 = (hi ? p.b[1] : p.b[0]) + d, p2 = (hi ? p.b[3] : p.b[2]) + d;
#pragma unroll
        for (int r = 0; r < kRegs; r += 2) {
            st[(r & 2 ? k2 : k0) + col_off<FROM_A>(r)] = v[r];
            st[(r & 2 ? p2 : p0) + col_off<FROM_A>(r)] = v[r | 1];
        }
    } else {
        __syncwarp();
#pragma unroll
        for (int r = 0; r < kRegs; r++) st[f.b[r & 3] + col_off<FROM_A>(r)] = v[r];
    }
    __syncwarp();
    const ColSlots t = FROM_A ? col_slots_b(x, c) : col_slots_a(x, c);
#pragma unroll
    for (int r = 0; r < kRegs; r++) v[r] = st[t.b[r & 3] + col_off<!FROM_A>(r)];
}

// RX (GM, A.gx) on A.tmask, the next layer's phase, RX (GM2, A.gx2) on
// A.tmask: k_pass's fused pass for tiles of 8-amplitude or wider rows and
// targets among tile bits 3..11, with the tables of A.img, A.tcut.
template <typename WT, int GM, int GM2>
__global__ void __launch_bounds__(kColThreads, 1)
    k_pass_col(const PassArgs A, const __grid_constant__ CUtensorMap tmap, const TmaGeom G) {
    extern __shared__ unsigned char smraw[];
    unsigned char* sm = reinterpret_cast<unsigned char*>(
        (reinterpret_cast<uintptr_t>(smraw) + 1023) & ~(uintptr_t)1023);
    double2* const stage = reinterpret_cast<double2*>(sm);
    using SM = ColSmem<WT>;
    unsigned long long* const full = reinterpret_cast<unsigned long long*>(sm + SM::bar);
    int* const ndone = reinterpret_cast<int*>(full + kColBars);  // warps done with a stage
    volatile int* const last = ndone + kColStages;  // the last tile loaded on each barrier, -1: none
    volatile int* const gave_up = last + kColBars;
    WT* const kring = reinterpret_cast<WT*>(sm + SM::kp);
    WT* const creg = reinterpret_cast<WT*>(sm + SM::creg);
    WT* const cthr = reinterpret_cast<WT*>(sm + SM::cthr);
    double2* const qt = reinterpret_cast<double2*>(sm + SM::qtab);
    double2* const zf = reinterpret_cast<double2*>(sm + SM::zf);
    double2* const smtab = reinterpret_cast<double2*>(sm + SM::smtab);
    constexpr bool INTW = sizeof(WT) == sizeof(int);
    const int l = A.l, a = A.a, nmid = a - l;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nunits = (int)(A.ntiles / 2);
    // Tile j of this CTA: 2U + (j & 1) of unit U = blockIdx.x + (j >> 1) grid.
    const int count = 2 * ((nunits - 1 - (int)blockIdx.x) / (int)gridDim.x + 1);
    auto tile_of = [&](int j) {
        return 2 * ((int)blockIdx.x + (j >> 1) * (int)gridDim.x) + (j & 1);
    };

    if (threadIdx.x == 0) {
        for (int b = 0; b < kColBars; b++) {
            mbar_init(&full[b], 1);
            last[b] = -1;
        }
        *gave_up = 0;
        for (int s = 0; s < kColStages; s++) ndone[s] = 0;
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    // Layout B's constants from the geometry's image (PassSmem from creg on):
    // its thread (lane, c) is thread t1 of layout L1.
    {
        using PS = PassSmem<WT>;
        const unsigned char* const img = reinterpret_cast<const unsigned char*>(A.img);
        const WT* const icreg = reinterpret_cast<const WT*>(img) + 16;
        const WT* const ithr =
            reinterpret_cast<const WT*>(img + (PS::thrc - PS::creg)) + 5 * kPassThreads;
        const int t = threadIdx.x & (kPassThreads - 1), ln = t & 31;
        const int t1 = (t >> 5) | ((ln & 1) << 3) | ((ln >> 1) << 4);
        for (int k = threadIdx.x >> 8; k < 4; k += 2)
            zf[k * kPassThreads + t] =
                unit_power(A.gamma, (double)ithr[(1 + k) * kPassThreads + t1]);
        if (threadIdx.x < kPassThreads) cthr[t] = ithr[t1];
        if (threadIdx.x < 16) {
            creg[threadIdx.x] = icreg[threadIdx.x];
            qt[threadIdx.x] = unit_power(A.gamma, (double)icreg[threadIdx.x]);
        }
        if (INTW) load_phase_tables(A, smtab, threadIdx.x, kColThreads);
    }
    __syncthreads();
    auto load = [&](int j) {
        const int T = tile_of(j), s = j % kColStages;
        const int lo = T & ((1 << nmid) - 1), hi = T >> nmid;
        unsigned long long* const bar = &full[j % kColBars];
        constexpr unsigned kb = kTcutStride * sizeof(WT);
        last[j % kColBars] = j;
        mbar_expect_tx(bar, kTileBytes + kb);
        bulk_load(kring + (j % kColBars) * kTcutStride,
                  reinterpret_cast<const WT*>(A.tcut) + (i64)T * kTcutStride, kb, bar);
        if (G.kind == TG_ROWS)
            tma_load_5d(stage + (size_t)s * kTile, &tmap, bar, 0, 0, lo, 0, hi);
        else
            tma_load_5d(stage + (size_t)s * kTile, &tmap, bar, 0, lo, 0, 0, hi);
    };
    if (threadIdx.x == 0)
        for (int j = 0; j < kColStages && j < count; j++) load(j);

    // Group grp, chunk c of every line.
    const int grp = warp >> 3, c = warp & 7;
    const unsigned m_hi = (A.tmask >> 8) & 15u, m_mid = (A.tmask >> 4) & 15u;
    const bool lane_rx = (A.tmask >> 3) & 1u;
    const bool tree = INTW || A.tree != 0;
    const int own = lane * 8 + (c ^ (lane & 7));  // layout A as landed: own + 256 r
    for (int j = grp; j < count; j += 2) {
        const int T = tile_of(j), s = j % kColStages;
        double2* const st = stage + (size_t)s * kTile;
        if (!mbar_wait_polls(&full[j % kColBars], (unsigned)((j / kColBars) & 1), A.polls)) {
            if (lane == 0) {
                *(volatile int*)A.err = 1;
                *gave_up = 1;
            }
            break;
        }
        double2 v[kRegs];
#pragma unroll
        for (int r = 0; r < kRegs; r++) v[r] = st[own + 256 * r];
        rx_regs<GM>(v, m_hi, A.gx, 0.0, 0.0);
        col_exchange<true, GM>(v, st, lane, c, lane_rx, A.gx);
        rx_regs<GM>(v, m_mid, A.gx, 0.0, 0.0);
        {  // the next layer's phase
            const WT* const kp = kring + (j % kColBars) * kTcutStride;
            int x = lane;
            asm volatile("" : "+r"(x));
            const int t = (c << 5) | x;
            // cbase: the thread's tile bits are 0..2 (c), 3 (lane bit 0) and
            // 8..11 (lane bits 1..4); the registers' are 4..7.
            WT cb = kp[0] + cthr[t];
#pragma unroll
            for (int b = 0; b < 3; b++)
                if ((c >> b) & 1) cb += kp[1 + b];
#pragma unroll
            for (int b = 0; b < 5; b++)
                if ((x >> b) & 1) cb += kp[b == 0 ? 4 : 8 + b];
            if (tree) {
                const double2 P = phase_of<WT>(A, smtab, cb);
                double2 E[4];
                if constexpr (INTW) {
#pragma unroll
                    for (int k = 0; k < 4; k++)
                        E[k] = cmul(zf[k * kPassThreads + t], tab_pow(A, smtab, kp[5 + k]));
                } else {
                    const double2 u = zpow<WT>(A, smtab, kp[5 + (x & 3)]);
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const double2 uk = make_double2(__shfl_sync(0xffffffffu, u.x, k),
                                                        __shfl_sync(0xffffffffu, u.y, k));
                        E[k] = cmul(zf[k * kPassThreads + t], uk);
                    }
                }
                phase_tree<PH_MUL>(v, P, qt, E[0], E[1], E[2], E[3]);
            } else {  // the reference's own argument per amplitude
                const WT* const ithr =
                    reinterpret_cast<const WT*>(reinterpret_cast<const unsigned char*>(A.img) +
                                                (PassSmem<WT>::thrc - PassSmem<WT>::creg)) +
                    5 * kPassThreads + (c | ((x & 1) << 3) | ((x >> 1) << 4));
#pragma unroll
                for (int r = 0; r < kRegs; r++) {
                    WT cr = cb + creg[r];
#pragma unroll
                    for (int k = 0; k < 4; k++)
                        if ((r >> k) & 1) cr += ithr[(1 + k) * kPassThreads] + kp[5 + k];
                    const double S = 2.0 * (double)cr - A.W;
                    double sn, cs;
                    sincos(S * A.gamma / 2, &sn, &cs);
                    v[r] = cmul(v[r], make_double2(cs * A.scale, sn * A.scale));
                }
            }
        }
        rx_regs<GM2>(v, m_mid, A.gx2, 0.0, 0.0);
        col_exchange<false, GM2>(v, st, lane, c, lane_rx, A.gx2);
        rx_regs<GM2>(v, m_hi, A.gx2, 0.0, 0.0);
        __syncwarp();  // the warp has read its chunks
#pragma unroll
        for (int r = 0; r < kRegs; r++) st[own + 256 * r] = v[r];
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) {
            __threadfence_block();
            if (atomicAdd(&ndone[s], 1) == kPassThreads / 32 - 1) {  // the tile's last warp
                __threadfence_block();
                ndone[s] = 0;
                const int lo = T & ((1 << nmid) - 1), hi = T >> nmid;
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                if (G.kind == TG_ROWS)
                    tma_store_5d(&tmap, st, 0, 0, lo, 0, hi);
                else
                    tma_store_5d(&tmap, st, 0, lo, 0, 0, hi);
                asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                // Once the store has read the stage the next tile may land in it.
                asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                if (j + kColStages < count) load(j + kColStages);
            }
        }
        __syncwarp();
    }
    asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    // After a wait that gave up, copies may be in flight, and the other group
    // may have started more: once no warp starts any, wait (bounded) for all of
    // them, so that none lands in shared memory that is no longer this CTA's.
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned char* at = smraw;
        asm volatile("" : "+l"(at));  // the addresses are not held across the tile loop
        at = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(at) + 1023) &
                                              ~(uintptr_t)1023);
        unsigned long long* const bars = reinterpret_cast<unsigned long long*>(at + SM::bar);
        volatile int* const loaded = reinterpret_cast<int*>(bars + kColBars) + kColStages;
        if (loaded[kColBars])  // gave_up
            for (int b = 0; b < kColBars; b++)
                if (loaded[b] >= 0)
                    mbar_wait_bounded(&bars[b], (unsigned)((loaded[b] / kColBars) & 1));
    }
}

}  // namespace fq
