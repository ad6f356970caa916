// fq_engine.cu -- fused QAOA engine and the reference-path cost / RX entry
// points, all built on the streaming tile pass (fq_pass.cuh).
#include <math.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "fq_ctx.h"
#include "fq_engine.h"
#include "fq_launch.cuh"

namespace fq {

// ---------------------------------------------------------------- kernels --

// Phase of every integer cut value c in [cmin, cmin + n): scale *
// (cos, sin)(S * gamma / 2), S = 2c - W, the same double argument the
// reference forms from its exact integer sum (src/rzz.cu:146).
__global__ void k_phase_table(double2* tab, int cmin, int n, long long W, double gamma,
                              double scale) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        const double S = (double)(2ll * (cmin + i) - W);
        double sn, cs;
        sincos(S * gamma / 2, &sn, &cs);
        tab[i] = make_double2(cs * scale, sn * scale);
    }
}

// Two-level table of powers of z = exp(i*gamma) used by the engine's
// passes: tab[j] = z^j for j < 32, tab[32 + h] = z^(dlo + 32h).
__global__ void k_phase_table2(double2* tab, int dlo, int nhi, double gamma) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < kPhaseLo)
        tab[i] = unit_power(gamma, (double)i);
    else if (i < kPhaseLo + nhi)
        tab[i] = unit_power(gamma, (double)(dlo + 32ll * (i - kPhaseLo)));
}

// Tables of k_phase_table2 for up to kMaxTableLayers layers in one launch:
// layer p's table at tab + p * kTableStride.
// The last block of x takes z^creg[r] of every geometry from the images at
// img (WT per entry) instead; FP64 weights have nothing else (nhi = 0).
struct LayerGammas {
    double g[kMaxTableLayers];
};

template <typename WT>
__global__ void k_phase_tables2(double2* tab, int dlo, int nhi, LayerGammas lg, int P,
                                const unsigned char* img, int ngeom) {
    const int p = blockIdx.y;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= P) return;
    double2* t = tab + (size_t)p * kTableStride;
    if (blockIdx.x == gridDim.x - 1) {
        const int j = threadIdx.x;
        if (j >= ngeom * kQtabStride) return;
        const WT* creg = reinterpret_cast<const WT*>(img + (j / kQtabStride) * kImgStride);
        t[kPhaseLo + kPhaseHiMax + j] = unit_power(lg.g[p], (double)creg[j % kQtabStride]);
    } else if (i < kPhaseLo) {
        t[i] = unit_power(lg.g[p], (double)i);
    } else if (i < kPhaseLo + nhi) {
        t[i] = unit_power(lg.g[p], (double)(dlo + 32ll * (i - kPhaseLo)));
    }
}

// Deterministic sum of n partials into out[0]: fixed strided split and a
// fixed tree, so the same inputs always give the same bits.
__global__ void k_reduce_partials(const double* partial, int n, double* out) {
    __shared__ double sh[256];
    double s = 0;
    for (int i = threadIdx.x; i < n; i += 256) s += partial[i];
    sh[threadIdx.x] = s;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[0] = sh[0];
}

// Per-block max|a-b|^2, max|b|^2, sum|a-b|^2, sum|b|^2 over a grid-stride
// split (fixed per launch geometry, so the same inputs give the same bits).
__global__ void k_state_diff(const double2* a, const double2* b, u64 n, double* part) {
    __shared__ double sh[4][256];
    double m = 0, mb = 0, s = 0, sb = 0;
    for (u64 i = blockIdx.x * 256ull + threadIdx.x; i < n; i += (u64)gridDim.x * 256ull) {
        const double2 x = a[i], y = b[i];
        const double dx = x.x - y.x, dy = x.y - y.y;
        const double d2 = dx * dx + dy * dy, b2 = y.x * y.x + y.y * y.y;
        m = fmax(m, d2);
        mb = fmax(mb, b2);
        s += d2;
        sb += b2;
    }
    sh[0][threadIdx.x] = m;
    sh[1][threadIdx.x] = mb;
    sh[2][threadIdx.x] = s;
    sh[3][threadIdx.x] = sb;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) {
            sh[0][threadIdx.x] = fmax(sh[0][threadIdx.x], sh[0][threadIdx.x + o]);
            sh[1][threadIdx.x] = fmax(sh[1][threadIdx.x], sh[1][threadIdx.x + o]);
            sh[2][threadIdx.x] += sh[2][threadIdx.x + o];
            sh[3][threadIdx.x] += sh[3][threadIdx.x + o];
        }
        __syncthreads();
    }
    if (threadIdx.x < 4) part[4 * blockIdx.x + threadIdx.x] = sh[threadIdx.x][0];
}

// Small states (N < 12, at most 2048 amplitudes): one CTA, the reference's
// per-amplitude pair-order sum (src/rzz.cu:127-156) on a symmetric FP64
// weight matrix.
__global__ void k_cost_small(double2* sv, int N, double angle, const double* w, int first,
                             double amp) {
    for (int b = threadIdx.x; b < (1 << N); b += blockDim.x) {
        double sum = 0;
        for (int i = 0; i < N; i++)
            for (int j = i + 1; j < N; j++) {
                const double wij = w[i * N + j];
                if (wij != 0) sum += (((b >> i) ^ (b >> j)) & 1) ? wij : -wij;
            }
        double sn, cs;
        sincos(sum * angle / 2, &sn, &cs);
        if (first) {
            sv[b] = make_double2(cs * amp, sn * amp);
        } else {
            const double2 in = sv[b];
            sv[b] = make_double2(in.x * cs - in.y * sn, in.x * sn + in.y * cs);
        }
    }
}

struct Targets {
    int t[kMaxQubits];
};

// src/rx.cu:32-53 applied target by target over a small state (one CTA).
__global__ void k_rx_small(double2* sv, int N, Targets T, int nt, double c, double s) {
    for (int g = 0; g < nt; g++) {
        const int t = T.t[g];
        for (int k = threadIdx.x; k < (1 << (N - 1)); k += blockDim.x) {
            const int up = ((k >> t) << (t + 1)) | (k & ((1 << t) - 1));
            const int lo = up + (1 << t);
            const double2 q0 = sv[up], q1 = sv[lo];
            sv[up] = make_double2(q0.x * c + q1.y * s, q0.y * c - q1.x * s);
            sv[lo] = make_double2(q0.y * s + q1.x * c, -q0.x * s + q1.y * c);
        }
        __syncthreads();
    }
}

// <C> or the cut diagonal of a small state (one CTA).
__global__ void k_cut_small(const double2* sv, int N, const double* w, double* energy,
                            double* diag) {
    __shared__ double sh[256];
    double acc = 0;
    for (int b = threadIdx.x; b < (1 << N); b += blockDim.x) {
        double cz = 0;
        for (int i = 0; i < N; i++)
            for (int j = i + 1; j < N; j++)
                if (((b >> i) ^ (b >> j)) & 1) cz += w[i * N + j];
        if (diag) diag[b] = cz;
        if (energy) {
            const double2 v = sv[b];
            acc = fma(fma(v.x, v.x, v.y * v.y), cz, acc);
        }
    }
    if (energy) {
        sh[threadIdx.x] = acc;
        __syncthreads();
        for (int o = 128; o > 0; o >>= 1) {
            if ((int)threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
            __syncthreads();
        }
        if (threadIdx.x == 0) energy[0] = sh[0];
    }
}

// ------------------------------------------------------------- planning --


static int passes_for(int N, int lrows) {
    return 1 + (N - kTileBits + (kTileBits - lrows) - 1) / (kTileBits - lrows);
}

// Row bits of the strided passes: the widest rows (best DRAM locality) that
// still give the fewest passes.
static int choose_lrows(int N) {
    int best = 4;
    for (int lr = 4; lr >= 1; lr--)
        if (passes_for(N, lr) < passes_for(N, best)) best = lr;
    return best;
}

// One layer's passes: the contiguous tile 0..11 and strided tiles bringing
// the next 12 - lrows qubits on chip each (the last strided pass widens its
// rows when fewer qubits remain).  The first pass of a layer carries its
// cost phase (layer 0: the launch-control init), and the fused schedule
// runs the first and last passes of consecutive layers as one sweep, so
// with three or more passes the contiguous or mirror pass (four exchanges
// when fused, two alone) goes second and never fuses.  The strided passes
// over the highest qubits lead and the one over the lowest closes each layer.
// A half state's passes cover the same number of qubits: the mirror tile
// takes qubits 0..10 and N-1, the strided ones 11..N-2.
// Circuits on half states on B200, three runs in turn in one call, ms:
//                            N=28 p=3     N=30 p=4     N=30 p=5   N=32 p=3 (FP64)
//   this order                5.39-5.40    31.8-32.1    37.9-38.2    124-125
//   mirror pass first         5.92-5.93    33.5-34.0    42.7-43.0    160-161
//   lowest strided one first  5.47-5.49    31.0-31.8    38.7-39.1    132
std::vector<PassPlan> plan_layer(int N, bool half) {
    std::vector<PassPlan> v;
    if (half)
        v.push_back({kTileBits - 1, N - 1, (1u << kTileBits) - 1, 1});
    else
        v.push_back({kTileBits, kTileBits, (1u << kTileBits) - 1});
    const int lrows = choose_lrows(N);
    const int end = half ? N - 1 : N;
    for (int q = half ? kTileBits - 1 : kTileBits; q < end;) {
        const int k = std::min(kTileBits - lrows, end - q);
        const int l = kTileBits - k;
        v.push_back({l, q, ((1u << k) - 1) << l});
        q += k;
    }
    if (v.size() >= 3) {  // [last strided, contiguous, ..., first strided]
        std::swap(v[0], v[v.size() - 1]);
        std::swap(v[1], v[v.size() - 1]);
    }
    for (size_t i = 0; i < v.size(); i++) v[i].geom = (int)i;
    return v;
}

// Reduced RX: RX(beta) = f * G with G = [[1,-it],[-it,1]] (t = s/c, f = c)
// or [[u,-i],[-i,u]] (u = c/s, f = s), whichever keeps |t|,|u| <= 1.  The
// factor f of every gate in a layer is folded into that layer's phase.
void gate_params(double beta, int& gm, double& g, double& f) {
    const double s = sin(beta / 2), c = cos(beta / 2);
    if (fabs(c) >= fabs(s)) {
        gm = GM_TAN;
        g = s / c;
        f = c;
    } else {
        gm = GM_COT;
        g = c / s;
        f = s;
    }
}

// Tiles a pass prefetches ahead into L2 (FQ_PREFETCH overrides, 0 = off).
static int prefetch_distance() {
    static int d = -1;
    if (d < 0) {
        const char* e = getenv("FQ_PREFETCH");
        d = e ? std::max(0, std::min(4, atoi(e))) : 1;
    }
    return d;
}

PassArgs base_args(fq_ctx* ctx, void* sv, int N, const GraphPrep& g) {
    PassArgs A;
    memset(&A, 0, sizeof(A));
    A.sv = (double2*)sv;
    A.w = ctx->d_w;
    A.ptab = ctx->d_ptab;
    A.partial = ctx->d_partial;
    A.diag = nullptr;
    A.ntiles = 1ll << (N - kTileBits);
    A.N = N;
    A.l = kTileBits;
    A.a = kTileBits;
    A.tmask = 0;
    A.cmin = (int)g.cmin;
    A.ntab = g.integer ? (int)(g.cmax - g.cmin + 1) : 1;
    A.nhi = 0;
    A.W = g.integer ? (double)g.W_int : g.W;
    A.scale = 1.0;
    A.pf_dist = prefetch_distance();
    A.err = ctx->err;
    A.polls = ctx->polls < 0 ? kWaitSpins : std::min(ctx->polls, kWaitSpins);
    return A;
}

PassArgs engine_args(fq_ctx* ctx, void* sv, int N, const GraphPrep& g, const PassPlan& p) {
    PassArgs A = base_args(ctx, sv, N, g);
    A.ntiles >>= 1;  // a half state's
    A.l = p.l;
    A.a = p.a;
    A.tmask = p.tmask;
    A.mir = p.mir;
    A.img = ctx->d_img + p.geom * kImgStride;
    return A;
}

void set_layer_tables(fq_ctx* ctx, PassArgs& A, const PassPlan& p, int layer) {
    A.ptab = ctx->d_ptab + (size_t)layer * kTableStride;
    A.qt = A.ptab + kPhaseLo + kPhaseHiMax + p.geom * kQtabStride;
}

// Range [dlo, dhi] of the powers of z the passes look up: every cut value
// and every single-qubit flip change g (|g| <= gmax).
static void table_range(const GraphPrep& g, long long& dlo, long long& dhi) {
    dlo = std::min(g.cmin, -g.gmax);
    dhi = std::max(g.cmax, g.gmax);
}

// High-part entries of the engine's two-level table (0: the range is too
// wide for shared memory and the one-level global phase table is used).
int engine_nhi(const GraphPrep& g) {
    long long dlo, dhi;
    table_range(g, dlo, dhi);
    const long long nhi = (dhi - dlo + 1 + kPhaseLo - 1) / kPhaseLo;
    return nhi <= kPhaseHiMax ? (int)nhi : 0;
}

int launch_tables2(fq_ctx* ctx, const GraphPrep& g, const double* gammas, int P, int ngeom) {
    const int nhi = g.integer ? engine_nhi(g) : 0;
    if ((g.integer && nhi == 0) || P > kMaxTableLayers) return FQ_ERR_INVALID;
    long long dlo, dhi;
    table_range(g, dlo, dhi);
    LayerGammas lg;
    for (int p = 0; p < kMaxTableLayers; p++) lg.g[p] = p < P ? gammas[p] : 0.0;
    const int n = g.integer ? kPhaseLo + nhi : 0;
    const int tok = prof_begin(ctx);
    const dim3 grid((n + 255) / 256 + 1, P);
    if (g.integer)
        k_phase_tables2<int><<<grid, 256, 0, ctx->stream>>>(ctx->d_ptab, (int)dlo, nhi, lg, P,
                                                            ctx->d_img, ngeom);
    else
        k_phase_tables2<double><<<grid, 256, 0, ctx->stream>>>(ctx->d_ptab, 0, 0, lg, P,
                                                               ctx->d_img, ngeom);
    FQ_CUDA(cudaGetLastError());
    prof_end(ctx, tok, FQ_KIND_OTHER, 0.0);
    ctx->launches++;
    return FQ_OK;
}

int launch_table2(fq_ctx* ctx, const GraphPrep& g, double gamma) {
    const int nhi = engine_nhi(g);
    if (nhi == 0) return FQ_ERR_INVALID;
    long long dlo, dhi;
    table_range(g, dlo, dhi);
    const int n = kPhaseLo + nhi;
    const int tok = prof_begin(ctx);
    k_phase_table2<<<(n + 255) / 256, 256, 0, ctx->stream>>>(ctx->d_ptab, (int)dlo, nhi, gamma);
    FQ_CUDA(cudaGetLastError());
    prof_end(ctx, tok, FQ_KIND_OTHER, 0.0);
    ctx->launches++;
    return FQ_OK;
}

bool phase_tree_ok(const GraphPrep& g, double gamma) { return fabs(gamma) * g.wabs <= 512.0; }

void set_table_args(PassArgs& A, const GraphPrep& g, double gamma, double scale) {
    A.nhi = engine_nhi(g);
    if (A.nhi > 0) {
        long long dlo, dhi;
        table_range(g, dlo, dhi);
        A.dlo = (int)dlo;
        A.ntab = (int)(dhi - dlo + 1);
        // exp(-i*gamma*W/2), turned by the product's rounding error (unit_power).
        const double W = (double)g.W_int, x = gamma * W, lo = fma(gamma, W, -x) / 2;
        const double c = cos(x / 2), s = sin(x / 2), cl = cos(lo), sl = sin(lo);
        A.ph0x = scale * (c * cl - s * sl);
        A.ph0y = -scale * (s * cl + c * sl);
    }
}

int launch_table(fq_ctx* ctx, const GraphPrep& g, double gamma, double scale) {
    const int n = (int)(g.cmax - g.cmin + 1);
    k_phase_table<<<(n + 255) / 256, 256, 0, ctx->stream>>>(ctx->d_ptab, (int)g.cmin, n, g.W_int,
                                                             gamma, scale);
    FQ_CUDA(cudaGetLastError());
    ctx->launches++;
    return FQ_OK;
}

int read_result(fq_ctx* ctx, double* host) {
    FQ_CUDA(cudaStreamSynchronize(ctx->stream));
    FQ_TRY(check_device_error(ctx));
    *host = *(volatile double*)ctx->result;
    return FQ_OK;
}

int reduce_partials(fq_ctx* ctx, const double* partial, int n, double* out_dev) {
    const int tok = prof_begin(ctx);
    k_reduce_partials<<<1, 256, 0, ctx->stream>>>(partial, n, out_dev);
    FQ_CUDA(cudaGetLastError());
    prof_end(ctx, tok, FQ_KIND_OTHER, 0.0);
    ctx->launches++;
    return FQ_OK;
}

int reduce_to_result(fq_ctx* ctx, int n) {
    k_reduce_partials<<<1, 256, 0, ctx->stream>>>(ctx->d_partial, n, ctx->result);
    FQ_CUDA(cudaGetLastError());
    ctx->launches++;
    return FQ_OK;
}

int check_state(void* sv, int N) {
    FQ_CHECK(sv != nullptr, FQ_ERR_INVALID, "null state pointer");
    FQ_CHECK(((uintptr_t)sv & 15) == 0, FQ_ERR_INVALID, "state pointer not 16-byte aligned");
    FQ_CHECK(N >= 1 && N <= kMaxQubits, FQ_ERR_INVALID, "N=%d out of range [1,%d]", N, kMaxQubits);
    return FQ_OK;
}

// Prepare the graph; small states always use the FP64 weights.
int setup_graph(fq_ctx* ctx, const double* graph, int N, GraphPrep& g) {
    FQ_TRY(prep_graph(graph, N, g));
    if (N < kTileBits) g.integer = false;
    FQ_TRY(upload_graph(ctx, g, graph));
    return FQ_OK;
}

// The tables of a circuit's pass geometries that depend on the graph alone,
// built by one launch (k_tile_cuts) and kept while the weights and N stay
// the same (upload_graph; a new graph costs 11 to 20 us a call on B200, upload
// and launch): every tile's cut constants in ctx->d_tcut (grown on demand,
// tabs[i] serves plan[i]; null when it cannot be had, the passes then
// compute them per tile) and the static tables of each geometry in
// ctx->d_img.  The tile constants are 64 B per tile (128 B with FP64
// weights), 1/1024 of the swept state per geometry, and replace per-tile
// work on two warps and the barrier after it.  The images replace each
// CTA's own set-up from the weights, a chain of dependent shared-memory
// reads and sincos before its first tile, which at one tile per CTA was half
// of a pass.  On B200 (calls on one graph, A/B in one call): forward N=20 p=5 112 against 140 us
// with the set-up in every pass, N=23 p=4 (FP64 weights) 291 against 315 us;
// gradient N=19 p=6 215 against 279 us; N >= 26 within 1%.
static int tile_cut_tables(fq_ctx* ctx, const GraphPrep& g, int N,
                           const std::vector<PassPlan>& plan, std::vector<const void*>& tabs) {
    tabs.assign(plan.size(), nullptr);
    FQ_CHECK(plan.size() <= kMaxGeoms, FQ_ERR_INVALID, "%zu passes per layer", plan.size());
    const size_t wt = g.integer ? sizeof(int) : sizeof(double);
    const i64 ntiles = 1ll << (N - kTileBits - 1);  // a half state's
    const size_t per = (size_t)ntiles * kTcutStride * wt;
    const size_t need = per * plan.size();
    // Built for these weights (no upload since) and this N: reuse them, as
    // an optimiser's calls on one graph do.
    if (ctx->tcut_version == ctx->g_version && ctx->tcut_n == N) {
        for (size_t i = 0; i < plan.size() && need <= ctx->tcut_bytes; i++)
            tabs[i] = (char*)ctx->d_tcut + i * per;
        return FQ_OK;
    }
    ctx->tcut_version = -1;
    if (need > ctx->tcut_bytes) {
        if (ctx->d_tcut && ctx->captured) {
            ctx->retired.push_back(ctx->d_tcut);  // captured calls still use it
        } else if (ctx->d_tcut) {
            FQ_CUDA(cudaStreamSynchronize(ctx->stream));
            FQ_CUDA(cudaFree(ctx->d_tcut));
        }
        ctx->d_tcut = nullptr;
        ctx->tcut_bytes = 0;
        if (alloc_any_time(&ctx->d_tcut, need) == cudaSuccess)
            ctx->tcut_bytes = need;
        else
            ctx->d_tcut = nullptr;
    }
    const bool fits = need <= ctx->tcut_bytes;
    const i64 nt = fits ? ntiles : 0;
    // Eight blocks a SM at most; block 0 of each geometry also writes its image.
    const int grid = (int)std::max<i64>(1, std::min<i64>((nt + 3) / 4, (i64)ctx->num_sms * 8));
    // The attribute is the same for every N: contexts on other threads (the
    // server's lanes) set it concurrently, and a launch needing more than
    // another thread's smaller setting would fail.
    const size_t smem = g.integer ? tcut_smem_bytes<int>(N) : tcut_smem_bytes<double>(N);
    if (g.integer)
        FQ_CUDA(cudaFuncSetAttribute(k_tile_cuts<int>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)tcut_smem_bytes<int>(kMaxQubits)));
    else
        FQ_CUDA(cudaFuncSetAttribute(k_tile_cuts<double>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)tcut_smem_bytes<double>(kMaxQubits)));
    TcutGeoms G;
    memset(&G, 0, sizeof(G));
    for (size_t i = 0; i < plan.size(); i++) {
        G.l[i] = plan[i].l;
        G.a[i] = plan[i].a;
    }
    const dim3 grid2(grid, (unsigned)plan.size());
    if (g.integer)
        k_tile_cuts<int><<<grid2, kPassThreads, smem, ctx->stream>>>(
            (const int*)ctx->d_w, N, G, nt, (int*)ctx->d_tcut, ctx->d_img);
    else
        k_tile_cuts<double><<<grid2, kPassThreads, smem, ctx->stream>>>(
            (const double*)ctx->d_w, N, G, nt, (double*)ctx->d_tcut, ctx->d_img);
    FQ_CUDA(cudaGetLastError());
    ctx->launches++;
    ctx->tcut_version = ctx->g_version;
    ctx->tcut_n = N;
    for (size_t i = 0; i < plan.size() && fits; i++) tabs[i] = (char*)ctx->d_tcut + i * per;
    return FQ_OK;
}

bool fuse_enabled() {
    static int m = -1;
    if (m < 0) {
        const char* e = getenv("FQ_FUSE");
        m = e ? (atoi(e) != 0) : 1;
    }
    return m != 0;
}

// The fused forward circuit (see fq_qaoa_forward); with energy
// != NULL the last sweep also sums <C> and *energy receives it.

// The fused schedule: layer p visits its passes in plan order when p is even
// and in reverse order when p is odd, so the last pass of layer p and the
// first of layer p+1 have the same tile geometry and run as one fused pass
// (RX of layer p, phase of layer p+1, RX of layer p+1).  The phase still
// precedes every RX of its layer and follows every RX of the layer before:
// RX gates on different qubits commute.  Sweeps: npass + (P-1)(npass-1)
// instead of P * npass (11 instead of 15 at N=30, p=5).
//
// last_order: the circuit's last pass writes both halves of the state, 32 B
// per amplitude, and a strided pass with 128-byte rows writes them at two
// thirds of the rate the mirror pass does with its runs of 32 KB.  With three
// passes in a layer the last layer takes its mirror pass last and the strided
// one before it (both follow the first pass, which carries the phase):
// 38.9-39.2 against 39.3-39.5 ms per N=30 p=5 circuit on B200 (three pairs
// in one call), N=28 8.73-8.97 against 8.85-8.97, smaller ones within 1%.
static int last_order(int npass, int j) { return npass == 3 && j > 0 ? 3 - j : j; }

// Whether a pass of ntiles tiles is launched in a chain (0: no, 1: as its
// first pass, 2: after another pass; PassArgs::chained).  Passes of a few
// tiles per SM spend a good part of their time on launch, set-up and the last
// wave.  Whole calls with five layers, one by one against chained:
//   forward, integer weights   N=20 84.2 / 76.2 us, N=21 106 / 95.2, N=22 166 / 158
//   forward, FP64 weights      N=20 89.9 / 81.3 us, N=22 175 / 168, N=23 336 / 347
//   gradient, integer weights  N=20 188 / 175 us, N=21 289 / 275, N=23 984 / 1004
//   gradient, FP64 weights     N=21 298 / 290 us, N=22 546 / 548, N=23 1045 / 1075
// hence forward passes up to 4 tiles per SM (N = 22), adjoint passes, whose
// CTAs have an SM each, up to 2 (N = 21).  Kernels that are timed one by one
// (profiling), and those of a server's lanes, are launched one by one.
int chain_pass(const fq_ctx* ctx, i64 ntiles, int per_sm, bool first) {
    if (!ctx->chain || ctx->profiling || ntiles > (i64)per_sm * ctx->num_sms) return 0;
    return first ? 1 : 2;
}

static int engine_forward_fused(fq_ctx* ctx, void* sv, int N, int P, const GraphPrep& g,
                                const double* gammas, const double* betas, double* energy,
                                const std::vector<PassPlan>& plan,
                                const std::vector<const void*>& tcut, int& last_grid,
                                bool skip_last) {
    const double amp0 = fq_init_amp(N);
    const int npass = (int)plan.size();
    std::vector<int> gm(P);
    std::vector<double> gx(P), scale(P);
    for (int p = 0; p < P; p++) {
        double f;
        gate_params(betas[p], gm[p], gx[p], f);
        scale[p] = pow(f, N) * (p == 0 ? amp0 : 1.0);
    }
    const bool tables = P <= kMaxTableLayers;
    if (tables) FQ_TRY(launch_tables2(ctx, g, gammas, P, npass));
    // Phase arguments of layer q on a pass over plan[idx].
    auto phase_args = [&](PassArgs& A, int q, int idx) {
        if (g.integer) set_table_args(A, g, gammas[q], scale[q]);
        if (tables) set_layer_tables(ctx, A, plan[idx], q);
        A.tree = phase_tree_ok(g, gammas[q]) ? 1 : 0;
        A.gamma = gammas[q];
        A.scale = g.integer ? 1.0 : scale[q];
    };
    for (int p = 0; p < P; p++) {
        for (int j = (p == 0 ? 0 : 1); j < npass; j++) {
            if (skip_last && p == P - 1 && j == npass - 1) break;
            // The last layer ends on the mirror pass, see last_order.
            const int q = p == P - 1 && !skip_last ? last_order(npass, j) : j;
            const int idx = (p % 2 == 0) ? q : npass - 1 - q;
            PassArgs A = engine_args(ctx, sv, N, g, plan[idx]);
            A.tcut = tcut[idx];
            A.gx = gx[p];
            A.chained = chain_pass(ctx, A.ntiles, 4, p == 0 && j == 0);
            const bool last_of_layer = j == npass - 1;
            int ph = PH_NONE;
            if (p == 0 && j == 0) {  // launch-control init + layer-0 phase + RX
                phase_args(A, 0, idx);
                ph = PH_INIT;
                FQ_TRY(dispatch_phase_pass(ctx, g.integer, PH_INIT, gm[0], A));
            } else if (last_of_layer && p + 1 < P) {
                phase_args(A, p + 1, idx);
                A.gx2 = gx[p + 1];
                ph = PH_MUL;
                FQ_TRY(dispatch_fused(ctx, g.integer, gm[p], gm[p + 1], A));
            } else {
                A.full = p == P - 1 && last_of_layer;
                const bool ex = energy && A.full;
                FQ_TRY(dispatch_rx(ctx, g.integer, gm[p], ex, A));
            }
            last_grid = pass_grid(ctx, A, ph, true);
        }
    }
    return FQ_OK;
}

bool engine_fused(const GraphPrep& g, int P) {
    return fuse_enabled() && P >= 2 &&
           (!g.integer || (engine_nhi(g) > 0 && P <= kMaxTableLayers));
}

int engine_last_pass(const GraphPrep& g, int N, int P) {
    const int npass = (int)plan_layer(N, true).size();
    return (engine_fused(g, P) && (P - 1) % 2 == 1) ? 0 : npass - 1;
}

int engine_forward(fq_ctx* ctx, void* sv, int N, int P, const GraphPrep& g, const double* gammas,
                   const double* betas, double* energy, bool skip_last) {
    const double amp0 = fq_init_amp(N);
    const std::vector<PassPlan> plan = plan_layer(N, true);
    int last_grid = 0;
    const bool fused = engine_fused(g, P);
    FQ_CHECK(!(skip_last && energy), FQ_ERR_INVALID,
             "the forward circuit can stop before its last pass only without <C>");
    std::vector<const void*> tcut;
    FQ_TRY(tile_cut_tables(ctx, g, N, plan, tcut));
    if (fused)
        FQ_TRY(engine_forward_fused(ctx, sv, N, P, g, gammas, betas, energy, plan, tcut,
                                    last_grid, skip_last));
    for (int p = 0; p < (fused ? 0 : P); p++) {
        int gm;
        double gx, f;
        gate_params(betas[p], gm, gx, f);
        const double scale = pow(f, N) * (p == 0 ? amp0 : 1.0);
        const int nhi = g.integer ? engine_nhi(g) : 0;
        // Two-level tables: all layers' in one launch (layer p's at slot p,
        // kept for the reverse sweep of a gradient); else one global table
        // per layer.
        const bool all_tables = (nhi > 0 || !g.integer) && P <= kMaxTableLayers;
        if (all_tables && p == 0) FQ_TRY(launch_tables2(ctx, g, gammas, P, (int)plan.size()));
        if (g.integer && !all_tables) {
            if (nhi > 0) {
                FQ_TRY(launch_table2(ctx, g, gammas[p]));
            } else {
                FQ_TRY(launch_table(ctx, g, gammas[p], scale));
            }
        }
        for (size_t j = 0; j < plan.size(); j++) {
            if (skip_last && p == P - 1 && j + 1 == plan.size()) break;
            const size_t i =
                p == P - 1 && !skip_last ? last_order((int)plan.size(), (int)j) : (int)j;
            PassArgs A = engine_args(ctx, sv, N, g, plan[i]);
            A.full = p == P - 1 && j + 1 == plan.size();
            A.tcut = tcut[i];
            A.gx = gx;
            if (nhi > 0) set_table_args(A, g, gammas[p], scale);
            if (all_tables) set_layer_tables(ctx, A, plan[i], p);
            A.tree = phase_tree_ok(g, gammas[p]) ? 1 : 0;
            A.gamma = gammas[p];
            A.scale = g.integer ? 1.0 : scale;
            const int ph = i == 0 ? (p == 0 ? PH_INIT : PH_MUL) : PH_NONE;
            const int ex = energy && A.full ? 1 : 0;
            if (ph != PH_NONE)
                FQ_TRY(dispatch_phase_pass(ctx, g.integer, ph, gm, A));
            else
                FQ_TRY(dispatch_rx(ctx, g.integer, gm, ex != 0, A));
            last_grid = pass_grid(ctx, A, ph, true);
        }
    }
    if (energy) {
        FQ_TRY(reduce_to_result(ctx, last_grid));
        FQ_TRY(read_result(ctx, energy));
        *energy *= 2.0;  // the swept half's sum
    }
    return FQ_OK;
}

}  // namespace fq

using namespace fq;

extern "C" {

int fq_qaoa_forward(fq_ctx* ctx, void* sv, int N, int P, const double* graph,
                    const double* gammas, const double* betas, double* energy) {
    FQ_TRY(validate_ctx(ctx));
    FQ_TRY(check_state(sv, N));
    FQ_CHECK(N >= 2, FQ_ERR_INVALID, "N=%d: need at least 2 qubits", N);
    FQ_CHECK(P >= 1 && gammas && betas, FQ_ERR_INVALID, "need P >= 1 and angle arrays");
    for (int p = 0; p < P; p++)
        FQ_CHECK(isfinite(gammas[p]) && isfinite(betas[p]), FQ_ERR_INVALID,
                 "non-finite angle at layer %d", p);
    GraphPrep g;
    if (N <= kSmallJobMaxQubits) {
        FQ_TRY(prep_graph(graph, N, g));
        FQ_TRY(run_small(ctx, g, P, gammas, betas, SJ_STATE, (double2*)sv, ctx->result));
        return energy ? read_result(ctx, energy) : FQ_OK;
    }
    if (mid_ok(ctx, N, P)) {
        FQ_TRY(prep_graph(graph, N, g));
        FQ_TRY(run_mid(ctx, g, P, gammas, betas, SJ_STATE, (double2*)sv, nullptr, ctx->result));
        if (mid_ok(ctx, N, P)) return energy ? read_result(ctx, energy) : FQ_OK;
    }
    FQ_TRY(setup_graph(ctx, graph, N, g));
    return engine_forward(ctx, sv, N, P, g, gammas, betas, energy);
}

int fq_expectation(fq_ctx* ctx, const void* sv, int N, const double* graph, double* energy) {
    FQ_TRY(validate_ctx(ctx));
    FQ_TRY(check_state((void*)sv, N));
    FQ_CHECK(energy != nullptr, FQ_ERR_INVALID, "null energy pointer");
    GraphPrep g;
    FQ_TRY(setup_graph(ctx, graph, N, g));
    if (N < kTileBits) {
        k_cut_small<<<1, 256, 0, ctx->stream>>>((const double2*)sv, N, (const double*)ctx->d_w,
                                                ctx->result, nullptr);
        FQ_CUDA(cudaGetLastError());
        ctx->launches++;
        return read_result(ctx, energy);
    }
    PassArgs A = base_args(ctx, (void*)sv, N, g);
    FQ_TRY(dispatch_readonly(ctx, g.integer, false, A));
    FQ_TRY(reduce_to_result(ctx, pass_grid(ctx, A, PH_NONE, false)));
    return read_result(ctx, energy);
}

int fq_cut_diagonal(fq_ctx* ctx, void* out, int N, const double* graph) {
    FQ_TRY(validate_ctx(ctx));
    FQ_CHECK(out != nullptr && ((uintptr_t)out & 7) == 0, FQ_ERR_INVALID, "bad output pointer");
    FQ_CHECK(N >= 1 && N <= kMaxQubits, FQ_ERR_INVALID, "N=%d out of range", N);
    GraphPrep g;
    FQ_TRY(setup_graph(ctx, graph, N, g));
    if (N < kTileBits) {
        k_cut_small<<<1, 256, 0, ctx->stream>>>(nullptr, N, (const double*)ctx->d_w, nullptr,
                                                (double*)out);
        FQ_CUDA(cudaGetLastError());
        ctx->launches++;
        return FQ_OK;
    }
    PassArgs A = base_args(ctx, nullptr, N, g);
    A.diag = (double*)out;
    return dispatch_readonly(ctx, g.integer, true, A);
}

// src/rzz.cu:173-206.  Layer 0 writes phase * init_amp (launch control,
// src/rzz.cu:148-150); later layers multiply (src/rzz.cu:152-154).
int fq_cost_phase(fq_ctx* ctx, void* sv, int N, double angle, const double* graph,
                  int is_first_layer, double init_amp) {
    FQ_TRY(validate_ctx(ctx));
    FQ_TRY(check_state(sv, N));
    FQ_CHECK(isfinite(angle) && isfinite(init_amp), FQ_ERR_INVALID, "non-finite angle");
    GraphPrep g;
    FQ_TRY(setup_graph(ctx, graph, N, g));
    if (N < kTileBits) {
        k_cost_small<<<1, 1024, 0, ctx->stream>>>((double2*)sv, N, angle, (const double*)ctx->d_w,
                                                  is_first_layer ? 1 : 0, init_amp);
        FQ_CUDA(cudaGetLastError());
        ctx->launches++;
        return FQ_OK;
    }
    PassArgs A = base_args(ctx, sv, N, g);
    A.gamma = angle;
    A.scale = is_first_layer ? init_amp : 1.0;
    if (g.integer) {
        FQ_TRY(launch_table(ctx, g, angle, 1.0));
    }
    return dispatch_phase_pass(ctx, g.integer, is_first_layer ? PH_INIT : PH_MUL, GM_NONE, A);
}

}  // extern "C"

namespace fq {

// RX(angle) (full form, src/rx.cu:47-50) on every qubit of `mask`: qubits
// below 12 share the contiguous tile, higher ones are covered by strided
// tiles of up to 9 qubits.
int rx_mask(fq_ctx* ctx, void* sv, int N, unsigned long long mask, double angle) {
    const double s = sin(angle / 2), c = cos(angle / 2);  // src/rx.cu:121
    if (!mask) return FQ_OK;
    if (N < kTileBits) {
        Targets T;
        int nt = 0;
        for (int q = 0; q < N; q++)
            if ((mask >> q) & 1ull) T.t[nt++] = q;
        k_rx_small<<<1, 1024, 0, ctx->stream>>>((double2*)sv, N, T, nt, c, s);
        FQ_CUDA(cudaGetLastError());
        ctx->launches++;
        return FQ_OK;
    }
    GraphPrep g;  // RX passes read no cost data
    g.N = N;
    if (mask & 0xFFFull) {
        PassArgs A = base_args(ctx, sv, N, g);
        A.tmask = (unsigned)(mask & 0xFFFull);
        A.c = c;
        A.s = s;
        FQ_TRY(dispatch_rx_full(ctx, A));
    }
    // Targets above bit 11: strided tiles whose high bits are a window of
    // k qubits, in 9-qubit windows; a window spans only as many qubits as
    // its targets do (at least one), so few targets, such as the one or two
    // a sharded state swaps in per layer, leave the rows wide (2^(12-k)
    // contiguous amplitudes) and the pass streams at the copy rate.
    unsigned long long rest = mask & ~0xFFFull;
    const int kmax = std::min(kTileBits - 3, N - kTileBits);
    while (rest) {
        const int t0 = __builtin_ctzll(rest);
        int hi = t0;
        for (int t = t0; t < t0 + kmax && t < N; t++)
            if ((rest >> t) & 1ull) hi = t;
        const int k = hi - t0 + 1;
        const int a = std::min(t0, N - k);
        PassArgs A = base_args(ctx, sv, N, g);
        A.l = kTileBits - k;
        A.a = a;
        A.tmask = 0;
        for (int t = a; t < a + k; t++)
            if ((rest >> t) & 1ull) {
                A.tmask |= 1u << (A.l + t - a);
                rest &= ~(1ull << t);
            }
        A.c = c;
        A.s = s;
        FQ_TRY(dispatch_rx_full(ctx, A));
    }
    return FQ_OK;
}

}  // namespace fq

using namespace fq;

extern "C" {

// src/rx.cu:118-174: RX(angle) on every listed target of the chunk.
int fq_rx_chunk(fq_ctx* ctx, void* sv, int N, int chunk_qubits, const int* targets, int gate_size,
                double angle) {
    FQ_TRY(validate_ctx(ctx));
    FQ_TRY(check_state(sv, N));
    FQ_CHECK(isfinite(angle), FQ_ERR_INVALID, "non-finite angle");
    FQ_CHECK(chunk_qubits >= 1 && chunk_qubits <= 13 && chunk_qubits <= N, FQ_ERR_INVALID,
             "chunk_qubits=%d must be in [1, min(13, N)]", chunk_qubits);
    FQ_CHECK(gate_size >= 0 && gate_size <= chunk_qubits && (gate_size == 0 || targets),
             FQ_ERR_INVALID, "gate_size=%d must be in [0, chunk_qubits]", gate_size);
    unsigned long long seen = 0;
    for (int i = 0; i < gate_size; i++) {
        const int t = targets[i];
        FQ_CHECK(t >= 0 && t < chunk_qubits, FQ_ERR_INVALID,
                 "target %d outside the %d-qubit chunk", t, chunk_qubits);
        FQ_CHECK(!((seen >> t) & 1ull), FQ_ERR_INVALID, "target %d repeated", t);
        seen |= 1ull << t;
    }
    return rx_mask(ctx, sv, N, seen, angle);
}

int fq_rx_targets(fq_ctx* ctx, void* sv, int N, const int* targets, int n, double angle) {
    FQ_TRY(validate_ctx(ctx));
    FQ_TRY(check_state(sv, N));
    FQ_CHECK(isfinite(angle), FQ_ERR_INVALID, "non-finite angle");
    FQ_CHECK(n >= 0 && n <= N && (n == 0 || targets), FQ_ERR_INVALID, "bad target list");
    unsigned long long seen = 0;
    for (int i = 0; i < n; i++) {
        const int t = targets[i];
        FQ_CHECK(t >= 0 && t < N, FQ_ERR_INVALID, "target %d out of range", t);
        FQ_CHECK(!((seen >> t) & 1ull), FQ_ERR_INVALID, "target %d repeated", t);
        seen |= 1ull << t;
    }
    return rx_mask(ctx, sv, N, seen, angle);
}

int fq_state_diff(fq_ctx* ctx, const void* a, const void* b, int N, double* out) {
    FQ_TRY(validate_ctx(ctx));
    FQ_TRY(check_state((void*)a, N));
    FQ_TRY(check_state((void*)b, N));
    FQ_CHECK(out != nullptr, FQ_ERR_INVALID, "null output");
    const u64 n = 1ull << N;
    const int grid = (int)std::min<u64>((n + 255) / 256, (u64)ctx->partial_cap / 4);
    k_state_diff<<<grid, 256, 0, ctx->stream>>>((const double2*)a, (const double2*)b, n,
                                                ctx->d_partial);
    FQ_CUDA(cudaGetLastError());
    ctx->launches++;
    std::vector<double> part(4 * (size_t)grid);
    FQ_CUDA(cudaMemcpyAsync(part.data(), ctx->d_partial, sizeof(double) * part.size(),
                            cudaMemcpyDeviceToHost, ctx->stream));
    FQ_CUDA(cudaStreamSynchronize(ctx->stream));
    double m = 0, mb = 0, s = 0, sb = 0;
    for (int i = 0; i < grid; i++) {
        m = std::max(m, part[4 * i]);
        mb = std::max(mb, part[4 * i + 1]);
        s += part[4 * i + 2];
        sb += part[4 * i + 3];
    }
    out[0] = sqrt(m);
    out[1] = sqrt(mb);
    out[2] = sqrt(s);
    out[3] = sqrt(sb);
    return FQ_OK;
}

}  // extern "C"
