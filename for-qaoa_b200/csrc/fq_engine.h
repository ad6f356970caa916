// fq_engine.h -- host-side pieces of the fused engine shared by the forward
// circuit (fq_engine.cu) and the gradient (fq_grad.cu).
#pragma once

#include <vector>

#include "fq_ctx.h"
#include "fq_pass.cuh"
#include "fq_small.h"

namespace fq {

// One pass of a layer: tile bits 0..l-1 = physical 0..l-1, tile bits
// l..11 = physical a..a+11-l, RX on the tile bits of tmask; mir: the mirror
// pass of a half state (fq_pass.cuh).
struct PassPlan {
    int l, a;
    unsigned tmask;
    int mir = 0;
    int geom = 0;  // index in its plan: the place of its tables
};

// Passes of one layer for N >= 12: the contiguous tile over qubits 0..11
// and strided tiles over the remaining qubits (the first strided one leads
// when there are three or more passes); the first pass carries the phase.
// half: the passes of a half state, the mirror tile over qubits 0..10 and
// N-1 and strided tiles over qubits 11..N-2.
std::vector<PassPlan> plan_layer(int N, bool half = false);
// Pass arguments of plan entry p on a whole circuit's half state
// (fq_pass.cuh).  The passes are bound by on-chip work and HBM traffic per
// amplitude, and both halve.  On B200, against sweeping the whole state (A/B
// in one call): forward N=30 p=5 40.0 against 77.6 ms, N=28 p=3 with FP64
// weights 6.20 against 11.87 ms, N=23 p=4 0.315 against 0.493 ms; gradient
// N=26 p=10 15.5 against 30.7 ms.
PassArgs engine_args(fq_ctx* ctx, void* sv, int N, const GraphPrep& g, const PassPlan& p);
// Reduced RX for angle beta: gate mode, t or u, and the factor f.
void gate_params(double beta, int& gm, double& g, double& f);
PassArgs base_args(fq_ctx* ctx, void* sv, int N, const GraphPrep& g);
// High-part entries of the two-level phase table (0: use the global table).
int engine_nhi(const GraphPrep& g);
// Two-level table of powers of exp(i*gamma) in ctx->d_ptab (nhi > 0), and
// the pass arguments that read it (nhi, dlo, ntab, ph0 = scale*exp(-i*gamma*W/2)).
int launch_table2(fq_ctx* ctx, const GraphPrep& g, double gamma);
// The same for layers 0..P-1 (P <= kMaxTableLayers) in one launch, layer p's
// table at ctx->d_ptab + p * kTableStride.
// (FP64 weights: only z^creg[r] of the plan's ngeom geometries, which integer
// weights get too; the images of tile_cut_tables come first).
int launch_tables2(fq_ctx* ctx, const GraphPrep& g, const double* gammas, int P, int ngeom);
// Points A at layer `layer`'s tables as launch_tables2 left them.
void set_layer_tables(fq_ctx* ctx, PassArgs& A, const PassPlan& p, int layer);
void set_table_args(PassArgs& A, const GraphPrep& g, double gamma, double scale);
// FP64 weights: whether product-tree phases keep the phase arguments within
// the reference's own rounding (|gamma| * sum|w| small).  Above the bound
// each amplitude takes sincos of the reference's argument (2C - W)*gamma/2,
// which is exact for integer-valued weights.
bool phase_tree_ok(const GraphPrep& g, double gamma);
int launch_table(fq_ctx* ctx, const GraphPrep& g, double gamma, double scale);
// Whether the fused two-layer schedules run (the forward circuit's and the
// gradient's reverse sweep); FQ_FUSE=0 turns them off (one sweep per pass of
// every layer).
bool fuse_enabled();
// Fixed-order sum of n partials into one device word.
int reduce_partials(fq_ctx* ctx, const double* partial, int n, double* out_dev);
int reduce_to_result(fq_ctx* ctx, int n);
// Waits for the stream and reads ctx->result[0].
int read_result(fq_ctx* ctx, double* host);
int check_state(void* sv, int N);
// RX(angle) (full form) on every qubit whose bit is set in mask (fq_rx_targets).
int rx_mask(fq_ctx* ctx, void* sv, int N, unsigned long long mask, double angle);
int setup_graph(fq_ctx* ctx, const double* graph, int N, GraphPrep& g);
// The forward circuit (fq_qaoa_forward); skip_last stops before the last
// pass of the last layer (the gradient's turnaround pass runs it).
int engine_forward(fq_ctx* ctx, void* sv, int N, int P, const GraphPrep& g, const double* gammas,
                   const double* betas, double* energy, bool skip_last = false);
// Whether engine_forward uses the fused two-layer schedule, and the plan
// index of the last pass it runs.
bool engine_fused(const GraphPrep& g, int P);
int engine_last_pass(const GraphPrep& g, int N, int P);
int chain_pass(const fq_ctx* ctx, i64 ntiles, int per_sm, bool first);

// The gradient of more than kSmallJobMaxQubits qubits split for asynchronous
// use: grad_enqueue puts every kernel on ctx's stream, the last of which write
// the results to ctx->result (pinned); once the stream has passed that point,
// and without an error, grad_collect assembles them.
int grad_enqueue(fq_ctx* ctx, void* sv, void* costate, int N, int P, const double* graph,
                 const double* gammas, const double* betas);
int grad_collect(fq_ctx* ctx, int N, int P, double* energy, double* grad_gamma,
                 double* grad_beta);

// Small instances (fq_small.cuh, N <= kSmallJobMaxQubits).  small_job fills a
// descriptor (its pointers apart) and its small_words(N, P) data words: the
// weights, then the layers.
// cap: phase-table entries there is room for; most: entries of one layer's
// table that are worth computing.
void small_job(const GraphPrep& g, int P, const double* gammas, const double* betas, int flags,
               int cap, long long most, SmallJob& J, double* data);
// Enqueues one instance on ctx's stream; out (1 + 2P words with SJ_GRAD,
// else 1) and state (SJ_STATE) are device-accessible.
int run_small(fq_ctx* ctx, const GraphPrep& g, int P, const double* gammas, const double* betas,
              int flags, double2* state, double* out);
// run_small's launch of size class c >= 4, one instance or njobs descriptors on
// the device.
struct SmallArgs;
int launch_small_cluster(int c, bool grad, const SmallArgs* one, const SmallJob* jobs, int njobs,
                         cudaStream_t stream);
// One whole circuit or gradient (SJ_STATE or SJ_GRAD) of 16..19 qubits as a
// cooperative launch (fq_mid.cuh), where mid_ok says so; results as run_small's.
// Nothing was launched if mid_ok says otherwise afterwards (a stream with too
// few SMs).
bool mid_ok(const fq_ctx* ctx, int N, int P);
int run_mid(fq_ctx* ctx, const GraphPrep& g, int P, const double* gammas, const double* betas,
            int flags, double2* state, double2* lam, double* out);
// Gradients of njobs instances of size class c, descriptors on the device.
int launch_small_batch(const SmallJob* jobs, int njobs, int c, cudaStream_t stream);

}  // namespace fq
