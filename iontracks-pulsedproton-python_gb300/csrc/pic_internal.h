// pic_internal.h -- host-side declarations shared by the translation units of
// libpic_gb300.so (not part of the public C ABI).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <string>

#include <nvtx3/nvToolsExt.h>

#include "../../include/pic_gb300.h"

namespace pic {

// Upper bound on the fused step's grid (blocks); sizes its tally workspace.
constexpr int64_t kMaxStepBlocks = 152 * 32;

struct Workspace {
    double *partials;       // [kMaxStepBlocks][4]
    unsigned int *counter;  // completion counter, zero between steps
    int *status;            // 0, or the code of a bounded wait that expired
};

inline Workspace workspace_layout(void *ws) {
    Workspace w;
    char *base = reinterpret_cast<char *>(ws);
    w.partials = reinterpret_cast<double *>(base);
    w.counter = reinterpret_cast<unsigned int *>(base + kMaxStepBlocks * 4 * sizeof(double));
    w.status = reinterpret_cast<int *>(base + kMaxStepBlocks * 4 * sizeof(double) + 128);
    return w;
}

// Largest CTA of the streaming step kernel: 16 consumer warps + 1 producer.
constexpr int kStreamMaxThreads = 17 * 32;
// Block-size bound of the streaming kernel instantiated for IPT items per
// consumer thread; a smaller bound leaves each thread more registers, so the
// IPT items of a plane can be unrolled without spilling.
__host__ __device__ constexpr int stream_max_threads(int ipt) {
    return ipt <= 1 ? 17 * 32 : (ipt == 2 ? 13 * 32 : (ipt == 3 ? 11 * 32 : 9 * 32));
}
// Wider instantiations for 2 to 4 items a thread allow up to 16 consumer
// warps: more warps per SM to hide latency, each thread held to fewer
// registers (65536 / the block rounded up to 128 threads). A launch takes the
// narrowest instantiation its threads fit.
constexpr int kStreamWide1 = 16 * 32, kStreamWide2 = 17 * 32;
__host__ __device__ constexpr int stream_thread_limit(int ipt) {
    return (ipt >= 2 && ipt <= 4) ? kStreamWide2 : stream_max_threads(ipt);
}
// items (k-vectors of a plane) per consumer thread: 1 .. kStreamMaxIpt
constexpr int kStreamMaxIpt = 6;
constexpr int kStreamMaxSmem = 227 * 1024;
// Division by an invariant divisor d >= 1 of dividends n < 2^31, by one
// multiply and shift (T. Granlund and P. Montgomery, "Division by invariant
// integers using multiplication", PLDI 1994): with l = ceil(log2 d) and
// m = ceil(2^(31+l) / d), n / d = (n * m) >> (31 + l) exactly (m < 2^33, so
// the product fits 64 bits).
struct FastDiv {
    uint64_t m;
    int sh;
};
__host__ __device__ inline FastDiv make_fastdiv(int64_t d) {
    int l = 0;
    while (((int64_t)1 << l) < d) ++l;
    const int sh = 31 + l;
    return FastDiv{(((uint64_t)1 << sh) + (uint64_t)d - 1) / (uint64_t)d, sh};
}
__host__ __device__ __forceinline__ uint32_t fast_div(uint32_t n, FastDiv f) {
    return (uint32_t)(((unsigned long long)n * f.m) >> f.sh);
}

// Warps per track of a deposition: a step's tracks alone rarely fill the GPU
// (a few to a few thousand per step), so with few tracks each box is shared by
// up to 8 warps.
__host__ __device__ inline int deposit_parts(int64_t m, int sms) {
    const int64_t warps = (int64_t)sms * 32;  // half the resident warps of the GPU
    int p = 8;
    while (p > 1 && m * p > warps) p >>= 1;
    return p;
}

// AUTO picks the streaming kernel from this many allocated cells (no_xy^2 * kpitch)
constexpr int64_t kStreamMinCells = 200000000;

// Launch shape of the streaming step kernel.
struct StreamShape {
    int tile_rows, planes_per_item, stages, consumer_warps, ctas_per_sm, sm_count;
};

int stream_smem_bytes(int tj, int kp, int stages);
int launch_stream_step(const pic_grid *g, const StreamShape &sh, const void *pos_in, const void *neg_in,
                       void *pos_out, void *neg_out, const void *dens, void *dens_zero, double *tally, void *ws,
                       cudaStream_t st);
// Fills the shape fields of *g (variant .. ctas_per_sm) where they are 0.
int resolve_shape(pic_grid *g);
constexpr int64_t kWorkspaceBytes = kMaxStepBlocks * 4 * (int64_t)sizeof(double) + 256;

// The scored-column test of the reference, (i - mid)^2 + (j - mid)^2 < r2
// with mid = no_xy / 2 (pulsed_ion_chamber/config.py:254-255), in exact
// integer form: with dx = 2 i - 2 mid and dy = 2 j - 2 mid (integers), the
// float64 comparison is exact (half-integer squares are exact) and equals
// dx^2 + dy^2 <= ceil(4 r2) - 1. Keeps float64 off the per-voxel path (the
// GPU's FP64 rate is ~1/64 of its FP32 rate).
struct ScoreTest {
    int64_t two_mid;
    int64_t thr4;
};
int score_test(const pic_grid *g, ScoreTest *out);
__host__ __device__ inline bool scored_column(const ScoreTest &t, int64_t i, int64_t j) {
    const int64_t dx = 2 * i - t.two_mid, dy = 2 * j - t.two_mid;
    return dx * dx + dy * dy <= t.thr4;
}

// Row pitch of the 2D density: no_xy rounded up to 4 elements, so every row
// starts 16-byte aligned and a row segment can be fetched by a bulk copy.
inline int64_t dens_pitch(int64_t no_xy) { return (no_xy + 3) / 4 * 4; }

// A named NVTX range over an entry point's host-side work (header-only NVTX:
// a no-op unless a profiler is attached), so that a kernel launch list taken
// with ncu --nvtx splits by phase: segments, graph replays, batched steps,
// gradient passes.
struct NvtxRange {
    explicit NvtxRange(const char *name) { nvtxRangePushA(name); }
    ~NvtxRange() { nvtxRangePop(); }
    NvtxRange(const NvtxRange &) = delete;
    NvtxRange &operator=(const NvtxRange &) = delete;
};

int set_error(int code, const std::string &msg);
int set_cuda_error(const char *what, cudaError_t e);
int check_launch(const char *what);

// Largest useful grid for the step kernel on the current device (SMs x
// resident blocks), cached per device.
int64_t step_grid_cap(int f64);
int sm_count();
int step_occupancy(int dtype, int *blocks_per_sm);

int launch_step(const pic_grid *g, const void *pos_in, const void *neg_in, void *pos_out, void *neg_out,
                const void *dens, void *dens_zero, double *tally, void *ws, cudaStream_t st);
// The `steps` steps of a segment of one grid, launched one by one on one
// stream. A flat step that finishes its own tallies ends in a chain of its blocks
// (store, fence, count, the last block's sum) that nothing runs beside: 2 to 4
// us. Here a step leaves its blocks' partials in the workspace (two buffers in
// turn) and the next step's block 0 sums them while the others step; the last
// one finishes its own, so a segment takes no launch more. Measured, us a step
// of a segment, finished in the step / by the next: 30^2 x 406 9.6 / 6.2, 61^2 x 606
// 14.4 / 10.3, 119^2 x 406 22.7 / 19.6, 208^2 x 406 57.0 / 53.3; float64 36^2 x 206
// 26.7 / 22.6. The streaming step finishes its own.
class StepRun {
public:
    StepRun(const pic_grid *g, void *ws, int64_t steps, cudaStream_t st) : g_(*g), ws_(ws), st_(st), left_(steps) {
        rc_ = resolve_shape(&g_);
    }
    int step(const void *pos_in, const void *neg_in, void *pos_out, void *neg_out, const void *dens, void *dens_zero,
             double *tally);

private:
    pic_grid g_;
    void *ws_;
    cudaStream_t st_;
    int64_t left_;  // steps not launched yet
    int rc_, prev_blocks_ = 0;
    double *prev_tally_ = nullptr;  // the step before's row, not summed yet
};

// The deposition of one step's m tracks into dens. ws / ws_bytes: the step
// workspace when the caller has one (null otherwise); its track lists, behind
// the fixed part, let the binned form run.
int launch_deposit(const pic_grid *g, const double *xs, const double *ys, int64_t m, void *dens,
                   uint32_t *counts, cudaStream_t st, void *ws = nullptr, int64_t ws_bytes = 0);

// Binned tile deposition (deposit.cu): a binning launch evaluates each
// track's Gaussian row and column factors once and lists the track in the
// tiles of kBinOut x kBinOut cells its written box meets; then one block per
// tile sums its tracks' outer products in a fixed order and stores each cell
// once. One pair of launches serves up to kBinSteps steps of a segment (their
// tracks together at most kBinTracks), each step a slot with its own track
// lists and its own pair buffer in the workspace. The scratch sits in the
// step workspace behind kWorkspaceBytes: a count per slot and tile (zero
// between launches; the tile's block clears it), kBinCap track indices per
// slot and tile (a tile with more scans its slot's tracks), the boxes and
// factors of kBinTracks tracks, and kBinSteps pair buffers.
constexpr int kBinOut = 62;
constexpr int kBinCap = 4096;
constexpr int kBinSteps = 8;
constexpr int kBinTracks = 65536;
constexpr int kBinBox = 64;               // factors kept per track and axis
constexpr int64_t kBinMaxNoXy = 4096;     // largest grid with track lists
// AUTO: the binned form for a segment's steps (up to eight per launch pair)
// where those launches give every SM a block (tiles x 8 >= SMs) or a tile
// meets about kBinAutoPerTile tracks of a step at most, so one block's serial
// sum stays short. Measured on GB300, per step against the per-track warps:
// 1068^2 with 8 500 tracks 20 against 64 us, 608^2 with 27 000 106 against
// 133, 208^2 with 300 6 against 11, 128^2 with 109 4.5 against 7.7, 48^2
// with 101 3.5 against 3.8 and with ~290 (~630 a tile) a 10 um column's
// whole run 18.3 against 22.1 ms; 108^2 with 632 (~350 a tile) 8.1 against
// 6.9; 48^2 with 1 011 (~2 200 a tile) 16 against 10.5. One step alone (the
// checkpointed gradient) only where the grid's tiles give at least
// kBinAutoTilesPerSm blocks per SM (no_xy >= 1055 on 152 SMs; 608^2 with
// 27 000 tracks 158 against 132 us, 208^2 20 against 11).
constexpr int kBinAutoTilesPerSm = 2;
constexpr int kBinAutoPerTile = 1024;
constexpr int kBinSpan = 256;  // steps one launch pair may span, idle steps between included
inline int64_t bin_tiles_per_side(int64_t n) { return (n + kBinOut - 1) / kBinOut; }
inline int64_t bin_align(int64_t b) { return (b + 255) / 256 * 256; }
inline int64_t bin_count_bytes(int64_t n) {
    const int64_t t = bin_tiles_per_side(n);
    return bin_align(kBinSteps * t * t * 4);
}
inline int64_t bin_list_bytes(int64_t n) {
    const int64_t t = bin_tiles_per_side(n);
    return kBinSteps * t * t * kBinCap * 4;
}
inline int64_t bin_box_bytes() { return bin_align((int64_t)kBinTracks * 8); }
inline int64_t bin_fac_bytes(int64_t es) { return (int64_t)kBinTracks * 2 * kBinBox * es; }
inline int64_t bin_dens_bytes(int64_t n, int64_t es) { return bin_align(n * dens_pitch(n) * 2 * es); }
// A grid takes the binned form when its track lists fit (no_xy <= 4096) and
// every truncation box, [ceil(c - cut), floor(c + cut)], spans at most
// kBinBox cells (floor(2 cut) + 1 of them at most).
inline bool bin_eligible(const pic_grid *g) {
    return g->no_xy <= kBinMaxNoXy && g->cutoff_voxels > 0.0 && 2.0 * g->cutoff_voxels + 1.0 < (double)kBinBox;
}
inline int64_t dep_bin_bytes(const pic_grid *g) {
    if (!bin_eligible(g)) return 0;
    const int64_t es = g->dtype == PIC_F64 ? 8 : 4;
    return bin_count_bytes(g->no_xy) + bin_list_bytes(g->no_xy) + bin_box_bytes() + bin_fac_bytes(es) +
           kBinSteps * bin_dens_bytes(g->no_xy, es);
}
// The binned deposition of a batched global step (batched.cu): its workspace
// (a slot per grid, per-tile counts and lists, per-track boxes and factors).
constexpr int kBinMaxSlots = 1024;
int64_t batched_deposit_bytes(int32_t n_cfgs, int32_t total_tiles, int64_t max_tracks, int64_t dens_bytes,
                              int32_t dtype);

// The resident step (resident.cu): how a float32 grid is divided over blocks
// that keep it on the chip for up to kResSteps steps of one launch. ti x tj
// columns and tkv k-vectors a block (nti x ntj x ntk of them), a patch of
// columns a thread (gi x gj patches, `threads` of them), `aux` threads beside
// the chain, `packets` a block publishes per step.
constexpr int kResSteps = 256;
constexpr int kResMinSteps = 4;  // shorter segments step by step (two launches a step)
constexpr int64_t kResMaxNoXy = 1024;
struct ResPlan {
    int patch, nti, ntj, ntk, ti, tj, tkv, gi, gj, blocks, threads, aux, smem, packets;
};
// The division of this grid; false when it does not fit the chip.
bool resident_plan(const pic_grid *g, ResPlan *out);
// `steps` steps from pos_in/neg_in. keep_stride 0: the last step's state into
// pos_out/neg_out (which may be the input for an even number of steps); > 0:
// step s's state at pos_out/neg_out + s * keep_stride. slot[s]: the pairs of
// step s at dens + slot[s] * dens_stride, -1: none. tally null: none wanted.
int launch_resident(const pic_grid *g, const ResPlan &p, const void *pos_in, const void *neg_in, void *pos_out,
                    void *neg_out, const void *dens, int64_t dens_stride, const int16_t *slot, int steps,
                    int64_t keep_stride, double *tally, void *packets, void *partials, int *status, cudaStream_t st);
// The division of this grid for the resident adjoint; false when it does not fit.
bool resident_adjoint_plan(const pic_grid *g, ResPlan *out);
// Adjoint steps steps - 1 .. 0 of a checkpoint segment: step 0 from the state
// pos0/neg0, step j > 0 from pos/neg + j * state_stride; lambda from lp_in/ln_in
// to lp_out/ln_out (the same buffers for an even number of steps only); the
// derivative sums join the blocks' slots (adjoint_accumulate_begin).
int launch_resident_adjoint(const pic_grid *g, const ResPlan &p, const void *pos0, const void *neg0, const void *pos,
                            const void *neg, int64_t state_stride, const void *dens, int64_t dens_stride,
                            const int16_t *slot, int steps, const void *lp_in, const void *ln_in, void *lp_out,
                            void *ln_out, double *slots, void *packets, int *status, cudaStream_t st);
// The resident step's part of the step workspace, behind the binned
// deposition's: the tile counts of kResSteps slots and the packets (one clear
// before a launch), the launch's tally partials and, where the binned
// deposition can run, the slots' track lists and pairs.
struct ResSpace {
    int64_t counts, packets, partials, lists, dens, end;  // byte offsets from the workspace's start
};
inline ResSpace resident_space(const pic_grid *g, const ResPlan &p) {
    ResPlan adj;
    int64_t packets = 2LL * p.blocks * p.packets * 16;
    if (resident_adjoint_plan(g, &adj)) packets = std::max<int64_t>(packets, 2LL * adj.blocks * adj.packets * 16);
    const int64_t tiles = bin_tiles_per_side(g->no_xy) * bin_tiles_per_side(g->no_xy);
    const bool bins = bin_eligible(g);
    ResSpace r;
    r.counts = kWorkspaceBytes + dep_bin_bytes(g);
    r.packets = r.counts + (bins ? bin_align(kResSteps * tiles * 4) : 0);
    r.partials = r.packets + bin_align(packets);
    r.lists = r.partials + bin_align((int64_t)kResSteps * p.blocks * p.aux);  // 32 bytes a warp
    r.dens = r.lists + (bins ? kResSteps * tiles * kBinCap * 4 : 0);
    r.end = r.dens + (bins ? kResSteps * bin_dens_bytes(g->no_xy, 4) : 0);
    return r;
}
// Whether the grid leaves the choice of kernels to the library.
inline bool resident_wanted(const pic_grid *g) {
    return g->variant == PIC_VARIANT_AUTO && g->steps_per_launch == 0 && g->deposit_variant != PIC_DEPOSIT_TRACKS;
}
// Whether a segment of these steps, in launches that end at every span-th,
// runs resident: the library's own choice of kernels (no variant, steps per
// launch or per-track deposition asked for), a workspace of
// pic_segment_workspace_bytes, and tracks the binned deposition takes and is no
// slower with. It deposits a launch's steps together, a block a step and tile, so
// it lasts as long as the tile with the most tracks: 80 to 110 ns a track; the
// per-track warps of the steps launched one by one take 5 us and 5 to 16 ns a
// track, one step after the other. So a tile's share is to be at most
// kBinAutoPerTile, as in the flat steps' groups, or, over the launches where it
// is more, a tenth of their tracks. Measured, us a step of 64, its deposition alone, binned / per track:
// 24^2 x 206 with 2000 tracks a step 6.6 / 31, 4000 23 / 66, 12000 141 / 139, 20000
// 383 / 206, 65000 3468 / 579; 18^2 x 56 with 4000 23 / 28, 8000 61 / 50, 20000 382
// / 109; four steps of 2000 tracks on 48^2 x 206 41 / 23.
bool resident_steps_eligible(const pic_grid *g, const void *ws, int64_t ws_bytes, const int64_t *off, int64_t n_steps,
                             int64_t span, ResPlan *plan);
// The end of the next resident launch's steps from s0 (at most kResSteps of
// them and kBinTracks tracks).
int64_t next_resident_group(const int64_t *off, int64_t s0, int64_t n_steps);
// Deposits and runs steps s0 .. s1 - 1 (a group of next_resident_group) from
// pos_in/neg_in into pos_out/neg_out. targets: where the pairs go, one slot of
// target_stride pairs per step with tracks (null: into the workspace).
// *last_pairs: the last step's pairs (null: no tracks).
int resident_steps(const pic_grid *g, const ResPlan &plan, const void *pos_in, const void *neg_in, void *pos_out,
                   void *neg_out, const double *xs, const double *ys, const int64_t *off, int64_t s0, int64_t s1,
                   uint32_t *counts, double *tally, void *targets, int64_t target_stride, const void **last_pairs,
                   void *ws, cudaStream_t st);
// The binned deposition of steps s0 .. s1 - 1 (up to kResSteps with tracks),
// a slot per step with tracks; slot[s - s0] receives step s's (-1: none). counts
// and lists: the slots' tile counts (zero) and lists, byte offsets in ws.
int launch_deposit_slots(const pic_grid *g, const double *xs, const double *ys, const int64_t *off, int64_t s0,
                         int64_t s1, uint32_t *hist, void *ws, int64_t counts, int64_t lists, void *dens,
                         int64_t dens_stride, int16_t *slot, cudaStream_t st);

// Clears the tile counts of the step workspace before a segment: another grid
// that shares it (a batch's grids that step alone) may have left its own lists
// where this one's counts are.
int clear_tile_counts(const pic_grid *g, void *ws, cudaStream_t st);
// Of a step's `most` tracks, those a tile of the binned form meets on average.
double bin_tile_tracks(const pic_grid *g, int64_t most);
// Whether the deposition takes the binned form for this grid and workspace:
// for a segment's steps together (most = the most tracks one of them has),
// or with most < 0 for one step alone.
bool deposit_binned(const pic_grid *g, const void *ws, int64_t ws_bytes, int64_t most);
// The end of the next launch pair's steps from s0: at most `slots` of them
// with tracks (*n_dep), kBinTracks tracks and kBinSpan steps.
int64_t next_deposit_group(const int64_t *off, int64_t s0, int64_t n_steps, int slots, int64_t *n_dep);
// The binned deposition of steps s0 .. s1 - 1 (tracks xs/ys[off[s] ..
// off[s + 1]), a group of next_deposit_group) into targets[k] for the k-th
// step with tracks, or with targets null into the workspace's pair buffers:
// dens[s - s0] is step s's pairs, or null for a step without tracks.
int launch_deposit_steps(const pic_grid *g, const double *xs, const double *ys, const int64_t *off, int64_t s0,
                         int64_t s1, uint32_t *counts, void *ws, void *const *targets, const void **dens,
                         cudaStream_t st);
// Kernel launches issued by this library so far (every launch site reports
// to check_launch; a captured graph's launches count at each replay).
void count_launches(int64_t n);

using BatchLaunch = pic_batch_launch;
int batched_workspace_bytes(int32_t n_blocks, int32_t n_cfgs, int64_t *bytes);
int batched_loop(const BatchLaunch &L, cudaStream_t st);
int batched_persistent(const BatchLaunch &L, const int64_t *step_task_off, const int64_t *step_tracks,
                       cudaStream_t st);
int batched_status(const BatchLaunch &L, cudaStream_t st, int32_t *status);
// The streaming batched step (batched_stream.cu).
int batched_stream_workspace_bytes(int32_t n_cfgs, int32_t n_items, int32_t consumer_warps, int64_t *bytes);
int batched_stream_prepare(const pic_batch_cfg *cfgs, int32_t n_cfgs, const int32_t *items, int32_t n_items,
                           const int32_t *tile_rows, int32_t consumer_warps, void *ws, int64_t ws_bytes,
                           cudaStream_t st, pic_batch_stream *out);
// dens: the step's deposition pairs in the packed layout; dens_zero: pairs the
// step clears for the next one (null: none)
int batched_stream_step(const BatchLaunch &L, const pic_batch_stream &B, int bi, int bo, int64_t step,
                        const void *dens, void *dens_zero, cudaStream_t st);
int batched_stream_status(const pic_batch_stream &B, int32_t reset, cudaStream_t st, int32_t *status);
// batched_loop with B non-null runs the streaming step instead of the flat one.
int batched_loop_stream(const BatchLaunch &L, const pic_batch_stream *B, cudaStream_t st);

// Several steps of one grid per cooperative launch (multistep.cu): for a
// resolved FLAT grid with steps_per_launch > 1.
constexpr int kMaxMultiSteps = 256;
bool multistep_eligible(const pic_grid *resolved);
int launch_multistep(const pic_grid *g, void *const pos[2], void *const neg[2], int parity, int n_steps,
                     const double *xs, const double *ys, const int64_t *off, void *const dens[2], int dens_parity,
                     uint32_t *counts, double *tally, void *ws, cudaStream_t st);

int step_noalloc(const pic_grid *g, const void *pos_in, const void *neg_in, void *pos_out, void *neg_out,
                 const double *xs, const double *ys, int64_t n_tracks, uint32_t *counts, double *tally,
                 cudaStream_t st);
int step_noalloc_status(int32_t reset, cudaStream_t st, int32_t *status);

int adjoint_workspace_bytes(int64_t *bytes);
int launch_adjoint(const pic_grid *g, const void *pos, const void *neg, const void *dens, void *lp_in, void *ln_in,
                   void *lp_out, void *ln_out, double *grad, void *ws, cudaStream_t st, bool accumulate = false);
int adjoint_accumulate_begin(const pic_grid *g, void *ws, cudaStream_t st);
// The streaming adjoint (adjoint_stream.cu): float32 grids with
// adjoint_variant STREAM, or AUTO and at least kAdjStreamMinCells cells: below,
// its items are too few to fill the SMs evenly and the eight-wide kernel is the
// faster one (330^2 x 406, 44 M cells: 221 us a step against 236), above, the
// plane ring saves neighbour traffic (608^2 x 406, 151 M: 728 against 718).
constexpr int64_t kAdjStreamMinCells = 100000000;
bool adjoint_stream_eligible(const pic_grid *g);
int launch_adjoint_stream(const pic_grid *g, const void *pos, const void *neg, const void *dens, const void *lp_in,
                          const void *ln_in, void *lp_out, void *ln_out, double *grad, unsigned int *counter,
                          int *status, double *partials, int64_t max_blocks, cudaStream_t st, bool accumulate);
double *adjoint_slots(void *ws);  // the blocks' running sums in the adjoint workspace
int adjoint_accumulate_end(const pic_grid *g, void *ws, double *grad, cudaStream_t st);

// Binomial checkpointing (revolve.cu).
int revolve_plan(int64_t n_steps, int64_t n_slots, int64_t *recompute_steps, int64_t *spine_levels);
int revolve_spine(int64_t n_steps, int64_t n_slots, int64_t *steps, int64_t cap, int64_t *n_levels);
int revolve_trace(int64_t n_steps, int64_t n_slots, int64_t *events, int64_t cap, int64_t *n_events,
                  int64_t *advanced);
int revolve_forward(const pic_grid *g, void *pos0, void *neg0, void *pos1, void *neg1, int64_t n_steps,
                    const double *xs, const double *ys, const int64_t *off, void *dens, uint32_t *counts,
                    double *tally, void *slots_pos, void *slots_neg, int64_t state_stride, int64_t n_slots, void *ws,
                    int64_t ws_bytes, cudaStream_t st);
int revolve_backward(const pic_grid *g, void *slots_pos, void *slots_neg, int64_t state_stride, int64_t n_slots,
                     int64_t n_steps, const double *xs, const double *ys, const int64_t *off, void *dens,
                     void *work_pos0, void *work_neg0, void *work_pos1, void *work_neg1, void *lam_pos0,
                     void *lam_neg0, void *lam_pos1, void *lam_neg1, double *grad, void *ws, int64_t ws_bytes,
                     void *adj_ws, cudaStream_t st);

int selftest_waits(int32_t *barrier_status, int32_t *mbarrier_status, cudaStream_t st);
int selftest_packets(const pic_grid *g, int32_t *step_status, int32_t *adjoint_status, int32_t *poisoned,
                     cudaStream_t st);

int sample_disc(const double *u, int64_t n_pairs, double scale, double mid, double radius_sq, int64_t n_wanted,
                double *xs, double *ys, int64_t *n_accepted, int64_t *n_pairs_used);
int arrival_counts_pcg64(uint64_t *st, int64_t n, double duration, const double *edges, int64_t n_edges,
                         int64_t *counts);
int sample_disc_pcg64(uint64_t *st, double scale, double mid, double radius_sq, int64_t n_wanted, int64_t max_pairs,
                      double *xs, double *ys, int64_t *n_accepted, int64_t *n_draws);

// Deposition further ahead than kBinSteps steps, for grids of few tiles whose
// eight steps leave most SMs without a block (a 36^2 grid: 8 blocks, one of them
// 59 us in float64): as many steps a launch pair as give kAheadBlocksPerSm blocks
// an SM, at most kResSteps, in slots of their own behind the step workspace. Only
// where the choice of deposition is the library's and the workspace is
// pic_segment_workspace_bytes large. slots = 0: not for this grid. Measured, us a
// step, eight steps a pair / ahead: float32 119^2 x 406 with 70 tracks 22.4 / 20.8,
// 208^2 x 406 with 300 57.5 / 55.9, with 1500 60.5 / 57.3, 330^2 x 206 with 500
// 70.4 / 69.4; a whole float64 run of 36^2 x 206 (2097 steps, 39 tracks each) 65.1
// / 50.7 ms.
constexpr int kAheadBlocksPerSm = 4;
struct AheadSpace {
    int64_t counts, lists, dens, end;  // byte offsets from the workspace's start
    int slots;
};
AheadSpace ahead_space(const pic_grid *g);

// The binned depositions of a segment, group by group.
class StepDeposits {
public:
    StepDeposits(const pic_grid *g, const double *xs, const double *ys, const int64_t *off, uint32_t *counts, void *ws,
                 int64_t ws_bytes, cudaStream_t st)
        : g_(g), xs_(xs), ys_(ys), off_(off), counts_(counts), ws_(ws), st_(st), space_(ahead_space(g)) {
        if (ws_bytes < space_.end) space_.slots = 0;
    }
    int begin();  // before the segment's first group
    // Deposits the next group's steps [s0, *s1), *n_dep of them with tracks:
    // the k-th of these into targets + k * target_bytes (targets null: into the
    // workspace); pairs[s - s0]: step s's pairs, null without tracks.
    int group(int64_t s0, int64_t n_steps, char *targets, int64_t target_bytes, int64_t *s1, int64_t *n_dep);
    const void *pairs[kBinSpan];

private:
    const pic_grid *g_;
    const double *xs_, *ys_;
    const int64_t *off_;
    uint32_t *counts_;
    void *ws_;
    cudaStream_t st_;
    AheadSpace space_;
};

}  // namespace pic
