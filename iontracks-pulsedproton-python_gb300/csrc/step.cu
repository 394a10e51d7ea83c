// step.cu -- the fused time step (deposition broadcast + Lax-Wendroff sweep +
// recombination sink + lateral wall + scored tallies) for one grid.
//
// One work item is consecutive k of one (i, j) column: eight for FP32 fields
// (pic_wide.cuh; four beyond 32-bit offsets), four for FP64. Every column of the output is written:
//   interior (1 <= i, j <= no_xy-2): the 7-point Lax-Wendroff update,
//     z-weights swapped for the negative species, minus alpha*dt*n+*n-;
//   outer ring, absorbing wall: the ring is carried with this step's
//     deposition added (the reference's deposit-then-carry, state.py:157-176);
//   outer ring, reflecting wall: the new value of the nearest interior column
//     (the reference's i-planes-then-j-planes mirror, state.py:151-154, which
//     maps corners to the diagonal interior column).
// The step's deposition is added to every value as it is read (gap layers
// only), the fused form of the reference's separate broadcast pass
// (solver_numba_parallel.py:222-277): each column reads one pair, its own
// G * density (added to its values) and the sum over its four lateral
// neighbours (added to the stencil's lateral sum). The z end planes
// k = 0 and k >= nzb-1 (and the row padding) are written as zero.
//
// Tallies over the scored set (interior, inside scoring_radius_sq, gap
// layers) follow _lax_wendroff_step_numba (solver_numba.py:204-211):
// recombined uses the pre-step densities, n+/n- the updated ones. The
// injected charge of the step is sum(G * density) over scored columns times
// no_z (solver_numba_parallel.py:271-276).
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "pic_device.cuh"
#include "pic_flat.cuh"
#include "pic_internal.h"
#include "pic_wide.cuh"

namespace pic {

// Whether the launch finishes its own tallies. It then lets the next one start
// only as it ends: that one's blocks, waiting on the SMs, slow the chain of its
// blocks and its last block's sum (float64 lone steps, us, started early / at the
// end: 24^2 x 206 18.3 / 14.7, 36^2 x 206 28.0 / 22.9; float32 59^2 x 406 10.1 / 9.7).
template <typename T>
__device__ __forceinline__ bool finishes(const StepArgs<T> &a) {
    return a.tally && a.counter;
}

// The end of a step: the tallies finished here, or (no counter) the block's
// partials left for the next step's block 0.
template <int BLOCK>
__device__ __forceinline__ void end_step(DF (&v)[4], const StepArgs<float> &a, unsigned block, unsigned blocks) {
    if (a.counter) finish_tally_df<BLOCK>(v, a.partials, a.counter, a.tally, a.injected_scale, block, blocks);
    else leave_partial<BLOCK>(v, a.partials + 4 * (int64_t)block);
}
template <int BLOCK>
__device__ __forceinline__ void end_step(double (&v)[4], const StepArgs<double> &a, unsigned block, unsigned blocks) {
    if (a.counter) finish_tally<BLOCK>(v, a.partials, a.counter, a.tally, a.injected_scale, block, blocks);
    else leave_partial<BLOCK>(v, a.partials + 4 * (int64_t)block);
}

// The blocks that step: all, or all but block 0, which sums the tallies of the
// step before (true: done, nothing to step).
template <typename T, int BLOCK>
__device__ __forceinline__ bool sums_prev(const StepArgs<T> &a, unsigned &block, unsigned &blocks) {
    block = blockIdx.x;
    blocks = gridDim.x;
    if (!a.prev_tally) return false;
    if (block == 0) {
        sum_partials<T, BLOCK>(a.prev_partials, a.prev_blocks, a.injected_scale, a.prev_tally);
        return true;
    }
    --block;
    --blocks;
    return false;
}

template <typename T, int BLOCK, typename I>
__global__ void __launch_bounds__(BLOCK) step_kernel(StepArgs<T> a) {
    wait_for_prev();
    unsigned block, blocks;
    if (sums_prev<T, BLOCK>(a, block, blocks)) return;
    Tally<T> t_rec, t_p, t_n, t_inj;
    const I stride = (I)blocks * BLOCK, items = (I)a.items;
    for (I item = (I)block * BLOCK + threadIdx.x; item < items; item += stride)
        flat_item<T, I>(a, item, t_rec, t_p, t_n, t_inj);
    if (!finishes(a)) let_next_start();
    if (!a.tally) return;  // no tallies wanted (a recomputation): no reduction
    if constexpr (sizeof(T) == 4) {
        DF v[4] = {df_of(t_inj), df_of(t_rec), df_of(t_p), df_of(t_n)};
        end_step<BLOCK>(v, a, block, blocks);
    } else {
        double v[4] = {t_inj.value(), t_rec.value(), t_p.value(), t_n.value()};
        end_step<BLOCK>(v, a, block, blocks);
    }
}

// The float32 step over eight-wide items (pic_wide.cuh).
constexpr int kWideBlock = 256, kWideBlocksPerSm = 2;
__global__ void __launch_bounds__(kWideBlock, kWideBlocksPerSm) wide_step_kernel(StepArgs<float> a) {
    wait_for_prev();
    unsigned block, blocks;
    if (sums_prev<float, kWideBlock>(a, block, blocks)) return;
    WideTally tl;
    wide_sweep(a, a.pos_in, a.neg_in, a.pos_out, a.neg_out, a.dens, a.dens_zero, block * kWideBlock + threadIdx.x,
               blocks * kWideBlock, tl);
    if (!finishes(a)) let_next_start();
    if (!a.tally) return;
    DF v[4];
    tl.store(v);
    end_step<kWideBlock>(v, a, block, blocks);
}

// How a flat step shares its tallies with its neighbours in a run: partials
// in buffer `slot`, left unsummed (leave), the step before to sum first
// (prev_tally, prev_blocks; its partials in the other buffer).
struct StepLink {
    int slot = 0;
    bool leave = false;
    double *prev_tally = nullptr;
    int prev_blocks = 0;
};

// Threads of a four-wide block. Float64 steps of a small grid are bound by the
// FP64 units, which an SM shares among its warps: small blocks spread the warps
// evenly (36^2 x 206: 264 blocks of 256 leave 40 of 152 SMs half the work of the
// rest). Measured with 90 tracks a step, us a step: 64 threads 19.7, 128 and 256
// 21.7, 32 23.8; 100^2 x 406 164 either way. A step that finishes its own tallies
// keeps blocks of 256: its last block reads every block's partials (60^2 x 206, lone
// steps: 49.4 us with 64 threads, 43.5 with 256).
template <typename T> constexpr int kFlatBlock = sizeof(T) == 8 ? 64 : 256;
constexpr int kFinishBlock = 256;

// Blocks of a flat step (wide: of the eight-wide form; finish: one that
// finishes its own tallies); in a run one block fewer than fit at once, so that
// the summing block runs beside them.
static int64_t flat_blocks(const pic_grid *g, bool wide, bool finish, bool run) {
    const bool small = g->dtype == PIC_F64 && !finish;
    const int64_t items = g->no_xy * g->no_xy * (g->kpitch / (wide ? 8 : 4)), block = wide ? kWideBlock : small ? kFlatBlock<double> : kFinishBlock;
    int64_t cap = wide ? (int64_t)kWideBlocksPerSm * sm_count() : step_grid_cap(g->dtype == PIC_F64 ? 1 : 0);
    if (g->dtype == PIC_F64 && finish) cap = std::max<int64_t>(1, cap * kFlatBlock<double> / kFinishBlock);
    return std::min({(items + block - 1) / block, std::max<int64_t>(1, cap - (run ? 1 : 0)), kMaxStepBlocks / 2});
}

template <typename T, int BLOCK>
static int launch_four_wide(const pic_grid *g, unsigned blocks, const StepArgs<T> &a, cudaStream_t st) {
    // (items + stride stays below 2^32 on the 32-bit path: items < 2^29; float32
    // grids come here beyond 32-bit offsets only)
    if constexpr (sizeof(T) == 8) {
        if (flat_index32(g->no_xy, g->kpitch)) {
            launch_linked(step_kernel<T, BLOCK, uint32_t>, blocks, BLOCK, st, a);
            return check_launch("step_kernel");
        }
    }
    launch_linked(step_kernel<T, BLOCK, int64_t>, blocks, BLOCK, st, a);
    return check_launch("step_kernel");
}

template <typename T>
static int launch_step_t(const pic_grid *g, const void *pos_in, const void *neg_in, void *pos_out, void *neg_out,
                         const void *dens, void *dens_zero, double *tally, void *ws, const StepLink *link, cudaStream_t st) {
    StepArgs<T> a;
    a.pos_in = (const T *)pos_in;
    a.neg_in = (const T *)neg_in;
    a.pos_out = (T *)pos_out;
    a.neg_out = (T *)neg_out;
    a.dens = (const pair_t<T> *)dens;
    a.dens_zero = (pair_t<T> *)dens_zero;
    a.tally = tally;
    Workspace w = workspace_layout(ws);
    a.partials = w.partials;
    a.counter = w.counter;
    a.n = g->no_xy;
    a.kp = g->kpitch;
    a.c4 = g->kpitch / 4;
    a.items = g->no_xy * g->no_xy * a.c4;
    a.dp = dens_pitch(g->no_xy);
    a.nzb = (int)g->nzb;
    a.nze = (int)g->nze;
    a.gap_end = (int)(g->nze + g->no_z);
    a.reflecting = g->wall == PIC_WALL_REFLECTING;
    a.p_lat = (T)g->p_lat; a.p_zm = (T)g->p_zm; a.p_zp = (T)g->p_zp;
    a.p_cen = centre_weight<T>(g->p_lat, g->p_zm, g->p_zp, g->p_cen);
    a.n_lat = (T)g->n_lat; a.n_zm = (T)g->n_zm; a.n_zp = (T)g->n_zp;
    a.n_cen = centre_weight<T>(g->n_lat, g->n_zm, g->n_zp, g->n_cen);
    a.alpha_dt = (T)g->alpha_dt;
    a.gfac = (T)g->gaussian_factor;
    int rc = score_test(g, &a.score);
    if (rc) return rc;
    a.injected_scale = (double)g->no_z;
    a.div_c4 = make_fastdiv(a.c4);
    a.div_n = make_fastdiv(a.n);
    const bool wide = sizeof(T) == 4 && wide_eligible(g->no_xy, g->kpitch, pos_in, neg_in, pos_out, neg_out);
    const bool finish = tally && !(link && link->leave);
    int64_t blocks = flat_blocks(g, wide, finish, link);
    a.prev_partials = nullptr;
    a.prev_tally = nullptr;
    a.prev_blocks = 0;
    if (link) {
        a.prev_tally = link->prev_tally;
        a.prev_blocks = link->prev_blocks;
        a.prev_partials = a.partials + 4 * (link->slot ^ 1) * (kMaxStepBlocks / 2);
        a.partials += 4 * link->slot * (kMaxStepBlocks / 2);
        if (link->leave) a.counter = nullptr;
        if (link->prev_tally) ++blocks;
    }
    if constexpr (sizeof(T) == 4) {
        if (wide) {
            launch_linked(wide_step_kernel, (unsigned)blocks, kWideBlock, st, a);
            return check_launch("wide_step_kernel");
        }
    }
    return finish ? launch_four_wide<T, kFinishBlock>(g, (unsigned)blocks, a, st)
                  : launch_four_wide<T, kFlatBlock<T>>(g, (unsigned)blocks, a, st);
}

static int launch_flat(const pic_grid *g, const void *pos_in, const void *neg_in, void *pos_out, void *neg_out,
                       const void *dens, void *dens_zero, double *tally, void *ws, const StepLink *link, cudaStream_t st) {
    if (g->dtype == PIC_F64)
        return launch_step_t<double>(g, pos_in, neg_in, pos_out, neg_out, dens, dens_zero, tally, ws, link, st);
    return launch_step_t<float>(g, pos_in, neg_in, pos_out, neg_out, dens, dens_zero, tally, ws, link, st);
}

int launch_step(const pic_grid *g_in, const void *pos_in, const void *neg_in, void *pos_out, void *neg_out,
                const void *dens, void *dens_zero, double *tally, void *ws, cudaStream_t st) {
    pic_grid r = *g_in;
    int rc = resolve_shape(&r);
    if (rc) return rc;
    const pic_grid *g = &r;
    if (g->variant == PIC_VARIANT_STREAM) {
        StreamShape sh{g->tile_rows, g->planes_per_item, g->stages, g->consumer_warps, g->ctas_per_sm, sm_count()};
        return launch_stream_step(g, sh, pos_in, neg_in, pos_out, neg_out, dens, dens_zero, tally, ws, st);
    }
    return launch_flat(g, pos_in, neg_in, pos_out, neg_out, dens, dens_zero, tally, ws, nullptr, st);
}

int StepRun::step(const void *pos_in, const void *neg_in, void *pos_out, void *neg_out, const void *dens,
                  void *dens_zero, double *tally) {
    if (rc_) return rc_;
    if (g_.variant == PIC_VARIANT_STREAM)
        return launch_step(&g_, pos_in, neg_in, pos_out, neg_out, dens, dens_zero, tally, ws_, st_);
    const bool wide = g_.dtype != PIC_F64 && wide_eligible(g_.no_xy, g_.kpitch, pos_in, neg_in, pos_out, neg_out);
    StepLink link;
    link.slot = (int)(left_ & 1);
    link.leave = --left_ > 0;
    link.prev_tally = prev_tally_;
    link.prev_blocks = prev_blocks_;
    prev_tally_ = link.leave ? tally : nullptr;
    prev_blocks_ = (int)flat_blocks(&g_, wide, !link.leave, true);
    return launch_flat(&g_, pos_in, neg_in, pos_out, neg_out, dens, dens_zero, tally, ws_, &link, st_);
}

int step_occupancy(int dtype, int *blocks_per_sm) {
    cudaError_t e = dtype == PIC_F64
                        ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, step_kernel<double, kFlatBlock<double>, uint32_t>, kFlatBlock<double>, 0)
                        : cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, step_kernel<float, 256, int64_t>, 256, 0);
    return e == cudaSuccess ? PIC_OK : set_cuda_error("cudaOccupancyMaxActiveBlocksPerMultiprocessor", e);
}

}  // namespace pic
