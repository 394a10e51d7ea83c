// resident.cu -- up to kResSteps time steps of a small float32 grid in ONE
// cooperative launch whose blocks keep the fields on the chip.
//
// A grid of up to about 1.7 million cells has less state than the SMs have
// registers and shared memory, but launched step by step it is rewritten
// through L2 every step, and a step costs two chains of L2 round trips (its
// neighbour loads, its tally reduction) and a launch gap: 5-15 us whatever
// the arithmetic. Here every block owns a box of ti x tj interior columns and
// tkv k-vectors for the whole launch. A thread owns a patch of RI x RJ columns
// of one k-vector: both species' values stay in its registers from step to
// step, with a copy in shared memory that its neighbours in the block read.
// What a block needs of other blocks, one layer on each of its six faces,
// comes as tagged packets through L2 (pic_packet.cuh): the step's only
// communication, with no device-wide barrier and no fence.
//
// A step of a block:
//   its patch threads compute, neighbours from registers inside the patch and
//     from shared memory around it, and store the new values into shared
//     memory (a second copy of the cells, for small patches);
//   the same threads then send the block's face items, evenly shared out, and
//     poll for the neighbours' into the halo cells.
// That chain is what a step costs, so what can be is off it: one to four more
// warps fetch the deposition pairs a step ahead and sum the block's tallies of
// the step before. A packet buffer is written every other step: a block sends
// step s + 2's packets only after it took in its neighbours' of step s + 1,
// which they sent after taking in its packets of step s.
//
// The wall's ring columns live in the halo cells next to the wall: mirrored
// by the column beside them (reflecting) or carried with the step's deposition
// (absorbing). The pairs of all the launch's steps are formed before it
// (deposit.cu, a slot per depositing step). resident_tally_kernel sums the
// blocks' partials in block order afterwards. Every sum is in a fixed order:
// two runs of one grid give the same bits.
//
// What bounds it: the chain of a step -- about 1 us of it the packets' trip
// through L2, the rest the patches' arithmetic and shared memory at 65 cycles a
// warp's item -- not bandwidth. Measured on GB300, us a step of a 256-step
// launch without tracks, against the flat step's launches: 11^2 x 56 1.6 (6.2),
// 24^2 x 206 2.1 (8.3), 48^2 x 206 2.8 (8.3), 53^2 x 206 3.1 (10.3), 76^2 x 206
// 5.0 (12.4), 48^2 x 406 3.6 (10.3), 59^2 x 406 5.4 (12.4); with 14 tracks a step
// on 24^2 x 206, their deposition included, 2.4.
//
// The arithmetic is the streaming step's (pic_stream.cuh; the reference's
// _lax_wendroff_step_numba, solver_numba.py:130-213, and the walls of
// state.py:113-176), in packed FP32x2.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <type_traits>

#include "pic_resident.cuh"

namespace pic {

namespace {

struct ResArgs : ResShape {
    const float *pos_in, *neg_in;
    float *pos_out, *neg_out;
    const float2 *dens;   // pairs of slot q at dens + q * dens_stride
    int64_t dens_stride;
    float2 *partials;     // [steps][blocks][aux warps][4] double-floats
    int64_t keep_stride;  // > 0: every step's state is stored, step s's at out + s * keep_stride; 0: the last one's
    int dp, steps;
    float2 p_lat, p_zm, p_zp, p_cen, n_lat, n_zm, n_zp, n_cen, alpha_dt;  // each twice, for packed arithmetic
    ScoreTest score;
    int16_t slot[kResSteps];  // pair slot of each step, -1: no tracks
};

// a + b, exactly (Knuth's TwoSum, as in df_add).
__device__ __forceinline__ DF two_sum(float a, float b) {
    const float s = a + b, v = s - a;
    return DF{s, (a - (s - v)) + (b - v)};
}

// Adds an item's sum (a scored one's) to a thread's tally of a step, the first as it is.
__device__ __forceinline__ void tally_item(Tally<float> &t, float2 v, bool scored, bool first) {
    const float x = scored ? v.x + v.y : 0.f;
    if (first) t.s = x;
    else t.add(x);
}

// Shared memory: two buffers of deposition pairs over the block's columns (ring
// and halo included), the threads' tallies (of a patch of several items
// double-floats; two buffers where no barrier stands between the sum of a step's,
// at the next one's start, and that one's own), one or two buffers of the cells ([row][column][species][4 + 4 TKV] and 4 floats more, a row and a
// column more on each side), and the table of what the block trades.
__host__ __device__ inline int res_pair_floats(int cells) { return (4 * cells + 3) / 4 * 4; }
__host__ __device__ constexpr bool res_small(int ri, int rj) { return ri * rj < 6; }
__host__ __device__ constexpr int res_tally_values(int ri, int rj) { return ri * rj > 1 ? 2 : 1; }
__host__ __device__ inline int res_tally_buffers(bool small, int blocks) { return small && blocks == 1 ? 2 : 1; }
template <int RI, int RJ, int TKV, int MAXT, bool MIRROR>
__global__ void __launch_bounds__(MAXT, 1) resident_kernel(const __grid_constant__ ResArgs a) {
    // Small patches keep two buffers of cells, so that a step's values need not
    // wait until all of the block has read the step before's (one barrier a
    // step, not two); large ones have no room, nor registers for the row before.
    constexpr bool SMALL = res_small(RI, RJ);
    constexpr int PITCH = res_pitch(TKV), COL = 2 * PITCH;  // floats of a row of k, of a column (P, then N)
    extern __shared__ __align__(16) float res_smem[];
    __shared__ volatile int s_abort;
    const int tid = threadIdx.x, T = a.patch_threads, lane = tid & 31;
    const int W = a.gj * RJ + 2, ROW = W * COL;
    ResTile<PITCH> tile(a, W);
    const int cta = tile.cta, bk = tile.bk, i0 = tile.i0, j0 = tile.j0, kv0 = tile.kv0;
    const int rows = tile.rows, cols = tile.cols, kvn = tile.kvn, n_side = tile.n_side, n_around = tile.n_around;
    const bool lo_i = tile.lo_i, hi_i = tile.hi_i, lo_j = tile.lo_j, hi_j = tile.hi_j;
    const int n = a.n, kp = a.kp, tkv = a.tkv, steps = a.steps;
    const int ncell = res_cells(a.gi, a.gj, RI, RJ);
    float2 *pairs = reinterpret_cast<float2 *>(res_smem);  // [2][ncell]
    constexpr int VALUES = res_tally_values(RI, RJ);
    float *const sums = res_smem + res_pair_floats(ncell);  // [1 or 2][3][T][VALUES]
    const int SUMS = res_tally_buffers(SMALL, gridDim.x) == 2 ? 3 * VALUES * T : 0;  // from one buffer to the other
    float *S = sums + 3 * VALUES * T + SUMS;
    const int BUF = SMALL ? ncell * COL + 4 : 0;  // floats from one buffer of cells to the other
    const bool trades = gridDim.x > 1;  // cells with other blocks

    // ---- load: cells to zero, then the block's values and its surroundings ----
    if (tid == 0) s_abort = 0;
    for (int u = tid; u < (ncell * COL + 4) / 4 * (SMALL ? 2 : 1); u += blockDim.x) st4s(S + 4 * u, make_float4(0.f, 0.f, 0.f, 0.f));
    for (int u = tid; u < 3 * VALUES * T + SUMS; u += blockDim.x) sums[u] = 0.f;
    __syncthreads();
    for (int u = tid; u < n_around * kvn; u += blockDim.x) {
        const int col = u / kvn, v = u - col * kvn;
        int r, c;
        tile.around(col, r, c);
        if (col >= n_side && !tile.ring_col(col, r, c)) continue;  // nobody's neighbour
        const int64_t o = ((int64_t)(i0 + r) * n + (j0 + c)) * kp + 4 * (kv0 + v);
        float *d = S + tile.cell_of(r, c) + 4 * v;
        st4s(d, *reinterpret_cast<const float4 *>(a.pos_in + o));
        st4s(d + PITCH, *reinterpret_cast<const float4 *>(a.neg_in + o));
    }
    for (int u = tid; u < rows * cols; u += blockDim.x) {
        const int r = u / cols, c = u - r * cols;
        const int64_t o = ((int64_t)(i0 + r) * n + (j0 + c)) * kp + 4 * kv0;
        float *d = S + tile.cell_of(r, c);
        if (tile.lo_k) d[-1] = a.pos_in[o - 1], d[PITCH - 1] = a.neg_in[o - 1];
        if (tile.hi_k) d[4 * kvn] = a.pos_in[o + 4 * kvn], d[PITCH + 4 * kvn] = a.neg_in[o + 4 * kvn];
    }

    tile.table(reinterpret_cast<int4 *>(S + (SMALL ? 2 : 1) * (ncell * COL + 4)));

    if (tid >= T) {
        // ---------------- the warps beside the steps' chain ----------------
        const int AT = a.aux_threads, at = tid - T, aw = at >> 5;
        auto fetch_pairs = [&](int s) {  // step s's pairs of the block's columns, asynchronously
            const int sl = s < steps ? a.slot[s] : -1;
            if (sl < 0) return;
            const float2 *src = a.dens + sl * a.dens_stride + (int64_t)(i0 - 1) * a.dp + (j0 - 1);
            for (int u = at; u < (rows + 2) * (cols + 2); u += AT) {
                const int r = u / (cols + 2), c = u - r * (cols + 2);
                const uint32_t dst = (uint32_t)__cvta_generic_to_shared(pairs + (s & 1) * ncell + r * W + c);
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src + (int64_t)r * a.dp + c)
                             : "memory");
            }
        };
        DF inj{0.f, 0.f};
        auto sum_step = [&](int s) {  // this warp's share of the block's tallies of step s
            const float *q = sums + (s & 1) * SUMS;
            DF v[4] = {inj, {0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
            for (int u = 4 / VALUES * at; u < T; u += 4 / VALUES * AT)
#pragma unroll
                for (int x = 0; x < 3; ++x) {
                    const float4 f = ld4s(q + VALUES * (x * T + u));
                    v[x + 1] = df_add(v[x + 1], VALUES == 1 ? df_add(two_sum(f.x, f.y), two_sum(f.z, f.w))
                                                            : df_add(DF{f.x, f.y}, DF{f.z, f.w}));
                }
            const DF w = warp_sum4(v, lane);
            if ((lane & 7) == 0)
                a.partials[(((int64_t)s * gridDim.x + cta) * (AT >> 5) + aw) * 4 + (lane >> 3)] = make_float2(w.hi, w.lo);
        };
        fetch_pairs(0);
        for (int s = 0; s < steps; ++s) {
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();
            if (s_abort) return;
            if (s > 0) sum_step(s - 1);
            inj = DF{0.f, 0.f};
            if (a.slot[s] >= 0 && bk == 0) {
                const float2 *Dp = pairs + (s & 1) * ncell;
                for (int u = at; u < rows * cols; u += AT) {
                    const int r = u / cols, c = u - r * cols;
                    if (scored_col_t<uint32_t>(a.score, i0 + r, j0 + c))
                        inj = df_add(inj, DF{Dp[(r + 1) * W + c + 1].x, 0.f});
                }
            }
            fetch_pairs(s + 1);
            if (!SMALL) __syncthreads();
            if (trades) __syncthreads();
        }
        __syncthreads();
        sum_step(steps - 1);
        return;
    }

    // ---------------- the threads with patches ----------------
    const int q = tid / tkv, kv = tid - q * tkv;
    const int g_i = q / a.gj, g_j = q - g_i * a.gj;
    const bool act = g_i < a.gi && kv < kvn;
    const int rb = act ? g_i * RI : 0, cb = act ? g_j * RJ : 0, kvt = act ? kv : 0;
    const int k0 = 4 * (kv0 + kvt);
    unsigned own = 0, scored = 0;
#pragma unroll
    for (int r = 0; r < RI; ++r)
#pragma unroll
        for (int c = 0; c < RJ; ++c)
            if (act && rb + r < rows && cb + c < cols) {
                own |= 1u << (r * RJ + c);
                if (scored_col_t<uint32_t>(a.score, i0 + rb + r, j0 + cb + c)) scored |= 1u << (r * RJ + c);
            }
    auto gap = [&](int k) { return k >= a.nze && k < a.gap_end ? 0xffffffffu : 0u; };
    uint32_t gm0 = gap(k0), gm1 = gap(k0 + 1), gm2 = gap(k0 + 2), gm3 = gap(k0 + 3);
    uint32_t gkm = gap(k0 - 1), gkp = gap(k0 + 4);
    // (opaque: one AND a use; the compiler would compare and select again)
    asm volatile("" : "+r"(gm0), "+r"(gm1), "+r"(gm2), "+r"(gm3), "+r"(gkm), "+r"(gkp));
    const bool all_valid = k0 >= 1 && k0 + 3 <= a.nzb - 2;
    const int r_last = rows - 1 - rb, c_last = cols - 1 - cb;
    float *const cell0 = S + tile.cell_of(rb, cb) + 4 * kvt;
    const float2 *const pair0 = pairs + (rb + 1) * W + cb + 1;
    // edges of the patch on a reflecting wall, whose ring mirrors them (the row or
    // column within the patch, -1: none)
    const bool w_im = MIRROR && !lo_i && rb == 0, w_jm = MIRROR && !lo_j && cb == 0;
    const int w_ip = MIRROR && !hi_i ? r_last : -1, w_jp = MIRROR && !hi_j ? c_last : -1;
    const bool walls = w_im || w_ip >= 0 || w_jm || w_jp >= 0;

    float4 P[RI][RJ], N[RI][RJ];
#pragma unroll
    for (int r = 0; r < RI; ++r)
#pragma unroll
        for (int c = 0; c < RJ; ++c) {
            P[r][c] = N[r][c] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (own >> (r * RJ + c) & 1) {
                const int64_t o = ((int64_t)(i0 + rb + r) * n + (j0 + cb + c)) * kp + k0;
                float *d = cell0 + r * ROW + c * COL;
                P[r][c] = *reinterpret_cast<const float4 *>(a.pos_in + o);
                N[r][c] = *reinterpret_cast<const float4 *>(a.neg_in + o);
                st4s(d, P[r][c]);
                st4s(d + PITCH, N[r][c]);
            }
        }

    // The absorbing ring from the cells of step s into those of step s + 1: its
    // own value and the step's deposition.
    const bool carries = !MIRROR && (!lo_i || !hi_i || !lo_j || !hi_j);
    auto carry_ring = [&](int s) {
        const bool dep = a.slot[s] >= 0, keep = a.keep_stride > 0 || s + 1 == steps;
        // with two buffers the other one still holds the ring of a step before,
        // the same unless that step or this one deposited
        if (!(dep || keep || (SMALL && (s == 0 || a.slot[s - 1] >= 0)))) return;
        const float2 *Dp = pairs + (s & 1) * ncell;
        const float *from = S + (s & 1 ? BUF : 0);
        float *to = S + (s & 1 ? 0 : BUF);
        for (int u = tid; u < n_around * kvn; u += T) {
            const int col = u / kvn, v = u - col * kvn;
            int r, c;
            tile.around(col, r, c);
            if (!tile.ring_col(col, r, c)) continue;
            const int d = tile.cell_of(r, c) + 4 * v;
            float4 RP = ld4s(from + d), RN = ld4s(from + d + PITCH);
            const float dd = dep ? Dp[(r + 1) * W + c + 1].x : 0.f;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int k = 4 * (kv0 + v) + e;
                const float x = k >= a.nze && k < a.gap_end ? dd : 0.f;
                (&RP.x)[e] += x;
                (&RN.x)[e] += x;
            }
            st4s(to + d, RP);
            st4s(to + d + PITCH, RN);
            if (keep) {
                const int64_t o = s * a.keep_stride + ((int64_t)(i0 + r) * n + (j0 + c)) * kp + 4 * (kv0 + v);
                *reinterpret_cast<float4 *>(a.pos_out + o) = RP;
                *reinterpret_cast<float4 *>(a.neg_out + o) = RN;
            }
        }
    };

    const float2 NEG1 = make_float2(-1.f, -1.f);
    // The pairwise sums of a k-vector's elements in the gap.
    auto gap_sum = [&](float4 v) {
        return __fadd2_rn(make_float2(masked(v.x, gm0), masked(v.y, gm1)), make_float2(masked(v.z, gm2), masked(v.w, gm3)));
    };
    // A step of the patch from the cells at `cells` (and, DEP, the pairs at
    // Dp); returns the sum of the scored recombination terms. No branch and no
    // store in it: the items' loads and arithmetic overlap.
    auto advance = [&](auto with_deposition, const float *cells, const float2 *Dp) {
        constexpr bool DEP = decltype(with_deposition)::value;
        Tally<float> t_rec;
        float4 pP[RJ], pN[RJ];  // the row before, as it was (large patches: from the cells, which still hold it)
        if (SMALL)
#pragma unroll
            for (int c = 0; c < RJ; ++c) {
                pP[c] = ld4s(cells - ROW + c * COL);
                pN[c] = ld4s(cells - ROW + c * COL + PITCH);
            }
#pragma unroll
        for (int r = 0; r < RI; ++r) {
            float4 oP[RJ], oN[RJ];
#pragma unroll
            for (int c = 0; c < RJ; ++c) {
                oP[c] = P[r][c];
                oN[c] = N[r][c];
            }
#pragma unroll
            for (int c = 0; c < RJ; ++c) {
                const float *const d = cells + r * ROW + c * COL;
                float4 Pc = oP[c], Nc = oN[c];
                float pkm = d[-1], pkp = d[4], nkm = d[PITCH - 1], nkp = d[PITCH + 4];
                float4 Pip, Nip, Pjm, Njm, Pjp, Njp;
                if (r + 1 < RI) Pip = P[r + 1][c], Nip = N[r + 1][c];
                if (r + 1 == RI || r == r_last) Pip = ld4s(d + ROW), Nip = ld4s(d + ROW + PITCH);
                if (c > 0) Pjm = oP[c - 1], Njm = oN[c - 1];
                else Pjm = ld4s(d - COL), Njm = ld4s(d - COL + PITCH);
                if (c + 1 < RJ) Pjp = oP[c + 1], Njp = oN[c + 1];
                if (c + 1 == RJ || c == c_last) Pjp = ld4s(d + COL), Njp = ld4s(d + COL + PITCH);
                const float4 Pim = SMALL ? pP[c] : ld4s(d - ROW), Nim = SMALL ? pN[c] : ld4s(d - ROW + PITCH);
                auto add = [](float a0, float a1, float b0, float b1) {
                    return __fadd2_rn(make_float2(a0, a1), make_float2(b0, b1));
                };
                float2 Llo = __fadd2_rn(add(Pjm.x, Pjm.y, Pjp.x, Pjp.y), add(Pim.x, Pim.y, Pip.x, Pip.y));
                float2 Lhi = __fadd2_rn(add(Pjm.z, Pjm.w, Pjp.z, Pjp.w), add(Pim.z, Pim.w, Pip.z, Pip.w));
                float2 Mlo = __fadd2_rn(add(Njm.x, Njm.y, Njp.x, Njp.y), add(Nim.x, Nim.y, Nip.x, Nip.y));
                float2 Mhi = __fadd2_rn(add(Njm.z, Njm.w, Njp.z, Njp.w), add(Nim.z, Nim.w, Nip.z, Nip.w));
                if (DEP) {
                    const float2 dd = Dp[r * W + c];
                    const float2 d01 = make_float2(masked(dd.x, gm0), masked(dd.x, gm1));
                    const float2 d23 = make_float2(masked(dd.x, gm2), masked(dd.x, gm3));
                    const float2 l01 = make_float2(masked(dd.y, gm0), masked(dd.y, gm1));
                    const float2 l23 = make_float2(masked(dd.y, gm2), masked(dd.y, gm3));
                    Pc.x += d01.x, Pc.y += d01.y, Pc.z += d23.x, Pc.w += d23.y;
                    Nc.x += d01.x, Nc.y += d01.y, Nc.z += d23.x, Nc.w += d23.y;
                    const float dm = masked(dd.x, gkm), dq = masked(dd.x, gkp);
                    pkm += dm, nkm += dm, pkp += dq, nkp += dq;
                    Llo = __fadd2_rn(Llo, l01), Lhi = __fadd2_rn(Lhi, l23);
                    Mlo = __fadd2_rn(Mlo, l01), Mhi = __fadd2_rn(Mhi, l23);
                }
                const float2 Plo = make_float2(Pc.x, Pc.y), Phi = make_float2(Pc.z, Pc.w);
                const float2 Nlo = make_float2(Nc.x, Nc.y), Nhi = make_float2(Nc.z, Nc.w);
                float2 plo = __ffma2_rn(a.p_cen, Plo, __ffma2_rn(a.p_lat, Llo, __ffma2_rn(a.p_zp, make_float2(Pc.y, Pc.z), __fmul2_rn(a.p_zm, make_float2(pkm, Pc.x)))));
                float2 phi = __ffma2_rn(a.p_cen, Phi, __ffma2_rn(a.p_lat, Lhi, __ffma2_rn(a.p_zp, make_float2(Pc.w, pkp), __fmul2_rn(a.p_zm, make_float2(Pc.y, Pc.z)))));
                float2 nlo = __ffma2_rn(a.n_cen, Nlo, __ffma2_rn(a.n_lat, Mlo, __ffma2_rn(a.n_zp, make_float2(nkm, Nc.x), __fmul2_rn(a.n_zm, make_float2(Nc.y, Nc.z)))));
                float2 nhi = __ffma2_rn(a.n_cen, Nhi, __ffma2_rn(a.n_lat, Mhi, __ffma2_rn(a.n_zp, make_float2(Nc.y, Nc.z), __fmul2_rn(a.n_zm, make_float2(Nc.w, nkp)))));
                const float2 rlo = __fmul2_rn(__fmul2_rn(a.alpha_dt, Plo), Nlo), rhi = __fmul2_rn(__fmul2_rn(a.alpha_dt, Phi), Nhi);
                plo = __ffma2_rn(rlo, NEG1, plo);
                phi = __ffma2_rn(rhi, NEG1, phi);
                nlo = __ffma2_rn(rlo, NEG1, nlo);
                nhi = __ffma2_rn(rhi, NEG1, nhi);
                P[r][c] = make_float4(plo.x, plo.y, phi.x, phi.y);
                N[r][c] = make_float4(nlo.x, nlo.y, nhi.x, nhi.y);
                const float2 rec = gap_sum(make_float4(rlo.x, rlo.y, rhi.x, rhi.y));
                tally_item(t_rec, rec, scored >> (r * RJ + c) & 1, r + c == 0);
            }
            if (SMALL)
#pragma unroll
                for (int c = 0; c < RJ; ++c) {
                    pP[c] = oP[c];
                    pN[c] = oN[c];
                }
        }
        return t_rec;
    };

    // what alternates from step to step: the cells read and written, the pairs,
    // the tallies
    int now = 0, pair_now = 0, sum_now = 0;
    for (int s = 0; s < steps; ++s) {
        __syncthreads();  // the cells of this step and its pairs are in
        if (s_abort) return;
        const float *const cells = cell0 + now;
        now = BUF - now;
        float *const next = cell0 + now;
        const bool send = s + 1 < steps;
        const Tally<float> t_rec = a.slot[s] >= 0 ? advance(std::true_type{}, cells, pair0 + pair_now)
                                            : advance(std::false_type{}, cells, pair0);
        if (!all_valid) {  // the end planes and the row padding stay zero
            const int top = a.nzb - 2 - k0;  // the last valid element
#pragma unroll
            for (int r = 0; r < RI; ++r)
#pragma unroll
                for (int c = 0; c < RJ; ++c) {
                    if (k0 < 1 || top < 0) P[r][c].x = N[r][c].x = 0.f;
                    if (top < 1) P[r][c].y = N[r][c].y = 0.f;
                    if (top < 2) P[r][c].z = N[r][c].z = 0.f;
                    if (top < 3) P[r][c].w = N[r][c].w = 0.f;
                }
        }
        if (!SMALL) __syncthreads();  // every cell of this step has been read
#pragma unroll
        for (int r = 0; r < RI; ++r)
#pragma unroll
            for (int c = 0; c < RJ; ++c)
                if (own >> (r * RJ + c) & 1) {
                    float *const d = next + r * ROW + c * COL;
                    st4s(d, P[r][c]);
                    st4s(d + PITCH, N[r][c]);
                }
        if (walls) {  // the reflecting ring mirrors the columns beside it
#pragma unroll
            for (int r = 0; r < RI; ++r)
#pragma unroll
                for (int c = 0; c < RJ; ++c)
                    if (own >> (r * RJ + c) & 1) {
                        float *const d = next + r * ROW + c * COL;
                        auto put = [&](float *x) {
                            st4s(x, P[r][c]);
                            st4s(x + PITCH, N[r][c]);
                        };
                        if (r == 0 && w_im) put(d - ROW);
                        if (r == w_ip) put(d + ROW);
                        if (c == 0 && w_jm) put(d - COL);
                        if (c == w_jp) put(d + COL);
                    }
        }
        pair_now = ncell - pair_now;
        if (trades) {
            __syncthreads();  // the block's new cells are in
            if (send) tile.give(S + now, (uint32_t)(s + 1));
        }
        // while the packets are on their way: the tallies (the aux warps sum
        // them during the next step), the wall's ring, the states to keep
        Tally<float> t_p, t_n;
#pragma unroll
        for (int r = 0; r < RI; ++r)
#pragma unroll
            for (int c = 0; c < RJ; ++c) {
                const bool in = scored >> (r * RJ + c) & 1;
                tally_item(t_p, gap_sum(P[r][c]), in, r + c == 0);
                tally_item(t_n, gap_sum(N[r][c]), in, r + c == 0);
            }
        auto leave = [&](int x, const Tally<float> &t) {
            float *const m = sums + sum_now + VALUES * (x * T + tid);
            if constexpr (VALUES == 1) *m = t.s;
            else *reinterpret_cast<float2 *>(m) = make_float2(t.s, -t.c);
        };
        leave(0, t_rec), leave(1, t_p), leave(2, t_n);
        sum_now = SUMS - sum_now;
        if (a.keep_stride > 0 || !send) {
#pragma unroll
            for (int r = 0; r < RI; ++r)
#pragma unroll
                for (int c = 0; c < RJ; ++c)
                    if (own >> (r * RJ + c) & 1) {
                        const int i = i0 + rb + r, j = j0 + cb + c;
                        // the column, and the reflecting ring's columns that mirror it
                        for (int ii = (MIRROR && i == 1 ? 0 : i); ii <= (MIRROR && i == n - 2 ? n - 1 : i); ++ii)
                            for (int jj = (MIRROR && j == 1 ? 0 : j); jj <= (MIRROR && j == n - 2 ? n - 1 : j); ++jj) {
                                const int64_t o = s * a.keep_stride + ((int64_t)ii * n + jj) * kp + k0;
                                *reinterpret_cast<float4 *>(a.pos_out + o) = P[r][c];
                                *reinterpret_cast<float4 *>(a.neg_out + o) = N[r][c];
                            }
                    }
        }
        if (!MIRROR && carries) carry_ring(s);
        if (trades && send && !tile.take(S + now, (uint32_t)(s + 1))) s_abort = 1;
    }
    __syncthreads();
}

// A warp per step: the step's tally from its blocks' partials, in order.
__global__ void __launch_bounds__(256) resident_tally_kernel(const float2 *partials, int steps, int parts,
                                                              double injected_scale, double *tally) {
    const int s = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (s >= steps) return;
    const float4 *p = reinterpret_cast<const float4 *>(partials + (int64_t)s * parts * 4);
    DF v[4] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
    for (int b = lane; b < parts; b += 32) {
        const float4 x = p[2 * b], y = p[2 * b + 1];
        v[0] = df_add(v[0], DF{x.x, x.y});
        v[1] = df_add(v[1], DF{x.z, x.w});
        v[2] = df_add(v[2], DF{y.x, y.y});
        v[3] = df_add(v[3], DF{y.z, y.w});
    }
    const DF w = warp_sum4(v, lane);
    if ((lane & 7) == 0) tally[4 * (int64_t)s + (lane >> 3)] = df_value(w) * (lane == 0 ? injected_scale : 1.0);
}

// The patches a thread may own, with the block size their registers allow.
constexpr ResPatch kPatches[] = {{1, 1, 640}, {2, 1, 512}, {2, 2, 512}, {3, 2, 448}, {4, 2, 384}};

int64_t step_smem(const ResPlan &p, const ResPatch &pt) {
    const int64_t cells = res_cells(p.gi, p.gj, pt.ri, pt.rj);
    const int64_t tallies = 3LL * res_tally_values(pt.ri, pt.rj) * res_tally_buffers(res_small(pt.ri, pt.rj), p.blocks);
    return 4 * (res_pair_floats((int)cells) + tallies * p.threads +
                (2 * cells * res_pitch(kResTkvMax) + 4) * (res_small(pt.ri, pt.rj) ? 2 : 1)) +
           16LL * (2 * (p.ti + p.tj) * p.tkv + 2 * p.ti * p.tj);
}

template <int RI, int RJ, int MAXT, bool MIRROR>
int launch_walled(const ResArgs &a, const ResPlan &p, cudaStream_t st) {
    return launch_cooperative(resident_kernel<RI, RJ, kResTkvMax, MAXT, MIRROR>, "resident_kernel", a, p, st);
}
template <int RI, int RJ, int MAXT>
int launch_patch(const ResArgs &a, const ResPlan &p, cudaStream_t st) {
    return a.reflecting ? launch_walled<RI, RJ, MAXT, true>(a, p, st) : launch_walled<RI, RJ, MAXT, false>(a, p, st);
}

constexpr int kResSmem = 227 * 1024 - 4096;  // less the kernel's static part

// The next larger piece that splits M into fewer pieces (M + 1 after M).
int next_split(int M, int piece) {
    const int pieces = (M + piece - 1) / piece;
    return pieces > 1 ? (M + pieces - 2) / (pieces - 1) : M + 1;
}

// Estimated microseconds of a step, fitted to measured ones (GB300, idle steps,
// 11^2 x 56 to 76^2 x 206 and 59^2 x 406, eleven divisions): a fixed part, the
// patches (a warp's item takes 65 cycles of its SM, with the larger patches'
// spills 75), and a round of packets with the faces' size.
double plan_cost(const ResPlan &p, const ResPatch &pt, double item_scale) {
    const double items = p.threads / 32 * pt.ri * pt.rj;  // of warps
    double t = 0.4 + (pt.ri * pt.rj >= 6 ? 0.038 : 0.0325) * item_scale * items;
    if (p.blocks > 1) {
        const double kb = (2.0 * (p.ti + p.tj) * p.tkv * 48.0 + 2.0 * (p.ntk > 1) * p.ti * p.tj * 16.0) / 1024.0;
        t += 0.95 + 0.032 * kb;
        const int faces = 2 * (p.ti + p.tj) * p.tkv, round = 2 * p.threads;  // two a thread at once
        t += 0.4 * ((faces + round - 1) / round - 1);
    }
    return t;
}

bool find_plan(int M, int c4, int sms, const ResPatch *patches, int count, ResSmem smem_of, double item_scale, ResPlan *out) {
    // more cells than the largest patches hold
    if ((int64_t)M * M * c4 > (int64_t)sms * 4608) return false;
    ResPlan best{};
    double best_t = 1e30;
    for (int pi = 0; pi < count; ++pi) {
        const ResPatch &pt = patches[pi];
        for (int ntk = (c4 + kResTkvMax - 1) / kResTkvMax, tries = 0; tries < 3 && (tries == 0 || c4 / ntk >= 4); ++tries, ++ntk) {
            ResPlan p{};
            p.patch = pi;
            p.tkv = (c4 + ntk - 1) / ntk;
            p.ntk = (c4 + p.tkv - 1) / p.tkv;
            if (p.ntk != ntk) continue;
            for (int ti = 1; ti <= M; ti = next_split(M, ti)) {
                p.ti = ti;
                p.nti = (M + ti - 1) / ti;
                p.gi = (ti + pt.ri - 1) / pt.ri;
                const int room = sms / (p.nti * ntk);
                if (room < 1) continue;
                // the finest splits of j that the SMs hold, and j in one piece
                int tj = (M + std::min(room, M) - 1) / std::min(room, M);
                for (int tries = 0; tries < 4 && tj <= M; ++tries) {
                    p.tj = tj;
                    tj = tries < 2 ? next_split(M, tj) : (tj < M ? M : M + 1);
                    p.ntj = (M + p.tj - 1) / p.tj;
                    p.gj = (p.tj + pt.rj - 1) / pt.rj;
                    p.blocks = p.nti * p.ntj * p.ntk;
                    const int64_t threads = (int64_t)p.gi * p.gj * p.tkv;
                    p.threads = (int)(threads + 31) / 32 * 32;
                    const int left = (pt.max_threads - p.threads) / 32;  // warps
                    if (left < 1) continue;
                    // a warp beside the chain per 128 patch threads
                    p.aux = 32 * std::min(left, (p.threads + 127) / 128);
                    const int64_t smem = smem_of(p, pt);
                    if (smem > kResSmem) continue;
                    p.smem = (int)smem;
                    const double t = plan_cost(p, pt, item_scale);
                    if (t < best_t) {
                        best_t = t;
                        best = p;
                    }
                }
            }
        }
    }
    if (best_t >= 1e30) return false;
    best.packets = res_faces(best.ti, best.tj, best.tkv).total;
    *out = best;
    return true;
}

}  // namespace

bool ResPlanMemo::plan(const pic_grid *g, const ResPatch *patches, int count, ResSmem smem_of, double item_scale,
                       ResPlan *out) {
    if (g->dtype != PIC_F32 || g->no_xy < 3 || g->no_xy > kResMaxNoXy) return false;
    const int M_ = (int)g->no_xy - 2, c4_ = (int)(g->kpitch / 4), sms_ = sm_count();
    if (M != M_ || c4 != c4_ || sms != sms_) {
        M = M_, c4 = c4_, sms = sms_;
        fits = find_plan(M, c4, sms, patches, count, smem_of, item_scale, &last);
    }
    if (fits) *out = last;
    return fits;
}

// Estimated microseconds of a flat step of a grid that stays in the L2
// (pic_wide.cuh): 30^2 x 406 3.9, 61^2 x 606 8.1, 119^2 x 406 17.4.
static double flat_cost(const pic_grid *g) { return 3.0 + 2.5e-6 * (double)(g->no_xy * g->no_xy * g->nzb); }

// Grids whose division is estimated slower than the flat step run flat: few and
// tall columns, which the SMs split badly (51^2 x 606, ms for 1500 steps, absorbing /
// reflecting: resident 12.6 / 12.3, flat 11.4 / 12.0; estimates 7.9 and 6.9 us a step.
// 61^2 x 406 the same either way, 86^2 x 206 11.5 resident, 12.1 flat).
bool resident_plan(const pic_grid *g, ResPlan *out) {
    static thread_local ResPlanMemo memo;
    if (!memo.plan(g, kPatches, (int)(sizeof(kPatches) / sizeof(kPatches[0])), step_smem, 1.0, out)) return false;
    return plan_cost(*out, kPatches[out->patch], 1.0) <= flat_cost(g);
}

int launch_resident(const pic_grid *g, const ResPlan &p, const void *pos_in, const void *neg_in, void *pos_out,
                    void *neg_out, const void *dens, int64_t dens_stride, const int16_t *slot, int steps,
                    int64_t keep_stride, double *tally, void *packets, void *partials, int *status, cudaStream_t st) {
    if (steps < 1 || steps > kResSteps) return set_error(PIC_E_INVALID, "resident launch: 1 .. kResSteps steps");
    auto twice = [](float x) { return make_float2(x, x); };
    ResArgs a;
    a.pos_in = static_cast<const float *>(pos_in);
    a.neg_in = static_cast<const float *>(neg_in);
    a.pos_out = static_cast<float *>(pos_out);
    a.neg_out = static_cast<float *>(neg_out);
    a.dens = static_cast<const float2 *>(dens);
    a.dens_stride = dens_stride;
    a.keep_stride = keep_stride;
    a.partials = static_cast<float2 *>(partials);
    a.dp = (int)dens_pitch(g->no_xy);
    a.steps = steps;
    res_shape(g, p, packets, status, &a);
    a.p_lat = twice((float)g->p_lat), a.p_zm = twice((float)g->p_zm), a.p_zp = twice((float)g->p_zp);
    a.p_cen = twice(centre_weight<float>(g->p_lat, g->p_zm, g->p_zp, g->p_cen));
    a.n_lat = twice((float)g->n_lat), a.n_zm = twice((float)g->n_zm), a.n_zp = twice((float)g->n_zp);
    a.n_cen = twice(centre_weight<float>(g->n_lat, g->n_zm, g->n_zp, g->n_cen));
    a.alpha_dt = twice((float)g->alpha_dt);
    int rc = score_test(g, &a.score);
    if (rc) return rc;
    for (int s = 0; s < steps; ++s) a.slot[s] = slot[s];
    switch (p.patch) {
        case 0: rc = launch_patch<1, 1, kPatches[0].max_threads>(a, p, st); break;
        case 1: rc = launch_patch<2, 1, kPatches[1].max_threads>(a, p, st); break;
        case 2: rc = launch_patch<2, 2, kPatches[2].max_threads>(a, p, st); break;
        case 3: rc = launch_patch<3, 2, kPatches[3].max_threads>(a, p, st); break;
        default: rc = launch_patch<4, 2, kPatches[4].max_threads>(a, p, st); break;
    }
    if (rc || !tally) return rc;
    resident_tally_kernel<<<(unsigned)((steps + 7) / 8), 256, 0, st>>>(static_cast<const float2 *>(partials), steps,
                                                                        p.blocks * (p.aux / 32), (double)g->no_z, tally);
    return check_launch("resident_tally_kernel");
}

bool resident_steps_eligible(const pic_grid *g, const void *ws, int64_t ws_bytes, const int64_t *off, int64_t n_steps,
                             int64_t span, ResPlan *plan) {
    if (!resident_wanted(g) || n_steps < kResMinSteps || !ws || !resident_plan(g, plan) || ws_bytes < resident_space(g, *plan).end)
        return false;
    if (off[n_steps] == off[0]) return true;
    if (!bin_eligible(g)) return false;
    double longest = 0.0, tracks = 0.0;  // of the launches with a tile of more than kBinAutoPerTile: its tracks, all tracks
    for (int64_t s0 = 0, s1; s0 < n_steps; s0 = s1) {
        s1 = next_resident_group(off, s0, std::min(n_steps, (s0 / span + 1) * span));
        if (s1 == s0) return false;  // a step of more than kBinTracks
        int64_t most = 0;
        for (int64_t s = s0; s < s1; ++s) most = std::max(most, off[s + 1] - off[s]);
        const double tile = bin_tile_tracks(g, most);
        if (tile <= kBinAutoPerTile) continue;
        longest += std::min(tile, (double)most);
        tracks += (double)(off[s1] - off[s0]);
    }
    return g->deposit_variant == PIC_DEPOSIT_BINNED || 10.0 * longest <= tracks;
}

int64_t next_resident_group(const int64_t *off, int64_t s0, int64_t n_steps) {
    int64_t s1 = s0;
    while (s1 < n_steps && s1 - s0 < kResSteps && off[s1 + 1] - off[s0] <= kBinTracks) ++s1;
    return s1;
}

int resident_steps(const pic_grid *g, const ResPlan &plan, const void *pos_in, const void *neg_in, void *pos_out,
                   void *neg_out, const double *xs, const double *ys, const int64_t *off, int64_t s0, int64_t s1,
                   uint32_t *counts, double *tally, void *targets, int64_t target_stride, const void **last_pairs,
                   void *ws, cudaStream_t st) {
    const ResSpace r = resident_space(g, plan);
    char *w = static_cast<char *>(ws);
    const bool tracks = off[s1] > off[s0];
    const int64_t clear0 = tracks ? r.counts : r.packets;
    if (tracks || plan.blocks > 1) {
        cudaError_t e = cudaMemsetAsync(w + clear0, 0, (size_t)(r.partials - clear0), st);
        if (e != cudaSuccess) return set_cuda_error("cudaMemsetAsync(packets)", e);
    }
    char *dens = targets ? static_cast<char *>(targets) : w + r.dens;
    const int64_t stride = targets ? target_stride : bin_dens_bytes(g->no_xy, 4) / 8;
    int16_t slot[kResSteps];
    int rc = launch_deposit_slots(g, xs, ys, off, s0, s1, counts, ws, r.counts, r.lists, dens, stride, slot, st);
    if (rc) return rc;
    const int16_t end = slot[s1 - 1 - s0];
    *last_pairs = end < 0 ? nullptr : dens + 8 * stride * end;
    return launch_resident(g, plan, pos_in, neg_in, pos_out, neg_out, dens, stride, slot, (int)(s1 - s0), 0, tally,
                           w + r.packets, w + r.partials, workspace_layout(ws).status, st);
}

}  // namespace pic
