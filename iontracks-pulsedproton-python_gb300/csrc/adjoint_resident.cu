// adjoint_resident.cu -- the adjoint steps of a checkpoint segment of a small
// float32 grid in one cooperative launch whose blocks keep lambda on the chip
// (adjoint.cu states the equations, resident.cu how such a launch works).
//
// Step by step the flat adjoint kernel takes 8 us on a grid of half a million
// cells, a launch and chains of L2 round trips for a microsecond of
// arithmetic. Here a thread keeps mu -- lambda_{s+1} with the reflecting ring's
// share folded in -- of its patch in registers, with two copies in shared
// memory that alternate by step, and the blocks trade their faces of mu as the
// resident step trades its fields. Of the recomputed states a step needs its
// own voxels' only, since the derivative sums are taken by parts
// (adjoint_stream.cu): each thread fetches them a step ahead into its own
// slots of shared memory, while packets fly. The aux warps fetch the deposition
// pairs and the ring columns' state. The five sums stay in compensated
// registers through the launch and join the block's slot at its end.
//
// Ring columns: mu there is zero in every stencil (their cells stay zero).
// Absorbing, a ring column's lambda is its own plus lat mu of the column beside
// it, summed in the output buffer by the one thread beside it; reflecting, it is
// lat mu alone, which the next step folds back into that column: the thread
// adds it at once, and stores it only with the launch's last lambda.
//
// What bounds it is the step's chain, as in resident.cu. Measured on GB300, the
// whole gradient of the 48^2 x 206 column (1622 steps, checkpoints every 64):
// 69.4 ms with a launch for every recomputed and every adjoint step, 21.8 ms so.
#include <cuda_runtime.h>
#include <stdint.h>

#include <mutex>
#include <type_traits>

#include "pic_adjoint.cuh"
#include "pic_resident.cuh"

namespace pic {

namespace {

struct AdjResArgs : ResShape {
    const float *pos0, *neg0;  // the state of the launch's earliest step
    const float *pos, *neg;    // the others': step j's at pos + j * state_stride
    int64_t state_stride;
    const float2 *dens;        // pairs of slot q at dens + q * dens_stride
    int64_t dens_stride;
    const float *lp_in, *ln_in;  // lambda after the latest step
    float *lp_out, *ln_out;      // lambda before the earliest one
    float2 *slots;               // [blocks][kAdjGrad] running sums (double-floats)
    int dp, steps;
    float2 p_lat, p_zm, p_zp, p_cen, n_lat, n_zm, n_zp, n_cen, alpha_dt, c_pos, c_neg;  // each twice
    ScoreTest score;
    int16_t slot[kResSteps];  // pair slot of step j, -1: no tracks
};

__device__ __forceinline__ float2 lo2(float4 v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(float4 v) { return make_float2(v.z, v.w); }
__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __fadd2_rn(a, neg2(b)); }
__device__ __forceinline__ float2 masked2(float2 v, uint32_t m0, uint32_t m1) {
    return make_float2(masked(v.x, m0), masked(v.y, m1));
}
__device__ __forceinline__ void copy_async16(float *dst, const float *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}

template <int RI, int RJ, int TKV, int MAXT, bool MIRROR>
__global__ void __launch_bounds__(MAXT, 1) adjoint_resident_kernel(const __grid_constant__ AdjResArgs a) {
    constexpr int PITCH = res_pitch(TKV), COL = 2 * PITCH;
    extern __shared__ __align__(16) float res_smem[];
    __shared__ volatile int s_abort;
    const int tid = threadIdx.x, T = a.patch_threads;
    const int W = a.gj * RJ + 2, ROW = W * COL;
    ResTile<PITCH> tile(a, W);
    const int i0 = tile.i0, j0 = tile.j0, kv0 = tile.kv0, rows = tile.rows, cols = tile.cols, kvn = tile.kvn;
    const int n = a.n, kp = a.kp, tkv = a.tkv, steps = a.steps;
    const int ncell = res_cells(a.gi, a.gj, RI, RJ), nring = tile.n_side * kvn;
    // shared memory: pairs [2], the ring's state [2][species], each thread's
    // own states [item][species], cells [2], the table of trades
    float2 *const pairs = reinterpret_cast<float2 *>(res_smem);
    float *const ring = res_smem + (4 * ncell + 3) / 4 * 4;
    const int RING = 4 * 2 * (a.ti + a.tj) * tkv;  // floats of one species of one buffer, as allocated
    float *const own_u = ring + 4 * RING;
    float *const S = own_u + 8 * RI * RJ * T;
    const int BUF = ncell * COL + 4;
    const bool trades = gridDim.x > 1;
    auto offset = [&](int i, int j, int k) { return ((int64_t)i * n + j) * kp + k; };
    // lambda of an interior column as the steps before it want it: a reflecting
    // ring's lambda folded into the columns it copies
    auto folded = [&](const float *lam, int i, int j, int k) {
        float4 v = *reinterpret_cast<const float4 *>(lam + offset(i, j, k));
        if (MIRROR)
            for (int ii = i == 1 ? 0 : i; ii <= (i == n - 2 ? n - 1 : i); ++ii)
                for (int jj = j == 1 ? 0 : j; jj <= (j == n - 2 ? n - 1 : j); ++jj)
                    if (ii != i || jj != j) {
                        const float4 w = *reinterpret_cast<const float4 *>(lam + offset(ii, jj, k));
                        v.x += w.x, v.y += w.y, v.z += w.z, v.w += w.w;
                    }
        return v;
    };

    // ---- load: cells to zero, then mu around the block ----
    if (tid == 0) s_abort = 0;
    for (int u = tid; u < BUF / 4 * 2; u += blockDim.x) st4s(S + 4 * u, make_float4(0.f, 0.f, 0.f, 0.f));
    for (int u = tid; u < 8 * RI * RJ * T / 4; u += blockDim.x) st4s(own_u + 4 * u, make_float4(0.f, 0.f, 0.f, 0.f));
    __syncthreads();
    for (int u = tid; u < nring; u += blockDim.x) {
        const int col = u / kvn, v = u - col * kvn;
        int r, c;
        tile.around(col, r, c);
        if (tile.ring_col(col, r, c)) continue;
        float *d = S + tile.cell_of(r, c) + 4 * v;
        st4s(d, folded(a.lp_in, i0 + r, j0 + c, 4 * (kv0 + v)));
        st4s(d + PITCH, folded(a.ln_in, i0 + r, j0 + c, 4 * (kv0 + v)));
    }
    for (int u = tid; u < rows * cols; u += blockDim.x) {
        const int r = u / cols, c = u - r * cols, k = 4 * kv0;
        float *d = S + tile.cell_of(r, c);
        if (tile.lo_k) {
            d[-1] = folded(a.lp_in, i0 + r, j0 + c, k - 4).w;
            d[PITCH - 1] = folded(a.ln_in, i0 + r, j0 + c, k - 4).w;
        }
        if (tile.hi_k) {
            d[4 * kvn] = folded(a.lp_in, i0 + r, j0 + c, k + 4 * kvn).x;
            d[PITCH + 4 * kvn] = folded(a.ln_in, i0 + r, j0 + c, k + 4 * kvn).x;
        }
    }
    tile.table(reinterpret_cast<int4 *>(S + 2 * BUF));
    // the grid's corners have no interior neighbour: an absorbing one is carried, a reflecting one zero
    for (int u = tid; u < 4 * kvn; u += blockDim.x) {
        const int q = tile.n_side + u / kvn, v = u % kvn;
        int r, c;
        tile.around(q, r, c);
        if (!tile.ring_col(q, r, c)) continue;
        const int64_t o = offset(i0 + r, j0 + c, 4 * (kv0 + v));
        const float4 Z = make_float4(0.f, 0.f, 0.f, 0.f);
        if (!MIRROR) {
            *reinterpret_cast<float4 *>(a.lp_out + o) = *reinterpret_cast<const float4 *>(a.lp_in + o);
            *reinterpret_cast<float4 *>(a.ln_out + o) = *reinterpret_cast<const float4 *>(a.ln_in + o);
        } else if (a.lp_out != a.lp_in) {  // (in place, the blocks beside still read it: zeroed with the last step)
            *reinterpret_cast<float4 *>(a.lp_out + o) = Z;
            *reinterpret_cast<float4 *>(a.ln_out + o) = Z;
        }
    }

    if (tid >= T) {
        // ---------------- the warps beside the steps' chain ----------------
        const int AT = a.aux_threads, at = tid - T;
        auto fetch = [&](int s) {  // the pairs and the ring's state of the s-th step taken, asynchronously
            if (s >= steps) return;
            const int j = steps - 1 - s, sl = a.slot[j];
            if (sl >= 0) {
                const float2 *src = a.dens + sl * a.dens_stride + (int64_t)(i0 - 1) * a.dp + (j0 - 1);
                for (int u = at; u < (rows + 2) * (cols + 2); u += AT) {
                    const int r = u / (cols + 2), c = u - r * (cols + 2);
                    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(pairs + (s & 1) * ncell + r * W + c);
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src + (int64_t)r * a.dp + c)
                                 : "memory");
                }
            }
            const float *pos = j == 0 ? a.pos0 : a.pos + j * a.state_stride;
            const float *neg = j == 0 ? a.neg0 : a.neg + j * a.state_stride;
            for (int u = at; u < nring; u += AT) {
                const int col = u / kvn, v = u - col * kvn;
                int r, c;
                tile.around(col, r, c);
                if (!tile.ring_col(col, r, c)) continue;
                const int64_t o = offset(i0 + r, j0 + c, 4 * (kv0 + v));
                copy_async16(ring + (s & 1) * 2 * RING + 4 * u, pos + o);
                copy_async16(ring + ((s & 1) * 2 + 1) * RING + 4 * u, neg + o);
            }
        };
        fetch(0);
        for (int s = 0; s < steps; ++s) {
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();
            if (s_abort) break;
            fetch(s + 1);
            if (trades) __syncthreads();
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
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
    asm volatile("" : "+r"(gm0), "+r"(gm1), "+r"(gm2), "+r"(gm3));  // (as in resident.cu)
    const bool all_valid = k0 >= 1 && k0 + 3 <= a.nzb - 2;
    const int r_last = rows - 1 - rb, c_last = cols - 1 - cb;
    float *const cell0 = S + tile.cell_of(rb, cb) + 4 * kvt;
    const float2 *const pair0 = pairs + (rb + 1) * W + cb + 1;
    float *const u0 = own_u + 4 * tid;  // item x's states: u0 + 8 x T (positive), + 4 T (negative)
    // edges of the patch on the wall (the row or column within it, -1: none)
    const bool w_im = act && !tile.lo_i && rb == 0, w_jm = act && !tile.lo_j && cb == 0;
    const int w_ip = act && !tile.hi_i ? r_last : -1, w_jp = act && !tile.hi_j ? c_last : -1;
    const bool walls = w_im || w_jm || (w_ip >= 0 && w_ip < RI) || (w_jp >= 0 && w_jp < RJ);

    // each side of the wall item (r, c) lies on: f(ring column i, j, its index beside the block)
    auto each_side = [&](int r, int c, auto f) {
        const int i = i0 + rb + r, j = j0 + cb + c;
        if (r == 0 && w_im) f(0, j, cb + c);
        if (r == w_ip) f(n - 1, j, cols + cb + c);
        if (c == 0 && w_jm) f(i, 0, 2 * cols + rb + r);
        if (c == w_jp) f(i, n - 1, 2 * cols + rows + rb + r);
    };
    auto fetch_own = [&](int s) {
        if (s >= steps) return;
        const int j = steps - 1 - s;
        const float *pos = j == 0 ? a.pos0 : a.pos + j * a.state_stride;
        const float *neg = j == 0 ? a.neg0 : a.neg + j * a.state_stride;
#pragma unroll
        for (int r = 0; r < RI; ++r)
#pragma unroll
            for (int c = 0; c < RJ; ++c)
                if (own >> (r * RJ + c) & 1) {
                    const int64_t o = offset(i0 + rb + r, j0 + cb + c, k0);
                    copy_async16(u0 + 8 * (r * RJ + c) * T, pos + o);
                    copy_async16(u0 + 8 * (r * RJ + c) * T + 4 * T, neg + o);
                }
    };
    float4 P[RI][RJ], N[RI][RJ];  // mu of both species
#pragma unroll
    for (int r = 0; r < RI; ++r)
#pragma unroll
        for (int c = 0; c < RJ; ++c) {
            P[r][c] = N[r][c] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (own >> (r * RJ + c) & 1) {
                float *d = cell0 + r * ROW + c * COL;
                P[r][c] = folded(a.lp_in, i0 + rb + r, j0 + cb + c, k0);
                N[r][c] = folded(a.ln_in, i0 + rb + r, j0 + cb + c, k0);
                st4s(d, P[r][c]);
                st4s(d + PITCH, N[r][c]);
            }
        }
    fetch_own(0);
    Tally<float> acc[kAdjGrad];
    const float2 M6 = make_float2(-6.f, -6.f), M2 = make_float2(-2.f, -2.f), HALF = make_float2(0.5f, 0.5f);

    // One adjoint step of the patch from the cells at `cells`: P, N become
    // lambda_s, with the reflecting ring's share folded in where `fold`.
    auto retreat = [&](auto with_deposition, const float *cells, const float2 *Dp, const float *ringu, bool fold) {
        constexpr bool DEP = decltype(with_deposition)::value;
        float4 pP[RJ], pN[RJ];
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
                float2 G0 = make_float2(0.f, 0.f), G1 = G0, G2 = G0, G3 = G0, G4 = G0;  // the item's terms
                const float4 MP = oP[c], MN = oN[c];
                const float mp_km = d[-1], mp_kp = d[4], mn_km = d[PITCH - 1], mn_kp = d[PITCH + 4];
                float4 A1, B1, A2, B2, A3, B3;
                if (r + 1 < RI) A1 = P[r + 1][c], B1 = N[r + 1][c];
                if (r + 1 == RI || r == r_last) A1 = ld4s(d + ROW), B1 = ld4s(d + ROW + PITCH);
                if (c > 0) A2 = oP[c - 1], B2 = oN[c - 1];
                else A2 = ld4s(d - COL), B2 = ld4s(d - COL + PITCH);
                if (c + 1 < RJ) A3 = oP[c + 1], B3 = oN[c + 1];
                if (c + 1 == RJ || c == c_last) A3 = ld4s(d + COL), B3 = ld4s(d + COL + PITCH);
                const float2 LPl = __fadd2_rn(__fadd2_rn(lo2(pP[c]), lo2(A1)), __fadd2_rn(lo2(A2), lo2(A3)));
                const float2 LPh = __fadd2_rn(__fadd2_rn(hi2(pP[c]), hi2(A1)), __fadd2_rn(hi2(A2), hi2(A3)));
                const float2 LNl = __fadd2_rn(__fadd2_rn(lo2(pN[c]), lo2(B1)), __fadd2_rn(lo2(B2), lo2(B3)));
                const float2 LNh = __fadd2_rn(__fadd2_rn(hi2(pN[c]), hi2(B1)), __fadd2_rn(hi2(B2), hi2(B3)));
                const float4 P0 = ld4s(u0 + 8 * (r * RJ + c) * T), N0 = ld4s(u0 + 8 * (r * RJ + c) * T + 4 * T);
                float2 Pl = lo2(P0), Ph = hi2(P0), Nl = lo2(N0), Nh = hi2(N0);
                const float2 MPl = lo2(MP), MPh = hi2(MP), MNl = lo2(MN), MNh = hi2(MN);
                if (DEP) {
                    // (a place without an item has state zero and must add nothing)
                    const float2 dd = own >> (r * RJ + c) & 1 ? Dp[r * W + c] : make_float2(0.f, 0.f);
                    const float2 D = make_float2(dd.x, dd.x), L = make_float2(dd.y, dd.y);
                    const float2 Dl = masked2(D, gm0, gm1), Dh = masked2(D, gm2, gm3);
                    const float2 Ll = masked2(L, gm0, gm1), Lh = masked2(L, gm2, gm3);
                    Pl = __fadd2_rn(Pl, Dl), Ph = __fadd2_rn(Ph, Dh), Nl = __fadd2_rn(Nl, Dl), Nh = __fadd2_rn(Nh, Dh);
                    G0 = __ffma2_rn(MPl, Ll, __ffma2_rn(MPh, Lh, G0));
                    G2 = __ffma2_rn(MNl, Ll, __ffma2_rn(MNh, Lh, G2));
                }
                const float2 mpu_l = make_float2(MP.y, MP.z), mpu_h = make_float2(MP.w, mp_kp);
                const float2 mpd_l = make_float2(mp_km, MP.x), mpd_h = make_float2(MP.y, MP.z);
                const float2 mnu_l = make_float2(MN.y, MN.z), mnu_h = make_float2(MN.w, mn_kp);
                const float2 mnd_l = make_float2(mn_km, MN.x), mnd_h = make_float2(MN.y, MN.z);
                const float2 Ssl = __fadd2_rn(MPl, MNl), Ssh = __fadd2_rn(MPh, MNh);
                const float2 ANl = __fmul2_rn(a.alpha_dt, Nl), ANh = __fmul2_rn(a.alpha_dt, Nh);
                const float2 APl = __fmul2_rn(a.alpha_dt, Pl), APh = __fmul2_rn(a.alpha_dt, Ph);
                float2 lpl = __ffma2_rn(a.p_cen, MPl, __ffma2_rn(a.p_lat, LPl, __ffma2_rn(a.p_zp, mpd_l, __fmul2_rn(a.p_zm, mpu_l))));
                float2 lph = __ffma2_rn(a.p_cen, MPh, __ffma2_rn(a.p_lat, LPh, __ffma2_rn(a.p_zp, mpd_h, __fmul2_rn(a.p_zm, mpu_h))));
                float2 lnl = __ffma2_rn(a.n_cen, MNl, __ffma2_rn(a.n_lat, LNl, __ffma2_rn(a.n_zp, mnu_l, __fmul2_rn(a.n_zm, mnd_l))));
                float2 lnh = __ffma2_rn(a.n_cen, MNh, __ffma2_rn(a.n_lat, LNh, __ffma2_rn(a.n_zp, mnu_h, __fmul2_rn(a.n_zm, mnd_h))));
                lpl = __ffma2_rn(neg2(ANl), Ssl, lpl);
                lph = __ffma2_rn(neg2(ANh), Ssh, lph);
                lnl = __ffma2_rn(neg2(APl), Ssl, lnl);
                lnh = __ffma2_rn(neg2(APh), Ssh, lnh);
                const float2 pnl = __fmul2_rn(Pl, Nl), pnh = __fmul2_rn(Ph, Nh);
                G4 = __ffma2_rn(neg2(Ssh), pnh, __ffma2_rn(neg2(Ssl), pnl, G4));
                if (scored >> (r * RJ + c) & 1) {  // scored gap voxels
                    lpl = __fadd2_rn(lpl, masked2(ANl, gm0, gm1)), lph = __fadd2_rn(lph, masked2(ANh, gm2, gm3));
                    lnl = __fadd2_rn(lnl, masked2(APl, gm0, gm1)), lnh = __fadd2_rn(lnh, masked2(APh, gm2, gm3));
                    G4 = __fadd2_rn(G4, __fadd2_rn(masked2(pnl, gm0, gm1), masked2(pnh, gm2, gm3)));
                }
                // the derivative sums, by parts (adjoint_stream.cu)
                const float2 zsp_l = __fadd2_rn(mpu_l, mpd_l), zsp_h = __fadd2_rn(mpu_h, mpd_h);
                const float2 zsn_l = __fadd2_rn(mnu_l, mnd_l), zsn_h = __fadd2_rn(mnu_h, mnd_h);
                const float2 plm_l = __ffma2_rn(M6, MPl, zsp_l), plm_h = __ffma2_rn(M6, MPh, zsp_h);
                const float2 nlm_l = __ffma2_rn(M6, MNl, zsn_l), nlm_h = __ffma2_rn(M6, MNh, zsn_h);
                const float2 pcm_l = __ffma2_rn(a.c_pos, __ffma2_rn(M2, MPl, zsp_l), __fmul2_rn(HALF, sub2(mpu_l, mpd_l)));
                const float2 pcm_h = __ffma2_rn(a.c_pos, __ffma2_rn(M2, MPh, zsp_h), __fmul2_rn(HALF, sub2(mpu_h, mpd_h)));
                const float2 ncm_l = __ffma2_rn(a.c_neg, __ffma2_rn(M2, MNl, zsn_l), __fmul2_rn(HALF, sub2(mnd_l, mnu_l)));
                const float2 ncm_h = __ffma2_rn(a.c_neg, __ffma2_rn(M2, MNh, zsn_h), __fmul2_rn(HALF, sub2(mnd_h, mnu_h)));
                G0 = __ffma2_rn(lo2(P0), LPl, __ffma2_rn(Pl, plm_l, G0));
                G0 = __ffma2_rn(hi2(P0), LPh, __ffma2_rn(Ph, plm_h, G0));
                G1 = __ffma2_rn(Ph, pcm_h, __ffma2_rn(Pl, pcm_l, G1));
                G2 = __ffma2_rn(lo2(N0), LNl, __ffma2_rn(Nl, nlm_l, G2));
                G2 = __ffma2_rn(hi2(N0), LNh, __ffma2_rn(Nh, nlm_h, G2));
                G3 = __ffma2_rn(Nh, ncm_h, __ffma2_rn(Nl, ncm_l, G3));
                if (walls) {
                    // a ring column's state enters the lateral sum of the column
                    // beside it; its lambda, reflecting, folds back into it
                    each_side(r, c, [&](int, int, int col) {
                        const float4 UP = ld4s(ringu + 4 * (col * kvn + kvt)), UN = ld4s(ringu + RING + 4 * (col * kvn + kvt));
                        if (own >> (r * RJ + c) & 1) {
                            G0 = __ffma2_rn(lo2(UP), MPl, __ffma2_rn(hi2(UP), MPh, G0));
                            G2 = __ffma2_rn(lo2(UN), MNl, __ffma2_rn(hi2(UN), MNh, G2));
                        }
                        if (MIRROR && fold) {
                            lpl = __ffma2_rn(a.p_lat, MPl, lpl), lph = __ffma2_rn(a.p_lat, MPh, lph);
                            lnl = __ffma2_rn(a.n_lat, MNl, lnl), lnh = __ffma2_rn(a.n_lat, MNh, lnh);
                        }
                    });
                }
                P[r][c] = make_float4(lpl.x, lpl.y, lph.x, lph.y);
                N[r][c] = make_float4(lnl.x, lnl.y, lnh.x, lnh.y);
                acc[0].add(G0.x + G0.y);
                acc[1].add(G1.x + G1.y);
                acc[2].add(G2.x + G2.y);
                acc[3].add(G3.x + G3.y);
                acc[4].add(G4.x + G4.y);
            }
#pragma unroll
            for (int c = 0; c < RJ; ++c) {
                pP[c] = oP[c];
                pN[c] = oN[c];
            }
        }
    };

    int now = 0, pair_now = 0, ring_now = 0;
    for (int s = 0; s < steps; ++s) {
        asm volatile("cp.async.wait_all;" ::: "memory");  // this thread's own states
        __syncthreads();  // mu, the pairs and the ring of this step are in
        if (s_abort) break;
        const float *const cells = cell0 + now;
        now = BUF - now;
        float *const next = cell0 + now;
        const bool last = s + 1 == steps;
        if (a.slot[steps - 1 - s] >= 0) retreat(std::true_type{}, cells, pair0 + pair_now, ring + ring_now, !last);
        else retreat(std::false_type{}, cells, pair0, ring + ring_now, !last);
        fetch_own(s + 1);
        pair_now = ncell - pair_now;
        ring_now = 2 * RING - ring_now;
        if (!all_valid) {
            const int top = a.nzb - 2 - k0;
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
#pragma unroll
        for (int r = 0; r < RI; ++r)
#pragma unroll
            for (int c = 0; c < RJ; ++c)
                if (own >> (r * RJ + c) & 1) {
                    float *const d = next + r * ROW + c * COL;
                    st4s(d, P[r][c]);
                    st4s(d + PITCH, N[r][c]);
                }
        if (trades) {
            __syncthreads();
            if (!last) tile.give(S + now, (uint32_t)(s + 1));
        }
        if (walls && (!MIRROR || last)) {
            // the ring columns beside the patch: lat mu, absorbing added to their own
#pragma unroll
            for (int r = 0; r < RI; ++r)
#pragma unroll
                for (int c = 0; c < RJ; ++c)
                    if (own >> (r * RJ + c) & 1) {
                        const float4 MP = ld4s(cells + r * ROW + c * COL), MN = ld4s(cells + r * ROW + c * COL + PITCH);
                        each_side(r, c, [&](int i, int j, int) {
                            const int64_t o = offset(i, j, k0);
                            float4 RP = make_float4(0.f, 0.f, 0.f, 0.f), RN = RP;
                            if (!MIRROR) {
                                RP = *reinterpret_cast<const float4 *>((s == 0 ? a.lp_in : a.lp_out) + o);
                                RN = *reinterpret_cast<const float4 *>((s == 0 ? a.ln_in : a.ln_out) + o);
                            }
                            const float2 pl = __ffma2_rn(a.p_lat, lo2(MP), lo2(RP)), ph = __ffma2_rn(a.p_lat, hi2(MP), hi2(RP));
                            const float2 nl = __ffma2_rn(a.n_lat, lo2(MN), lo2(RN)), nh = __ffma2_rn(a.n_lat, hi2(MN), hi2(RN));
                            *reinterpret_cast<float4 *>(a.lp_out + o) = make_float4(pl.x, pl.y, ph.x, ph.y);
                            *reinterpret_cast<float4 *>(a.ln_out + o) = make_float4(nl.x, nl.y, nh.x, nh.y);
                        });
                    }
        }
        if (trades && !last && !tile.take(S + now, (uint32_t)(s + 1))) s_abort = 1;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    const bool failed = s_abort != 0;
    if (!failed) {
#pragma unroll
        for (int r = 0; r < RI; ++r)
#pragma unroll
            for (int c = 0; c < RJ; ++c)
                if (own >> (r * RJ + c) & 1) {
                    const int i = i0 + rb + r, j = j0 + cb + c;
                    const int64_t o = offset(i, j, k0);
                    *reinterpret_cast<float4 *>(a.lp_out + o) = P[r][c];
                    *reinterpret_cast<float4 *>(a.ln_out + o) = N[r][c];
                    if (MIRROR && a.lp_out == a.lp_in && (i == 1 || i == n - 2) && (j == 1 || j == n - 2)) {
                        const float4 Z = make_float4(0.f, 0.f, 0.f, 0.f);
                        for (int ii = i == 1 ? 0 : n - 1; ii < n; ii += i == 1 && i == n - 2 ? n - 1 : n)
                            for (int jj = j == 1 ? 0 : n - 1; jj < n; jj += j == 1 && j == n - 2 ? n - 1 : n) {
                                *reinterpret_cast<float4 *>(a.lp_out + offset(ii, jj, k0)) = Z;
                                *reinterpret_cast<float4 *>(a.ln_out + offset(ii, jj, k0)) = Z;
                            }
                    }
                }
    }
    // the block's sums of the launch, into its slot (NaN after a wait that expired)
    DF v[kAdjGrad];
    DF *const red = reinterpret_cast<DF *>(own_u);  // the states are read
    const int lane = tid & 31, warp = tid >> 5;
#pragma unroll
    for (int x = 0; x < kAdjGrad; ++x) {
        v[x] = warp_sum(df_of(acc[x]));
        if (lane == 0) red[warp * kAdjGrad + x] = v[x];
    }
    asm volatile("bar.sync 1, %0;" ::"r"(T) : "memory");  // (the aux warps have left)
    if (tid < kAdjGrad) {
        DF s{0.f, 0.f};
        for (int w = 0; w < T / 32; ++w) s = df_add(s, red[w * kAdjGrad + tid]);
        adj_accumulate(reinterpret_cast<double *>(a.slots + (int64_t)kAdjGrad * blockIdx.x + tid),
                       failed ? DF{__int_as_float(0x7fc00000), 0.f} : s);
    }
}

// Patches and block sizes of the adjoint.
constexpr ResPatch kAdjPatches[] = {{1, 1, 512}, {2, 1, 512}, {2, 2, 384}};

int64_t adj_smem(const ResPlan &p, const ResPatch &pt) {
    const int64_t cells = res_cells(p.gi, p.gj, pt.ri, pt.rj);
    return 4 * ((4 * cells + 3) / 4 * 4 + 4 * 8LL * (p.ti + p.tj) * p.tkv + 8LL * pt.ri * pt.rj * p.threads +
                2 * (2 * cells * res_pitch(kResTkvMax) + 4)) +
           16LL * (2 * (p.ti + p.tj) * p.tkv + 2 * p.ti * p.tj);
}

template <int RI, int RJ, int MAXT, bool MIRROR>
int launch_walled(const AdjResArgs &a, const ResPlan &p, cudaStream_t st) {
    return launch_cooperative(adjoint_resident_kernel<RI, RJ, kResTkvMax, MAXT, MIRROR>, "adjoint_resident_kernel", a, p, st);
}
template <int RI, int RJ, int MAXT>
int launch_patch(const AdjResArgs &a, const ResPlan &p, cudaStream_t st) {
    return a.reflecting ? launch_walled<RI, RJ, MAXT, true>(a, p, st) : launch_walled<RI, RJ, MAXT, false>(a, p, st);
}

}  // namespace

// Taken wherever it fits. Measured, us a reverse step, resident / eight-wide, absorbing
// wall: 10^2 x 56 4.3 / 6.0, 24^2 x 206 4.9 / 6.7, 48^2 x 206 8.2 / 9.5, 28^2 x 406 7.9 / 9.4,
// 20^2 x 606 5.8 / 7.8; near its limits 56^2 x 206 12.5 / 11.1, 108^2 x 56 13.3 / 12.5;
// reflecting (the other one folds the ring in a launch of its own) 4.4 / 8.1, 4.9 /
// 8.6, 8.2 / 11.7, 8.0 / 11.4, 5.8 / 9.4, 11.0 / 12.8, 12.5 / 14.4.
bool resident_adjoint_plan(const pic_grid *g, ResPlan *out) {
    static thread_local ResPlanMemo memo;
    return memo.plan(g, kAdjPatches, (int)(sizeof(kAdjPatches) / sizeof(kAdjPatches[0])), adj_smem, 1.7, out);
}

int launch_resident_adjoint(const pic_grid *g, const ResPlan &p, const void *pos0, const void *neg0, const void *pos,
                            const void *neg, int64_t state_stride, const void *dens, int64_t dens_stride,
                            const int16_t *slot, int steps, const void *lp_in, const void *ln_in, void *lp_out,
                            void *ln_out, double *slots, void *packets, int *status, cudaStream_t st) {
    if (steps < 1 || steps > kResSteps) return set_error(PIC_E_INVALID, "resident adjoint: 1 .. kResSteps steps");
    auto twice = [](float x) { return make_float2(x, x); };
    AdjResArgs a;
    res_shape(g, p, packets, status, &a);
    a.pos0 = static_cast<const float *>(pos0);
    a.neg0 = static_cast<const float *>(neg0);
    a.pos = static_cast<const float *>(pos);
    a.neg = static_cast<const float *>(neg);
    a.state_stride = state_stride;
    a.dens = static_cast<const float2 *>(dens);
    a.dens_stride = dens_stride;
    a.lp_in = static_cast<const float *>(lp_in);
    a.ln_in = static_cast<const float *>(ln_in);
    a.lp_out = static_cast<float *>(lp_out);
    a.ln_out = static_cast<float *>(ln_out);
    a.slots = reinterpret_cast<float2 *>(slots);
    a.dp = (int)dens_pitch(g->no_xy);
    a.steps = steps;
    a.p_lat = twice((float)g->p_lat), a.p_zm = twice((float)g->p_zm), a.p_zp = twice((float)g->p_zp);
    a.p_cen = twice(centre_weight<float>(g->p_lat, g->p_zm, g->p_zp, g->p_cen));
    a.n_lat = twice((float)g->n_lat), a.n_zm = twice((float)g->n_zm), a.n_zp = twice((float)g->n_zp);
    a.n_cen = twice(centre_weight<float>(g->n_lat, g->n_zm, g->n_zp, g->n_cen));
    a.alpha_dt = twice((float)g->alpha_dt);
    a.c_pos = twice((float)(g->p_zm - g->p_zp)), a.c_neg = twice((float)(g->n_zm - g->n_zp));
    int rc = score_test(g, &a.score);
    if (rc) return rc;
    for (int s = 0; s < steps; ++s) a.slot[s] = slot[s];
    switch (p.patch) {
        case 0: return launch_patch<1, 1, kAdjPatches[0].max_threads>(a, p, st);
        case 1: return launch_patch<2, 1, kAdjPatches[1].max_threads>(a, p, st);
        default: return launch_patch<2, 2, kAdjPatches[2].max_threads>(a, p, st);
    }
}

}  // namespace pic
