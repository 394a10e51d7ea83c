// pic_wide.cuh -- the float32 body of the flat fused step: eight consecutive
// k of one column a thread and pass, shared by the single-grid kernel
// (step.cu) and the batched multi-grid kernel (batched.cu). Semantics as
// flat_item (pic_flat.cuh), which float64 fields, grids beyond 32-bit offsets,
// batched grids whose rows are not 32-byte aligned and the persistent kernels use.
//
// Why eight: decoding an item, its masks, offsets, scoring test and tallies
// cost as much as its stencil, so the four-wide item took 305 instructions for
// four k (428 batched); this one takes about 290 for eight, its arithmetic in
// packed FP32x2, its loads 256 bits wide. 16 warps an SM keep ten such loads each
// in flight (at 96 registers, 20 warps, the loads spill: 25 % slower; at 140, 12
// warps, 10 %). What bounds it: the memory system, not the instructions. With the
// neighbour loads or the arithmetic left out 330^2 x 406 takes the same time
// within 3 %, 119^2 x 406, which stays in the L2, 10-18 % less. Two rows or
// columns a thread (fewer loads a cell), prefetches of the next pass into L2 and
// planes marched in registers measured no faster. Measured on GB300, us a step of
// a segment without tracks, four-wide / here (the tallies' share in pic_internal.h):
// 30^2 x 406 9.6 / 6.2, 61^2 x 606 14.4 / 10.3, 119^2 x 406 26.0 / 19.6, 208^2 x 406
// 60.5 / 53.3, 330^2 x 406 137.5 / 124.2, 608^2 x 406 449 / 412; with 1500 tracks a
// step, their deposition included, 208^2 x 406 68.9 / 59.0. With linked launches
// (pic_device.cuh), absorbing / reflecting wall: 51^2 x 606 6.6 / 6.7, 119^2 x 406 17.3 /
// 17.8, 208^2 x 406 50.8 / 51.4, 330^2 x 406 121 absorbing (the reflecting ring's
// writes as a loop over its eight sides: 6.7 / 7.5, 17.6 / 18.9, 51.2 / 52.0).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "pic_device.cuh"
#include "pic_flat.cuh"
#include "pic_internal.h"

namespace pic {

// Whether the wide body takes a grid's step: 32-bit offsets, 32-byte aligned rows.
inline bool wide_eligible(int64_t n, int64_t kp, const void *a, const void *b, const void *c, const void *d) {
    return flat_index32(n, kp) && kp % 8 == 0 &&
           (((uintptr_t)a | (uintptr_t)b | (uintptr_t)c | (uintptr_t)d) & 31) == 0;
}

struct Oct {
    float2 v[4];  // eight consecutive k
};

// (volatile and coherent: a linked kernel, pic_device.cuh, is resident while its
// input is written, so no load of it may move above wait_for_prev() or take the
// read-only path)
__device__ __forceinline__ Oct load8(const float *p) {
    Oct o;
    asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(o.v[0].x), "=f"(o.v[0].y), "=f"(o.v[1].x), "=f"(o.v[1].y), "=f"(o.v[2].x), "=f"(o.v[2].y),
          "=f"(o.v[3].x), "=f"(o.v[3].y)
        : "l"(p)
        : "memory");
    return o;
}
__device__ __forceinline__ void store8(float *p, const Oct &o) {
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(o.v[0].x), "f"(o.v[0].y),
                 "f"(o.v[1].x), "f"(o.v[1].y), "f"(o.v[2].x), "f"(o.v[2].y), "f"(o.v[3].x), "f"(o.v[3].y)
                 : "memory");
}

// Byte b of m has its sign bit set where the mask holds: spread to the word.
template <int B>
__device__ __forceinline__ uint32_t spread(uint32_t m) {
    uint32_t d;
    asm("prmt.b32 %0, %1, 0, %2;" : "=r"(d) : "r"(m), "n"(0x8888 + 0x1111 * B));
    return d;
}
__device__ __forceinline__ float keep(float v, uint32_t m) { return __uint_as_float(__float_as_uint(v) & m); }
__device__ __forceinline__ float2 keep2(float2 v, const uint32_t *m) { return {keep(v.x, m[0]), keep(v.y, m[1])}; }

// Two running sums side by side as double-floats s + c, each addition Knuth's
// TwoSum in packed operations (a - b as fma(b, -1, a), the same rounding): the
// sums do not depend on how the items fall to threads beyond 2^-44.
struct Tally2 {
    float2 s = {0.f, 0.f}, c = {0.f, 0.f};
    __device__ __forceinline__ void add(float2 v) {
        const float2 m1 = {-1.f, -1.f};
        const float2 t = __fadd2_rn(s, v), z = __ffma2_rn(s, m1, t);
        const float2 e = __ffma2_rn(__ffma2_rn(z, m1, t), m1, s);
        c = __fadd2_rn(c, __fadd2_rn(e, __ffma2_rn(z, m1, v)));
        s = t;
    }
};
__device__ __forceinline__ DF df_of(const Tally2 &t) {
    return df_add(DF{t.s.x, t.c.x}, DF{t.s.y, t.c.y});
}

struct WideTally {
    Tally2 neg_rec, p, n;  // -recombined
    Tally<float> inj;
    __device__ __forceinline__ void store(DF (&v)[4]) const {
        const DF r = df_of(neg_rec);
        v[0] = pic::df_of(inj), v[1] = DF{-r.hi, -r.lo}, v[2] = df_of(p), v[3] = df_of(n);
    }
};

// Thread r of T steps the whole grid's items together with the others: an item
// is eight k of an interior column; the ring's columns follow as items of
// their own (carried with the deposition where the wall absorbs; a reflecting
// wall's are written by the interior columns beside them, their items only
// clear the next step's pairs). With T >= kpitch/8 each thread keeps one k and
// the threads advance T / (kpitch/8) columns a pass, so masks and offsets along
// k are fixed for the whole sweep (fewer than kpitch/8 threads of a launch stay
// idle); else the threads take one column a pass, T vectors of k at a time.
// The launch sweeps one front through the grid: a column's i-1 / i+1
// neighbours are in L2, its j neighbours mostly in L1. Threads of a warp take
// consecutive vectors of a column, so the k neighbours come from the next
// lanes and only the warp's first and last lane read one value more. r is
// 32-aligned per warp; every lane of a warp runs every pass.
__device__ __forceinline__ void wide_sweep(const StepArgs<float> &a, const float *pos_in, const float *neg_in,
                                           float *pos_out, float *neg_out, const float2 *dens, float2 *dens_zero,
                                           uint32_t r, uint32_t T, WideTally &tl) {
    const uint32_t n = (uint32_t)a.n, kp = (uint32_t)a.kp, c8 = kp / 8, dp = (uint32_t)a.dp, di = n * kp, w = n - 2;
    const uint32_t inner = w * w, all = n * n;
    const bool many = T >= c8;
    const uint32_t step = many ? T / c8 : 1;
    const uint32_t step_i = step / w, step_j = step - step_i * w;
    const uint32_t out_step = (step_i * n + step_j) * kp;
    const int lane = threadIdx.x & 31;
    const bool scores = a.score.thr4 >= 0;
    const uint32_t thr = a.score.thr4 >= 0xffffffffLL ? 0xffffffffu : (uint32_t)a.score.thr4;
    const int two_mid = (int)a.score.two_mid;
    const float2 p_lat = {a.p_lat, a.p_lat}, p_cen = {a.p_cen, a.p_cen}, n_lat = {a.n_lat, a.n_lat},
                 n_cen = {a.n_cen, a.n_cen}, nalpha = {-a.alpha_dt, -a.alpha_dt};
    const float p_zm = a.p_zm, p_zp = a.p_zp, n_zm = a.n_zm, n_zp = a.n_zp;

    for (uint32_t pass = 0;; ++pass) {
        const uint32_t col0 = many ? r / c8 : 0;
        uint32_t c = many ? r - col0 * c8 : pass * T + r;
        const bool ok = many ? col0 < step : c < c8;
        if (!__any_sync(0xffffffffu, ok)) return;
        if (!ok) c = c8 - 1;
        const int k0 = (int)(8 * c);
        // masks of the eight outputs: gap layers (deposition, tallies), layers
        // that are stepped (1 .. nzb-2), and the edge lanes' outer neighbour
        uint32_t g_lo = 0, g_hi = 0, v_lo = 0, v_hi = 0;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const uint32_t bit = 0x80u << (8 * e);
            const int k = k0 + e, q = k0 + 4 + e;
            g_lo |= (k >= a.nze && k < a.gap_end) ? bit : 0u;
            g_hi |= (q >= a.nze && q < a.gap_end) ? bit : 0u;
            v_lo |= (k >= 1 && k <= a.nzb - 2) ? bit : 0u;
            v_hi |= (q >= 1 && q <= a.nzb - 2) ? bit : 0u;
        }
        const bool ends = (v_lo & v_hi) != 0x80808080u;
        const int ke = lane == 0 ? k0 - 1 : k0 + 8;
        const uint32_t g_edge = (ke >= a.nze && ke < a.gap_end) ? 0xffffffffu : 0u;
        const bool edge_lane = lane == 0 || lane == 31;
        const uint32_t edge_off = lane == 0 ? 0xffffffffu : 8u;

        uint32_t v = ok ? col0 : all;
        uint32_t i = ok ? 1 + col0 / w : 1, j = ok ? 1 + col0 - (i - 1) * w : 1;
        uint32_t at = (i * n + j) * kp + (uint32_t)k0;
        while (__any_sync(0xffffffffu, v < inner)) {
            const bool act = v < inner;
            const uint32_t base = act ? at : n * kp + kp + (uint32_t)k0;  // (column (1, 1) for a lane without one)
            const uint32_t dcol = act ? i * dp + j : dp + 1;
            float2 d = {0.f, 0.f};
            if (dens) d = dens[dcol];  // (in flight with the fields)
            Oct P = load8(pos_in + base), N = load8(neg_in + base);
            const Oct Pim = load8(pos_in + (base - di)), Pip = load8(pos_in + (base + di));
            const Oct Pjm = load8(pos_in + (base - kp)), Pjp = load8(pos_in + (base + kp));
            const Oct Nim = load8(neg_in + (base - di)), Nip = load8(neg_in + (base + di));
            const Oct Njm = load8(neg_in + (base - kp)), Njp = load8(neg_in + (base + kp));
            float ep = 0.f, en = 0.f;
            if (edge_lane) {
                ep = pos_in[base + edge_off];
                en = neg_in[base + edge_off];
            }
            Oct LP, LN;
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                LP.v[h] = __fadd2_rn(__fadd2_rn(Pjm.v[h], Pjp.v[h]), __fadd2_rn(Pim.v[h], Pip.v[h]));
                LN.v[h] = __fadd2_rn(__fadd2_rn(Njm.v[h], Njp.v[h]), __fadd2_rn(Nim.v[h], Nip.v[h]));
            }
            const uint32_t m[8] = {spread<0>(g_lo), spread<1>(g_lo), spread<2>(g_lo), spread<3>(g_lo),
                                   spread<0>(g_hi), spread<1>(g_hi), spread<2>(g_hi), spread<3>(g_hi)};
            if (dens) {
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    const float2 dch = keep2(float2{d.x, d.x}, m + 2 * h), dlh = keep2(float2{d.y, d.y}, m + 2 * h);
                    P.v[h] = __fadd2_rn(P.v[h], dch);
                    N.v[h] = __fadd2_rn(N.v[h], dch);
                    LP.v[h] = __fadd2_rn(LP.v[h], dlh);
                    LN.v[h] = __fadd2_rn(LN.v[h], dlh);
                }
                const float de = keep(d.x, g_edge);
                ep += de;
                en += de;
            }
            // (a lane whose neighbour in the warp is another column's end
            // takes any value there: its own end layer is not stepped)
            float pkm = __shfl_up_sync(0xffffffffu, P.v[3].y, 1), nkm = __shfl_up_sync(0xffffffffu, N.v[3].y, 1);
            float pkp = __shfl_down_sync(0xffffffffu, P.v[0].x, 1), nkp = __shfl_down_sync(0xffffffffu, N.v[0].x, 1);
            if (lane == 0) pkm = ep, nkm = en;
            if (lane == 31) pkp = ep, nkp = en;
            const float pk[10] = {pkm,      P.v[0].x, P.v[0].y, P.v[1].x, P.v[1].y,
                                  P.v[2].x, P.v[2].y, P.v[3].x, P.v[3].y, pkp};
            const float nk[10] = {nkm,      N.v[0].x, N.v[0].y, N.v[1].x, N.v[1].y,
                                  N.v[2].x, N.v[2].y, N.v[3].x, N.v[3].y, nkp};
            float2 R[4];
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                R[h] = __fmul2_rn(__fmul2_rn(nalpha, P.v[h]), N.v[h]);  // -recombined
                float2 p = __fmul2_rn(p_lat, LP.v[h]), q = __fmul2_rn(n_lat, LN.v[h]);
                p.x = fmaf(p_zm, pk[2 * h], fmaf(p_zp, pk[2 * h + 2], p.x));
                p.y = fmaf(p_zm, pk[2 * h + 1], fmaf(p_zp, pk[2 * h + 3], p.y));
                q.x = fmaf(n_zm, nk[2 * h + 2], fmaf(n_zp, nk[2 * h], q.x));
                q.y = fmaf(n_zm, nk[2 * h + 3], fmaf(n_zp, nk[2 * h + 1], q.y));
                LP.v[h] = __fadd2_rn(__ffma2_rn(p_cen, P.v[h], p), R[h]);
                LN.v[h] = __fadd2_rn(__ffma2_rn(n_cen, N.v[h], q), R[h]);
            }
            if (ends) {
                const uint32_t u[8] = {spread<0>(v_lo), spread<1>(v_lo), spread<2>(v_lo), spread<3>(v_lo),
                                       spread<0>(v_hi), spread<1>(v_hi), spread<2>(v_hi), spread<3>(v_hi)};
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    LP.v[h] = keep2(LP.v[h], u + 2 * h);
                    LN.v[h] = keep2(LN.v[h], u + 2 * h);
                }
            }
            if (act) {
                const int dx = 2 * (int)i - two_mid, dy = 2 * (int)j - two_mid;
                if (scores && (uint32_t)(dx * dx) + (uint32_t)(dy * dy) <= thr) {
                    float2 sr[4], sp[4], sn[4];
#pragma unroll
                    for (int h = 0; h < 4; ++h) {
                        sr[h] = keep2(R[h], m + 2 * h);
                        sp[h] = keep2(LP.v[h], m + 2 * h);
                        sn[h] = keep2(LN.v[h], m + 2 * h);
                    }
                    tl.neg_rec.add(__fadd2_rn(__fadd2_rn(sr[0], sr[1]), __fadd2_rn(sr[2], sr[3])));
                    tl.p.add(__fadd2_rn(__fadd2_rn(sp[0], sp[1]), __fadd2_rn(sp[2], sp[3])));
                    tl.n.add(__fadd2_rn(__fadd2_rn(sn[0], sn[1]), __fadd2_rn(sn[2], sn[3])));
                    if (k0 == 0 && dens) tl.inj.add(d.x);
                }
                store8(pos_out + base, LP);
                store8(neg_out + base, LN);
                if (k0 == 0 && dens_zero) dens_zero[dcol] = float2{0.f, 0.f};
                if (a.reflecting) {
                    // the ring columns whose nearest interior column this is
                    const bool up = i == 1, down = i == w, left = j == 1, right = j == w;
                    auto ring = [&](uint32_t o) {
                        store8(pos_out + o, LP);
                        store8(neg_out + o, LN);
                    };
                    if (up) ring(base - di);
                    if (down) ring(base + di);
                    if (left || right) {
                        if (left) ring(base - kp);
                        if (right) ring(base + kp);
                        if (up && left) ring(base - di - kp);
                        if (up && right) ring(base - di + kp);
                        if (down && left) ring(base + di - kp);
                        if (down && right) ring(base + di + kp);
                    }
                }
                v += step;
                at += out_step;
                i += step_i;
                j += step_j;
                if (j > w) j -= w, ++i, at += 2 * kp;
            }
        }
        if (a.reflecting && !dens_zero) v = all;
        for (; v < all; v += step) {
            const uint32_t u = v - inner;  // ring: row 0, row n-1, then the two ends of each row between
            if (u < 2 * n) i = u < n ? 0 : n - 1, j = u < n ? u : u - n;
            else i = 1 + (u - 2 * n) / 2, j = (u & 1) ? n - 1 : 0;
            if (!a.reflecting) {
                const uint32_t o = (i * n + j) * kp + (uint32_t)k0;
                Oct P = load8(pos_in + o), N = load8(neg_in + o);
                if (dens) {
                    const float d = dens[i * dp + j].x;
                    const uint32_t m[8] = {spread<0>(g_lo), spread<1>(g_lo), spread<2>(g_lo), spread<3>(g_lo),
                                           spread<0>(g_hi), spread<1>(g_hi), spread<2>(g_hi), spread<3>(g_hi)};
#pragma unroll
                    for (int h = 0; h < 4; ++h) {
                        const float2 dh = keep2(float2{d, d}, m + 2 * h);
                        P.v[h] = __fadd2_rn(P.v[h], dh);
                        N.v[h] = __fadd2_rn(N.v[h], dh);
                    }
                }
                store8(pos_out + o, P);
                store8(neg_out + o, N);
            }
            if (k0 == 0 && dens_zero) dens_zero[i * dp + j] = float2{0.f, 0.f};
        }
        if (many) return;
    }
}

}  // namespace pic
