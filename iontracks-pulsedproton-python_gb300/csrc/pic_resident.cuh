// pic_resident.cuh -- what the resident kernels share (resident.cu: the step;
// adjoint_resident.cu: its adjoint): how a block finds its box of the grid,
// and how it trades the faces of its cells with the blocks around it.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <mutex>
#include <type_traits>

#include "pic_device.cuh"
#include "pic_flat.cuh"
#include "pic_internal.h"
#include "pic_packet.cuh"

namespace pic {

__device__ __forceinline__ float4 ld4s(const float *p) { return *reinterpret_cast<const float4 *>(p); }
__device__ __forceinline__ void st4s(float *p, float4 v) { *reinterpret_cast<float4 *>(p) = v; }
__device__ __forceinline__ float masked(float x, uint32_t m) { return __uint_as_float(__float_as_uint(x) & m); }

// Offsets of a block's six faces in its packet region. A lateral face holds
// [packet][column][k-vector], three packets an item (i_side or j_side apart);
// a k face one packet a column.
struct Faces {
    int i_side, j_side, im, ip, jm, jp, km, kp, total;
};
__host__ __device__ inline Faces res_faces(int ti, int tj, int tkv) {
    Faces f;
    f.i_side = tj * tkv;
    f.j_side = ti * tkv;
    f.im = 0;
    f.ip = f.im + 3 * f.i_side;
    f.jm = f.ip + 3 * f.i_side;
    f.jp = f.jm + 3 * f.j_side;
    f.km = f.jp + 3 * f.j_side;
    f.kp = f.km + ti * tj;
    f.total = f.kp + ti * tj;
    return f;
}

__device__ __forceinline__ void send_item(uint4 *p, int side, float4 P, float4 N, uint32_t tag) {
    packet_store(p, __float_as_uint(P.x), __float_as_uint(P.y), __float_as_uint(P.z), tag);
    packet_store(p + side, __float_as_uint(P.w), __float_as_uint(N.x), __float_as_uint(N.y), tag);
    packet_store(p + 2 * side, __float_as_uint(N.z), __float_as_uint(N.w), 0u, tag);
}

// The grid and its division over the blocks (ResPlan).
struct ResShape {
    uint4 *packets;  // [2][blocks][Faces::total]
    int *status;
    int n, kp, c4, nzb, nze, gap_end, reflecting;
    int nti, ntj, ntk, ti, tj, tkv, gi, gj;
    int patch_threads, aux_threads;  // the roles of a block's threads, in this order
};
inline void res_shape(const pic_grid *g, const ResPlan &p, void *packets, int *status, ResShape *a) {
    a->packets = static_cast<uint4 *>(packets);
    a->status = status;
    a->n = (int)g->no_xy;
    a->kp = (int)g->kpitch;
    a->c4 = a->kp / 4;
    a->nzb = (int)g->nzb;
    a->nze = (int)g->nze;
    a->gap_end = (int)(g->nze + g->no_z);
    a->reflecting = g->wall == PIC_WALL_REFLECTING;
    a->nti = p.nti, a->ntj = p.ntj, a->ntk = p.ntk;
    a->ti = p.ti, a->tj = p.tj, a->tkv = p.tkv, a->gi = p.gi, a->gj = p.gj;
    a->patch_threads = p.threads, a->aux_threads = p.aux;
}

// (four floats between two rows of k: the one above the lower row's end, ..,
// the one below the next row's start; 120 floats a column, so that the lanes
// of a warp that go on into the next column of 13 or 14 k-vectors also go on
// through the banks)
__host__ __device__ constexpr int res_pitch(int tkv_max) { return 4 * tkv_max + 4; }
// columns of a block's cells, one more on each side of its patches
__host__ __device__ inline int res_cells(int gi, int gj, int RI, int RJ) { return (gi * RI + 2) * (gj * RJ + 2); }

// A block's box of the grid: interior columns [i0, i0 + rows) x [j0, j0 + cols)
// and k-vectors [kv0, kv0 + kvn), its cells in shared memory
// ([row][column][species][4 + 4 TKV], PITCH floats a species, from row and
// column -1 to one past the patches) and its neighbours.
template <int PITCH>
struct ResTile {
    static constexpr int COL = 2 * PITCH;
    const ResShape &a;
    int cta, bk, i0, j0, kv0, rows, cols, kvn, W;
    bool lo_i, hi_i, lo_j, hi_j, lo_k, hi_k;  // a block beyond that face
    Faces F;
    int64_t region;                 // packets of one parity of steps
    int n_side, n_around;           // columns beside the block; with its corners
    int h_im, h_jm, h_km, h_i, h_lat, h_k;  // items traded: i-, j-, k-, both i, all lateral, all k
    int4 *trade;

    __device__ __forceinline__ ResTile(const ResShape &a_, int W_) : a(a_), W(W_) {
        cta = blockIdx.x;
        bk = cta % a.ntk;
        const int bj = (cta / a.ntk) % a.ntj, bi = cta / (a.ntk * a.ntj);
        i0 = 1 + bi * a.ti, j0 = 1 + bj * a.tj, kv0 = bk * a.tkv;
        rows = min(a.ti, a.n - 1 - i0), cols = min(a.tj, a.n - 1 - j0), kvn = min(a.tkv, a.c4 - kv0);
        lo_i = bi > 0, hi_i = bi + 1 < a.nti, lo_j = bj > 0, hi_j = bj + 1 < a.ntj;
        lo_k = bk > 0, hi_k = bk + 1 < a.ntk;
        F = res_faces(a.ti, a.tj, a.tkv);
        region = (int64_t)gridDim.x * F.total;
        n_side = 2 * cols + 2 * rows, n_around = n_side + 4;
        h_im = lo_i ? cols * kvn : 0, h_jm = lo_j ? rows * kvn : 0, h_km = lo_k ? rows * cols : 0;
        h_i = h_im + (hi_i ? cols * kvn : 0);
        h_lat = h_i + h_jm + (hi_j ? rows * kvn : 0);
        h_k = h_km + (hi_k ? rows * cols : 0);
    }
    __device__ __forceinline__ int cell_of(int r, int c) const { return ((r + 1) * W + c + 1) * COL + 4; }

    // The columns around the block: the sides i-, i+, j-, j+, then the corners.
    __device__ __forceinline__ void around(int u, int &r, int &c) const {
        if (u < cols) r = -1, c = u;
        else if (u < 2 * cols) r = rows, c = u - cols;
        else if (u < 2 * cols + rows) c = -1, r = u - 2 * cols;
        else if (u < n_side) c = cols, r = u - 2 * cols - rows;
        else r = (u - n_side) & 1 ? rows : -1, c = (u - n_side) & 2 ? cols : -1;
    }
    // Whether column u of them is a ring column this block keeps (a corner of
    // the block is one where it is the grid's corner).
    __device__ __forceinline__ bool ring_col(int u, int r, int c) const {
        const int i = i0 + r, j = j0 + c;
        return (i == 0 || i == a.n - 1) + (j == 0 || j == a.n - 1) >= (u < n_side ? 1 : 2);
    }

    // What the block trades: lateral item u of trade[] is a cell of the block's
    // edge, sent, and the cell beyond it, taken in; item h_lat + u the same of
    // the k faces (one element). x: its packet to send, y: to take, z and w:
    // the cells from and to (lateral: z both, in units of four floats; w the
    // distance of its three packets).
    __device__ __forceinline__ void table(int4 *at) {
        trade = at;
        for (int q = threadIdx.x; q < h_lat; q += blockDim.x) {
            int u = q, nb, own_face, its_face, r, c, dr = 0, dc = 0, along;
            if (u < h_i) {
                const bool up = u >= h_im;
                if (up) u -= h_im;
                c = along = u / kvn, u -= c * kvn;
                r = up ? rows - 1 : 0, dr = up ? 1 : -1;
                nb = dr * a.ntj * a.ntk, own_face = up ? F.ip : F.im, its_face = up ? F.im : F.ip;
            } else {
                u -= h_i;
                const bool up = u >= h_jm;
                if (up) u -= h_jm;
                r = along = u / kvn, u -= r * kvn;
                c = up ? cols - 1 : 0, dc = up ? 1 : -1;
                nb = dc * a.ntk, own_face = up ? F.jp : F.jm, its_face = up ? F.jm : F.jp;
            }
            const int o = along * a.tkv + u;
            trade[q] = make_int4(cta * F.total + own_face + o, (cta + nb) * F.total + its_face + o,
                                 (cell_of(r, c) / 4 + u) | (cell_of(r + dr, c + dc) / 4 + u) << 16, dr ? F.i_side : F.j_side);
        }
        for (int q = threadIdx.x; q < h_k; q += blockDim.x) {
            const bool up = q >= h_km;
            const int u = up ? q - h_km : q, r = u / cols, c = u - r * cols, o = r * a.tj + c, d = cell_of(r, c);
            trade[h_lat + q] = make_int4(cta * F.total + (up ? F.kp : F.km) + o, (cta + (up ? 1 : -1)) * F.total + (up ? F.km : F.kp) + o,
                                         d + (up ? 4 * kvn - 1 : 0), d + (up ? 4 * kvn : -1));
        }
    }

    // Sends the block's face cells of the step that gives `tag`.
    __device__ __forceinline__ void give(const float *B, uint32_t tag) const {
        const int tid = threadIdx.x, T = a.patch_threads;
        uint4 *const out = a.packets + (tag & 1 ? region : 0);
#pragma unroll 1
        for (int u = tid; u < h_lat; u += T) {
            const int4 e = trade[u];
            const float *d = B + (e.z & 0xffff) * 4;
            send_item(out + e.x, e.w, ld4s(d), ld4s(d + PITCH), tag);
        }
#pragma unroll 1
        for (int u = tid; u < h_k; u += T) {
            const int4 e = trade[h_lat + u];
            packet_store(out + e.x, __float_as_uint(B[e.z]), __float_as_uint(B[e.z + PITCH]), 0u, tag);
        }
    }
    // Takes in the cells beyond them; false when they did not come. A thread
    // polls for LAT lateral items and K k items at once, from items u and v on,
    // every T-th; past the last one it takes that one again (the same values).
    template <int LAT, int KS>
    __device__ __forceinline__ bool take_some(const uint4 *in, float *B, uint32_t tag, int u, int v) const {
        const int T = a.patch_threads;
        const uint4 *p[LAT + 1], *pk = nullptr;
        int side[LAT + 1], d[LAT + 1], dk = 0;
#pragma unroll
        for (int x = 0; x < LAT; ++x) {
            const int4 e = trade[min(u + x * T, h_lat - 1)];
            p[x] = in + e.y, side[x] = e.w, d[x] = (int)((unsigned)e.z >> 16) * 4;
        }
        if (KS) {
            const int4 e = trade[h_lat + min(v, h_k - 1)];
            pk = in + e.y, dk = e.w;
        }
        uint4 V[LAT + 1][3], K;
        for (int polls = 0;; ++polls) {
#pragma unroll
            for (int x = 0; x < LAT; ++x)
#pragma unroll
                for (int y = 0; y < 3; ++y) V[x][y] = packet_load(p[x] + y * side[x]);
            if (KS) K = packet_load(pk);
            uint32_t off = KS ? K.w ^ tag : 0u;
#pragma unroll
            for (int x = 0; x < LAT; ++x) off |= (V[x][0].w ^ tag) | (V[x][1].w ^ tag) | (V[x][2].w ^ tag);
            if (off == 0) break;
            if ((polls & 1023) == 1023 && (polls > kPacketPolls || *reinterpret_cast<volatile int *>(a.status) != 0)) {
                atomicCAS(a.status, 0, kPacketTimeout);
                return false;
            }
        }
#pragma unroll
        for (int x = 0; x < LAT; ++x) {
            st4s(B + d[x], make_float4(__uint_as_float(V[x][0].x), __uint_as_float(V[x][0].y),
                                       __uint_as_float(V[x][0].z), __uint_as_float(V[x][1].x)));
            st4s(B + d[x] + PITCH, make_float4(__uint_as_float(V[x][1].y), __uint_as_float(V[x][1].z),
                                               __uint_as_float(V[x][2].x), __uint_as_float(V[x][2].y)));
        }
        if (KS) {
            B[dk] = __uint_as_float(K.x);
            B[dk + PITCH] = __uint_as_float(K.y);
        }
        return true;
    }
    __device__ __forceinline__ bool take(float *B, uint32_t tag) const {
        const int T = a.patch_threads;
        const uint4 *const in = a.packets + (tag & 1 ? region : 0);
        int u = threadIdx.x, v = u, left = h_lat, left_k = h_k;  // the block's items still to take
        bool ok = true;
        if (left > 0 && left_k > 0)
            ok = left > T ? take_some<2, 1>(in, B, tag, u, v) : take_some<1, 1>(in, B, tag, u, v),
            u += 2 * T, v += T, left -= 2 * T, left_k -= T;
        for (; ok && left > 0; u += 2 * T, left -= 2 * T) ok = take_some<2, 0>(in, B, tag, u, v);
        for (; ok && left_k > 0; v += T, left_k -= T) ok = take_some<0, 1>(in, B, tag, u, v);
        return ok;
    }
};

// A patch of columns a thread may own, with the most threads a block of them
// may have, and the longest k range of a block.
struct ResPatch {
    int ri, rj, max_threads;
};
constexpr int kResTkvMax = 14;

// The division of a grid over blocks of one kernel's patches (smem: the bytes
// of shared memory a division takes; item_scale: what an item costs against
// the step's). A segment asks for its grid's plan again and again: the last
// one is kept (it depends on the grid's size and the SM count alone).
using ResSmem = int64_t (*)(const ResPlan &, const ResPatch &);
struct ResPlanMemo {
    int M = 0, c4 = 0, sms = 0;
    bool fits = false;
    ResPlan last{};
    bool plan(const pic_grid *g, const ResPatch *patches, int count, ResSmem smem_of, double item_scale, ResPlan *out);
};

// Launches a resident kernel: cooperative, since its blocks wait on one another.
template <typename K, typename A>
int launch_cooperative(K kernel, const char *name, const A &args, const ResPlan &p, cudaStream_t st) {
    static std::mutex mu;  // one per kernel type and so shared by its instances: the limit is set for each pointer
    static const void *known[64] = {nullptr};
    static int configured[64][64] = {{0}};  // [kernel][device]: largest dynamic shared memory set so far
    {
        int dev = 0, slot = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e != cudaSuccess) return set_cuda_error("cudaGetDevice", e);
        std::lock_guard<std::mutex> lock(mu);
        const void *f = reinterpret_cast<const void *>(kernel);
        while (slot < 63 && known[slot] && known[slot] != f) ++slot;
        known[slot] = f;
        if (dev < 0 || dev >= 64 || slot == 63 || p.smem > configured[slot][dev]) {
            e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, p.smem);
            if (e != cudaSuccess) return set_cuda_error(name, e);
            if (dev >= 0 && dev < 64) configured[slot][dev] = p.smem;
        }
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)p.blocks);
    cfg.blockDim = dim3((unsigned)(p.threads + p.aux));
    cfg.dynamicSmemBytes = (size_t)p.smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, args);
    if (e != cudaSuccess) return set_cuda_error(name, e);
    count_launches(1);
    return PIC_OK;
}

}  // namespace pic
