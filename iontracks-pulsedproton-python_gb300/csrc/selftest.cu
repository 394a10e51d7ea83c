// selftest.cu -- the bounded waits of the kernels, run against partners that
// never come, so that a test can check on the GPU that an expired wait
// returns an error status and leaves the context usable (no fault, no hang).
//
// barrier: two blocks; block 1 leaves at once, block 0 waits at the
//   device-wide barrier of the persistent and multi-step kernels
//   (pic_barrier.cuh) with a short poll limit;
// mbarrier: one block initialises an mbarrier that nothing arrives on and
//   waits on its first phase with the streaming kernels' bounded wait
//   (pic_async.cuh), with a short try-wait limit;
// packets: the resident step and its adjoint without the last block of their
//   division, whose packets never come: the blocks beside it give up after
//   kPacketPolls rounds, the others when they see the status. (What a block
//   would read of the missing one's lies inside the packet buffer of the whole
//   division and is zero or of the other parity, so no tag of it matches.)
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>

#include "pic_adjoint.cuh"
#include "pic_async.cuh"
#include "pic_barrier.cuh"
#include "pic_internal.h"

namespace pic {

namespace {

constexpr long long kSelftestPolls = 1LL << 12;
constexpr int kSelftestMbarCode = 91;

__global__ void selftest_barrier_kernel(unsigned int *count, unsigned int *gen, int *status) {
    if (blockIdx.x == 1) return;  // the partner that never arrives
    grid_barrier(BarrierRef{count, gen, status}, kSelftestPolls);
}

__global__ void selftest_mbarrier_kernel(int *status) {
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        mbar_fence_init();
    }
    __syncthreads();
    if (threadIdx.x == 0) mbar_wait(&bar, 0u, status, kSelftestMbarCode, kSelftestPolls);
}

}  // namespace

int selftest_waits(int32_t *barrier_status, int32_t *mbarrier_status, cudaStream_t st) {
    // [count, gen, barrier status, mbarrier status]
    int *d = nullptr;
    cudaError_t e = cudaMallocAsync(reinterpret_cast<void **>(&d), 4 * sizeof(int), st);
    if (e != cudaSuccess) return set_cuda_error("cudaMallocAsync(selftest)", e);
    int host[4] = {0, 0, 0, 0};
    e = cudaMemsetAsync(d, 0, 4 * sizeof(int), st);
    if (e == cudaSuccess) {
        selftest_barrier_kernel<<<2, 32, 0, st>>>(reinterpret_cast<unsigned int *>(d),
                                                  reinterpret_cast<unsigned int *>(d + 1), d + 2);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) {
        selftest_mbarrier_kernel<<<1, 32, 0, st>>>(d + 3);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(host, d, sizeof(host), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    cudaFreeAsync(d, st);
    if (e != cudaSuccess) return set_cuda_error("selftest_waits", e);
    *barrier_status = host[2];
    *mbarrier_status = host[3];
    return PIC_OK;
}

int selftest_packets(const pic_grid *g, int32_t *step_status, int32_t *adjoint_status, int32_t *poisoned,
                     cudaStream_t st) {
    constexpr int kSteps = 64;  // more than a division's blocks along an axis: all of them come to wait
    constexpr int kMaxBlocks = 256;
    ResPlan p, adj;
    if (!resident_plan(g, &p) || p.blocks < 3 || p.blocks > kMaxBlocks)
        return set_error(PIC_E_INVALID, "the grid does not run resident in 3 to 256 blocks");
    const bool has_adj = resident_adjoint_plan(g, &adj) && adj.blocks >= 3 && adj.blocks <= kMaxBlocks;
    int64_t packets = 2LL * p.blocks * p.packets * 16;
    if (has_adj) packets = std::max<int64_t>(packets, 2LL * adj.blocks * adj.packets * 16);
    const int64_t field = g->no_xy * g->no_xy * g->kpitch * 4, partials = (int64_t)kSteps * p.blocks * p.aux;
    const int64_t slots = (int64_t)kMaxBlocks * kAdjGrad * 8;
    char *d = nullptr;
    cudaError_t e = cudaMallocAsync(reinterpret_cast<void **>(&d), (size_t)(4 * field + packets + partials + slots + 8), st);
    if (e != cudaSuccess) return set_cuda_error("cudaMallocAsync(selftest)", e);
    char *const pk = d + 4 * field, *const part = pk + packets, *const sl = part + partials;
    int *const status = reinterpret_cast<int *>(sl + slots);
    int host[2] = {0, 0};
    float2 sums[kMaxBlocks * kAdjGrad];
    int16_t slot[kSteps];
    std::fill(slot, slot + kSteps, (int16_t)-1);
    int rc = PIC_OK;
    e = cudaMemsetAsync(d, 0, (size_t)(4 * field + packets + partials + slots + 8), st);
    if (e == cudaSuccess) {
        --p.blocks;
        rc = launch_resident(g, p, d, d + field, d + 2 * field, d + 3 * field, nullptr, 0, slot, kSteps, 0, nullptr, pk,
                             part, status, st);
    }
    if (e == cudaSuccess && rc == PIC_OK && has_adj) {
        --adj.blocks;
        e = cudaMemsetAsync(pk, 0, (size_t)packets, st);
        if (e == cudaSuccess)
            rc = launch_resident_adjoint(g, adj, d, d + field, d, d + field, 0, nullptr, 0, slot, kSteps, d, d + field,
                                         d + 2 * field, d + 3 * field, reinterpret_cast<double *>(sl), pk, status + 1, st);
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(host, status, sizeof(host), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(sums, sl, (size_t)slots, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    cudaFreeAsync(d, st);
    if (rc) return rc;
    if (e != cudaSuccess) return set_cuda_error("selftest_packets", e);
    *step_status = host[0];
    *adjoint_status = has_adj ? host[1] : -1;
    *poisoned = 0;
    for (int b = 0; has_adj && b < adj.blocks; ++b) {
        bool all = true;
        for (int q = 0; q < kAdjGrad; ++q) all = all && isnan(sums[b * kAdjGrad + q].x);
        *poisoned += all;
    }
    if (has_adj) *poisoned = *poisoned == adj.blocks;
    return PIC_OK;
}

}  // namespace pic
