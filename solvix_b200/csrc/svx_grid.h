// svx_grid.h - the bounded grid-wide barrier of the cooperative kernels
// (the persistent PCG kernels, the direct path's substitution kernel).
// Device code: included by the .cu units only.
#ifndef SVX_GRID_H
#define SVX_GRID_H
#ifdef __CUDACC__

#include "svx_internal.h"
#include "svx_warp.h"

namespace svx {

// polls of a grid barrier before it gives up (about a second)
constexpr long long BARRIER_SPIN_LIMIT = 1LL << 25;
// back-off between two polls of a grid barrier's arrival count
#ifndef SVX_BARRIER_SLEEP_NS
#define SVX_BARRIER_SLEEP_NS 32
#endif

// Bounded grid-wide barrier (all blocks co-resident: cooperative launch).
// gb->count only grows during a launch (the host zeroes it before each
// launch); every block keeps its own running target, nblocks more per
// barrier.  After bar.sync, thread 0 arrives with a gpu-scope release add
// (cumulative over the block's writes ordered before it by the bar.sync)
// and polls with acquire loads until the count reaches the target; the
// closing bar.sync passes that on to the block.  A block that polls
// spin_limit times raises gb->error and returns false, and so does a block
// that finds the flag raised by another while it waits.
__device__ __forceinline__ void barrier_arrive(unsigned int* p) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(p) : "memory");
}
__device__ __forceinline__ unsigned int barrier_count(const unsigned int* p) {
    unsigned int v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ bool grid_sync(GridBarrier* gb, unsigned int nblocks,
                                          unsigned int& target,
                                          long long spin_limit = BARRIER_SPIN_LIMIT) {
    __shared__ int ok;
    target += nblocks;
    __syncthreads();
    if (threadIdx.x == 0) {
        int good = 1;
        barrier_arrive(&gb->count);
        long long spins = 0;
        while (barrier_count(&gb->count) < target) {
            if (++spins > spin_limit) {
                atomicExch(&gb->error, 1);
                good = 0;
                break;
            }
            if ((spins & 255) == 0 && *((volatile int*)&gb->error) != 0) {
                good = 0;
                break;
            }
#if SVX_BARRIER_SLEEP_NS > 0
            __nanosleep(SVX_BARRIER_SLEEP_NS);
#endif
        }
        ok = good;
    }
    __syncthreads();
    return ok != 0;
}

// Sums of (a, b) over the grid, the same bits in every thread: warp sums on
// the tensor cores, the block's pair to `pt` (one pair a block, 16-byte
// aligned), the barrier, and one warp reads the other blocks' pairs (read by
// all warps of 148 blocks their few cache lines are a hot spot of the L2).
// sh: 66 doubles.  The reductions of an iteration use different `pt`: a block
// past the first one's barrier may publish its next pair while a late block
// still reads this one; with a barrier between two uses of a `pt` no block can
// overwrite what another still reads.
__device__ __forceinline__ bool grid_pair_sum(GridBarrier* gb, unsigned int nblocks,
                                              unsigned int& target, double* pt, double* sh,
                                              double a, double b, double& ta, double& tb) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = int(blockDim.x) >> 5;
    const double v = lane_sum_pair(a, b, lane);
    if ((lane & 15) == 0) sh[2 * warp + (lane >> 4)] = v;
    __syncthreads();
    if (warp == 0) {
        const double w = lane_sum_pair(lane < warps ? sh[2 * lane] : 0.0,
                                       lane < warps ? sh[2 * lane + 1] : 0.0, lane);
        if ((lane & 15) == 0) pt[2 * blockIdx.x + (lane >> 4)] = w;
    }
    if (!grid_sync(gb, nblocks, target)) return false;
    if (warp == 0) {
        double x = 0.0, y = 0.0;
        for (int k = lane; k < int(nblocks); k += 32) {
            const double2 w = __ldcg(reinterpret_cast<const double2*>(pt) + k);
            x += w.x;
            y += w.y;
        }
        x = lane_sum(x);
        y = lane_sum(y);
        if (lane == 0) {
            sh[64] = x;
            sh[65] = y;
        }
    }
    __syncthreads();
    ta = sh[64];
    tb = sh[65];
    return true;
}

}  // namespace svx

#endif  // __CUDACC__
#endif  // SVX_GRID_H
