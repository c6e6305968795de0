// Bounded grid-wide barrier of the persistent cooperative kernels (the propagators).
#pragma once

#include "common.cuh"

namespace paces {

// All blocks are co-resident (cooperative launch).  bar[0] counts arrivals over all barriers of
// the launch (zeroed before it); barrier `gen` is passed when it reaches (gen + 1) * nblocks, so
// an arrival is one atomic and a waiting block only reads.  A wait longer than `limit_ns` raises
// PACES_ERR_TIMEOUT on `status` (if given) and returns false instead of spinning on.  `skip` (a
// test hook) makes this block give up without arriving: it raises the timeout itself, and every
// other block's wait runs out.

// By all lanes of one warp, for a block whose other warps' accesses this warp has synchronised
// with; the caller advances `gen` and synchronises the block afterwards.  Lane 0 acquires the
// other blocks' writes; the warp barrier behind its wait (a shuffle orders no memory) lets every
// lane of the warp read them, as the callers that fold the blocks' values do.
__device__ __forceinline__ bool grid_barrier_warp(unsigned* bar, unsigned nblocks, unsigned gen, int* status,
                                                  uint64_t limit_ns = kWaitLimitNs, bool skip = false) {
    int ok = 1;
    if ((threadIdx.x & 31) == 0) {
        if (skip) {
            raise_status(status, PACES_ERR_TIMEOUT);
            ok = 0;
        } else {
            const unsigned target = (gen + 1) * nblocks;
            asm volatile("fence.acq_rel.gpu;\n\tred.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
            const uint64_t t0 = global_ns();
            unsigned seen;
            for (;;) {
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(bar) : "memory");
                if (int(seen - target) >= 0) break;
                if (global_ns() - t0 > limit_ns) {
                    raise_status(status, PACES_ERR_TIMEOUT);
                    ok = 0;
                    break;
                }
            }
        }
    }
    __syncwarp();
    return __shfl_sync(0xffffffffu, ok, 0) != 0;
}

__device__ __forceinline__ bool grid_barrier(unsigned* bar, unsigned nblocks, unsigned& gen, int* status,
                                             uint64_t limit_ns = kWaitLimitNs, bool skip = false) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x < 32) {
        const bool ok = grid_barrier_warp(bar, nblocks, gen, status, limit_ns, skip);
        if (threadIdx.x == 0) s_ok = ok ? 1 : 0;
    }
    ++gen;
    __syncthreads();
    return s_ok != 0;
}

}  // namespace paces
