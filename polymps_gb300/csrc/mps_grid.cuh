// mps_grid.cuh — grid barriers and grid-wide sums inside one cooperative launch.
//
// A block stores its partials, adds one to a 64-bit arrival counter (release) and one lane
// polls the counter; then warp 0 of every block reads all blocks' partials itself, so no block
// publishes a result and releases the others.  The poll is a relaxed load without back-off
// and one fence follows it (an acquire load per poll, with a sleep between polls, measured
// 2.64 us a sum over 152 blocks of 1024 threads; this form 1.65 us).  Carrying the partials in
// tagged 16-byte slots that every block polls saves the second trip to the L2 at 2 blocks
// (1.07 us) but 152 x 152 polled slots contend: 4.1 us.  Clusters of 2 to 16 blocks summing
// through distributed shared memory first measured 2.3 to 3.3 us, and clusters above 2 do
// not cover the 152 SMs.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#define GRID_SPIN (1 << 22)   // polls of the counter before a wait gives up (about two seconds)
#define GRID_NV 4             // values of one sum at most
#define GRID_PER_LANE 8       // partials a lane of warp 0 reads: up to 256 blocks

struct GridBar {
    unsigned long long* arrivals;   // zeroed before the launch
    unsigned int* abortWord;        // zeroed before the launch; set when a wait ran out
    unsigned int gen;               // barriers passed (the same in every thread)
};

__device__ __forceinline__ unsigned long long ldRelaxed(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
// Arrival and wait of warp 0, after a __syncthreads of the block: the block's writes before
// that are visible to every block's reads after its own wait.  True in every lane when all
// blocks arrived, false when the (bounded) wait ran out here or in another block.
__device__ __forceinline__ bool gridWaitWarp0(GridBar& g) {
    const unsigned long long target = (unsigned long long)g.gen * gridDim.x;
    int ok = 1;
    if (threadIdx.x == 0) {
        asm volatile("red.release.gpu.global.add.u64 [%0], 1;" ::"l"(g.arrivals) : "memory");
        for (int spins = 1; ldRelaxed(g.arrivals) < target; spins++) {
            if (spins >= GRID_SPIN) { atomicExch(g.abortWord, 1u); ok = 0; break; }
            if ((spins & 63) == 0 && *(volatile unsigned int*)g.abortWord) { ok = 0; break; }
        }
    }
    ok = __shfl_sync(0xffffffffu, ok, 0);
    asm volatile("fence.acq_rel.gpu;" ::: "memory");
    return ok != 0;
}
// Grid barrier of all threads.
__device__ __forceinline__ bool gridBarrier(GridBar& g) {
    g.gen++;
    __syncthreads();
    int ok = 1;
    if (threadIdx.x < 32) ok = gridWaitWarp0(g);
    return __syncthreads_and(ok) != 0;
}
// The blocks' partials of NV values: pv is thread 0's, part holds 2 GRID_NV gridDim.x words (the
// sets of consecutive barriers alternate: a block is at most one barrier ahead of another's
// reads).  Warp 0 only: got[q][m] is block lane + 32 m's (absent blocks: none).  The caller
// has passed a __syncthreads since the block's last global write, and g.gen is advanced by all.
template <int NV>
__device__ __forceinline__ bool gridCollectWarp0(const unsigned long long (&pv)[NV], GridBar& g, unsigned long long* part,
                                                 unsigned long long none, unsigned long long (&got)[NV][GRID_PER_LANE]) {
    unsigned long long* const set = part + (size_t)(g.gen & 1u) * GRID_NV * gridDim.x;
    if (threadIdx.x == 0)
#pragma unroll
        for (int q = 0; q < NV; q++)
            asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(set + q * gridDim.x + blockIdx.x), "l"(pv[q]) : "memory");
    if (!gridWaitWarp0(g)) return false;
#pragma unroll
    for (int q = 0; q < NV; q++)
#pragma unroll
        for (int m = 0; m < GRID_PER_LANE; m++) {
            const unsigned b = threadIdx.x + 32 * m;
            got[q][m] = b < gridDim.x ? ldRelaxed(set + q * gridDim.x + b) : none;
        }
    return true;
}
