// gbp_barrier.cuh -- the arithmetic of the coarse-level kernels' grid barrier
// (grid_barrier in batch_kernels.cu): one word counts arrivals and is never
// reset within a solve, so it wraps in a long one. Every barrier adds a power of
// two to it, whatever the grid (block 0 adds what the others leave), which
// keeps a barrier's end a multiple of that power beyond the wrap. (Adding the
// grid's size, no divisor of 2^32, lost the multiples there: 152 blocks at 16
// barriers an iteration after 1.8 million iterations, with 30 sweeps a level after
// 60 thousand.) The same source compiles for the host
// (tests/test_grid_barrier.py).
#pragma once

namespace gbp {

// the power of two that a barrier of `grid` blocks adds, at least grid
__host__ __device__ __forceinline__ unsigned barrier_span(unsigned grid) {
#ifdef __CUDA_ARCH__
    return 1u << ((32 - __clz((int)(grid - 1u))) & 31);
#else
    unsigned s = 1u;
    while (s < grid) s *= 2u;
    return s;
#endif
}
// what block `block` adds when it arrives
__host__ __device__ __forceinline__ unsigned barrier_step(unsigned block, unsigned grid) {
    return block == 0u ? barrier_span(grid) - (grid - 1u) : 1u;
}
// the count at which a barrier ends, from the count a block found there
__host__ __device__ __forceinline__ unsigned barrier_end(unsigned seen, unsigned grid) {
    return (seen | (barrier_span(grid) - 1u)) + 1u;
}
__host__ __device__ __forceinline__ bool barrier_reached(unsigned now, unsigned end) { return (int)(now - end) >= 0; }

}  // namespace gbp
