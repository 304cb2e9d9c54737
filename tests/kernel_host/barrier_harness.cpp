// TEST INFRASTRUCTURE: the grid barrier's arithmetic (shiokaze_gb300/csrc/
// gbp_barrier.cuh) compiled for the host, its blocks' arrivals in a given order.
#include <vector>
#define __host__
#define __device__
#define __forceinline__ inline
#include "gbp_barrier.cuh"

// Barriers one after another from `count`; order holds each one's arrival order.
// Returns the number of times that a block would pass before all have arrived,
// or wait although they have (also with the next barrier's first arrivals in).
extern "C" long long host_barriers(unsigned count, unsigned grid, int barriers, const int *order) {
    long long bad = 0;
    std::vector<unsigned> end(grid), last;
    for (int b = 0; b < barriers; ++b) {
        for (unsigned n = 0; n < grid; ++n) {
            const unsigned block = (unsigned)order[(long long)b * grid + n];
            end[block] = gbp::barrier_end(count, grid);
            count += gbp::barrier_step(block, grid);
            for (unsigned m = 0; m <= n; ++m) {
                const unsigned other = (unsigned)order[(long long)b * grid + m];
                bad += gbp::barrier_reached(count, end[other]) != (n + 1 == grid);
            }
            for (unsigned e : last) bad += !gbp::barrier_reached(count, e);
        }
        last = end;
    }
    return bad;
}
