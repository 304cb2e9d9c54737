// gbp_internal.cuh -- shared device/host definitions of libgbp.
//
// Data layout in HBM (one scene): every per-cell array is a dense nx*ny*nz
// array, x fastest. The operator is stored matrix-free as four per-cell
// arrays: diag (0 off the unknowns) and the coupling weight of the cell's
// +x/+y/+z face, cx/cy/cz, which is the negated off-diagonal
// -A[c][c+e_d] and is 0 unless both cells are unknowns. Vectors are dense
// with 0 off the unknowns, so A*x is the 7-point (5-point in 2D) stencil
//   (A x)_c = diag_c x_c - sum_d (cd_c x_{c+e_d} + cd_{c-e_d} x_{c-e_d}).
//
// Work is split into tiles of 32 (x) by 8 (y) by TZ (z) cells. A launch runs
// a fixed number of blocks (a multiple of the SM count); block b handles
// tiles b, b+G, b+2G, ... in order. Reductions keep one partial per block
// and the last block to finish sums them in block order, so every result is
// bitwise reproducible run to run.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace gbp {

constexpr int TILE_X = 32;
constexpr int TILE_Y = 8;
constexpr int BLOCK_THREADS = TILE_X * TILE_Y;  // 256
constexpr int MAX_GRID = 152 * 8;               // partial-array capacity

// Exact unsigned division by a divisor fixed at run time: one multiply-high,
// an add and two shifts instead of a division routine (Granlund and
// Montgomery, "Division by invariant integers using multiplication",
// PLDI 1994, fig. 4.1). Exact for every 32-bit dividend and divisor >= 1.
struct FastDiv {
    unsigned d, m;
    int s1, s2;
};

__host__ __device__ inline FastDiv make_fastdiv(unsigned d) {
    FastDiv f;
    f.d = d;
    int l = 0;
    while ((1ull << l) < d) ++l;  // l = ceil(log2 d)
    f.m = (unsigned)(((1ull << 32) * ((1ull << l) - d)) / d + 1);
    f.s1 = l < 1 ? l : 1;
    f.s2 = l > 1 ? l - 1 : 0;
    return f;
}

__host__ __device__ __forceinline__ unsigned fdiv(unsigned n, const FastDiv &f) {
#ifdef __CUDA_ARCH__
    const unsigned t1 = __umulhi(f.m, n);
#else
    const unsigned t1 = (unsigned)(((unsigned long long)f.m * n) >> 32);
#endif
    return (t1 + ((n - t1) >> f.s1)) >> f.s2;
}

struct Grid {
    int nx, ny, nz;   // cells (nz == 1 in 2D)
    int dim;          // 2 or 3
    int tz;           // tile depth in z
    int ntx, nty, ntz;
    long long ntiles;
    long long ncell;
    // divisors of the tile decompositions: ntx (32-wide cell tiles), ntx2
    // (64-wide pair tiles), nty; and of the node grid: nx+1, (nx+1)(ny+1)
    FastDiv ftx, ftx2, fty;
    FastDiv fn1, fn2;
};

// deep_min: the fewest cells for tiles 4 planes deep. Deep tiles give a
// block more cells and the gather-first column kernels their 4 planes;
// thin ones spread small grids over all SMs. A scene's fine grid takes deep
// tiles above 2^18 cells (64^3): mixed MGPCG with thin and deep tiles, ms, at
// 64^3 liquid 1.66 / 1.69, 80^3 2.27 / 2.20, 96^3 2.49 / 2.39, 112^3 3.33 /
// 3.07, a batch of 64 liquids up to 160^3 73.5 / 69.4, six served scenes 30.0 /
// 26.9. Coarse levels take them only above 2^21 (their 2^21-cell level, under
// a 256^3 grid, balances better in thin tiles: 11.17 against 11.25 ms).
constexpr long long DEEP_MIN_FINE = (1LL << 18) + 1;
constexpr long long DEEP_MIN_COARSE = (1LL << 21) + 1;
constexpr long long DEEP_MIN_CG = 1LL << 21;  // plain CG (Solver::solve_cg)
inline Grid make_grid(int dim, int nx, int ny, int nz, long long deep_min = DEEP_MIN_FINE) {
    Grid g;
    g.dim = dim;
    g.nx = nx;
    g.ny = ny;
    g.nz = dim == 3 ? nz : 1;
    g.tz = (g.nz == 1 || (long long)nx * ny * g.nz < deep_min) ? 1 : 4;
    g.ntx = (nx + TILE_X - 1) / TILE_X;
    g.nty = (ny + TILE_Y - 1) / TILE_Y;
    g.ntz = (g.nz + g.tz - 1) / g.tz;
    g.ntiles = (long long)g.ntx * g.nty * g.ntz;
    g.ncell = (long long)nx * ny * g.nz;
    g.ftx = make_fastdiv((unsigned)g.ntx);
    g.ftx2 = make_fastdiv((unsigned)((nx + 63) / 64));
    g.fty = make_fastdiv((unsigned)g.nty);
    g.fn1 = make_fastdiv((unsigned)(nx + 1));
    g.fn2 = make_fastdiv((unsigned)((nx + 1) * (ny + 1)));
    return g;
}

// Reduction scratch of one solve: per-block partials and scalars that the
// last block of a launch writes. Lives in device memory.
struct Scalars {
    double rho;      // r . z of the current iterate
    double alpha;
    double beta;
    double pap;      // p . A p
    double tol;      // absolute stopping threshold on |r|_inf
    double res0;     // |r0|_inf
    double res;      // |r|_inf of the latest iterate
    double r2;       // r . r of the latest iterate (for reporting)
    double aux[4];
    double inner_tol;   // mixed: absolute threshold of the current inner solve
    double inner_res0;  // mixed: |r_f|_inf at the start of the inner solve
    int iter;        // completed (inner) iterations
    int done;        // nonzero once the solve has stopped
    int status;      // 0 running, 1 converged, 2 max iterations, 3 breakdown (0/0 or NaN)
    int max_iter;
    int fluid_exists;
    int first;        // next preconditioned dot starts a new direction (beta = 0)
    int first_update; // next update overwrites (rather than adds to) the correction
    int inner_done;   // mixed: the current inner solve has stopped
    int inner_iter;   // mixed: iterations of the current inner solve
    int inner_max;    // mixed: iteration cap of one inner solve
    int outer_iter;   // mixed: refinement steps taken
    int pad;
    unsigned long long unknowns;
    unsigned long long bits_max;  // max of non-negative doubles through their bit patterns
    unsigned int counter[8];      // last-block tickets, one per reduction site
};

struct Partials {
    double a[MAX_GRID];
    double b[MAX_GRID];
    double c[MAX_GRID];
};

#ifdef __CUDACC__

__device__ __forceinline__ long long cell_index(const Grid &g, int i, int j, int k) {
    return (long long)i + (long long)g.nx * ((long long)j + (long long)g.ny * k);
}

// Coordinates of node t of the (nx+1)(ny+1)(nz+1) node grid, x fastest
// (node counts fit 32 bits).
__device__ __forceinline__ void node_coords(const Grid &g, long long t, int &i, int &j, int &k) {
    const unsigned tt = (unsigned)t;
    const unsigned q = fdiv(tt, g.fn1);
    const unsigned kk = fdiv(tt, g.fn2);
    i = (int)(tt - q * g.fn1.d);
    j = (int)(q - kk * (unsigned)(g.ny + 1));
    k = (int)kk;
}

// Tiles are numbered x fastest, then y, then z (tile counts fit 32 bits).
__device__ __forceinline__ void tile_origin(const Grid &g, long long t, int &i0, int &j0, int &k0) {
    const unsigned tt = (unsigned)t;
    const unsigned r = fdiv(tt, g.ftx);
    const unsigned tk = fdiv(r, g.fty);
    i0 = (int)(tt - r * (unsigned)g.ntx) * TILE_X;
    j0 = (int)(r - tk * (unsigned)g.nty) * TILE_Y;
    k0 = (int)tk * g.tz;
}

// Block-wide reductions of BLOCK_THREADS FP64 values. A warp instruction
// holds this GPU's FP64 pipe 16 cycles and its result takes over 100, so a
// shuffle tree in every warp (45 instructions a block, most lanes adding
// nothing) cost more than the pass that fed it on small grids. The values go
// through shared memory instead and one warp adds them, eight to a lane: 12
// instructions, in the shuffle tree's association (bitwise the same sum:
// within a warp's 32 values halves are added, 16 apart, then 8, 4, 2, 1; then
// the 8 warps' sums 4, 2, 1 apart). Maxima of magnitudes run on bit patterns, with
// integer instructions alone.

// where thread t's value goes: 4 apart per warp's 32, so that the lanes of
// tree256 read different banks
constexpr int TREE_PAD = 288;
__device__ __forceinline__ int tree_at(int t) { return t + (t >> 5) * 4; }

// The sum of 256 values placed by tree_at, by one warp; result in lane 0.
// Lane 4w + q adds the values q, q + 4, ... of warp w's 32.
__device__ __forceinline__ double tree256(const double *v) {
    const int lane = threadIdx.x & 31;
    const double *p = v + (lane >> 2) * 36 + (lane & 3);
    double a[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) a[k] = p[4 * k] + p[4 * k + 16];
    double s = (a[0] + a[2]) + (a[1] + a[3]);
    s += __shfl_down_sync(0xffffffffu, s, 2);
    s += __shfl_down_sync(0xffffffffu, s, 1);
    s += __shfl_down_sync(0xffffffffu, s, 16);
    s += __shfl_down_sync(0xffffffffu, s, 8);
    s += __shfl_down_sync(0xffffffffu, s, 4);
    return s;
}

// |x|'s bit pattern (ordered as |x| is), 0 for a NaN, which fmax ignores
__device__ __forceinline__ unsigned long long abs_bits(double x) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffull;
    return b > 0x7ff0000000000000ull ? 0ull : b;
}

__device__ __forceinline__ unsigned long long warp_max_bits(unsigned long long b) {
    const unsigned hi = (unsigned)(b >> 32), mh = __reduce_max_sync(0xffffffffu, hi);
    const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? (unsigned)b : 0u);
    return (unsigned long long)mh << 32 | ml;
}

// Block-wide sum in a fixed order; result valid in thread 0.
__device__ __forceinline__ double block_sum(double v) {
    __shared__ double vals[TREE_PAD];
    __syncthreads();
    vals[tree_at(threadIdx.x)] = v;
    __syncthreads();
    return threadIdx.x < 32 ? tree256(vals) : 0.0;
}

// Block-wide maximum of abs_bits patterns; result valid in warp 0.
__device__ __forceinline__ unsigned long long block_max_bits(unsigned long long b) {
    __shared__ unsigned long long maxs[BLOCK_THREADS / 32];
    b = warp_max_bits(b);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) maxs[threadIdx.x >> 5] = b;
    __syncthreads();
    return threadIdx.x < 32 ? warp_max_bits(threadIdx.x < BLOCK_THREADS / 32 ? maxs[threadIdx.x] : 0ull) : 0ull;
}

// Publishes this block's partial(s) and returns true in every thread of the
// block that finished last. Must be called by all threads of the block.
__device__ __forceinline__ bool last_block(unsigned int *counter) {
    __shared__ bool is_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned int ticket = atomicAdd(counter, 1u);
        is_last = (ticket == gridDim.x - 1);
    }
    __syncthreads();
    if (is_last) __threadfence();
    return is_last;
}

// Sums partial[0..n) in a fixed order (strided per thread, then the block
// tree); result valid in thread 0.
__device__ __forceinline__ double reduce_partials_sum(const double *partial, int n) {
    double v = 0.0;
    for (int t = threadIdx.x; t < n; t += blockDim.x) v += __ldcg(partial + t);
    return block_sum(v);
}

__device__ __forceinline__ double reduce_partials_max(const double *partial, int n) {
    unsigned long long v = 0;
    for (int t = threadIdx.x; t < n; t += blockDim.x) v = max(v, abs_bits(__ldcg(partial + t)));
    return __longlong_as_double((long long)block_max_bits(v));
}

#endif  // __CUDACC__

}  // namespace gbp
