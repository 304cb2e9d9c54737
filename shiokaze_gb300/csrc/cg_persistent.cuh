// cg_persistent.cuh -- a whole conjugate-gradient solve in one launch, for
// systems whose vectors fit the SMs' shared memory.
//
// The launched form of CG (cg_kernels.cu, csr_solver.cu) takes three launches
// an iteration, whose time on a small system is latency. Here the blocks stay
// resident, keep x, r, s and z of their rows in shared memory and exchange s
// through L2.
//
// Results equal the launched form's bit for bit, as they have to: CG from
// these right-hand sides multiplies a difference of 1e-15 to 3e-4 in thirty
// iterations, so a sum in another order stops elsewhere. The rows, the order
// in which a thread adds its terms and the shape of every sum are therefore
// the launched form's: the work is cut into its blocks of 256 threads
// ("virtual blocks"); a physical block carries `sub` of them, and every virtual
// block sums its 256 values in block_sum's tree, the partials in
// reduce_partials_sum's. Virtual blocks without a row keep partial 0. What
// need not keep that shape does not: the stencil and the vector updates run
// over the block's rows packed into full warps (of the 32 x 8 tiles of a
// liquid many lanes have none), and the stop test is a flag, the sign bit of
// the partial of r.r (read only where r.r is no NaN).
//
// Exchange of the partials: a cluster's blocks push them into each other's
// shared memory and meet at the hardware barrier; blocks of a cooperative
// launch write them to L2, meet at a counter and read them all. (Polling the
// slots themselves instead of the counter, 379 to 912 of them from 152 blocks,
// held up the writes: 17.8 against 12.3 ms on the matrix below.)
//
// Measured on one GB300, launched form and here: 2D liquid 128^2 (a cluster)
// 9.37 and 5.2 ms for 575 iterations, 3D liquid 75 x 92 x 61 47.9 and 21.0 ms
// for 1057, a 64^3 liquid's matrix in rows 21.5 and 12.0 ms for 920. (One
// thread a lane of the virtual blocks instead of packed rows, partials through
// L2 in the cluster too: 5.6, 21.1 and 12.3 ms.) What is left is latency: over
// 100 cycles a level of the FP64 trees, 800 for each of the two divisions, and
// the L2 round trips.
//
// Waits: the cluster form uses the hardware barrier; the cooperative form
// polls, bounded (about two seconds), and leaves with status 4 if a wait runs
// out (tests/test_gpu_cg_forms.py makes it).
#pragma once

#include "gbp_internal.cuh"
#include "gbp_kernels.h"

namespace gbp {

struct CgPersistentArgs {
    double *x, *r, *s;
    Scalars *sc;
    Partials *pt;   // the partials of s.z (a) and r.r (c)
    int nb;         // virtual blocks, as many as the launched form has blocks
    int sub;        // virtual blocks of a physical block
    int per_block;  // rows a thread has in one virtual block (the launched form's tiles and planes)
    int max_steps;  // iterations in this launch
    int polls = 0, fail_block = 0;  // of CgDebug (the TEST form of the kernel)
};

#ifdef __CUDACC__
namespace cgp {

constexpr int kPolls = 1 << 22;  // about two seconds
constexpr int kClusterBlocks = 16, kClusterSlots = 64;

// Rows of the matrix-free operator: thread t of virtual block vb has the
// cells of tiles vb, vb + nb, ..., tz planes each, as for_each_cell walks them.
struct GridRows {
    Grid g;
    Operator<double> A;
    // the cell of item c and its neighbours that exist (bits 0..5: -x +x -y +y -z +z); -1: none, or not an unknown
    __device__ __forceinline__ int row(int vb, int nb, int c, int t, unsigned &nbr) const {
        const int q = g.tz == 1 ? c : c / g.tz;
        const long long tile = vb + (long long)q * nb;
        if (tile >= g.ntiles) return -1;
        int i, j, k;
        tile_origin(g, tile, i, j, k);
        i += t & (TILE_X - 1);
        j += t / TILE_X;
        k += c - q * g.tz;
        if (i >= g.nx || j >= g.ny || k >= g.nz) return -1;
        const int e = (int)cell_index(g, i, j, k);
        nbr = (i > 0 ? 1u : 0u) | (i + 1 < g.nx ? 2u : 0u) | (j > 0 ? 4u : 0u) | (j + 1 < g.ny ? 8u : 0u) |
              (g.dim == 3 && k > 0 ? 16u : 0u) | (g.dim == 3 && k + 1 < g.nz ? 32u : 0u);
        // a cell off the unknowns has a zero row, r, s and x
        return (__double_as_longlong(__ldg(A.diag + e)) << 1) != 0 ? e : -1;
    }
    // apply_A's terms in its order, every load first
    __device__ __forceinline__ double apply(int e, unsigned nbr, double s, const double *sv) const {
        const int sy = g.nx, sz = g.nx * g.ny;
        double c[6], v[6];
#pragma unroll
        for (int n = 0; n < 6; ++n) {
            const int step = n < 2 ? 1 : (n < 4 ? sy : sz);
            const double *cp = n < 2 ? A.cx : (n < 4 ? A.cy : A.cz);
            const bool on = nbr >> n & 1u;
            c[n] = on ? __ldg(cp + (n & 1 ? e : e - step)) : 0.0;
            v[n] = on ? __ldcg(sv + (n & 1 ? e + step : e - step)) : 0.0;
        }
        double acc = __ldg(A.diag + e) * s;
#pragma unroll
        for (int n = 0; n < 6; ++n)
            if (nbr >> n & 1u) acc = fma(-c[n], v[n], acc);
        return acc;
    }
};

// Rows of a matrix in compressed rows, as for_each_row walks them
struct CsrRows {
    long long n;
    const long long *rowstart;
    const int *cols;
    const double *vals;
    __device__ __forceinline__ int row(int vb, int nb, int c, int t, unsigned &nbr) const {
        const long long e = (long long)vb * BLOCK_THREADS + t + (long long)c * nb * BLOCK_THREADS;
        nbr = 0;
        return e < n ? (int)e : -1;
    }
    __device__ __forceinline__ double apply(int e, unsigned, double, const double *sv) const {
        const long long e0 = __ldg(rowstart + e), e1 = __ldg(rowstart + e + 1);
        double acc = 0.0;
        for (long long q = e0; q < e1; q += 8) {
            const int m = (int)(e1 - q < 8 ? e1 - q : 8);
            double a[8], v[8];
#pragma unroll
            for (int n = 0; n < 8; ++n) {
                a[n] = n < m ? __ldg(vals + q + n) : 0.0;
                v[n] = n < m ? __ldcg(sv + __ldg(cols + q + n)) : 0.0;
            }
#pragma unroll
            for (int n = 0; n < 8; ++n)
                if (n < m) acc = fma(a[n], v[n], acc);
        }
        return acc;
    }
};

// x != x without an FP64 instruction on the iteration's critical path
__device__ __forceinline__ bool nan_bits(double x) {
    return ((unsigned long long)__double_as_longlong(x) << 1) > 0xffe0000000000000ull;
}

// All blocks; false if a wait ran out. Writes before it are visible after it.
// TEST: block a.fail_block leaves instead of arriving, waits poll a.polls times.
template <bool CLUSTER, bool TEST>
__device__ __forceinline__ bool meet(unsigned *count, unsigned &target, const CgPersistentArgs &a) {
    if (CLUSTER) {
        asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
        return true;
    }
    target += gridDim.x;
    __syncthreads();
    int good = 1;
    if (TEST && (int)blockIdx.x == a.fail_block) {
        good = 0;
    } else if (threadIdx.x == 0) {
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
        unsigned seen;
        for (int it = 0;; ++it) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(count) : "memory");
            if (seen >= target) break;
            if (it > (TEST ? a.polls : kPolls)) {
                good = 0;
                break;
            }
        }
    }
    return __syncthreads_and(good) != 0;
}

template <class Rows, bool CLUSTER, bool TEST>
__global__ void __launch_bounds__(CLUSTER ? 512 : 768, 1) cg_persistent_kernel(const Rows rows, const CgPersistentArgs a) {
    extern __shared__ double smem[];
    Scalars *sc = a.sc;
    if (sc->done) return;  // (written after every block's last wait, so all threads read the same)
    const int T = blockDim.x, tid = threadIdx.x, nvb = a.sub, slots = nvb * a.per_block * 256;
    // home order: virtual block, item, thread
    double *R = smem, *S = R + slots, *Z = S + slots, *X = Z + slots;
    double *red = smem + 4 * slots;                // padded values of every virtual block
    double *fin = red + nvb * TREE_PAD;            // the partials' 256 strided sums
    double *box = fin + TREE_PAD;                  // the cluster's partials, by parity
    int *cell = (int *)(box + 2 * kClusterSlots);  // the block's rows packed: row,
    int *home = cell + slots;                      // slot << 6 | neighbour bits
    __shared__ int warp_n[32], active[32], has[32];
    __shared__ double sh_scalar;
    __shared__ int sh_status, sh_large, n_active, n_rows;
    const int warp = tid >> 5, lane = tid & 31, nwarps = T >> 5;
    auto virtual_block = [&](int q) { return (int)blockIdx.x + (int)gridDim.x * q; };
    if (tid < 32) has[tid] = 0;
    if (tid == 0) n_rows = 0, sh_large = 0;
    __syncthreads();
    // the block's rows, packed in home order
    for (int h0 = 0; h0 < slots; h0 += T) {
        const int h = h0 + tid;
        int e = -1, q = 0;
        unsigned nbr = 0;
        if (h < slots) {
            q = h / (a.per_block * 256);
            const int rest = h - q * a.per_block * 256, vb = virtual_block(q);
            if (vb < a.nb) e = rows.row(vb, a.nb, rest >> 8, rest & 255, nbr);
            R[h] = e >= 0 ? a.r[e] : 0.0;
            S[h] = e >= 0 ? a.s[e] : 0.0;
            X[h] = e >= 0 ? a.x[e] : 0.0;
            Z[h] = 0.0;
            if (e >= 0) has[q] = 1;
        }
        const unsigned vote = __ballot_sync(0xffffffffu, e >= 0);
        if (lane == 0) warp_n[warp] = __popc(vote);
        __syncthreads();
        const int mine = lane < nwarps ? warp_n[lane] : 0;
        const int at = n_rows + __reduce_add_sync(0xffffffffu, lane < warp ? mine : 0) + __popc(vote & ((1u << lane) - 1u));
        if (e >= 0) {
            cell[at] = e;
            home[at] = h << 6 | (int)nbr;
        }
        const int all = __reduce_add_sync(0xffffffffu, mine);
        __syncthreads();
        if (tid == 0) n_rows += all;
        __syncthreads();
    }
    if (tid == 0) {
        int n = 0;
        for (int q = 0; q < nvb; ++q)
            if (has[q]) active[n++] = q;
        n_active = n;
    }
    // virtual blocks without a row have partial 0
    if (CLUSTER) {
        for (int q = tid; q < 2 * kClusterSlots; q += T) box[q] = 0.0;
    } else if (tid < nvb && !has[tid] && virtual_block(tid) < a.nb) {
        __stcg(a.pt->a + virtual_block(tid), 0.0);
        __stcg(a.pt->c + virtual_block(tid), 0.0);
    }
    double rho = sc->rho, alpha = 0.0, beta = sc->beta;
    const unsigned long long tol = abs_bits(sc->tol);
    int iter = sc->iter, status = 0, sums = 0;
    const int max_iter = sc->max_iter;
    unsigned target = 0;
    unsigned *count = &sc->counter[4];
    bool good = meet<CLUSTER, TEST>(count, target, a);

    // Every thread's items of the active virtual blocks, term by term in
    // order, then the trees: a partial per virtual block (negative if `large`)
    // to every block.
    auto partials = [&](auto term, bool large, double *out) {
        if (large) sh_large = 1;
        __syncthreads();
        for (int v = tid; v < n_active * 256; v += T) {
            const int q = active[v >> 8], t = v & 255;
            double sum = 0.0;
            for (int c = 0; c < a.per_block; ++c) sum = term((q * a.per_block + c) * 256 + t, sum);
            red[q * TREE_PAD + tree_at(t)] = sum;
        }
        __syncthreads();
        const bool mark = sh_large != 0;
        for (int n = warp; n < n_active; n += nwarps) {
            const int q = active[n], vb = virtual_block(q);
            double p = tree256(red + q * TREE_PAD);
            if (mark) p = -p;
            if (CLUSTER) {
                p = __shfl_sync(0xffffffffu, p, 0);
                if (lane < (int)gridDim.x) {
                    const unsigned mine = (unsigned)__cvta_generic_to_shared(box + (sums & 1) * kClusterSlots + vb);
                    unsigned to;
                    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(to) : "r"(mine), "r"(lane));
                    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(to), "d"(p) : "memory");
                }
            } else if (lane == 0) {
                __stcg(out + vb, p);
            }
        }
    };
    // reduce_partials_sum, in every block alike: valid in thread 0. With
    // `marks` the partials are magnitudes and any tells whether one came
    // marked. False if a wait ran out.
    auto total = [&](double &sum, bool &any, const double *in, bool marks) {
        if (!meet<CLUSTER, TEST>(count, target, a)) return false;
        if (tid == 0) sh_large = 0;
        int marked = 0;
        if (tid < 256) {
            double v = 0.0;
            for (int q = tid; q < a.nb; q += 256) {
                double p = CLUSTER ? box[(sums & 1) * kClusterSlots + q] : __ldcg(in + q);
                if (marks) {
                    marked |= __double_as_longlong(p) < 0;
                    p = fabs(p);
                }
                v += p;
            }
            fin[tree_at(tid)] = v;
        }
        ++sums;
        any = __syncthreads_or(marked) != 0;
        sum = warp == 0 ? tree256(fin) : 0.0;
        return true;
    };

    double r2 = sc->r2;
    for (int step = 0; good && step < a.max_steps; ++step) {
        // z = A s, s.z
        for (int e = tid; e < n_rows; e += T) {
            const int h = home[e] >> 6;
            Z[h] = rows.apply(cell[e], (unsigned)home[e] & 63u, S[h], a.s);
        }
        bool more;
        double pap, rho_new;
        partials([&](int h, double sum) { return fma(S[h], Z[h], sum); }, false, a.pt->a);
        good = total(pap, more, a.pt->a, false);
        if (!good) break;
        if (tid == 0) sh_scalar = rho / pap;
        __syncthreads();
        alpha = sh_scalar;
        // x += alpha s, r -= alpha z, r.r, whether |r| exceeds the threshold
        bool large = false;
        for (int e = tid; e < n_rows; e += T) {
            const int h = home[e] >> 6;
            X[h] = fma(alpha, S[h], X[h]);
            const double rv = fma(-alpha, Z[h], R[h]);
            R[h] = rv;
            large = large || abs_bits(rv) > tol;
        }
        partials([&](int h, double sum) { return fma(R[h], R[h], sum); }, large, a.pt->c);
        good = total(rho_new, more, a.pt->c, true);
        if (!good) break;
        ++iter;
        if (tid == 0) {
            r2 = rho_new;
            // NaN first: |r|_inf and the marks pass over it (a NaN's sign says nothing)
            sh_status = nan_bits(rho_new) || nan_bits(alpha) ? 3 : (!more ? 1 : (iter >= max_iter ? 2 : 0));
            sh_scalar = rho_new / rho;
            if (!sh_status) rho = rho_new;
        }
        __syncthreads();
        status = sh_status;
        if (status) break;
        beta = sh_scalar;
        // s = r + beta s
        for (int e = tid; e < n_rows; e += T) {
            const int h = home[e] >> 6;
            const double s = fma(beta, S[h], R[h]);
            S[h] = s;
            __stcg(a.s + cell[e], s);
        }
        good = meet<CLUSTER, TEST>(count, target, a);
    }
    if (!good) status = 4;
    if (status < 4) {
        unsigned long long mx = 0;
        for (int e = tid; e < n_rows; e += T) {
            const int h = home[e] >> 6;
            a.x[cell[e]] = X[h];
            a.r[cell[e]] = R[h];
            mx = max(mx, abs_bits(R[h]));
        }
        mx = warp_max_bits(mx);
        if (lane == 0 && mx) atomicMax(&sc->bits_max, mx);
        if (!meet<CLUSTER, TEST>(count, target, a)) status = 4;
    }
    if ((blockIdx.x == 0 || status == 4) && tid == 0) {
        if (status < 4) {
            sc->rho = rho;
            sc->r2 = r2;
            sc->alpha = alpha;
            sc->beta = beta;
            sc->res = __longlong_as_double((long long)__ldcg(&sc->bits_max));
            sc->iter = iter;
        }
        // a run-out wait leaves done as it is: a block that starts only now
        // must not find it set in some of its threads (it runs out too)
        sc->status = status;
        if (status < 4) sc->done = status != 0;
    }
}

}  // namespace cgp
#endif  // __CUDACC__

// Shape of a persistent solve of nb virtual blocks with per_block rows a
// thread: up to 64 virtual blocks (the 2D grids, 24^3) run as one cluster of
// 16 blocks, whose barrier and shared memory beat L2; larger ones as
// a cooperative grid of one block an SM. Used while x, r, s, z and the row
// table fit the shared memory (about 800,000 grid cells); beyond, the launched
// form's passes are long enough to hide their launches.
struct CgPersistentPlan {
    bool use = false, cluster = false;
    int blocks = 0, threads = 0;
    size_t shared = 0;
    CgPersistentArgs args{};
};

inline CgPersistentPlan cg_persistent_plan(int nb, int per_block, int sms, const CgDebug &debug = {}) {
    CgPersistentPlan p;
    p.cluster = nb <= 64;
    p.blocks = p.cluster ? 16 : (nb < sms ? nb : sms);
    const int each = (nb + p.blocks - 1) / p.blocks;
    p.args.sub = each;
    p.args.nb = nb;
    p.args.per_block = per_block;
    p.args.max_steps = debug.steps > 0 ? debug.steps : CG_PERSISTENT_STEPS;
    p.args.polls = debug.polls;
    p.args.fail_block = debug.block;
    p.threads = p.cluster ? 512 : 768;
    const size_t slots = (size_t)each * per_block * 256;
    p.shared = slots * (4 * sizeof(double) + 2 * sizeof(int)) + (((size_t)each + 1) * TREE_PAD + 2 * 64) * sizeof(double);
    p.use = !debug.launched && p.shared <= 216 * 1024 && each <= 32 && nb <= MAX_GRID;
    return p;
}

#ifdef __CUDACC__
// One launch of a planned solve on `stream`; sc->done tells whether it ended.
template <class Rows>
cudaError_t cg_persistent_launch(const CgPersistentPlan &p, const Rows &rows, cudaStream_t stream) {
    const void *fn = p.cluster ? (const void *)cgp::cg_persistent_kernel<Rows, true, false>
                     : p.args.polls > 0 ? (const void *)cgp::cg_persistent_kernel<Rows, false, true>
                                        : (const void *)cgp::cg_persistent_kernel<Rows, false, false>;
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)p.shared);
    if (e == cudaSuccess && p.cluster) e = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    // the maximum, and the barrier's count
    if (e == cudaSuccess) e = cudaMemsetAsync(&p.args.sc->bits_max, 0, sizeof(unsigned long long), stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(&p.args.sc->counter[4], 0, sizeof(unsigned), stream);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)p.blocks);
    cfg.blockDim = dim3((unsigned)p.threads);
    cfg.dynamicSmemBytes = p.shared;
    cfg.stream = stream;
    cudaLaunchAttribute at[1];
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (p.cluster) {
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = (unsigned)p.blocks;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        int n = 0;
        if ((e = cudaOccupancyMaxActiveClusters(&n, fn, &cfg)) != cudaSuccess) return e;
        if (n < 1) return cudaErrorCooperativeLaunchTooLarge;
    } else {
        at[0].id = cudaLaunchAttributeCooperative;
        at[0].val.cooperative = 1;
    }
    Rows r = rows;
    CgPersistentArgs a = p.args;
    void *args[] = {&r, &a};
    return cudaLaunchKernelExC(&cfg, fn, args);
}
#endif  // __CUDACC__

}  // namespace gbp
