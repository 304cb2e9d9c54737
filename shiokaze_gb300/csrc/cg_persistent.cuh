// cg_persistent.cuh -- a whole conjugate-gradient solve in one launch, for
// systems whose vectors fit the SMs' shared memory.
//
// The launched form of CG (cg_kernels.cu, csr_solver.cu) takes three launches
// an iteration, whose time on a small system is latency: the launch, the
// partial sums read back by the last block, and a shuffle tree in every warp
// on the FP64 pipe (a warp instruction holds it 16 cycles). Here the blocks
// stay resident, keep x, r, s and z of their rows in shared memory, exchange
// s through L2 and meet at three barriers an iteration. Measured on one
// GB300, launched and here: 2D liquid 128^2 (one cluster) 9.37 and 5.64 ms for
// 575 iterations, 3D liquid 75 x 92 x 61 47.9 and 21.1 ms for 1057, a 64^3
// liquid's matrix in rows 21.5 and 12.3 ms for 920. What bounds it now is the
// latency of dependent FP64 operations (over 100 cycles a level of the sums'
// trees, 800 for a division) and the L2 round trips of the barriers.
//
// Results equal the launched form's bit for bit: the rows, the order in which
// a thread adds them, and the shape of every sum are the same. The work is
// cut into the launched form's blocks of 256 threads ("virtual blocks"); a
// physical block carries `sub` of them side by side, `rounds` times over, and
// every virtual block sums its 256 values in block_sum's tree, the partials
// in reduce_partials_sum's. Virtual blocks without a row keep partial 0.
// The maximum is order-free; it runs on integers (bit patterns of the
// absolute values), off the FP64 pipe.
//
// Waits: the cluster form uses the hardware barrier; the cooperative form
// polls a counter, bounded, and leaves with status 4 if a wait runs out.
#pragma once

#include "gbp_internal.cuh"
#include "gbp_kernels.h"

namespace gbp {

struct CgPersistentArgs {
    double *x, *r, *s;
    Scalars *sc;
    Partials *pt;
    int nb;         // virtual blocks, as many as the launched form has blocks
    int sub;        // virtual blocks side by side in a physical block
    int rounds;     // virtual blocks one after the other
    int per_block;  // rows a thread has in one virtual block (the launched form's tiles and planes)
    int max_steps;  // iterations in this launch
};

#ifdef __CUDACC__
namespace cgp {

constexpr int kPolls = 1 << 22;  // about two seconds
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
            for (int n = 0; n < 8; ++n)
                if (n < m) {
                    a[n] = __ldg(vals + q + n);
                    v[n] = __ldcg(sv + __ldg(cols + q + n));
                }
#pragma unroll
            for (int n = 0; n < 8; ++n)
                if (n < m) acc = fma(a[n], v[n], acc);
        }
        return acc;
    }
};

// All blocks; false if a wait ran out. Writes before it are visible after it.
template <bool CLUSTER> __device__ __forceinline__ bool meet(unsigned *count, unsigned &target) {
    if (CLUSTER) {
        asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
        return true;
    }
    target += gridDim.x;
    __syncthreads();
    int good = 1;
    if (threadIdx.x == 0) {
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
        unsigned seen;
        for (int it = 0;; ++it) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(count) : "memory");
            if (seen >= target) break;
            if (it > kPolls) {
                good = 0;
                break;
            }
        }
    }
    return __syncthreads_and(good) != 0;
}

template <class Rows, bool CLUSTER>
__global__ void __launch_bounds__(CLUSTER ? 1024 : 768, 1) cg_persistent_kernel(const Rows rows, const CgPersistentArgs a) {
    extern __shared__ double smem[];
    Scalars *sc = a.sc;
    if (sc->done) return;
    const int T = blockDim.x, tid = threadIdx.x, items = a.rounds * a.per_block;
    double *R = smem + tid, *S = R + items * T, *Z = S + items * T, *X = Z + items * T;
    double *red = smem + 4 * items * T;                    // padded values of every virtual block
    double *fin = red + a.rounds * a.sub * TREE_PAD;           // the partials' 256 strided sums
    int *meta = (int *)(fin + TREE_PAD) + tid;                 // row and neighbour bits of each item
    unsigned *nbrs = (unsigned *)((int *)(fin + TREE_PAD) + items * T) + tid;
    __shared__ unsigned long long smax[32];
    __shared__ int active[32];  // virtual blocks with rows: r * sub + s
    __shared__ int has[32];
    __shared__ double sh_alpha, sh_beta;
    __shared__ int sh_done, n_active;
    const int sub = tid >> 8, t = tid & 255, warp = tid >> 5, lane = tid & 31, nwarps = T >> 5;
    auto virtual_block = [&](int r, int s) { return (int)blockIdx.x + (int)gridDim.x * (s + a.sub * r); };
    if (tid < 32) has[tid] = 0;
    __syncthreads();
    for (int r = 0; r < a.rounds; ++r) {
        const int vb = virtual_block(r, sub);
        bool any = false;
        for (int c = 0; c < a.per_block; ++c) {
            const int m = (r * a.per_block + c) * T;
            unsigned nbr = 0;
            const int e = vb < a.nb ? rows.row(vb, a.nb, c, t, nbr) : -1;
            meta[m] = e;
            nbrs[m] = nbr;
            if (e >= 0) {
                any = true;
                R[m] = a.r[e];
                S[m] = a.s[e];
                X[m] = a.x[e];
            }
        }
        if (any) has[r * a.sub + sub] = 1;
    }
    __syncthreads();
    if (tid == 0) {
        int n = 0;
        for (int q = 0; q < a.rounds * a.sub; ++q) {
            const int vb = virtual_block(q / a.sub, q % a.sub);
            if (has[q]) {
                active[n++] = q;
            } else if (vb < a.nb) {
                a.pt->a[vb] = 0.0;
                a.pt->c[vb] = 0.0;
            }
        }
        n_active = n;
    }
    double rho = sc->rho, res = sc->res, alpha = 0.0, beta = sc->beta;
    const double tol = sc->tol;
    int iter = sc->iter, status = 0;
    const int max_iter = sc->max_iter;
    unsigned target = 0;
    unsigned *count = &sc->counter[4];
    __syncthreads();
    bool good = true;

    // one partial per virtual block with rows, by a warp each
    auto partials = [&](double *out) {
        __syncthreads();
        for (int q = warp; q < n_active; q += nwarps) {
            const double s = tree256(red + active[q] * TREE_PAD);
            if (lane == 0) __stcg(out + virtual_block(active[q] / a.sub, active[q] % a.sub), s);
        }
    };
    // reduce_partials_sum, in every block alike; valid in thread 0
    auto total = [&](const double *p) {
        if (tid < 256) {
            double v = 0.0;
            for (int q = tid; q < a.nb; q += 256) v += __ldcg(p + q);
            fin[tree_at(tid)] = v;
        }
        __syncthreads();
        return warp == 0 ? tree256(fin) : 0.0;
    };

    for (int step = 0; step < a.max_steps; ++step) {
        // z = A s, s.z
        for (int r = 0; r < a.rounds; ++r) {
            double dot = 0.0;
            for (int c = 0; c < a.per_block; ++c) {
                const int m = (r * a.per_block + c) * T;
                if (meta[m] < 0) continue;
                const double z = rows.apply(meta[m], nbrs[m], S[m], a.s);
                Z[m] = z;
                dot = fma(S[m], z, dot);
            }
            if (has[r * a.sub + sub]) red[(r * a.sub + sub) * TREE_PAD + tree_at(t)] = dot;
        }
        partials(a.pt->a);
        if (!(good = meet<CLUSTER>(count, target))) break;
        const double pap = total(a.pt->a);
        if (tid == 0) sh_alpha = rho / pap;
        __syncthreads();
        alpha = sh_alpha;
        // x += alpha s, r -= alpha z, |r|_inf, r.r
        unsigned long long mx = 0;
        for (int r = 0; r < a.rounds; ++r) {
            double r2 = 0.0;
            for (int c = 0; c < a.per_block; ++c) {
                const int m = (r * a.per_block + c) * T;
                if (meta[m] < 0) continue;
                X[m] = fma(alpha, S[m], X[m]);
                const double rv = fma(-alpha, Z[m], R[m]);
                R[m] = rv;
                const unsigned long long b = abs_bits(rv);
                mx = b > mx ? b : mx;
                r2 = fma(rv, rv, r2);
            }
            if (has[r * a.sub + sub]) red[(r * a.sub + sub) * TREE_PAD + tree_at(t)] = r2;
        }
        mx = warp_max_bits(mx);
        if (lane == 0) smax[warp] = mx;
        partials(a.pt->c);
        if (warp == nwarps - 1) {
            mx = warp_max_bits(lane < nwarps ? smax[lane] : 0ull);
            if (lane == 0) __stcg((unsigned long long *)a.pt->b + blockIdx.x, mx);
        }
        if (!(good = meet<CLUSTER>(count, target))) break;
        unsigned long long gm = 0;
        if (warp == 0) {
            for (int q = lane; q < (int)gridDim.x; q += 32) {
                const unsigned long long b = __ldcg((const unsigned long long *)a.pt->b + q);
                gm = b > gm ? b : gm;
            }
            gm = warp_max_bits(gm);
        }
        const double rho_new = total(a.pt->c);
        ++iter;
        if (tid == 0) {
            res = __longlong_as_double((long long)gm);
            int done = 0;
            if (res <= tol) done = 1;
            else if (iter >= max_iter) done = 2;
            else if (rho_new != rho_new || alpha != alpha) done = 3;
            sh_beta = rho_new / rho;
            sc->r2 = rho_new;  // every block writes the same value
            if (!done) rho = rho_new;
            sh_done = done;
        }
        __syncthreads();
        status = sh_done;
        if (status) break;
        beta = sh_beta;
        // s = r + beta s
        for (int m = 0; m < items * T; m += T) {
            if (meta[m] < 0) continue;
            const double s = fma(beta, S[m], R[m]);
            S[m] = s;
            __stcg(a.s + meta[m], s);
        }
        if (step + 1 < a.max_steps && !(good = meet<CLUSTER>(count, target))) break;
    }
    for (int m = 0; m < items * T; m += T) {
        if (meta[m] < 0) continue;
        a.x[meta[m]] = X[m];
        a.r[meta[m]] = R[m];
    }
    if (!good) status = 4;
    if ((blockIdx.x == 0 || !good) && tid == 0) {
        sc->rho = rho;
        sc->alpha = alpha;
        sc->beta = beta;
        sc->res = res;
        sc->iter = iter;
        sc->status = status;
        sc->done = status != 0;
    }
}

}  // namespace cgp
#endif  // __CUDACC__

// Shape of a persistent solve of nb virtual blocks with per_block rows a
// thread: up to 64 virtual blocks (the 2D grids, 24^3) run as one cluster of
// 16 blocks of at most four, whose hardware barrier beats a polled counter;
// larger ones as a cooperative grid of one block an SM, three virtual blocks
// side by side (85 registers a thread). Used while x, r, s, z and the row
// table fit the shared memory (about 900,000 grid cells); beyond, the launched
// form's passes are long enough to hide their launches.
struct CgPersistentPlan {
    bool use = false, cluster = false;
    int blocks = 0, threads = 0;
    size_t shared = 0;
    CgPersistentArgs args{};
};

inline CgPersistentPlan cg_persistent_plan(int nb, int per_block, int sms) {
    CgPersistentPlan p;
    p.cluster = nb <= 64;
    p.blocks = p.cluster ? 16 : (nb < sms ? nb : sms);
    while (p.cluster && p.blocks > 1 && p.blocks / 2 >= nb) p.blocks /= 2;
    const int each = (nb + p.blocks - 1) / p.blocks;
    p.args.sub = each < (p.cluster ? 4 : 3) ? each : (p.cluster ? 4 : 3);
    p.args.rounds = (each + p.args.sub - 1) / p.args.sub;
    p.args.nb = nb;
    p.args.per_block = per_block;
    p.args.max_steps = CG_PERSISTENT_STEPS;
    p.threads = p.args.sub * BLOCK_THREADS;
    const size_t items = (size_t)p.args.rounds * per_block * p.threads;
    p.shared = items * (4 * sizeof(double) + 2 * sizeof(int)) +
               ((size_t)p.args.rounds * p.args.sub + 1) * TREE_PAD * sizeof(double);
    p.use = p.shared <= 220 * 1024 && p.args.rounds * p.args.sub <= 32 && nb <= MAX_GRID;
    return p;
}

#ifdef __CUDACC__
// One launch of a planned solve on `stream`; sc->done tells whether it ended.
template <class Rows>
cudaError_t cg_persistent_launch(const CgPersistentPlan &p, const Rows &rows, cudaStream_t stream) {
    const void *fn = p.cluster ? (const void *)cgp::cg_persistent_kernel<Rows, true>
                               : (const void *)cgp::cg_persistent_kernel<Rows, false>;
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)p.shared);
    if (e == cudaSuccess && p.cluster) e = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e == cudaSuccess) e = cudaMemsetAsync(&p.args.sc->counter[4], 0, sizeof(unsigned), stream);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)p.blocks);
    cfg.blockDim = dim3((unsigned)p.threads);
    cfg.dynamicSmemBytes = p.shared;
    cfg.stream = stream;
    cudaLaunchAttribute at[1];
    if (p.cluster) {
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = (unsigned)p.blocks;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        int n = 0;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        if ((e = cudaOccupancyMaxActiveClusters(&n, fn, &cfg)) != cudaSuccess) return e;
        if (n < 1) return cudaErrorCooperativeLaunchTooLarge;
    } else {
        at[0].id = cudaLaunchAttributeCooperative;
        at[0].val.cooperative = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
    }
    Rows r = rows;
    CgPersistentArgs a = p.args;
    void *args[] = {&r, &a};
    return cudaLaunchKernelExC(&cfg, fn, args);
}
#endif  // __CUDACC__

}  // namespace gbp
