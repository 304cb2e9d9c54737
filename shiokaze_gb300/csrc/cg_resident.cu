// cg_resident.cu -- conjugate gradients on the matrix-free operator in one
// launch: the unknowns of a grid whose vectors fit the SMs' shared memory.
//
// The algorithm is cg_kernels.cu's (the reference's plain CG: the same
// iteration, stopping rule and status). That form takes three launches an
// iteration, whose time on such grids is latency, and walks every cell of the
// grid, liquid or not. Here the blocks stay resident (one cluster of 16 for
// grids up to 128^2, else one block an SM in a cooperative launch), share out
// the unknowns alone, keep x, r, s, z of theirs in shared memory and exchange
// s through L2. Three meetings an iteration: s written; s.As; r.r.
//
// Sums. On this GPU a dependent FP64 operation takes over 100 cycles and a
// warp holds the FP64 pipe 16 cycles an instruction, so the FP64 tree of a dot
// product (8 levels in a block, 9 more over the blocks) took longer than the
// stencil. Each thread's FP64 partial is instead added as a fixed-point number
// of 130 bits: five 26-bit limbs in the unit 2^(E - 104), E the binary
// exponent of the sum's previous value, summed by integer warp reductions and,
// between blocks, by atomics on five words that also count their arrivals. The
// sum of the partials is exact to 2^-87 of the previous value, whatever their
// order, and rounded once: closer to the true dot product than a tree, and the
// same for every distribution of the unknowns. A partial above 2^(E + 12), a
// non-finite one, or a sum below 2^(E - 34) ends the launch with status 5, and
// the solve is done again by the launched form.
//
// Measured on one GB300 (launched form, one launch with FP64 trees, this):
// 2D liquid 128^2, 575 iterations, 9.37 / 5.64 / TP ms; 3D liquid
// 75 x 92 x 61, 1057 iterations, 47.9 / 21.1 / TR ms.
//
// Waits: the cluster form uses the hardware barrier; the cooperative form
// polls, bounded, and leaves with status 4 if a wait runs out.
#include "gbp_internal.cuh"
#include "gbp_kernels.h"

namespace gbp {
namespace {

constexpr int THREADS = 1024;
constexpr int POLLS = 1 << 22;  // about two seconds
constexpr int CLUSTER_BLOCKS = 16;
constexpr long long CLUSTER_CELLS = 16384;
constexpr int LIMBS = 5, LIMB_BITS = 26, LIMB_MASK = (1 << LIMB_BITS) - 1;
constexpr int ITEM_BYTES = 4 * 8 + 2 * 4;  // x, r, s, z, cell, neighbour bits
constexpr size_t SHARED = 216 * 1024;
constexpr int SET_WORDS = LIMBS * 16;  // a sum's words, 128 bytes apart
constexpr unsigned long long BIAS = 1ull << 32, VALUE_MASK = (1ull << 48) - 1;

struct Args {
    Grid g;
    Operator<double> A;
    double *x, *r, *s;
    int *list;  // the unknowns' cells, one int a cell
    Scalars *sc;
    Partials *pt;  // zeroed: words of the sums, block counts, maxima, barrier
    int max_steps;
};

// scratch within Partials
__device__ __forceinline__ unsigned long long *sum_words(Partials *pt, int set) {
    return reinterpret_cast<unsigned long long *>(pt->a) + set * SET_WORDS;
}
__device__ __forceinline__ int *block_counts(Partials *pt) { return reinterpret_cast<int *>(pt->b); }
__device__ __forceinline__ unsigned long long *max_words(Partials *pt) {
    return reinterpret_cast<unsigned long long *>(pt->c);
}
__device__ __forceinline__ unsigned *barrier_word(Partials *pt) { return reinterpret_cast<unsigned *>(pt->c + 32); }

__device__ __forceinline__ int exponent_of(double v) {
    return (int)((unsigned long long)__double_as_longlong(v) >> 52 & 0x7ffu) - 1023;
}

// d in units of 2^base as signed limbs; false if it does not fit (E is base + 104)
__device__ __forceinline__ bool to_limbs(double d, int base, int (&l)[LIMBS]) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(d);
    const int e = (int)(b >> 52 & 0x7ffu), at = e - 1075 - base;  // bit 0 of the significand
    unsigned long long m = e ? (b & 0xfffffffffffffull) | 1ull << 52 : 0ull;
    const bool fits = e == 0 || e - 1023 < base + 104 + 12;
    if (!fits) m = 0;
    int sh = at;
    if (at < 0) {
        m = at > -64 ? m >> -at : 0ull;
        sh = 0;
    }
    if (!fits) sh = 0;
    const int q = sh / LIMB_BITS, r = sh - q * LIMB_BITS;
    const unsigned long long lo = m << r, hi = r ? m >> (64 - r) : 0ull;
    const int p0 = (int)(lo & LIMB_MASK), p1 = (int)(lo >> LIMB_BITS & LIMB_MASK),
              p2 = (int)((lo >> 2 * LIMB_BITS | hi << (64 - 2 * LIMB_BITS)) & LIMB_MASK),
              p3 = (int)(hi >> (3 * LIMB_BITS - 64));
    const int sign = (long long)b < 0 ? -1 : 1;
#pragma unroll
    for (int k = 0; k < LIMBS; ++k)
        l[k] = sign * (k == q ? p0 : (k == q + 1 ? p1 : (k == q + 2 ? p2 : (k == q + 3 ? p3 : 0))));
    return fits;
}

// sum L[k] 2^(26 k + base), rounded to nearest; 0 for a negative sum (as no sum here is)
__device__ __forceinline__ double from_limbs(long long (&L)[LIMBS], int base) {
#pragma unroll
    for (int k = 0; k + 1 < LIMBS; ++k) {
        L[k + 1] += L[k] >> LIMB_BITS;
        L[k] &= LIMB_MASK;
    }
    if (L[4] < 0) return 0.0;
    unsigned long long hi = (unsigned long long)L[4] << LIMB_BITS | (unsigned long long)L[3];
    unsigned long long mid = (unsigned long long)L[2] << LIMB_BITS | (unsigned long long)L[1], lo = (unsigned long long)L[0];
    int ex = base + 3 * LIMB_BITS;
    if (hi == 0) {  // below 2^(E - 26)
        hi = mid;
        mid = lo << LIMB_BITS;
        lo = 0;
        ex -= 2 * LIMB_BITS;
    }
    if (hi == 0) return 0.0;
    // the top 64 bits of hi (below 2^58) and mid (52 bits), the rest as a sticky bit
    const int z = __clzll((long long)hi);
    unsigned long long m = hi << z;
    if (z <= 52) {
        m |= mid >> (52 - z);
        if ((mid & ((1ull << (52 - z)) - 1)) | lo) m |= 1ull;
    } else {
        const int rest = LIMB_BITS - (z - 52);  // bits of lo beyond the 64
        m |= mid << (z - 52) | lo >> rest;
        if (lo & ((1ull << rest) - 1)) m |= 1ull;
    }
    return __longlong_as_double(__double_as_longlong(__ull2double_rn(m)) + ((long long)(ex - z) << 52));
}

template <bool CLUSTER> __device__ __forceinline__ bool meet(Partials *pt, unsigned &target) {
    if (CLUSTER) {
        asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
        return true;
    }
    target += gridDim.x;
    unsigned *count = barrier_word(pt);
    __syncthreads();
    int good = 1;
    if (threadIdx.x == 0) {
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
        unsigned seen;
        for (int it = 0;; ++it) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(count) : "memory");
            if (seen >= target) break;
            if (it > POLLS) {
                good = 0;
                break;
            }
        }
    }
    return __syncthreads_and(good) != 0;
}

struct SumShared {
    int warp[32][8];                    // a warp's limbs, its flags, its overflow
    int slot[2][CLUSTER_BLOCKS][8];     // a cluster's blocks' (by parity)
};

// The sum over all blocks of every thread's v, and of one flag per block: in
// thread 0, value (0 if it overflowed, total[1] counts those) and total[0] =
// blocks whose flag is set. False if a wait ran out.
template <bool CLUSTER>
__device__ __forceinline__ bool grid_sum(double v, bool flag, int base, int set, int parity, Partials *pt, SumShared &sh,
                                         double &value, int (&total)[2]) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int l[LIMBS];
    const bool over = !to_limbs(v, base, l);
#pragma unroll
    for (int k = 0; k < LIMBS; ++k) l[k] = __reduce_add_sync(0xffffffffu, l[k]);
    const bool wflag = __any_sync(0xffffffffu, flag), wover = __any_sync(0xffffffffu, over);
    if (lane == 0) {
#pragma unroll
        for (int k = 0; k < LIMBS; ++k) sh.warp[warp][k] = l[k];
        sh.warp[warp][5] = wflag ? 1 : 0;
        sh.warp[warp][6] = wover ? 1 : 0;
    }
    __syncthreads();
    bool good = true;
    if (warp == 0) {
        // the block's limbs: each warp's normalised (26 bits, the top one signed), then added
        long long t[LIMBS];
#pragma unroll
        for (int k = 0; k < LIMBS; ++k) t[k] = sh.warp[lane][k];
#pragma unroll
        for (int k = 0; k + 1 < LIMBS; ++k) {
            t[k + 1] += t[k] >> LIMB_BITS;
            t[k] &= LIMB_MASK;
        }
        int b[LIMBS];
#pragma unroll
        for (int k = 0; k < LIMBS; ++k) b[k] = (int)__reduce_add_sync(0xffffffffu, (unsigned)(int)t[k]);
        const bool bflag = __any_sync(0xffffffffu, sh.warp[lane][5] != 0),
                   bover = __any_sync(0xffffffffu, sh.warp[lane][6] != 0);
        long long L[LIMBS];
        if (CLUSTER) {
            // to every block's slots; the limbs normalised again, so that 16 add within an int
            long long u[LIMBS];
#pragma unroll
            for (int k = 0; k < LIMBS; ++k) u[k] = k + 1 < LIMBS ? (long long)(unsigned)b[k] : (long long)b[k];
#pragma unroll
            for (int k = 0; k + 1 < LIMBS; ++k) {
                u[k + 1] += u[k] >> LIMB_BITS;
                u[k] &= LIMB_MASK;
            }
            unsigned rank;
            asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
            if (lane < (int)gridDim.x) {
                const unsigned mine = (unsigned)__cvta_generic_to_shared(&sh.slot[parity][rank][0]);
                unsigned at;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(mine), "r"(lane));
#pragma unroll
                for (int k = 0; k < 7; ++k) {
                    const int w = k < LIMBS ? (int)u[k < LIMBS ? k : 0] : (k == 5 ? (int)bflag : (int)bover);
                    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(at + 4 * k), "r"(w) : "memory");
                }
            }
        } else {
            unsigned long long *w = sum_words(pt, set);
            int mine = 0;
#pragma unroll
            for (int k = 0; k < LIMBS; ++k) mine = lane == k ? b[k] : mine;
            if (lane < LIMBS) {
                const unsigned long long add =
                    BIAS + (lane + 1 < LIMBS ? (long long)(unsigned)mine : (long long)mine);
                unsigned long long word = add | 1ull << 48;
                if (lane == 0 && bflag) word |= 1ull << 56;
                if (lane == LIMBS - 1 && bover) word |= 1ull << 56;
                asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(w + lane * 16), "l"(word) : "memory");
            }
            unsigned long long seen = 0;
            if (lane < LIMBS)
                for (int it = 0;; ++it) {
                    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(seen) : "l"(w + lane * 16) : "memory");
                    if ((seen >> 48 & 0xff) == gridDim.x) break;
                    if (it > POLLS) {
                        good = false;
                        break;
                    }
                }
            good = __all_sync(0xffffffffu, good);
            const long long part = (long long)(seen & VALUE_MASK) - (long long)(BIAS * gridDim.x);
#pragma unroll
            for (int k = 0; k < LIMBS; ++k) L[k] = __shfl_sync(0xffffffffu, part, k);
            const unsigned hi = (unsigned)(seen >> 56);
            total[0] = (int)__shfl_sync(0xffffffffu, hi, 0);
            total[1] = (int)__shfl_sync(0xffffffffu, hi, LIMBS - 1);
            value = from_limbs(L, base);
        }
    }
    if (CLUSTER) {
        unsigned none = 0;
        meet<true>(pt, none);
        if (warp == 0) {
            int b[7];
#pragma unroll
            for (int k = 0; k < 7; ++k)
                b[k] = __reduce_add_sync(0xffffffffu, lane < (int)gridDim.x ? sh.slot[parity][lane][k] : 0);
            long long L[LIMBS];
#pragma unroll
            for (int k = 0; k < LIMBS; ++k) L[k] = b[k];
            total[0] = b[5];
            total[1] = b[6];
            value = from_limbs(L, base);
        }
    }
    return good;
}

template <bool CLUSTER>
__global__ void __launch_bounds__(THREADS, 1) cg_resident_kernel(const __grid_constant__ Args a) {
    extern __shared__ double smem[];
    __shared__ SumShared sum;
    __shared__ int warp_n[32], sh_status, sh_exp;
    __shared__ double sh_scalar;
    Scalars *sc = a.sc;
    if (sc->done) return;
    const Grid &g = a.g;
    const Operator<double> A = a.A;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int n = (int)g.ncell, P = gridDim.x, me = blockIdx.x;
    unsigned target = 0;

    // the unknowns' cells, in order: counted and listed by a stretch of cells a block
    const int chunk = ((n + P - 1) / P + THREADS - 1) / THREADS * THREADS;
    const int lo = min(n, me * chunk), hi = min(n, lo + chunk);
    unsigned long long mdiag = 0;
    int found = 0;
    for (int c = lo + tid; c < hi; c += THREADS) {
        const unsigned long long d = abs_bits(__ldg(A.diag + c));
        mdiag = max(mdiag, d);
        found += d != 0;
    }
    found = __reduce_add_sync(0xffffffffu, found);
    mdiag = warp_max_bits(mdiag);
    if (lane == 0) {
        warp_n[warp] = found;
        if (mdiag) atomicMax(max_words(a.pt), mdiag);
    }
    __syncthreads();
    if (warp == 0) {
        found = __reduce_add_sync(0xffffffffu, warp_n[lane]);
        if (lane == 0) __stcg(block_counts(a.pt) + me, found);
    }
    bool good = meet<CLUSTER>(a.pt, target);
    int before = 0, all = 0;
    for (int b = lane; b < P; b += 32) {
        const int v = __ldcg(block_counts(a.pt) + b);
        all += v;
        before += b < me ? v : 0;
    }
    all = __reduce_add_sync(0xffffffffu, all);
    before = __reduce_add_sync(0xffffffffu, before);
    for (int c0 = lo; c0 < hi; c0 += THREADS) {
        const int c = c0 + tid;
        const bool on = c < hi && abs_bits(__ldg(A.diag + c)) != 0;
        const unsigned vote = __ballot_sync(0xffffffffu, on);
        __syncthreads();
        if (lane == 0) warp_n[warp] = __popc(vote);
        __syncthreads();
        const int mine = warp_n[lane];
        const int ahead = __reduce_add_sync(0xffffffffu, lane < warp ? mine : 0);
        if (on) __stcg(a.list + before + ahead + __popc(vote & ((1u << lane) - 1u)), c);
        before += __reduce_add_sync(0xffffffffu, mine);
    }
    good = good && meet<CLUSTER>(a.pt, target);

    // this block's stretch of them
    const int per = (all + P - 1) / P, items = (per + THREADS - 1) / THREADS;
    const int first = min(all, me * per), count = min(all, first + per) - first;
    int status = 0;
    if ((size_t)items * THREADS * ITEM_BYTES > SHARED) status = 6;  // they do not fit: the same in every block
    double *R = smem + tid, *S = R + items * THREADS, *Z = S + items * THREADS, *X = Z + items * THREADS;
    int *cell = reinterpret_cast<int *>(smem + 4 * items * THREADS) + tid;
    int *nbrs = cell + items * THREADS;
    const int sy = g.nx, sz = g.nx * g.ny;
    if (!status && good)
        for (int m = 0; m < items; ++m) {
            const int o = m * THREADS;
            const int c = o + tid < count ? __ldcg(a.list + first + o + tid) : -1;
            cell[o] = c;
            if (c < 0) continue;
            const int k = c / sz, j = (c - k * sz) / sy, i = c - k * sz - j * sy;
            nbrs[o] = (i > 0) | (i + 1 < g.nx) << 1 | (j > 0) << 2 | (j + 1 < g.ny) << 3 |
                      (g.dim == 3 && k > 0) << 4 | (g.dim == 3 && k + 1 < g.nz) << 5;
            R[o] = a.r[c];
            S[o] = a.s[c];
            X[o] = a.x[c];
        }
    double rho = sc->rho, alpha = 0.0, beta = sc->beta, r2 = sc->r2;
    const double tol = sc->tol;
    const unsigned long long tol_bits = abs_bits(tol);
    int iter = sc->iter, sums = 0;
    const int max_iter = sc->max_iter;
    // exponents of the sums' previous values; s.As is at most twice the largest diagonal times s.s
    int e_rho = exponent_of(rho);
    int e_pap = e_rho + exponent_of(__longlong_as_double((long long)__ldcg(max_words(a.pt)))) + 1;
    __syncthreads();

    for (int step = 0; good && !status && step < a.max_steps; ++step) {
        // z = A s (apply_A's order), s.z
        double dot = 0.0;
        for (int m = 0; m < items; ++m) {
            const int o = m * THREADS, c = cell[o];
            if (c < 0) break;
            const int nb = nbrs[o];
            double w[6], v[6];
#pragma unroll
            for (int q = 0; q < 6; ++q) {
                const int d = q < 2 ? 1 : (q < 4 ? sy : sz);
                const double *cp = q < 2 ? A.cx : (q < 4 ? A.cy : A.cz);
                const bool on = nb >> q & 1;
                w[q] = on ? __ldg(cp + (q & 1 ? c : c - d)) : 0.0;
                v[q] = on ? __ldcg(a.s + (q & 1 ? c + d : c - d)) : 0.0;
            }
            const double s = S[o];
            // two chains of three terms: half the dependent latency
            double z0 = __ldg(A.diag + c) * s, z1 = w[3] * v[3];
            z0 = fma(-w[0], v[0], z0);
            z1 = fma(w[4], v[4], z1);
            z0 = fma(-w[1], v[1], z0);
            z1 = fma(w[5], v[5], z1);
            z0 = fma(-w[2], v[2], z0);
            const double z = z0 - z1;
            Z[o] = z;
            dot = fma(s, z, dot);
        }
        double pap = 0.0, rho_new = 0.0;
        int total[2] = {0, 0};
        // the sum, and whether a wait ran out, are warp 0's: thread 0 tells the others
        good = grid_sum<CLUSTER>(dot, false, e_pap - 104, step & 1, sums++ & 1, a.pt, sum, pap, total);
        if (tid == 0) {
            sh_status = !good ? 4 : (total[1] || exponent_of(pap) < e_pap - 34 ? 5 : 0);
            sh_scalar = rho / pap;
            sh_exp = exponent_of(pap);
        }
        __syncthreads();
        status = sh_status;
        if (status) break;
        alpha = sh_scalar;
        e_pap = sh_exp;
        // x += alpha s, r -= alpha z, r.r, whether |r| exceeds the threshold
        bool large = false;
        double part = 0.0;
        for (int m = 0; m < items; ++m) {
            const int o = m * THREADS;
            if (cell[o] < 0) break;
            X[o] = fma(alpha, S[o], X[o]);
            const double r = fma(-alpha, Z[o], R[o]);
            R[o] = r;
            large = large || abs_bits(r) > tol_bits;
            part = fma(r, r, part);
        }
        total[0] = total[1] = 0;
        good = grid_sum<CLUSTER>(part, large, e_rho - 104, 2 + (step & 1), sums++ & 1, a.pt, sum, rho_new, total);
        ++iter;
        if (tid == 0) {
            int st = !good ? 4 : (total[1] ? 5 : 0);
            if (!st) {
                r2 = rho_new;
                if (total[0] == 0) st = 1;
                else if (iter >= max_iter) st = 2;
                else if (alpha != alpha) st = 3;
                else if (exponent_of(rho_new) < e_rho - 34) st = 5;
            }
            if (!st) {
                sh_scalar = rho_new / rho;
                rho = rho_new;
                sh_exp = exponent_of(rho_new);
            }
            sh_status = st;
        }
        __syncthreads();
        status = sh_status;
        if (status) break;
        beta = sh_scalar;
        e_rho = sh_exp;
        // s = r + beta s
        for (int m = 0; m < items; ++m) {
            const int o = m * THREADS;
            if (cell[o] < 0) break;
            const double s = fma(beta, S[o], R[o]);
            S[o] = s;
            __stcg(a.s + cell[o], s);
        }
        if (!CLUSTER && me == 0 && tid < 2 * LIMBS) {
            // every block has read this step's s.As and the last step's r.r: clear
            // their words, which are next used after the barrier below
            const int set = tid < LIMBS ? (step & 1) : 2 + ((step + 1) & 1);
            __stcg(sum_words(a.pt, set) + tid % LIMBS * 16, 0ull);
        }
        good = meet<CLUSTER>(a.pt, target);
    }
    if (!good) status = 4;
    if (status < 4) {
        unsigned long long mx = 0;
        for (int m = 0; m < items; ++m) {
            const int o = m * THREADS, c = cell[o];
            if (c < 0) break;
            a.x[c] = X[o];
            a.r[c] = R[o];
            mx = max(mx, abs_bits(R[o]));
        }
        mx = warp_max_bits(mx);
        if (lane == 0 && mx) atomicMax(max_words(a.pt) + 16, mx);
        if (!meet<CLUSTER>(a.pt, target)) status = 4;
    }
    if ((me == 0 || status == 4) && tid == 0) {
        if (status < 4) {
            sc->rho = rho;
            sc->r2 = r2;
            sc->alpha = alpha;
            sc->beta = beta;
            sc->res = __longlong_as_double((long long)__ldcg(max_words(a.pt) + 16));
            sc->iter = iter;
        }
        sc->status = status;
        sc->done = status != 0;
    }
}

}  // namespace

cudaError_t launch_cg_resident(const Grid &g, Operator<double> A, double *x, double *r, double *s, void *list,
                               Scalars *sc, Partials *pt, int grid_blocks, cudaStream_t stream) {
    const bool cluster = g.ncell <= CLUSTER_CELLS;
    const void *fn = cluster ? (const void *)cg_resident_kernel<true> : (const void *)cg_resident_kernel<false>;
    // the words' counts hold 255 blocks
    const int sms = grid_blocks / 6 < 1 ? 1 : (grid_blocks / 6 > 250 ? 250 : grid_blocks / 6);
    int blocks = cluster ? CLUSTER_BLOCKS : sms;
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SHARED);
    if (e == cudaSuccess && cluster) e = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e == cudaSuccess) e = cudaMemsetAsync(pt, 0, sizeof(Partials), stream);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = SHARED;
    cfg.stream = stream;
    cudaLaunchAttribute at[1];
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (cluster) {
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = (unsigned)blocks;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        int fit = 0;
        if ((e = cudaOccupancyMaxActiveClusters(&fit, fn, &cfg)) != cudaSuccess) return e;
        if (fit < 1) return cudaErrorCooperativeLaunchTooLarge;
    } else {
        at[0].id = cudaLaunchAttributeCooperative;
        at[0].val.cooperative = 1;
    }
    Args a{g, A, x, r, s, static_cast<int *>(list), sc, pt, CG_RESIDENT_STEPS};
    void *args[] = {&a};
    return cudaLaunchKernelExC(&cfg, fn, args);
}

// A grid the one launch may take: its unknowns fit the shared memory if there
// are at most 5120 an SM (778,000 on 152), which the kernel finds out (status
// 6); grids of more than 2^21 cells are left to the launched form, whose
// passes are long enough to hide their launches.
bool cg_resident_grid(const Grid &g) { return g.ncell <= (1LL << 21); }

}  // namespace gbp
