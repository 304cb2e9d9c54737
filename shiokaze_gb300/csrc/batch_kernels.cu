// batch_kernels.cu -- the MGPCG iteration over a work list of (level, tile)
// items spanning every scene of a batch (see gbp_batch.h).
//
// Red (i+j+k even) / black Gauss-Seidel, Galerkin restriction by summing the
// 4 red children's residuals (the black ones' are zero after the pre-smoothing),
// post-smoothing black (adding the coarse correction's effect alone) then red, a
// tail of one block per scene for the small levels, and CG with
// FP64-accumulated dot products.
//
// Every kernel walks pair tiles (64 x 8 x tz cells): a thread owns the two
// x-adjacent cells (i, i+1) of a row, i even, one of each colour. On levels
// with an even row length and suitably aligned arrays (the host checks both
// and sets BLevel::vec) the pair and its y/z neighbour pairs move as one
// 8-byte (FP32) or 16-byte (FP64) access; elsewhere as two scalar accesses.
// The arithmetic, including the order of every sum, is the same either way.
//
// Algorithmic DRAM bytes per fine cell (s = sizeof(T)): presmooth 6 s,
// sweep 7 s, restrict 6 s + s/8, post_black 6 s + s/8, red_dot 7 s,
// direction and product 9 s in one pass (staged levels: direction 3 s, spmv
// 6 s), update 6 s; the mixed refinement after an inner
// solve (refine_residual, refine_update_pair) 4 (d) + 32 (level-0 operator
// and its low floats) + 8 + 8 (r64 read and write) + 4 (r_f) + 16 (x64 read
// and write) = 72 B.
#include <type_traits>

#include "gbp_barrier.cuh"
#include "gbp_batch.h"
#include "gbp_convert.cuh"
#include "gbp_floatfloat.cuh"

namespace gbp {
namespace {

// T -> double: exact; from integer instructions for FP32 (gbp_convert.cuh),
// off the FP64 pipe
__device__ __forceinline__ double widen(double v) { return v; }
__device__ __forceinline__ double widen(float v) { return f2d_exact(v); }

// FP64 to T; to FP32 by integer instructions (gbp_convert.cuh), off the
// FP64 pipe
template <class T> __device__ __forceinline__ T narrow_to(double v) {
    if constexpr (sizeof(T) == 4) return d2f_rn(v);
    else return v;
}

constexpr int SITE_DOT = 4, SITE_SPMV = 5, SITE_UPDATE = 6, SITE_REFINE = 7;

__device__ __forceinline__ bool gated(const Scalars *sc, int gate) {
    const volatile Scalars *v = sc;
    if (v->done) return true;
    if (gate == 1) return v->inner_done != 0;
    if (gate == 2) return v->inner_done == 0;
    return false;
}

// Every scene of the batch is done (the rest of a graph chunk after the
// last scene stopped): a launch returns at once.
__device__ __forceinline__ bool batch_idle(const BatchCounters *cnt) {
    return cnt != nullptr && *(const volatile int *)&cnt->remaining <= 0;
}

// Ticket of one item of a scene; true in every thread of the block whose
// item took the scene's last ticket (all threads must call it).
__device__ __forceinline__ bool item_last(unsigned int *counter, int count) {
    __shared__ bool is_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) is_last = atomicAdd(counter, 1u) == (unsigned)(count - 1);
    __syncthreads();
    if (is_last) __threadfence();
    return is_last;
}

__device__ __forceinline__ double sum_range(const double *part, int begin, int count) {
    double v = 0.0;
    for (int t = threadIdx.x; t < count; t += blockDim.x) v += __ldcg(part + begin + t);
    return block_sum(v);
}

// The largest of partial maxima of magnitudes, by their bit patterns: a NaN
// outranks every number.
__device__ __forceinline__ double max_range(const double *part, int begin, int count) {
    unsigned long long v = 0;
    for (int t = threadIdx.x; t < count; t += blockDim.x)
        v = max(v, (unsigned long long)__double_as_longlong(__ldcg(part + begin + t)));
    return __longlong_as_double((long long)block_max_bits(v));
}

// ---- pairs -----------------------------------------------------------------------

// Values of the cells (i, i+1) of a pair.
template <class T> struct Pair {
    T a, b;
};
template <class T> struct Vec2;
template <> struct Vec2<float> {
    using type = float2;
};
template <> struct Vec2<double> {
    using type = double2;
};

// v + alpha q as one fused multiply-add, written out so that every form of
// the prolongation (plane by plane, gather-first, staged) rounds alike
// whatever the compiler shares between them.
__device__ __forceinline__ float prolong(float v, float alpha, float q) { return __fmaf_rn(alpha, q, v); }
__device__ __forceinline__ double prolong(double v, double alpha, double q) { return __fma_rn(alpha, q, v); }
// s + c v, fused, for the same reason (every neighbour sum of the stencils)
__device__ __forceinline__ float fmadd(float s, float c, float v) { return __fmaf_rn(c, v, s); }
__device__ __forceinline__ double fmadd(double s, double c, double v) { return __fma_rn(c, v, s); }

// Read-only pair load: one 2-wide load when V (c even, array aligned), else
// the cells one by one (the second only if it exists).
template <class T, bool V> __device__ __forceinline__ Pair<T> ld2(const T *p, long long c, bool second) {
    if constexpr (V) {
        const typename Vec2<T>::type v = __ldg(reinterpret_cast<const typename Vec2<T>::type *>(p + c));
        return Pair<T>{v.x, v.y};
    } else {
        return Pair<T>{__ldg(p + c), second ? __ldg(p + c + 1) : T(0)};
    }
}
template <class T, bool V> __device__ __forceinline__ void st2(T *p, long long c, Pair<T> v, bool second) {
    if constexpr (V) {
        typename Vec2<T>::type w;
        w.x = v.a;
        w.y = v.b;
        *reinterpret_cast<typename Vec2<T>::type *>(p + c) = w;
    } else {
        p[c] = v.a;
        if (second) p[c + 1] = v.b;
    }
}

// The pair tile t of grid g: f(i, j, k, c, second) for each of the thread's
// tz pairs, c = index of cell i, second = (i+1 < nx).
template <class F> __device__ __forceinline__ void pair_tile1(const Grid &g, unsigned t, F f) {
    const int px = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const unsigned r = fdiv(t, g.ftx2);
    const unsigned tk = fdiv(r, g.fty);
    const int i = (int)(t - r * g.ftx2.d) * 64 + 2 * px;
    const int j = (int)(r - tk * (unsigned)g.nty) * TILE_Y + ty;
    const int k0 = (int)tk * g.tz;
    if (i >= g.nx || j >= g.ny) return;
    const int kend = min(k0 + g.tz, g.nz);
    const bool second = i + 1 < g.nx;
    const long long sz = (long long)g.nx * g.ny;
    long long c = cell_index(g, i, j, k0);
    for (int k = k0; k < kend; ++k, c += sz) f(i, j, k, c, second);
}

// cells of the cell tile t (32 x 8 x tz, one cell per thread and plane)
template <class F> __device__ __forceinline__ void cell_tile1(const Grid &g, unsigned t, F f) {
    int i0, j0, k0;
    tile_origin(g, t, i0, j0, k0);
    const int i = i0 + (threadIdx.x & (TILE_X - 1)), j = j0 + threadIdx.x / TILE_X;
    if (i >= g.nx || j >= g.ny) return;
    const int kend = min(k0 + g.tz, g.nz);
    const long long sz = (long long)g.nx * g.ny;
    long long c = cell_index(g, i, j, k0);
    for (int k = k0; k < kend; ++k, c += sz) f(i, j, k, c);
}

template <class F> __device__ __forceinline__ void pair_tile(const Grid &g, const BItem &it, F f) {
    for (int t = 0; t < it.ntiles; ++t) pair_tile1(g, (unsigned)(it.tile + t), f);
}
template <class F> __device__ __forceinline__ void cell_tile(const Grid &g, const BItem &it, F f) {
    for (int t = 0; t < it.ntiles; ++t) cell_tile1(g, (unsigned)(it.tile + t), f);
}

// A one-tile item whose tile has all 4 planes: fz(i, j, k0, c0) once per
// thread for its whole column of 4 pairs (the gather-first kernels, which
// issue every load of the column before the arithmetic); otherwise f per
// plane as pair_tile.
template <class FZ, class F>
__device__ __forceinline__ void pair_tile_z4(const Grid &g, const BItem &it, FZ fz, F f) {
    if (it.ntiles != 1 || g.tz != 4) {
        pair_tile(g, it, f);
        return;
    }
    const unsigned t = (unsigned)it.tile;
    const int px = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const unsigned r = fdiv(t, g.ftx2);
    const unsigned tk = fdiv(r, g.fty);
    const int i = (int)(t - r * g.ftx2.d) * 64 + 2 * px;
    const int j = (int)(r - tk * (unsigned)g.nty) * TILE_Y + ty;
    const int k0 = (int)tk * 4;
    if (k0 + 4 > g.nz) {
        pair_tile1(g, t, f);
        return;
    }
    if (i >= g.nx || j >= g.ny) return;
    fz(i, j, k0, cell_index(g, i, j, k0));
}

// Runs body(std::true_type) on vector levels, body(std::false_type) elsewhere.
template <class B> __device__ __forceinline__ void with_vec(int vec, B body) {
    if (vec) body(std::true_type{});
    else body(std::false_type{});
}
// body(V, U) with V as in with_vec and U = uniform couplings (tile class
// >= 0): each combination is its own straight-line code, so no load waits
// behind a branch on the class.
template <class B> __device__ __forceinline__ void with_vu(int vec, bool uni, B body) {
    if (vec) {
        if (uni) body(std::true_type{}, std::true_type{});
        else body(std::true_type{}, std::false_type{});
    } else {
        if (uni) body(std::false_type{}, std::true_type{});
        else body(std::false_type{}, std::false_type{});
    }
}

// The couplings a stencil reads: the level's arrays, or (u >= 0) the one
// value that every coupling of the current tile has (its tile class).
template <class T> struct Cpl {
    const T *cx, *cy, *cz;
    T u;
};

// The class of an item's tile (TILE_MIXED for items of several tiles, or
// without classes).
template <class T> __device__ __forceinline__ T item_class(const T *cls, const BItem &it) {
    return (cls != nullptr && it.ntiles == 1) ? __ldg(cls + it.tile) : T(TILE_MIXED);
}
// Class tests on the bit pattern (integer compares: no FP64 instruction,
// which this GPU issues at a small fraction of its FP32 rate).
__device__ __forceinline__ long long class_bits(double u) { return __double_as_longlong(u); }
__device__ __forceinline__ long long class_bits(float u) { return __float_as_int(u); }
template <class T> __device__ __forceinline__ bool tile_empty(T u) { return class_bits(u) == class_bits(T(TILE_EMPTY)); }
// Uniform tiles take the coupling-free path in FP32 only: the FP64 kernels
// are bound by the FP64 pipe, not by loads, and measure faster reading the
// couplings (empty tiles are skipped in both).
template <class T> __device__ __forceinline__ bool tile_uniform(T u) {
    return sizeof(T) == 4 && class_bits(u) >= 0;
}

// The class of item w of a list (TILE_MIXED past the end), with R the
// restriction tiling. Kernels load the class of the block's next item
// (w + G) while item w runs, so no stencil load waits on a class; `seg` is
// a copy of the caller's segment cursor.
template <class T, bool R>
__device__ __forceinline__ T class_at(const BLevel<T> *levels, const BSeg *segs, int nseg, int n, int w, int seg) {
    if (w >= n) return T(TILE_MIXED);
    const BItem it = item_at(segs, nseg, w, seg);
    return item_class(R ? levels[it.ref].tcr : levels[it.ref].tcp, it);
}
// The same for the block's next item, with the current item's level `ref`
// and class array (from the shared descriptors), used when the next item
// is of the same level (the common case: one global load instead of two).
template <class T, bool R>
__device__ __forceinline__ T class_next(const BLevel<T> *levels, const BSeg *segs, int nseg, int n, int w, int seg,
                                        int ref, const T *cls) {
    if (w >= n) return T(TILE_MIXED);
    const BItem it = item_at(segs, nseg, w, seg);
    return item_class(it.ref == ref ? cls : (R ? levels[it.ref].tcr : levels[it.ref].tcp), it);
}

// Neighbour sums of the pair (i, i+1) at c = index of cell i:
//   s.a = sum over the neighbours f of cell i of c_f v_f, s.b for cell i+1,
// in the order -x, +x, -y, +y, -z, +z. W selects the sums wanted: 0 (s.a),
// 1 (s.b) or 2 (both); the other's arithmetic and single-cell loads are
// dead code. `own` holds the pair's own values (each cell is the other's x
// neighbour); nb2(c', j', k', second) gives the neighbour pair at c' (row
// j', plane k'; its second cell exists exactly when the pair's does),
// nb1(c', i') one cell of the same row outside the pair. U: the tile's
// couplings all equal w.u, which replaces the coupling loads (the same
// products in the same order).
template <class T, bool V, bool U, int W, class NB2, class NB1>
__device__ __forceinline__ Pair<T> pair_nsum(const Grid &g, const Cpl<T> &w, int i, int j, int k, long long c,
                                              bool second, Pair<T> own, NB2 nb2, NB1 nb1) {
    constexpr bool A = W != 1, B = W != 0;
    const long long sy = g.nx, sz = (long long)g.nx * g.ny;
    Pair<T> s{T(0), T(0)};
    auto cw2 = [&](const T *a, long long m) {
        if constexpr (U) return Pair<T>{w.u, w.u};
        else return ld2<T, V>(a, m, second);
    };
    auto cw1 = [&](const T *a, long long m) {
        if constexpr (U) return w.u;
        else return __ldg(a + m);
    };
    const Pair<T> cxp = cw2(w.cx, c);  // faces (i|i+1), (i+1|i+2)
    if (A && i > 0) s.a = fmadd(s.a, cw1(w.cx, c - 1), nb1(c - 1, i - 1));
    if (second) {
        if (A) s.a = fmadd(s.a, cxp.a, own.b);
        if (B) s.b = fmadd(s.b, cxp.a, own.a);
        if (B && i + 2 < g.nx) s.b = fmadd(s.b, cxp.b, nb1(c + 2, i + 2));
    }
    auto add = [&](const Pair<T> &cw, const Pair<T> &v) {
        if (A) s.a = fmadd(s.a, cw.a, v.a);
        if (B) s.b = fmadd(s.b, cw.b, v.b);
    };
    if (j > 0) add(cw2(w.cy, c - sy), nb2(c - sy, j - 1, k, second));
    if (j + 1 < g.ny) add(cw2(w.cy, c), nb2(c + sy, j + 1, k, second));
    if (g.dim == 3) {
        if (k > 0) add(cw2(w.cz, c - sz), nb2(c - sz, j, k - 1, second));
        if (k + 1 < g.nz) add(cw2(w.cz, c), nb2(c + sz, j, k + 1, second));
    }
    return s;
}

// The neighbour sum of one cell h (0: i, 1: i+1) of the pair. h is uniform
// across a warp (a warp holds one row of pairs, i even, so the colour of
// cell i is that of j + k), so the branch does not diverge.
template <class T, bool V, bool U, class NB2, class NB1>
__device__ __forceinline__ T pair_nsum1(int h, const Grid &g, const Cpl<T> &w, int i, int j, int k, long long c,
                                        bool second, Pair<T> own, NB2 nb2, NB1 nb1) {
    if (h == 0) return pair_nsum<T, V, U, 0>(g, w, i, j, k, c, second, own, nb2, nb1).a;
    return pair_nsum<T, V, U, 1>(g, w, i, j, k, c, second, own, nb2, nb1).b;
}

// The level and scene of the current item, held in shared memory and
// reloaded only when the item's level changes (each work list holds one
// level per scene, so once per scene per block). Kernels then read the
// descriptors from shared memory instead of chasing item -> level -> scene
// pointers in global memory for every item.
template <class T> struct ItemCtx {
    BLevel<T> L;
    BScene<T> S;
    int skip;
    double alpha, beta;
    int overwrite;
};

template <class T>
__device__ __forceinline__ void refresh(ItemCtx<T> &c, int &cur_ref, const BItem &it, const BLevel<T> *levels,
                                        const BScene<T> *scenes, int gate) {
    if (it.ref == cur_ref) return;
    static_assert(sizeof(BLevel<T>) % 4 == 0 && sizeof(BScene<T>) % 4 == 0, "descriptors copied by words");
    __syncthreads();
    // the two descriptors side by side, a word a thread; the scalars' address
    // is read ahead of them
    if (threadIdx.x < 64) {
        const unsigned *src = reinterpret_cast<const unsigned *>(levels + it.ref);
        for (int q = threadIdx.x; q < (int)(sizeof(BLevel<T>) / 4); q += 64)
            reinterpret_cast<unsigned *>(&c.L)[q] = __ldg(src + q);
    } else if (threadIdx.x < 192) {
        const unsigned *src = reinterpret_cast<const unsigned *>(scenes + it.scene);
        for (int q = threadIdx.x - 64; q < (int)(sizeof(BScene<T>) / 4); q += 128)
            reinterpret_cast<unsigned *>(&c.S)[q] = __ldg(src + q);
    } else if (threadIdx.x == 192) {
        const Scalars *sc = scenes[it.scene].sc;
        c.skip = gate < 0 ? 0 : gated(sc, gate);
        c.alpha = sc->alpha;
        c.beta = sc->beta;
        c.overwrite = sc->first_update;
    }
    __syncthreads();
    cur_ref = it.ref;
}

// Blocks walk a list in groups of 2^gs consecutive items, group g on block
// g mod gridDim.x. Lists of one scene go item by item (gs = 0): neighbouring
// tiles then run at the same time and share their halos in cache. In a list of
// several scenes a block pays for every scene it meets (descriptors, gating,
// a flush of its partial: 2-4 us), so its share is dealt in groups, at least
// six a block to balance scenes of different fill. With this, the sums of
// block_sum and the descriptors copied side by side (refresh), a batch of 64
// liquids of 32^3 to 160^3 (96 items a block) went from 110.8 to 74.1 ms, six
// served scenes from 38.4 to 31.0 ms, 32^3 alone from 1.49 to 1.22 ms.
__device__ __forceinline__ int item_group(int n, int nseg) {
    if (nseg <= 1) return 0;
    const int share = n / (int)gridDim.x / 6;
    return share < 2 ? 0 : min(31 - __clz(share), 4);
}
__device__ __forceinline__ int first_item(int gs) { return (int)blockIdx.x << gs; }
__device__ __forceinline__ int next_item(int w, int gs) {
    ++w;
    return (w & ((1 << gs) - 1)) ? w : w + (((int)gridDim.x - 1) << gs);
}

// Reductions over a work list: a block walks its items (sorted by scene) and takes
// a ticket for each scene, after its last item there; the one that takes the
// scene's last ticket combines the partials. A scene whose items lie in the
// groups [g0, g1] of the list (item_group) meets min(g1 - g0 + 1, gridDim.x)
// blocks.

// Sums of a list of several scenes have one partial an item, combined in item
// order: they depend on the scene alone, not on its company, its place in the
// list or the grid. A block holds the threads' values of up to HELD items in
// shared memory and adds them with a warp an item. (One partial per block and
// scene took its items from the list's groups, and so depended on all three; a
// batch of 64 liquids took 49.4 ms with it, 51.0 here, and 53.8 with one partial
// per block over items dealt one by one.) The list of a single scene has one
// partial per block, its items w, w + grid, ...: the same bits where no block has
// two (256^3 mixed with one an item 10.36 instead of 9.88 ms).
// Acc may keep a maximum beside the sum (MAXS), as in max_items; the sums are at
// part + n then. finish(item, visits, sums): visits blocks met the scene, which
// has `sums` partial sums.
constexpr int HELD = 4;
template <class T, class Acc, class Body, class Finish>
__device__ __forceinline__ void sum_items(const BSeg *__restrict__ segs, int nseg, int n, double *part,
                                          const BLevel<T> *levels, const BScene<T> *scenes, int gate,
                                          ItemCtx<T> &ctx, Body body, Finish finish) {
    __shared__ double vals[HELD * TREE_PAD];
    const int gs = item_group(n, nseg);
    const int stride = gs ? 1 : (int)gridDim.x;  // between the items held
    int cur = -1, held = 0, newest = 0, sgc = 0;
    BItem first{};
    Acc acc;
    acc.reset();
    T cls_next = class_at<T, false>(levels, segs, nseg, n, first_item(gs), 0);
    for (int w = first_item(gs);; w = next_item(w, gs)) {
        // one level per scene in a list: a new level is a new scene
        const BItem it = w < n ? item_at(segs, nseg, w, sgc) : BItem{-1, 0, 0, 0, 0, 0};
        const bool leaves = it.ref != cur;
        if (held && (leaves || held == HELD || (gs && (w & ((1 << gs) - 1)) == 0))) {
            __syncthreads();
            const int j = threadIdx.x >> 5;
            if (j < held) {
                const double p = tree256(vals + j * TREE_PAD);
                if ((threadIdx.x & 31) == 0) part[(Acc::MAXS ? n : 0) + newest - (held - 1 - j) * stride] = p;
            }
            __syncthreads();
            held = 0;
        }
        if (leaves) {
            if (cur >= 0 && !ctx.skip) {
                const int B = gridDim.x, g0 = first.begin >> gs, g1 = (first.begin + first.count - 1) >> gs;
                if constexpr (Acc::MAXS) acc.store_max(part, first.begin + ((int)blockIdx.x - g0 % B + B) % B);
                finish(first, min(g1 - g0 + 1, B), nseg > 1 ? first.count : min(first.count, B));
            }
            if (w >= n) return;
            refresh(ctx, cur, it, levels, scenes, gate);
            first = it;
            acc.reset();
        }
        const T cls = cls_next;
        cls_next = class_next<T, false>(levels, segs, nseg, n, next_item(w, gs), sgc, it.ref, ctx.L.tcp);
        if (ctx.skip) continue;
        body(it, acc, cls);
        if (nseg > 1 || next_item(w, gs) >= n) {
            vals[held * TREE_PAD + tree_at(threadIdx.x)] = acc.sum();
            acc.reset_sum();
            ++held;
            newest = nseg > 1 ? w : (int)blockIdx.x;
        }
    }
}

// A maximum is the same in any order: one partial per (block, scene), at slot
// (b - g0) mod gridDim.x of the scene's range for block b.
template <class T, class Acc, class Body, class Finish>
__device__ __forceinline__ void max_items(const BSeg *__restrict__ segs, int nseg, int n, double *part,
                                          const BLevel<T> *levels, const BScene<T> *scenes, int gate,
                                          ItemCtx<T> &ctx, Body body, Finish finish) {
    int cur = -1;
    BItem first{};
    Acc acc;
    acc.reset();
    const int gs = item_group(n, nseg);
    auto flush = [&]() {
        const int B = gridDim.x, g0 = first.begin >> gs, g1 = (first.begin + first.count - 1) >> gs;
        const int slot = (int)((((long long)blockIdx.x - g0) % B + B) % B);
        acc.store_max(part, first.begin + slot);
        finish(first, min(g1 - g0 + 1, B));
    };
    int sgc = 0;
    T cls_next = class_at<T, false>(levels, segs, nseg, n, first_item(gs), 0);
    for (int w = first_item(gs); w < n; w = next_item(w, gs)) {
        const BItem it = item_at(segs, nseg, w, sgc);
        const T cls = cls_next;
        if (it.ref != cur) {
            if (cur >= 0 && !ctx.skip) flush();
            refresh(ctx, cur, it, levels, scenes, gate);
            first = it;
            acc.reset();
        }
        cls_next = class_next<T, false>(levels, segs, nseg, n, next_item(w, gs), sgc, it.ref, ctx.L.tcp);
        if (!ctx.skip) body(it, acc, cls);
    }
    if (cur >= 0 && !ctx.skip) flush();
}

// Per-thread partials of the reductions. FP64 path: FP64 FMA per term.
// FP32 path: FloatFloat::add_product (gbp_floatfloat.cuh: the product split
// exactly by an FMA, TwoSum, renormalised after every term; a thread's n
// terms within gamma_n^2 sum |a_i b_i|); a partial is converted to FP64 once,
// when its item or block ends, and partials add across threads and blocks in FP64. The
// FP32 path then issues no FP64 instruction per cell (the FP64 pipe of this
// GPU runs at a small fraction of its FP32 rate). It assumes |a b| stays
// inside the FP32 range, as the FP32 inner solve does for its vectors.
// sum() is the thread's partial; store() (the staged kernels) adds the block's and
// publishes it at slot idx of the list's partials, store_max() its maximum.
template <class T> struct DotAcc;
template <> struct DotAcc<double> {
    static constexpr bool MAXS = false;
    double v;
    __device__ void reset() { v = 0.0; }
    __device__ void add(double a, double b) { v = fma(a, b, v); }
    __device__ double sum() const { return v; }
    __device__ void reset_sum() { reset(); }
    __device__ double block() { return block_sum(v); }
    __device__ void store(double *part, int idx) {
        const double b = block();
        if (threadIdx.x == 0) part[idx] = b;
    }
};
template <> struct DotAcc<float> {
    static constexpr bool MAXS = false;
    FloatFloat f;
    __device__ void reset() { f.reset(); }
    __device__ void add(float a, float b) { f.add_product(a, b); }
    __device__ double sum() const { return f.value_fp64(); }
    __device__ void reset_sum() { reset(); }
    __device__ double block() { return block_sum(f.value_fp64()); }
    __device__ void store(double *part, int idx) {
        const double b = block();
        if (threadIdx.x == 0) part[idx] = b;
    }
};
// max |x|, exact, on bit patterns: no FP64 comparison per cell (which takes
// an FP64 pipe slot). NaN terms are ignored, as fmax ignores them; NaN is
// caught through alpha.
template <class T> struct MaxAcc;
template <> struct MaxAcc<double> {
    unsigned long long v;
    __device__ void reset() { v = 0ull; }
    __device__ void add(double x) { v = max(v, abs_bits(x)); }
    __device__ void store_max(double *part, int idx) {
        const unsigned long long b = block_max_bits(v);
        if (threadIdx.x == 0) part[idx] = __longlong_as_double((long long)b);
    }
};
template <> struct MaxAcc<float> {
    float v;
    __device__ void reset() { v = 0.0f; }
    __device__ void add(float x) { v = fmaxf(v, fabsf(x)); }
    __device__ void store_max(double *part, int idx) {
        __shared__ unsigned maxs[BLOCK_THREADS / 32];
        unsigned b = __reduce_max_sync(0xffffffffu, __float_as_uint(v));
        __syncthreads();
        if ((threadIdx.x & 31) == 0) maxs[threadIdx.x >> 5] = b;
        __syncthreads();
        if (threadIdx.x < 32) {
            b = __reduce_max_sync(0xffffffffu, threadIdx.x < BLOCK_THREADS / 32 ? maxs[threadIdx.x] : 0u);
            if (threadIdx.x == 0) part[idx] = widen(__uint_as_float(b));
        }
    }
};
// The refinement residual's norms (partials at idx and n + idx): max |x|
// of the FP64 residual, exact, taken on the bit patterns (integer compares:
// no FP64 instruction; a NaN outranks every number, so it reaches the
// stopping rule), and the sum of squares of its T copy with the dot
// product's accumulation (float-float for T = float), which only reports
// the L2 norm.
template <class T> struct MaxSumAcc {
    static constexpr bool MAXS = true;
    unsigned long long m;
    DotAcc<T> s;
    __device__ void reset() {
        m = 0ull;
        s.reset();
    }
    __device__ void add(double x, T xt) {
        const unsigned long long b = (unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffull;
        m = b > m ? b : m;
        s.add(xt, xt);
    }
    __device__ double sum() const { return s.sum(); }
    __device__ void reset_sum() { s.reset(); }
    __device__ void store_max(double *part, int idx) {
        const unsigned long long b = block_max_bits(m);
        if (threadIdx.x == 0) part[idx] = __longlong_as_double((long long)b);
    }
};

// ---- smoothing and transfers on the global-memory levels --------------------------

// First pre-smoothing pass over a gather-first column (the form of
// spmv_col4): red cells x = b inv, black cells from their red neighbours'
// b inv, with the products and sums of the plane-by-plane form. The black
// cell of each pair is cell i+1 where i + j + k is even, else cell i; only
// that side of each neighbour pair is read.
template <class T>
__device__ __forceinline__ void presmooth_col4(const Grid &g, T u, T *x, const T *b, const T *inv, int i, int j,
                                               int k0, long long c0) {
    const long long sy = g.nx, sz = (long long)g.nx * g.ny;
    Pair<T> bo[4], io[4];
    T yb[4][2], yi[4][2], xb[4], xi[4];
    const int h0 = ((i + j + k0) & 1) ^ 1;  // black side of plane k0 (alternates with z)
    T zb[2] = {T(0), T(0)}, zi[2] = {T(0), T(0)};
    if (k0 > 0) {
        zb[0] = __ldg(b + c0 - sz + h0);
        zi[0] = __ldg(inv + c0 - sz + h0);
    }
    if (k0 + 4 < g.nz) {
        zb[1] = __ldg(b + c0 + 4 * sz + (h0 ^ 1));
        zi[1] = __ldg(inv + c0 + 4 * sz + (h0 ^ 1));
    }
#pragma unroll
    for (int z = 0; z < 4; ++z) {
        const long long c = c0 + z * sz;
        const int h = h0 ^ (z & 1);
        bo[z] = ld2<T, true>(b, c, true);
        io[z] = ld2<T, true>(inv, c, true);
        yb[z][0] = yi[z][0] = yb[z][1] = yi[z][1] = T(0);
        if (j > 0) {
            yb[z][0] = __ldg(b + c - sy + h);
            yi[z][0] = __ldg(inv + c - sy + h);
        }
        if (j + 1 < g.ny) {
            yb[z][1] = __ldg(b + c + sy + h);
            yi[z][1] = __ldg(inv + c + sy + h);
        }
        const long long xc = h == 0 ? c - 1 : c + 2;
        const bool xin = h == 0 ? i > 0 : i + 2 < g.nx;
        xb[z] = xin ? __ldg(b + xc) : T(0);
        xi[z] = xin ? __ldg(inv + xc) : T(0);
    }
#pragma unroll
    for (int z = 0; z < 4; ++z) {
        const int k = k0 + z;
        const int h = h0 ^ (z & 1);
        const Pair<T> red{bo[z].a * io[z].a, bo[z].b * io[z].b};
        // the black side's z neighbours (red): the same side of the planes around
        const T zm = z == 0 ? zb[0] * zi[0] : (h ? bo[z - 1].b * io[z - 1].b : bo[z - 1].a * io[z - 1].a);
        const T zp = z == 3 ? zb[1] * zi[1] : (h ? bo[z + 1].b * io[z + 1].b : bo[z + 1].a * io[z + 1].a);
        T s = T(0);
        if (h == 0) {
            if (i > 0) s = fmadd(s, u, (xb[z] * xi[z]));
            s = fmadd(s, u, red.b);
        } else {
            s = fmadd(s, u, red.a);
            if (i + 2 < g.nx) s = fmadd(s, u, (xb[z] * xi[z]));
        }
        if (j > 0) s = fmadd(s, u, (yb[z][0] * yi[z][0]));
        if (j + 1 < g.ny) s = fmadd(s, u, (yb[z][1] * yi[z][1]));
        if (k > 0) s = fmadd(s, u, zm);
        if (k + 1 < g.nz) s = fmadd(s, u, zp);
        Pair<T> out = red;
        if (h) out.b = (bo[z].b + s) * io[z].b;
        else out.a = (bo[z].a + s) * io[z].a;
        st2<T, true>(x, c0 + z * sz, out, true);
    }
}

// First pre-smoothing pass from x = 0: red x = b / diag, then black from the
// red neighbours (computed on the fly as b inv), both written.
// COL: use presmooth_col4 where it applies (the cooperative coarse kernels,
// whose levels seldom have 4-plane tiles, leave it out to save registers).
template <class T, bool COL>
__device__ __forceinline__ void presmooth_items(const BLevel<T> *__restrict__ levels, const BSeg *__restrict__ segs, int nseg,
        int n, const BScene<T> *__restrict__ scenes, int gate, ItemCtx<T> &ctx) {
    int cur = -1;
    int sgc = 0;
    const int gs = item_group(n, nseg);
    T cls_next = class_at<T, false>(levels, segs, nseg, n, first_item(gs), 0);
    for (int w = first_item(gs); w < n; w = next_item(w, gs)) {
        const BItem it = item_at(segs, nseg, w, sgc);
        const T cls = cls_next;
        refresh(ctx, cur, it, levels, scenes, gate);
        cls_next = class_next<T, false>(levels, segs, nseg, n, next_item(w, gs), sgc, it.ref, ctx.L.tcp);
        if (ctx.skip) continue;
        const BLevel<T> L = ctx.L;  // registers: stores through generic pointers would force reloads from shared memory
        const Cpl<T> cw{L.cx, L.cy, L.cz, cls};
        with_vu(L.vec, tile_uniform(cw.u), [&](auto vt, auto ut) {
            constexpr bool V = decltype(vt)::value;
            constexpr bool U = decltype(ut)::value;
            if (tile_empty(cw.u)) {  // no unknown: x = 0
                pair_tile(L.g, it, [&](int, int, int, long long c, bool second) {
                    st2<T, V>(L.x, c, Pair<T>{T(0), T(0)}, second);
                });
                return;
            }
            auto nb2 = [&](long long m, int, int, bool sec) {
                const Pair<T> bb = ld2<T, V>(L.b, m, sec), ii = ld2<T, V>(L.inv, m, sec);
                return Pair<T>{bb.a * ii.a, bb.b * ii.b};
            };
            auto nb1 = [&](long long m, int) { return __ldg(L.b + m) * __ldg(L.inv + m); };
            auto plane = [&](int i, int j, int k, long long c, bool second) {
                const bool a_red = ((i + j + k) & 1) == 0;
                const Pair<T> b2 = ld2<T, V>(L.b, c, second), iv = ld2<T, V>(L.inv, c, second);
                const Pair<T> red{b2.a * iv.a, b2.b * iv.b};
                Pair<T> out = red;
                if (a_red) {
                    if (second)
                        out.b = (b2.b + pair_nsum1<T, V, U>(1, L.g, cw, i, j, k, c, second, red, nb2, nb1)) *
                                iv.b;
                } else {
                    out.a = (b2.a + pair_nsum1<T, V, U>(0, L.g, cw, i, j, k, c, second, red, nb2, nb1)) *
                            iv.a;
                }
                st2<T, V>(L.x, c, out, second);
            };
            if constexpr (COL && U && V)
                pair_tile_z4(L.g, it, [&](int i, int j, int k0, long long c0) {
                    presmooth_col4<T>(L.g, cw.u, L.x, L.b, L.inv, i, j, k0, c0);
                }, plane);
            else
                pair_tile(L.g, it, plane);
        });
    }
}

template <class T, int OCC, bool COL>
__global__ void __launch_bounds__(BLOCK_THREADS, OCC)
    presmooth_kernel(const BLevel<T> *__restrict__ levels, const BSeg *__restrict__ segs, int nseg, int n,
                  const BScene<T> *__restrict__ scenes, int gate, const BatchCounters *live) {
    if (batch_idle(live)) return;
    __shared__ ItemCtx<T> ctx;
    presmooth_items<T, COL>(levels, segs, nseg, n, scenes, gate, ctx);
}

// One colour of a Gauss-Seidel sweep (extra smoothing sweeps, and the final
// red pass of the post-smoothing on coarse levels).
template <class T>
__device__ __forceinline__ void sweep_items(const BLevel<T> *__restrict__ levels, const BSeg *__restrict__ segs, int nseg,
        int n, const BScene<T> *__restrict__ scenes, int gate, int color, ItemCtx<T> &ctx) {
    int cur = -1;
    int sgc = 0;
    const int gs = item_group(n, nseg);
    T cls_next = class_at<T, false>(levels, segs, nseg, n, first_item(gs), 0);
    for (int w = first_item(gs); w < n; w = next_item(w, gs)) {
        const BItem it = item_at(segs, nseg, w, sgc);
        const T cls = cls_next;
        refresh(ctx, cur, it, levels, scenes, gate);
        cls_next = class_next<T, false>(levels, segs, nseg, n, next_item(w, gs), sgc, it.ref, ctx.L.tcp);
        if (ctx.skip) continue;
        const BLevel<T> L = ctx.L;  // registers: stores through generic pointers would force reloads from shared memory
        const Cpl<T> cw{L.cx, L.cy, L.cz, cls};
        if (tile_empty(cw.u)) continue;  // x stays 0 (written by the presmoothing)
        with_vu(L.vec, tile_uniform(cw.u), [&](auto vt, auto ut) {
            constexpr bool V = decltype(vt)::value;
            constexpr bool U = decltype(ut)::value;
            auto nb2 = [&](long long m, int, int, bool sec) { return ld2<T, V>(L.x, m, sec); };
            auto nb1 = [&](long long m, int) { return __ldg(L.x + m); };
            pair_tile(L.g, it, [&](int i, int j, int k, long long c, bool second) {
                const int h = ((i + j + k) & 1) == color ? 0 : 1;
                if (h == 1 && !second) return;
                const Pair<T> x2 = ld2<T, V>(L.x, c, second);
                const T sh = pair_nsum1<T, V, U>(h, L.g, cw, i, j, k, c, second, x2, nb2, nb1);
                const long long ch = c + h;
                L.x[ch] = (__ldg(L.b + ch) + sh) * __ldg(L.inv + ch);
            });
        });
    }
}

template <class T, int OCC>
__global__ void __launch_bounds__(BLOCK_THREADS, OCC)
    sweep_kernel(const BLevel<T> *__restrict__ levels, const BSeg *__restrict__ segs, int nseg, int n,
                  const BScene<T> *__restrict__ scenes, int gate, int color, const BatchCounters *live) {
    if (batch_idle(live)) return;
    __shared__ ItemCtx<T> ctx;
    sweep_items<T>(levels, segs, nseg, n, scenes, gate, color, ctx);
}

// b - (d x - s), the residual of a cell from its neighbour sum s, with
// explicit roundings so that every form of the restriction rounds alike
__device__ __forceinline__ float resid(float b, float d, float x, float s) { return __fsub_rn(b, __fmaf_rn(d, x, -s)); }
__device__ __forceinline__ double resid(double b, double d, double x, double s) {
    return __dsub_rn(b, __fma_rn(d, x, -s));
}

// The restriction's residual of the red children (i + h, j0 + b2, k0 + c2)
// of a coarse cell, one per child pair: the pre-smoothing ends on a black
// half-sweep, after which the black cells' residual is zero (to rounding), so
// only the red half is formed. Each red cell's neighbours are black. All loads
// come before the arithmetic; U: every coupling of the tile is w.u. The sums
// keep the order -x, +x, -y, +y, -z, +z and the children's (z, y) order.
// 256^3: FP64 281 -> 146 us (half the FP64 operations), mixed 57 -> 46 us; a
// batch of 64 liquids 224 -> 150 us.
template <class T, bool U>
__device__ __forceinline__ T restrict_cell(const Grid &g, const Cpl<T> &w, const T *x, const T *b, const T *diag,
                                           int i, int j0, int k0) {
    const long long sy = g.nx, sz = (long long)g.nx * g.ny;
    const bool d3 = g.dim == 3;
    T sum = T(0);
    if (U && i + 1 < g.nx && j0 + 1 < g.ny && (!d3 || k0 + 1 < g.nz) && d3) {
        // all eight children: red R, black B, the outer neighbours of the reds
        T R[2][2], B[2][2], bb[2][2], dd[2][2], ox[2][2], oy[2][2], oz[2][2];
        bool hx[2][2];
        const bool hy[2] = {j0 > 0, j0 + 2 < g.ny}, hz[2] = {k0 > 0, k0 + 2 < g.nz};
        const long long f0 = cell_index(g, i, j0, k0);
#pragma unroll
        for (int c2 = 0; c2 < 2; ++c2)
#pragma unroll
            for (int b2 = 0; b2 < 2; ++b2) {
                const int h = (b2 + c2) & 1;
                const long long f = f0 + c2 * sz + b2 * sy;
                R[c2][b2] = __ldg(x + f + h);
                B[c2][b2] = __ldg(x + f + 1 - h);
                bb[c2][b2] = __ldg(b + f + h);
                dd[c2][b2] = __ldg(diag + f + h);
                hx[c2][b2] = h == 0 ? i > 0 : i + 2 < g.nx;
                ox[c2][b2] = hx[c2][b2] ? __ldg(x + (h == 0 ? f - 1 : f + 2)) : T(0);
                oy[c2][b2] = hy[b2] ? __ldg(x + f + h + (b2 ? sy : -sy)) : T(0);
                oz[c2][b2] = hz[c2] ? __ldg(x + f + h + (c2 ? sz : -sz)) : T(0);
            }
#pragma unroll
        for (int c2 = 0; c2 < 2; ++c2)
#pragma unroll
            for (int b2 = 0; b2 < 2; ++b2) {
                const int h = (b2 + c2) & 1;
                T s = T(0);
                if (h == 0) {
                    if (hx[c2][b2]) s = fmadd(s, w.u, ox[c2][b2]);
                    s = fmadd(s, w.u, B[c2][b2]);
                } else {
                    s = fmadd(s, w.u, B[c2][b2]);
                    if (hx[c2][b2]) s = fmadd(s, w.u, ox[c2][b2]);
                }
                const T yi = B[c2][1 - b2], zi = B[1 - c2][b2];
                if (b2) s = fmadd(s, w.u, yi);
                if (hy[b2]) s = fmadd(s, w.u, oy[c2][b2]);
                if (!b2) s = fmadd(s, w.u, yi);
                if (c2) s = fmadd(s, w.u, zi);
                if (hz[c2]) s = fmadd(s, w.u, oz[c2][b2]);
                if (!c2) s = fmadd(s, w.u, zi);
                sum += resid(bb[c2][b2], dd[c2][b2], R[c2][b2], s);
            }
        return sum;
    }
    const int kmax = d3 ? 2 : 1;
    for (int c2 = 0; c2 < kmax; ++c2)
        for (int b2 = 0; b2 < 2; ++b2) {
            const int j = j0 + b2, k = k0 + c2, ii = i + ((j + k) & 1);
            if (j >= g.ny || k >= g.nz || ii >= g.nx) continue;
            const long long f = cell_index(g, ii, j, k);
            const bool on[6] = {ii > 0, ii + 1 < g.nx, j > 0, j + 1 < g.ny, d3 && k > 0, d3 && k + 1 < g.nz};
            T c[6], v[6];
#pragma unroll
            for (int q = 0; q < 6; ++q) {
                const long long step = q < 2 ? 1 : (q < 4 ? sy : sz);
                const T *cp = q < 2 ? w.cx : (q < 4 ? w.cy : w.cz);
                c[q] = U ? w.u : (on[q] ? __ldg(cp + (q & 1 ? f : f - step)) : T(0));
                v[q] = on[q] ? __ldg(x + (q & 1 ? f + step : f - step)) : T(0);
            }
            const T bb = __ldg(b + f), dd = __ldg(diag + f), xx = __ldg(x + f);
            T s = T(0);
#pragma unroll
            for (int q = 0; q < 6; ++q)
                if (on[q]) s = fmadd(s, c[q], v[q]);
            sum += resid(bb, dd, xx, s);
        }
    return sum;
}

// Items are cell tiles of the coarse grid gc; a thread sums the residuals
// b - A x of the red children of its coarse cell (restrict_cell).
template <class T>
__device__ __forceinline__ void restrict_items(const BLevel<T> *__restrict__ levels, const BSeg *__restrict__ segs, int nseg,
        int n, const BScene<T> *__restrict__ scenes, int gate, ItemCtx<T> &ctx) {
    int cur = -1;
    int sgc = 0;
    const int gs = item_group(n, nseg);
    T cls_next = class_at<T, true>(levels, segs, nseg, n, first_item(gs), 0);
    for (int w = first_item(gs); w < n; w = next_item(w, gs)) {
        const BItem it = item_at(segs, nseg, w, sgc);
        const T cls = cls_next;
        refresh(ctx, cur, it, levels, scenes, gate);
        cls_next = class_next<T, true>(levels, segs, nseg, n, next_item(w, gs), sgc, it.ref, ctx.L.tcr);
        if (ctx.skip) continue;
        const BLevel<T> L = ctx.L;  // registers: stores through generic pointers would force reloads from shared memory
        const Cpl<T> cw{L.cx, L.cy, L.cz, cls};
        if (tile_empty(cw.u)) {  // no unknown among the children: b_c = 0
            cell_tile(L.gc, it, [&](int, int, int, long long cc) { L.bc[cc] = T(0); });
        } else if (tile_uniform(cw.u)) {
            cell_tile(L.gc, it, [&](int I, int J, int K, long long cc) {
                L.bc[cc] = restrict_cell<T, true>(L.g, cw, L.x, L.b, L.diag, 2 * I, 2 * J, 2 * K);
            });
        } else {
            cell_tile(L.gc, it, [&](int I, int J, int K, long long cc) {
                L.bc[cc] = restrict_cell<T, false>(L.g, cw, L.x, L.b, L.diag, 2 * I, 2 * J, 2 * K);
            });
        }
    }
}

template <class T, int OCC>
__global__ void __launch_bounds__(BLOCK_THREADS, OCC)
    restrict_kernel(const BLevel<T> *__restrict__ levels, const BSeg *__restrict__ segs, int nseg, int n,
                  const BScene<T> *__restrict__ scenes, int gate, const BatchCounters *live) {
    if (batch_idle(live)) return;
    __shared__ ItemCtx<T> ctx;
    restrict_items<T>(levels, segs, nseg, n, scenes, gate, ctx);
}

// Prolongation and black half-sweep of one thread's NP planes from k0 (its
// pairs (i, i+1) of row j). The pre-smoothing left every black cell at
// (b + sum c x_red) / d with the red values that are still there, so the sweep
// after the coarse correction e (piecewise constant, times alpha) adds only
//   alpha / d (sum c e)
// and reads neither b nor a neighbour's x: per black cell its own value, its
// inverse diagonal and the parents' corrections. Half of its neighbours share
// its own parent (one per axis), whose couplings are added first. U: every
// coupling is w.u. The operations and their order are the same for every NP
// and U (a coupling or parent that is not there counts as 0).
// 256^3: mixed 73 -> 40 us, FP64 216 -> 132 us; a batch of 64 liquids 279 ->
// 126 us.
template <class T, bool U, int NP>
__device__ __forceinline__ void post_black_planes(const Grid &g, const Grid &cg, const Cpl<T> &w, T alpha, T *x,
                                                  const T *inv, const T *xc, int i, int j, int k0, long long c0) {
    const long long sy = g.nx, sz = (long long)g.nx * g.ny;
    const long long csy = cg.nx, csz = (long long)cg.nx * cg.ny;
    const bool d3 = g.dim == 3, second = i + 1 < g.nx, yodd = (j & 1) != 0;
    const bool yin = yodd || j + 1 < g.ny, yout = yodd ? j + 1 < g.ny : j > 0;
    const long long pyo = yodd ? csy : -csy;
    T xo[NP], iv[NP], eo[NP], ex[NP], ey[NP], ez[NP], cix[NP], ciy[NP], ciz[NP], cox[NP], coy[NP], coz[NP];
    bool on[NP];
#pragma unroll
    for (int z = 0; z < NP; ++z) {
        const int k = k0 + z, h = ((j + k) & 1) == 1 ? 0 : 1;  // i is even
        const long long c = c0 + z * sz + h;
        const long long P = cell_index(cg, i >> 1, j >> 1, d3 ? (k >> 1) : 0);
        const bool zodd = (k & 1) != 0, xout = h == 0 ? i > 0 : i + 2 < g.nx;
        const bool zin = d3 && (zodd || k + 1 < g.nz), zout = d3 && (zodd ? k + 1 < g.nz : k > 0);
        on[z] = h == 0 || second;
        xo[z] = on[z] ? __ldg(x + c) : T(0);
        iv[z] = on[z] ? __ldg(inv + c) : T(0);
        eo[z] = __ldg(xc + P);
        ex[z] = xout ? __ldg(xc + P + (h == 0 ? -1 : 1)) : T(0);
        ey[z] = yout ? __ldg(xc + P + pyo) : T(0);
        ez[z] = zout ? __ldg(xc + P + (zodd ? csz : -csz)) : T(0);
        if constexpr (U) {
            cix[z] = second ? w.u : T(0);
            ciy[z] = yin ? w.u : T(0);
            ciz[z] = zin ? w.u : T(0);
            cox[z] = xout ? w.u : T(0);
            coy[z] = yout ? w.u : T(0);
            coz[z] = zout ? w.u : T(0);
        } else {
            // the pair's own face is at its first cell, the faces to j - 1 and
            // k - 1 one row and plane back
            cix[z] = on[z] && second ? __ldg(w.cx + c - h) : T(0);
            cox[z] = on[z] && xout ? __ldg(w.cx + (h == 0 ? c - 1 : c)) : T(0);
            ciy[z] = on[z] && yin ? __ldg(w.cy + (yodd ? c - sy : c)) : T(0);
            coy[z] = on[z] && yout ? __ldg(w.cy + (yodd ? c : c - sy)) : T(0);
            ciz[z] = on[z] && zin ? __ldg(w.cz + (zodd ? c - sz : c)) : T(0);
            coz[z] = on[z] && zout ? __ldg(w.cz + (zodd ? c : c - sz)) : T(0);
        }
    }
#pragma unroll
    for (int z = 0; z < NP; ++z) {
        if (!on[z]) continue;
        const int h = ((j + k0 + z) & 1) == 1 ? 0 : 1;
        T s = ((cix[z] + ciy[z]) + ciz[z]) * eo[z];
        s = fmadd(s, cox[z], ex[z]);
        s = fmadd(s, coy[z], ey[z]);
        s = fmadd(s, coz[z], ez[z]);
        x[c0 + z * sz + h] = fmadd(xo[z], alpha * iv[z], s);
    }
}

// Prolongation fused with the black half of the post-smoothing (see
// post_black_planes), four planes at a time in uniform tiles, two in FP32
// tiles with arrays of couplings.
template <class T, bool COL>
__device__ __forceinline__ void post_black_items(const BLevel<T> *__restrict__ levels, const BSeg *__restrict__ segs, int nseg,
        int n, const BScene<T> *__restrict__ scenes, int gate, T alpha, ItemCtx<T> &ctx) {
    int cur = -1;
    int sgc = 0;
    const int gs = item_group(n, nseg);
    T cls_next = class_at<T, false>(levels, segs, nseg, n, first_item(gs), 0);
    for (int w = first_item(gs); w < n; w = next_item(w, gs)) {
        const BItem it = item_at(segs, nseg, w, sgc);
        const T cls = cls_next;
        refresh(ctx, cur, it, levels, scenes, gate);
        cls_next = class_next<T, false>(levels, segs, nseg, n, next_item(w, gs), sgc, it.ref, ctx.L.tcp);
        if (ctx.skip) continue;
        const BLevel<T> L = ctx.L;  // registers: stores through generic pointers would force reloads from shared memory
        const Cpl<T> cw{L.cx, L.cy, L.cz, cls};
        if (tile_empty(cw.u)) continue;  // x stays 0 (written by the presmoothing)
        auto tile = [&](auto ut) {
            constexpr bool U = decltype(ut)::value;
            auto plane = [&](int i, int j, int k, long long c, bool) {
                post_black_planes<T, U, 1>(L.g, L.gc, cw, alpha, L.x, L.inv, L.xc, i, j, k, c);
            };
            if constexpr (COL && sizeof(T) == 4)
                pair_tile_z4(L.g, it, [&](int i, int j, int k0, long long c0) {
                    if constexpr (U) {
                        post_black_planes<T, U, 4>(L.g, L.gc, cw, alpha, L.x, L.inv, L.xc, i, j, k0, c0);
                    } else {
                        const long long sz = (long long)L.g.nx * L.g.ny;
                        post_black_planes<T, U, 2>(L.g, L.gc, cw, alpha, L.x, L.inv, L.xc, i, j, k0, c0);
                        post_black_planes<T, U, 2>(L.g, L.gc, cw, alpha, L.x, L.inv, L.xc, i, j, k0 + 2, c0 + 2 * sz);
                    }
                }, plane);
            else
                pair_tile(L.g, it, plane);
        };
        if (tile_uniform(cw.u)) tile(std::true_type{});
        else tile(std::false_type{});
    }
}

template <class T, int OCC, bool COL>
__global__ void __launch_bounds__(BLOCK_THREADS, OCC)
    post_black_kernel(const BLevel<T> *__restrict__ levels, const BSeg *__restrict__ segs, int nseg, int n,
                  const BScene<T> *__restrict__ scenes, int gate, T alpha, const BatchCounters *live) {
    if (batch_idle(live)) return;
    __shared__ ItemCtx<T> ctx;
    post_black_items<T, COL>(levels, segs, nseg, n, scenes, gate, alpha, ctx);
}

// ---- coarse levels in two cooperative launches -------------------------------------

// Grid-wide barrier of a cooperative launch (every block resident): the blocks
// add to cnt->bar_count, never reset within a solve, and wait until the count
// reaches the barrier's end (gbp_barrier.cuh; one atomic and polls of the
// same word; a reset and a separate generation word took two more trips to L2,
// and a sleep between polls another 0.1 us: the two cooperative kernels went
// from 50 to 42 us an iteration at 128^3, 155 to 123 us at 256^3). The wait is bounded (about two
// seconds); a block whose wait runs out records cnt->bar_err and leaves the
// kernel, the others run out the same way, and the host reports the error.
__device__ __forceinline__ bool grid_barrier(BatchCounters *cnt) {
    __syncthreads();
    int good = 1;
    if (threadIdx.x == 0) {
        if (cnt->test_what == 1 && (int)blockIdx.x == cnt->test_block) {
            // test hook: this block never arrives (as if it had stopped);
            // the others' waits run out
            good = 0;
        } else {
            unsigned seen;
            const unsigned step = barrier_step(blockIdx.x, gridDim.x);
            asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], %2;"
                         : "=r"(seen) : "l"(&cnt->bar_count), "r"(step) : "memory");
            const unsigned end = barrier_end(seen, gridDim.x);
            const int limit = cnt->test_polls > 0 ? cnt->test_polls : (1 << 22);
            seen += step;
            for (int it = 0; !barrier_reached(seen, end); ++it) {
                if (it > limit) {
                    good = 0;
                    atomicExch(&cnt->bar_err, 1);
                    break;
                }
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(&cnt->bar_count) : "memory");
            }
        }
    }
    return __syncthreads_and(good) != 0;
}

// Levels first..last top-down: presmooth, extra sweeps, restriction. The
// idle test at the start reads a counter no block changes during the
// launch, so either every block returns there or none does.
template <class T, int OCCB>
__global__ void __launch_bounds__(BLOCK_THREADS, OCCB)
    coarse_descend_kernel(const BLevel<T> *__restrict__ levels, const CoarseLists cl,
                          const BScene<T> *__restrict__ scenes, int gate, MgSettings ms, BatchCounters *cnt) {
    if (batch_idle(cnt)) return;
    __shared__ ItemCtx<T> ctx;
    for (int l = cl.first; l <= cl.last; ++l) {
        presmooth_items<T, false>(levels, cl.pair[l], cl.pair_seg[l], cl.pair_n[l], scenes, gate, ctx);
        if (!grid_barrier(cnt)) return;
        for (int sw = 1; sw < ms.smooth; ++sw)
            for (int color = 0; color < 2; ++color) {
                sweep_items<T>(levels, cl.pair[l], cl.pair_seg[l], cl.pair_n[l], scenes, gate, color, ctx);
                if (!grid_barrier(cnt)) return;
            }
        restrict_items<T>(levels, cl.restr[l], cl.restr_seg[l], cl.restr_n[l], scenes, gate, ctx);
        if (l < cl.last && !grid_barrier(cnt)) return;
    }
}

// Levels last..first bottom-up: prolongation with the black sweep, extra
// sweeps, the red sweep.
template <class T, int OCCB>
__global__ void __launch_bounds__(BLOCK_THREADS, OCCB)
    coarse_ascend_kernel(const BLevel<T> *__restrict__ levels, const CoarseLists cl,
                         const BScene<T> *__restrict__ scenes, int gate, MgSettings ms, T alpha, BatchCounters *cnt) {
    if (batch_idle(cnt)) return;
    __shared__ ItemCtx<T> ctx;
    for (int l = cl.last; l >= cl.first; --l) {
        post_black_items<T, false>(levels, cl.pair[l], cl.pair_seg[l], cl.pair_n[l], scenes, gate, alpha, ctx);
        if (!grid_barrier(cnt)) return;
        for (int sw = 1; sw < ms.smooth; ++sw)
            for (int color = 0; color < 2; ++color) {
                sweep_items<T>(levels, cl.pair[l], cl.pair_seg[l], cl.pair_n[l], scenes, gate, color, ctx);
                if (!grid_barrier(cnt)) return;
            }
        sweep_items<T>(levels, cl.pair[l], cl.pair_seg[l], cl.pair_n[l], scenes, gate, 0, ctx);
        if (l > cl.first && !grid_barrier(cnt)) return;
    }
}

// Gather-first columns: one thread's 4 pairs (i, i+1) x rows j x planes
// k0..k0+3 of a uniform tile (coupling u) on a vector level (nx even, so
// every pair is whole). Every load of the column is issued before the
// arithmetic: the planes' own pairs k0-1..k0+4 (whose neighbours in z are
// each other), the +-y pairs and the +-x cells. The plane-by-plane form
// cannot hoist them, as its stores could alias the next plane's loads.
// Products, their order (that of pair_nsum: -x, +x, -y, +y, -z, +z) and the
// dot-product terms are those of the plane-by-plane form, so the results
// are bitwise the same.
template <class T> struct Col4 {
    Pair<T> z[6];        // own pairs of planes k0-1 .. k0+4 (0 outside the grid)
    Pair<T> ym[4], yp[4];  // rows j-1, j+1
};
template <class T>
__device__ __forceinline__ void load_col4(Col4<T> &q, const T *v, const Grid &g, int j, int k0, long long c0) {
    const long long sy = g.nx, sz = (long long)g.nx * g.ny;
    const Pair<T> zero{T(0), T(0)};
    q.z[0] = k0 > 0 ? ld2<T, true>(v, c0 - sz, true) : zero;
    q.z[5] = k0 + 4 < g.nz ? ld2<T, true>(v, c0 + 4 * sz, true) : zero;
#pragma unroll
    for (int z = 0; z < 4; ++z) {
        const long long c = c0 + z * sz;
        q.z[z + 1] = ld2<T, true>(v, c, true);
        q.ym[z] = j > 0 ? ld2<T, true>(v, c - sy, true) : zero;
        q.yp[z] = j + 1 < g.ny ? ld2<T, true>(v, c + sy, true) : zero;
    }
}

// q = A p and p . q over a column (spmv)
template <class T>
__device__ __forceinline__ void spmv_col4(const Grid &g, T u, const T *p, const T *diag, T *qv, int i, int j, int k0,
                                          long long c0, DotAcc<T> &acc) {
    const long long sz = (long long)g.nx * g.ny;
    Col4<T> P;
    load_col4(P, p, g, j, k0, c0);
    T xm[4], xp[4];
    Pair<T> dv[4];
#pragma unroll
    for (int z = 0; z < 4; ++z) {
        const long long c = c0 + z * sz;
        xm[z] = i > 0 ? __ldg(p + c - 1) : T(0);
        xp[z] = i + 2 < g.nx ? __ldg(p + c + 2) : T(0);
        dv[z] = ld2<T, true>(diag, c, true);
    }
#pragma unroll
    for (int z = 0; z < 4; ++z) {
        const int k = k0 + z;
        const Pair<T> own = P.z[z + 1];
        Pair<T> s{T(0), T(0)};
        if (i > 0) s.a = fmadd(s.a, u, xm[z]);
        s.a = fmadd(s.a, u, own.b);
        s.b = fmadd(s.b, u, own.a);
        if (i + 2 < g.nx) s.b = fmadd(s.b, u, xp[z]);
        if (j > 0) {
            s.a = fmadd(s.a, u, P.ym[z].a);
            s.b = fmadd(s.b, u, P.ym[z].b);
        }
        if (j + 1 < g.ny) {
            s.a = fmadd(s.a, u, P.yp[z].a);
            s.b = fmadd(s.b, u, P.yp[z].b);
        }
        if (k > 0) {
            s.a = fmadd(s.a, u, P.z[z].a);
            s.b = fmadd(s.b, u, P.z[z].b);
        }
        if (k + 1 < g.nz) {
            s.a = fmadd(s.a, u, P.z[z + 2].a);
            s.b = fmadd(s.b, u, P.z[z + 2].b);
        }
        const Pair<T> q2{dv[z].a * own.a - s.a, dv[z].b * own.b - s.b};
        st2<T, true>(qv, c0 + z * sz, q2, true);
        acc.add(own.a, q2.a);
        acc.add(own.b, q2.b);
    }
}

// p = z + beta p, q = A z + beta q and p . q over a column (direction_spmv):
// A z is r on the red cells, the stencil's sum of red neighbours on the black
template <class T>
__device__ __forceinline__ void direction_spmv_col4(const Grid &g, T u, const T *zv, const T *rv, const T *diag, T *pv,
                                                    T *qv, T beta, bool fresh, int i, int j, int k0, long long c0,
                                                    DotAcc<T> &acc) {
    const long long sy = g.nx, sz = (long long)g.nx * g.ny;
    const Pair<T> zero{T(0), T(0)};
    Pair<T> own[4], po[4], qo[4];
    T xs[4], ym[4], yp[4], rr[4], dv[4];
    const int h0 = (i + j + k0 + 1) & 1;  // black side of plane k0 (alternates with z)
    const T zlo = k0 > 0 ? __ldg(zv + c0 - sz + h0) : T(0);
    const T zhi = k0 + 4 < g.nz ? __ldg(zv + c0 + 4 * sz + (h0 ^ 1)) : T(0);
#pragma unroll
    for (int z = 0; z < 4; ++z) {
        const long long c = c0 + z * sz;
        const int hb = h0 ^ (z & 1);
        own[z] = ld2<T, true>(zv, c, true);
        ym[z] = j > 0 ? __ldg(zv + c - sy + hb) : T(0);
        yp[z] = j + 1 < g.ny ? __ldg(zv + c + sy + hb) : T(0);
        xs[z] = hb == 0 ? (i > 0 ? __ldg(zv + c - 1) : T(0)) : (i + 2 < g.nx ? __ldg(zv + c + 2) : T(0));
        rr[z] = __ldg(rv + c + (hb ^ 1));
        dv[z] = __ldg(diag + c + hb);
        po[z] = fresh ? zero : ld2<T, true>(pv, c, true);
        qo[z] = fresh ? zero : ld2<T, true>(qv, c, true);
    }
#pragma unroll
    for (int z = 0; z < 4; ++z) {
        const int k = k0 + z;
        const int hb = h0 ^ (z & 1);
        const T zm = z == 0 ? zlo : (hb ? own[z - 1].b : own[z - 1].a);
        const T zp = z == 3 ? zhi : (hb ? own[z + 1].b : own[z + 1].a);
        T s = T(0);
        if (hb == 0) {
            if (i > 0) s = fmadd(s, u, xs[z]);
            s = fmadd(s, u, own[z].b);
        } else {
            s = fmadd(s, u, own[z].a);
            if (i + 2 < g.nx) s = fmadd(s, u, xs[z]);
        }
        if (j > 0) s = fmadd(s, u, ym[z]);
        if (j + 1 < g.ny) s = fmadd(s, u, yp[z]);
        if (k > 0) s = fmadd(s, u, zm);
        if (k + 1 < g.nz) s = fmadd(s, u, zp);
        const T az = fmadd(-s, dv[z], hb ? own[z].b : own[z].a);
        Pair<T> p2 = own[z], q2{hb ? rr[z] : az, hb ? az : rr[z]};
        if (!fresh) {
            p2 = Pair<T>{fmadd(p2.a, beta, po[z].a), fmadd(p2.b, beta, po[z].b)};
            q2 = Pair<T>{fmadd(q2.a, beta, qo[z].a), fmadd(q2.b, beta, qo[z].b)};
        }
        st2<T, true>(pv, c0 + z * sz, p2, true);
        st2<T, true>(qv, c0 + z * sz, q2, true);
        acc.add(p2.a, q2.a);
        acc.add(p2.b, q2.b);
    }
}

// red half-sweep of x (b = r) and z . r over a column (red_dot): the red
// cell of each pair is cell i where i + j + k is even, else cell i+1; its
// neighbours are black and not written here
template <class T>
__device__ __forceinline__ void red_dot_col4(const Grid &g, T u, T *x, const T *b, const T *inv, int i, int j,
                                             int k0, long long c0, DotAcc<T> &acc) {
    // only the red cell's side of each neighbour pair is read: single cells
    const long long sy = g.nx, sz = (long long)g.nx * g.ny;
    Pair<T> own[4], bv[4];
    T xs[4], iv[4], ym[4], yp[4];
    const int h0 = (i + j + k0) & 1;  // red side of plane k0 (alternates with z)
    const T zlo = k0 > 0 ? __ldg(x + c0 - sz + h0) : T(0);
    const T zhi = k0 + 4 < g.nz ? __ldg(x + c0 + 4 * sz + (h0 ^ 1)) : T(0);
#pragma unroll
    for (int z = 0; z < 4; ++z) {
        const long long c = c0 + z * sz;
        const int hr = h0 ^ (z & 1);
        own[z] = ld2<T, true>(x, c, true);
        ym[z] = j > 0 ? __ldg(x + c - sy + hr) : T(0);
        yp[z] = j + 1 < g.ny ? __ldg(x + c + sy + hr) : T(0);
        xs[z] = hr == 0 ? (i > 0 ? __ldg(x + c - 1) : T(0)) : (i + 2 < g.nx ? __ldg(x + c + 2) : T(0));
        iv[z] = __ldg(inv + c + hr);
        bv[z] = ld2<T, true>(b, c, true);
    }
#pragma unroll
    for (int z = 0; z < 4; ++z) {
        const int k = k0 + z;
        const int hr = h0 ^ (z & 1);
        // the red side's z neighbours: the same side of the planes around
        const T zm = z == 0 ? zlo : (hr ? own[z - 1].b : own[z - 1].a);
        const T zp = z == 3 ? zhi : (hr ? own[z + 1].b : own[z + 1].a);
        T s = T(0);
        if (hr == 0) {
            if (i > 0) s = fmadd(s, u, xs[z]);
            s = fmadd(s, u, own[z].b);
        } else {
            s = fmadd(s, u, own[z].a);
            if (i + 2 < g.nx) s = fmadd(s, u, xs[z]);
        }
        if (j > 0) s = fmadd(s, u, ym[z]);
        if (j + 1 < g.ny) s = fmadd(s, u, yp[z]);
        if (k > 0) s = fmadd(s, u, zm);
        if (k + 1 < g.nz) s = fmadd(s, u, zp);
        const T xv = ((hr ? bv[z].b : bv[z].a) + s) * iv[z];
        Pair<T> out = own[z];
        if (hr) out.b = xv;
        else out.a = xv;
        x[c0 + z * sz + hr] = xv;
        acc.add(out.a, bv[z].a);
        acc.add(out.b, bv[z].b);
    }
}

// Last red pass of the fine level, with rho' = z . r (z = x, r = b there)
// per scene; the scene's last flush sets beta (0 for a new direction).
template <class T, int OCC, bool COL>
__global__ void __launch_bounds__(BLOCK_THREADS, OCC)
    red_dot_kernel(const BLevel<T> *__restrict__ levels, const BSeg *__restrict__ segs, int nseg, int n,
                   const BScene<T> *__restrict__ scenes, int gate, double *part, const int *__restrict__ scene_of,
                   const BatchCounters *live) {
    if (batch_idle(live)) return;
    __shared__ ItemCtx<T> ctx;
    sum_items<T, DotAcc<T>>(
        segs, nseg, n, part, levels, scenes, gate, ctx,
        [&](const BItem &it, DotAcc<T> &acc, T cls) {
            const BLevel<T> L = ctx.L;  // registers: stores through generic pointers would force reloads from shared memory
            const Cpl<T> cw{L.cx, L.cy, L.cz, cls};
            if (tile_empty(cw.u)) return;  // z = 0 there: nothing to write or add
            with_vu(L.vec, tile_uniform(cw.u), [&](auto vt, auto ut) {
                constexpr bool V = decltype(vt)::value;
                constexpr bool U = decltype(ut)::value;
                auto nb2 = [&](long long m, int, int, bool sec) { return ld2<T, V>(L.x, m, sec); };
                auto nb1 = [&](long long m, int) { return __ldg(L.x + m); };
                auto plane = [&](int i, int j, int k, long long c, bool second) {
                    const int hr = ((i + j + k) & 1) == 0 ? 0 : 1;
                    const Pair<T> x2 = ld2<T, V>(L.x, c, second), b2 = ld2<T, V>(L.b, c, second);
                    Pair<T> out = x2;
                    if (hr == 0 || second) {
                        const T sh = pair_nsum1<T, V, U>(hr, L.g, cw, i, j, k, c, second, x2, nb2, nb1);
                        const long long ch = c + hr;
                        const T xv = ((hr ? b2.b : b2.a) + sh) * __ldg(L.inv + ch);
                        if (hr) out.b = xv;
                        else out.a = xv;
                        L.x[ch] = xv;
                    }
                    acc.add(out.a, b2.a);
                    if (second) acc.add(out.b, b2.b);
                };
                if constexpr (COL && U && V)
                    pair_tile_z4(L.g, it, [&](int i, int j, int k0, long long c0) {
                        red_dot_col4<T>(L.g, cw.u, L.x, L.b, L.inv, i, j, k0, c0, acc);
                    }, plane);
                else
                    pair_tile(L.g, it, plane);
            });
        },
        [&](const BItem &it, int visits, int sums) {
            Scalars *sc = ctx.S.sc;
            if (item_last(&sc->counter[SITE_DOT], visits)) {
                const double rho_new = sum_range(part, it.begin, sums);
                if (threadIdx.x == 0) {
                    if (sc->first) {
                        sc->beta = 0.0;
                        sc->first = 0;
                    } else {
                        sc->beta = rho_new / sc->rho;
                    }
                    sc->rho = rho_new;
                    if (rho_new != rho_new) {
                        sc->done = 1;
                        sc->status = 3;
                    }
                    sc->counter[SITE_DOT] = 0;
                }
            }
        });
}

// ---- tail, one block per scene --------------------------------------------------

// A tail level, in place in global memory; its descriptor lives in shared memory
// (one copy per block, read as broadcasts).
template <class T> struct SLevel {
    int nx, ny, nz, dim, n;
    int hx;             // pair slots per row, (nx + 1) / 2
    FastDiv fhx, fhxy;  // hx and hx ny, to split pair-slot indices
    T *b, *x, *inv, *diag, *cx, *cy, *cz;
};

// Neighbour sum of cell (i, j, k) = c, in the order -x, +x, -y, +y, -z,
// +z; xat(m, i', j', k') is the value at neighbour m = (i', j', k'). Every
// load is issued before the sum.
template <class T, class X>
__device__ __forceinline__ T snb(const SLevel<T> &L, int i, int j, int k, int c, X xat) {
    const int sy = L.nx, sz = L.nx * L.ny;
    const bool on[6] = {i > 0, i + 1 < L.nx, j > 0, j + 1 < L.ny, L.dim == 3 && k > 0, L.dim == 3 && k + 1 < L.nz};
    T w[6], v[6];
    w[0] = on[0] ? L.cx[c - 1] : T(0);
    v[0] = on[0] ? xat(c - 1, i - 1, j, k) : T(0);
    w[1] = on[1] ? L.cx[c] : T(0);
    v[1] = on[1] ? xat(c + 1, i + 1, j, k) : T(0);
    w[2] = on[2] ? L.cy[c - sy] : T(0);
    v[2] = on[2] ? xat(c - sy, i, j - 1, k) : T(0);
    w[3] = on[3] ? L.cy[c] : T(0);
    v[3] = on[3] ? xat(c + sy, i, j + 1, k) : T(0);
    w[4] = on[4] ? L.cz[c - sz] : T(0);
    v[4] = on[4] ? xat(c - sz, i, j, k - 1) : T(0);
    w[5] = on[5] ? L.cz[c] : T(0);
    v[5] = on[5] ? xat(c + sz, i, j, k + 1) : T(0);
    T s = T(0);
#pragma unroll
    for (int n = 0; n < 6; ++n)
        if (on[n]) s = fmadd(s, w[n], v[n]);
    return s;
}

// Thread mapping of the tail: pair slots (2 ip, j, k), ip < hx. A pass that
// updates one colour gives each thread the slot's cell of that colour
// (i = 2 ip + ((j + k + color) & 1)), so no thread idles on the other
// colour; a pass over every cell gives it both cells of the slot. A thread
// takes its slots two at a time and stores their values after computing both,
// so that their loads overlap (a store could alias the next slot's loads).
struct Slot {
    int i, j, k, c;
    bool on;
};
template <class T> __device__ __forceinline__ Slot slot_cell(const SLevel<T> &L, int p, int slots, int color) {
    Slot s;
    const int q = p < slots ? p : 0;
    const int t = (int)fdiv((unsigned)q, L.fhx);
    s.k = (int)fdiv((unsigned)q, L.fhxy);
    s.j = t - s.k * L.ny;
    s.i = 2 * (q - t * L.hx) + (color < 0 ? 0 : ((s.j + s.k + color) & 1));
    s.on = p < slots && s.i < L.nx;
    if (s.i >= L.nx) s.i = 0;
    s.c = s.i + L.nx * (s.j + L.ny * s.k);
    return s;
}
// x of one colour's cells = f(cell)
template <class T, class F> __device__ __forceinline__ void s_for_color(const SLevel<T> &L, int color, F f) {
    const int slots = L.hx * L.ny * L.nz;
    for (int p = threadIdx.x; p < slots; p += 2 * blockDim.x) {
        const Slot a = slot_cell(L, p, slots, color), b = slot_cell(L, p + (int)blockDim.x, slots, color);
        const T va = f(a.i, a.j, a.k, a.c), vb = b.on ? f(b.i, b.j, b.k, b.c) : T(0);
        if (a.on) L.x[a.c] = va;
        if (b.on) L.x[b.c] = vb;
    }
    __syncthreads();
}
// out(cell) = f(cell) for every cell
template <class T, class F>
__device__ __forceinline__ void s_for_cells(const SLevel<T> &L, T *out, F f) {
    const int slots = L.hx * L.ny * L.nz;
    for (int p = threadIdx.x; p < slots; p += blockDim.x) {
        const Slot a = slot_cell(L, p, slots, -1);
        const bool second = a.i + 1 < L.nx;
        const T va = f(a.i, a.j, a.k, a.c), vb = second ? f(a.i + 1, a.j, a.k, a.c + 1) : T(0);
        out[a.c] = va;
        if (second) out[a.c + 1] = vb;
    }
    __syncthreads();
}

// The coarsest level of at most one warp's slots (64 cells, 4^3): its
// coarsest_pairs_warp symmetric FP64 sweep pairs from x = 0 are a linear map
// of b, whose matrix the solve forms once, a warp per column (unit b). Run
// directly they were 32 half-sweeps, each a chain of seven dependent FP64
// operations and a barrier: 10 us of a 256^3 or 32^3 iteration's 40 or 33 us
// tail; the matrix takes 4096 FP64 products. With it and the passes below
// the tail went from 37 to 20 us an iteration at 128^3, 40 to 22 us at 256^3.
constexpr int TAIL_DENSE = 64;
__device__ __forceinline__ bool tail_dense(int hx, int ny, int nz) { return hx * ny * nz <= 32; }
template <class T>
__global__ void __launch_bounds__(32) tail_matrix_kernel(const BTail<T> *__restrict__ tails, MgSettings ms) {
    const BTail<T> &A = tails[blockIdx.x / TAIL_DENSE];
    const int col = blockIdx.x % TAIL_DENSE;
    if (A.nt <= 0) return;
    const MgLevel<T> &G = A.lv[A.nt - 1];
    const int nx = G.g.nx, ny = G.g.ny, nz = G.g.nz, hx = (nx + 1) / 2, n = nx * ny * nz;
    if (!tail_dense(hx, ny, nz) || col >= n) return;
    __shared__ double x[TAIL_DENSE + 1];
    if (threadIdx.x == 0) x[TAIL_DENSE] = 0.0;
    const int p = threadIdx.x, sy = nx, sz = nx * ny;
    x[p] = 0.0;
    x[p + 32] = 0.0;
    __syncwarp();
    const int t = p / hx, k = p / (hx * ny), j = t - k * ny, i0 = 2 * (p - t * hx);
    const int order[4] = {0, 1, 1, 0};
    // the slot's two cells: couplings and right-hand side over the diagonal,
    // and the neighbours (one past the cells, where x stays 0, if there is
    // none); two sums of three keep the dependent chain at four operations
    const int step[6] = {-1, 1, -sy, sy, -sz, sz};
    double w[2][6], b[2];
    int nb[2][6];
    bool have[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int i = i0 + h, c = i + nx * (j + ny * k);
        have[h] = p < hx * ny * nz && i < nx;
        const bool on[6] = {i > 0, i + 1 < nx, j > 0, j + 1 < ny, G.g.dim == 3 && k > 0, G.g.dim == 3 && k + 1 < nz};
        const T *a[6] = {G.cx + c - 1, G.cx + c, G.cy + c - sy, G.cy + c, G.cz + c - sz, G.cz + c};
        const double inv = have[h] ? (double)G.inv[c] : 0.0;
#pragma unroll
        for (int q = 0; q < 6; ++q) {
            w[h][q] = have[h] && on[q] ? (double)*a[q] * inv : 0.0;
            nb[h][q] = have[h] && on[q] ? c + step[q] : TAIL_DENSE;
        }
        b[h] = c == col ? inv : 0.0;
    }
    auto relax = [&](auto side) {
        constexpr int h = decltype(side)::value;
        if (!have[h]) return;
        const double u = fma(w[h][2], x[nb[h][2]], fma(w[h][1], x[nb[h][1]], fma(w[h][0], x[nb[h][0]], b[h])));
        const double v = fma(w[h][5], x[nb[h][5]], fma(w[h][4], x[nb[h][4]], w[h][3] * x[nb[h][3]]));
        x[i0 + h + nx * (j + ny * k)] = u + v;
    };
    for (int pr = 0; pr < ms.coarsest_pairs_warp; ++pr)
        for (int q = 0; q < 4; ++q) {
            if ((j + k + order[q]) & 1) relax(std::integral_constant<int, 1>{});
            else relax(std::integral_constant<int, 0>{});
            __syncwarp();
        }
    for (int r = p; r < n; r += 32) A.m64[r * TAIL_DENSE + col] = x[r];
}

// The V-cycle of the levels lv[0..nt) in one block per scene: b of lv[0]
// in, x of lv[0] out, same smoother, transfers and coarsest solve (FP64
// symmetric sweep pairs, as a matrix where tail_dense, else with the coarsest
// operator and right-hand side held in FP64) as the global levels. The levels
// (a few hundred KB at most) are read and written in place in global memory,
// where the block's L1 holds them between passes; __syncthreads orders a
// pass's writes before the next pass's reads within the block. (A copy into
// shared memory needs a carveout of the SM's L1 different from every other
// kernel's, and the switch costs more than the copy saves.) The block is
// bound by latency: passes issue their loads first, and the restriction goes
// through residuals in shared memory, a thread per fine pair.
template <class T>
__global__ void __launch_bounds__(MG_TAIL_THREADS) tail_kernel(const BTail<T> *__restrict__ tails,
                                                               const BScene<T> *__restrict__ scenes, int gate,
                                                               MgSettings ms, const BatchCounters *live) {
    if (batch_idle(live)) return;
    const int s = blockIdx.x;
    const BTail<T> &A = tails[s];
    if (A.nt <= 0) return;
    if (gated(scenes[s].sc, gate)) return;
    __shared__ SLevel<T> S[MG_MAX_LEVELS];
    __shared__ double *cd[6];  // coarsest: x, b, inv, cx, cy, cz in FP64
    __shared__ T res[MG_TAIL_BYTES_MAX / (7 * sizeof(T)) + 1];  // a level's residuals
    __shared__ double bc[TAIL_DENSE];
    if (threadIdx.x < A.nt) {
        const MgLevel<T> &G = A.lv[threadIdx.x];
        const Grid &g = G.g;
        SLevel<T> &L = S[threadIdx.x];
        L.nx = g.nx;
        L.ny = g.ny;
        L.nz = g.nz;
        L.dim = g.dim;
        L.n = (int)g.ncell;
        L.hx = (g.nx + 1) / 2;
        L.fhx = make_fastdiv((unsigned)L.hx);
        L.fhxy = make_fastdiv((unsigned)(L.hx * g.ny));
        L.b = G.b;
        L.x = G.x;
        L.inv = const_cast<T *>(G.inv);
        L.diag = const_cast<T *>(G.diag);
        L.cx = const_cast<T *>(G.cx);
        L.cy = const_cast<T *>(G.cy);
        L.cz = const_cast<T *>(G.cz);  // == cy in 2D, never read there
    }
    if (threadIdx.x < 6) cd[threadIdx.x] = A.c64 + (size_t)threadIdx.x * MG_COARSEST_MAX;
    __syncthreads();
    const T alpha = T(ms.alpha);
    for (int l = 0; l + 1 < A.nt; ++l) {
        const SLevel<T> &L = S[l];
        s_for_cells(L, L.x, [&](int i, int j, int k, int c) {
            const T inv = L.inv[c];
            if (((i + j + k) & 1) == 0) return L.b[c] * inv;
            return (L.b[c] + snb(L, i, j, k, c, [&](int m, int, int, int) { return L.b[m] * L.inv[m]; })) * inv;
        });
        for (int sw = 1; sw < ms.smooth; ++sw)
            for (int color = 0; color < 2; ++color)
                s_for_color(L, color, [&](int i, int j, int k, int c) {
                    return (L.b[c] + snb(L, i, j, k, c, [&](int m, int, int, int) { return L.x[m]; })) * L.inv[c];
                });
        const SLevel<T> &C = S[l + 1];
        s_for_cells(L, res, [&](int i, int j, int k, int c) {
            return resid(L.b[c], L.diag[c], L.x[c],
                         snb(L, i, j, k, c, [&](int m, int, int, int) { return L.x[m]; }));
        });
        s_for_cells(C, C.b, [&](int I, int J, int K, int) {
            T sum = T(0);
            const int kmax = L.dim == 3 ? 2 : 1;
            for (int c2 = 0; c2 < kmax; ++c2)
                for (int b2 = 0; b2 < 2; ++b2)
                    for (int a2 = 0; a2 < 2; ++a2) {
                        const int i = 2 * I + a2, j = 2 * J + b2, k = 2 * K + c2;
                        if (i >= L.nx || j >= L.ny || k >= L.nz) continue;
                        sum += res[i + L.nx * (j + L.ny * k)];
                    }
            return sum;
        });
    }
    {
        const SLevel<T> &L = S[A.nt - 1];
        const int slots = L.hx * L.ny * L.nz;
        if (tail_dense(L.hx, L.ny, L.nz)) {
            // x = M b, four threads a row
            if (threadIdx.x < 4 * TAIL_DENSE) {
                const int r = threadIdx.x >> 2, q = threadIdx.x & 3;
                double m[TAIL_DENSE / 4];
#pragma unroll
                for (int e = 0; e < TAIL_DENSE / 4; ++e)
                    m[e] = r < L.n && 4 * e + q < L.n ? __ldcg(A.m64 + r * TAIL_DENSE + 4 * e + q) : 0.0;
                if (threadIdx.x < TAIL_DENSE) bc[threadIdx.x] = threadIdx.x < L.n ? widen(L.b[threadIdx.x]) : 0.0;
                asm volatile("bar.sync 1, %0;" ::"n"(4 * TAIL_DENSE) : "memory");
                double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
#pragma unroll
                for (int e = 0; e < TAIL_DENSE / 4; e += 4) {
                    a0 = fma(m[e], bc[4 * e + q], a0);
                    a1 = fma(m[e + 1], bc[4 * e + 4 + q], a1);
                    a2 = fma(m[e + 2], bc[4 * e + 8 + q], a2);
                    a3 = fma(m[e + 3], bc[4 * e + 12 + q], a3);
                }
                double v = (a0 + a1) + (a2 + a3);
                v += __shfl_xor_sync(0xffffffffu, v, 1);
                v += __shfl_xor_sync(0xffffffffu, v, 2);
                if (q == 0 && r < L.n) L.x[r] = narrow_to<T>(v);
            }
            __syncthreads();
        } else {
            double *xc = cd[0], *bd = cd[1], *ivd = cd[2], *cxd = cd[3], *cyd = cd[4], *czd = cd[5];
            for (int c = threadIdx.x; c < L.n; c += blockDim.x) {
                xc[c] = 0.0;
                bd[c] = (double)L.b[c];
                ivd[c] = (double)L.inv[c];
                cxd[c] = (double)L.cx[c];
                cyd[c] = (double)L.cy[c];
                czd[c] = (double)L.cz[c];
            }
            __syncthreads();
            const int sy = L.nx, sz = L.nx * L.ny;
            const int order[4] = {0, 1, 1, 0};
            for (int p = 0; p < ms.coarsest_pairs; ++p)
                for (int q = 0; q < 4; ++q) {
                    for (int e = threadIdx.x; e < slots; e += blockDim.x) {
                        const Slot a = slot_cell(L, e, slots, order[q]);
                        if (!a.on) continue;
                        const int i = a.i, j = a.j, k = a.k, c = a.c;
                        double acc = 0.0;
                        if (i > 0) acc += cxd[c - 1] * xc[c - 1];
                        if (i + 1 < L.nx) acc += cxd[c] * xc[c + 1];
                        if (j > 0) acc += cyd[c - sy] * xc[c - sy];
                        if (j + 1 < L.ny) acc += cyd[c] * xc[c + sy];
                        if (L.dim == 3) {
                            if (k > 0) acc += czd[c - sz] * xc[c - sz];
                            if (k + 1 < L.nz) acc += czd[c] * xc[c + sz];
                        }
                        xc[c] = (bd[c] + acc) * ivd[c];
                    }
                    __syncthreads();
                }
            for (int c = threadIdx.x; c < L.n; c += blockDim.x) L.x[c] = T(xc[c]);
            __syncthreads();
        }
    }
    for (int l = A.nt - 2; l >= 0; --l) {
        const SLevel<T> &L = S[l];
        const SLevel<T> &C = S[l + 1];
        const bool d3 = L.dim == 3;
        s_for_color(L, 1, [&](int i, int j, int k, int c) {
            return (L.b[c] + snb(L, i, j, k, c, [&](int m, int mi, int mj, int mk) {
                        return prolong(L.x[m], alpha,
                                       C.x[(mi >> 1) + C.nx * ((mj >> 1) + C.ny * (d3 ? (mk >> 1) : 0))]);
                    })) * L.inv[c];
        });
        for (int sw = 1; sw < ms.smooth; ++sw)
            for (int color = 0; color < 2; ++color)
                s_for_color(L, color, [&](int i, int j, int k, int c) {
                    return (L.b[c] + snb(L, i, j, k, c, [&](int m, int, int, int) { return L.x[m]; })) * L.inv[c];
                });
        s_for_color(L, 0, [&](int i, int j, int k, int c) {
            return (L.b[c] + snb(L, i, j, k, c, [&](int m, int, int, int) { return L.x[m]; })) * L.inv[c];
        });
    }
}

// ---- CG on the fine level -----------------------------------------------------------

template <class T, int OCC>
__global__ void __launch_bounds__(BLOCK_THREADS, OCC)
    direction_kernel(const BLevel<T> *__restrict__ levels, const BSeg *__restrict__ segs, int nseg, int n,
                     const BScene<T> *__restrict__ scenes, int gate, const BatchCounters *live) {
    if (batch_idle(live)) return;
    __shared__ ItemCtx<T> ctx;
    int cur = -1;
    int sgc = 0;
    const int gs = item_group(n, nseg);
    T cls_next = class_at<T, false>(levels, segs, nseg, n, first_item(gs), 0);
    for (int w = first_item(gs); w < n; w = next_item(w, gs)) {
        const BItem it = item_at(segs, nseg, w, sgc);
        const T cls = cls_next;
        refresh(ctx, cur, it, levels, scenes, gate);
        cls_next = class_next<T, false>(levels, segs, nseg, n, next_item(w, gs), sgc, it.ref, ctx.L.tcp);
        if (ctx.skip) continue;
        const BLevel<T> L = ctx.L;  // registers: stores through generic pointers would force reloads from shared memory
        const BScene<T> S = ctx.S;
        const T beta = T(ctx.beta);
        const bool empty = tile_empty(cls);
        // no unknown: p = 0, written when a direction starts (beta = 0) and
        // unchanged after that
        if (empty && beta != T(0)) continue;
        with_vec(L.vec, [&](auto vt) {
            constexpr bool V = decltype(vt)::value;
            if (empty) {
                pair_tile(L.g, it, [&](int, int, int, long long c, bool second) {
                    st2<T, V>(S.p, c, Pair<T>{T(0), T(0)}, second);
                });
                return;
            }
            const bool fresh = beta == T(0);
            auto plane = [&](int, int, int, long long c, bool second) {
                const Pair<T> z2 = ld2<T, V>(S.z, c, second);
                Pair<T> p2;
                if (fresh) {
                    p2 = z2;
                } else {
                    const Pair<T> o = ld2<T, V>(S.p, c, second);
                    p2 = Pair<T>{fmadd(z2.a, beta, o.a), fmadd(z2.b, beta, o.b)};
                }
                st2<T, V>(S.p, c, p2, second);
            };
            if constexpr (V)
                // the column's loads first (see pair_tile_z4)
                pair_tile_z4(L.g, it, [&](int, int, int, long long c0) {
                    const long long sz = (long long)L.g.nx * L.g.ny;
                    Pair<T> z2[4], o[4];
#pragma unroll
                    for (int z = 0; z < 4; ++z) {
                        z2[z] = ld2<T, true>(S.z, c0 + z * sz, true);
                        o[z] = fresh ? Pair<T>{T(0), T(0)} : ld2<T, true>(S.p, c0 + z * sz, true);
                    }
#pragma unroll
                    for (int z = 0; z < 4; ++z)
                        st2<T, true>(S.p, c0 + z * sz,
                                     fresh ? z2[z] : Pair<T>{fmadd(z2[z].a, beta, o[z].a), fmadd(z2[z].b, beta, o[z].b)},
                                     true);
                }, plane);
            else
                pair_tile(L.g, it, plane);
        });
    }
}

template <class T, int OCC, bool COL>
__global__ void __launch_bounds__(BLOCK_THREADS, OCC)
    spmv_kernel(const BLevel<T> *__restrict__ levels, const BSeg *__restrict__ segs, int nseg, int n,
                const BScene<T> *__restrict__ scenes, int gate, double *part, const int *__restrict__ scene_of,
                const BatchCounters *live) {
    if (batch_idle(live)) return;
    __shared__ ItemCtx<T> ctx;
    sum_items<T, DotAcc<T>>(
        segs, nseg, n, part, levels, scenes, gate, ctx,
        [&](const BItem &it, DotAcc<T> &acc, T cls) {
            const BLevel<T> L = ctx.L;  // registers: stores through generic pointers would force reloads from shared memory
            const BScene<T> S = ctx.S;
            const Cpl<T> cw{L.cx, L.cy, L.cz, cls};
            // no unknown: q = A p = 0 there, and q is read nowhere else (the
            // update skips such tiles too)
            if (tile_empty(cw.u)) return;
            with_vu(L.vec, tile_uniform(cw.u), [&](auto vt, auto ut) {
                constexpr bool V = decltype(vt)::value;
                constexpr bool U = decltype(ut)::value;
                auto nb2 = [&](long long m, int, int, bool sec) { return ld2<T, V>(S.p, m, sec); };
                auto nb1 = [&](long long m, int) { return __ldg(S.p + m); };
                auto plane = [&](int i, int j, int k, long long c, bool second) {
                    const Pair<T> p2 = ld2<T, V>(S.p, c, second), d2 = ld2<T, V>(L.diag, c, second);
                    const Pair<T> s = pair_nsum<T, V, U, 2>(L.g, cw, i, j, k, c, second, p2, nb2, nb1);
                    const Pair<T> q2{d2.a * p2.a - s.a, d2.b * p2.b - s.b};
                    st2<T, V>(S.q, c, q2, second);
                    acc.add(p2.a, q2.a);
                    if (second) acc.add(p2.b, q2.b);
                };
                if constexpr (COL && U && V)
                    pair_tile_z4(L.g, it, [&](int i, int j, int k0, long long c0) {
                        spmv_col4<T>(L.g, cw.u, S.p, L.diag, S.q, i, j, k0, c0, acc);
                    }, plane);
                else
                    pair_tile(L.g, it, plane);
            });
        },
        [&](const BItem &it, int visits, int sums) {
            Scalars *sc = ctx.S.sc;
            if (item_last(&sc->counter[SITE_SPMV], visits)) {
                const double pq = sum_range(part, it.begin, sums);
                if (threadIdx.x == 0) {
                    sc->pap = pq;
                    sc->alpha = sc->rho / pq;
                    sc->counter[SITE_SPMV] = 0;
                }
            }
        });
}

// The new direction and its product in one pass: p = z + beta p and, by the
// same recurrence, q = A p = A z + beta q (beta = 0: p = z, q = A z). The
// V-cycle ends on a red half-sweep, which solves the red rows of A z = r, so
// A z is r there and the stencil runs on the black cells only. Two passes
// (p, then the stencil of p: the staged fine levels still take them) move 6
// words a cell (+ 3 couplings in mixed tiles) and take 9 FP64 operations; this
// one 6 (+ 3) and 6.5, in one launch. The FP64 solver is bound by its
// operations: a 256^3 solve went from 19.8 to 19.2 ms; the small ones by
// launches and latency: 32^3 mixed 1.03 to 0.98 ms, six served scenes 22.2 to
// 21.8 ms. At 256^3 mixed and in the batch of 64, bound by instructions, the
// two forms take the same time.
template <class T, int OCC, bool COL>
__global__ void __launch_bounds__(BLOCK_THREADS, OCC)
    direction_spmv_kernel(const BLevel<T> *__restrict__ levels, const BSeg *__restrict__ segs, int nseg, int n,
                          const BScene<T> *__restrict__ scenes, int gate, double *part, const BatchCounters *live) {
    if (batch_idle(live)) return;
    __shared__ ItemCtx<T> ctx;
    sum_items<T, DotAcc<T>>(
        segs, nseg, n, part, levels, scenes, gate, ctx,
        [&](const BItem &it, DotAcc<T> &acc, T cls) {
            const BLevel<T> L = ctx.L;  // registers: stores through generic pointers would force reloads from shared memory
            const BScene<T> S = ctx.S;
            const Cpl<T> cw{L.cx, L.cy, L.cz, cls};
            // no unknown: p and q are read nowhere (z = 0 there)
            if (tile_empty(cw.u)) return;
            const T beta = T(ctx.beta);
            const bool fresh = beta == T(0);
            with_vu(L.vec, tile_uniform(cw.u), [&](auto vt, auto ut) {
                constexpr bool V = decltype(vt)::value;
                constexpr bool U = decltype(ut)::value;
                auto nb2 = [&](long long m, int, int, bool sec) { return ld2<T, V>(S.z, m, sec); };
                auto nb1 = [&](long long m, int) { return __ldg(S.z + m); };
                auto plane = [&](int i, int j, int k, long long c, bool second) {
                    const int hb = ((i + j + k) & 1) ^ 1;  // black side
                    Pair<T> p2 = ld2<T, V>(S.z, c, second), po{T(0), T(0)}, qo{T(0), T(0)};
                    if (!fresh) {
                        po = ld2<T, V>(S.p, c, second);
                        qo = ld2<T, V>(S.q, c, second);
                    }
                    const T rr = hb == 1 || second ? __ldg(S.r + c + (hb ^ 1)) : T(0);
                    T az = T(0);
                    if (hb == 0 || second) {
                        const T d = __ldg(L.diag + c + hb);
                        const T s = pair_nsum1<T, V, U>(hb, L.g, cw, i, j, k, c, second, p2, nb2, nb1);
                        az = fmadd(-s, d, hb ? p2.b : p2.a);
                    }
                    Pair<T> q2{hb ? rr : az, hb ? az : rr};
                    if (!fresh) {
                        p2 = Pair<T>{fmadd(p2.a, beta, po.a), fmadd(p2.b, beta, po.b)};
                        q2 = Pair<T>{fmadd(q2.a, beta, qo.a), fmadd(q2.b, beta, qo.b)};
                    }
                    st2<T, V>(S.p, c, p2, second);
                    st2<T, V>(S.q, c, q2, second);
                    acc.add(p2.a, q2.a);
                    if (second) acc.add(p2.b, q2.b);
                };
                if constexpr (COL && U && V)
                    pair_tile_z4(L.g, it, [&](int i, int j, int k0, long long c0) {
                        direction_spmv_col4<T>(L.g, cw.u, S.z, S.r, L.diag, S.p, S.q, beta, fresh, i, j, k0, c0, acc);
                    }, plane);
                else
                    pair_tile(L.g, it, plane);
            });
        },
        [&](const BItem &it, int visits, int sums) {
            Scalars *sc = ctx.S.sc;
            if (item_last(&sc->counter[SITE_SPMV], visits)) {
                const double pq = sum_range(part, it.begin, sums);
                if (threadIdx.x == 0) {
                    sc->pap = pq;
                    sc->alpha = sc->rho / pq;
                    sc->counter[SITE_SPMV] = 0;
                }
            }
        });
}

// x += alpha p (x = alpha p on the first update of a solve), r -= alpha q,
// |r|_inf. mode 0: the solve's stopping rule; mode 1: inner solve.
template <class T, int OCC>
__global__ void __launch_bounds__(BLOCK_THREADS, OCC)
    update_kernel(const BLevel<T> *__restrict__ levels, const BSeg *__restrict__ segs, int nseg, int n,
                  const BScene<T> *__restrict__ scenes, int gate, double *part, int mode, BatchCounters *cnt,
                  const int *__restrict__ scene_of) {
    // as in refine_residual_kernel: this launch lowers the counter
    if (__syncthreads_or(threadIdx.x == 0 && batch_idle(cnt))) return;
    __shared__ ItemCtx<T> ctx;
    max_items<T, MaxAcc<T>>(
        segs, nseg, n, part, levels, scenes, gate, ctx,
        [&](const BItem &it, MaxAcc<T> &acc, T cls) {
            const BLevel<T> L = ctx.L;  // registers: stores through generic pointers would force reloads from shared memory
            const BScene<T> S = ctx.S;
            const T alpha = T(ctx.alpha);
            const bool overwrite = ctx.overwrite != 0;
            // no unknown: p = q = r = 0 there; x = 0 is written by the
            // solve's first update and unchanged after that
            const bool empty = tile_empty(cls);
            if (empty && !overwrite) return;
            with_vec(L.vec, [&](auto vt) {
                constexpr bool V = decltype(vt)::value;
                if (empty) {
                    pair_tile(L.g, it, [&](int, int, int, long long c, bool second) {
                        st2<T, V>(S.x, c, Pair<T>{T(0), T(0)}, second);
                    });
                    return;
                }
                auto plane = [&](int, int, int, long long c, bool second) {
                    const Pair<T> p2 = ld2<T, V>(S.p, c, second), q2 = ld2<T, V>(S.q, c, second);
                    const Pair<T> r2 = ld2<T, V>(S.r, c, second);
                    Pair<T> x2;
                    if (overwrite) {
                        x2 = Pair<T>{alpha * p2.a, alpha * p2.b};
                    } else {
                        const Pair<T> o = ld2<T, V>(S.x, c, second);
                        x2 = Pair<T>{fmadd(o.a, alpha, p2.a), fmadd(o.b, alpha, p2.b)};
                    }
                    const Pair<T> rn{fmadd(r2.a, -alpha, q2.a), fmadd(r2.b, -alpha, q2.b)};
                    st2<T, V>(S.x, c, x2, second);
                    st2<T, V>(S.r, c, rn, second);
                    acc.add(rn.a);
                    if (second) acc.add(rn.b);
                };
                if constexpr (V)
                    // the column's loads first (see pair_tile_z4)
                    pair_tile_z4(L.g, it, [&](int, int, int, long long c0) {
                        const long long sz = (long long)L.g.nx * L.g.ny;
                        Pair<T> p2[4], q2[4], r2[4], o[4];
#pragma unroll
                        for (int z = 0; z < 4; ++z) {
                            const long long c = c0 + z * sz;
                            p2[z] = ld2<T, true>(S.p, c, true);
                            q2[z] = ld2<T, true>(S.q, c, true);
                            r2[z] = ld2<T, true>(S.r, c, true);
                            o[z] = overwrite ? Pair<T>{T(0), T(0)} : ld2<T, true>(S.x, c, true);
                        }
#pragma unroll
                        for (int z = 0; z < 4; ++z) {
                            const long long c = c0 + z * sz;
                            const Pair<T> x2 = overwrite ? Pair<T>{alpha * p2[z].a, alpha * p2[z].b}
                                                         : Pair<T>{fmadd(o[z].a, alpha, p2[z].a),
                                                                   fmadd(o[z].b, alpha, p2[z].b)};
                            const Pair<T> rn{fmadd(r2[z].a, -alpha, q2[z].a), fmadd(r2[z].b, -alpha, q2[z].b)};
                            st2<T, true>(S.x, c, x2, true);
                            st2<T, true>(S.r, c, rn, true);
                            acc.add(rn.a);
                            acc.add(rn.b);
                        }
                    }, plane);
                else
                    pair_tile(L.g, it, plane);
            });
        },
        [&](const BItem &it, int visits) {
            Scalars *sc = ctx.S.sc;
            if (item_last(&sc->counter[SITE_UPDATE], visits)) {
                const double res = max_range(part, it.begin, visits);
                if (threadIdx.x == 0) {
                    sc->first_update = 0;
                    sc->iter += 1;
                    const bool bad = res != res || sc->alpha != sc->alpha;
                    int finished = 0;
                    if (mode == 0) {
                        sc->res = res;
                        if (bad) {
                            sc->status = 3;
                            finished = 1;
                        } else if (res <= sc->tol) {
                            sc->status = 1;
                            finished = 1;
                        } else if (sc->iter >= sc->max_iter) {
                            sc->status = 2;
                            finished = 1;
                        }
                    } else {
                        sc->inner_iter += 1;
                        if (bad) {
                            sc->status = 3;
                            finished = 1;
                        } else if (res <= sc->inner_tol || sc->inner_iter >= sc->inner_max ||
                                   sc->iter >= sc->max_iter) {
                            sc->inner_done = 1;
                            atomicAdd(&cnt->refine, 1);
                        }
                    }
                    if (finished) {
                        sc->done = 1;
                        atomicSub(&cnt->remaining, 1);
                    }
                    sc->counter[SITE_UPDATE] = 0;
                }
            }
        });
}

// ---- mixed precision: FP64 refinement -------------------------------------------------

// The mixed solver's refinement after an inner solve, without FP64
// multiplications: with d the inner solve's correction (FP32) and A = hi +
// lo the FP64 operator as level 0's FP32 operator plus the low floats
// (within 2^-48 of each value),
//   x64 += d,   r64 -= A d,
// A d formed per cell in float-float: every product c d as hi*d split
// exactly by an FMA plus lo*d, summed by TwoSum (about 2^-47 |A||d| from the
// exact value), then subtracted from r64 in FP64. The result is the FP64
// residual b - A x64 updated recursively (each update exact to about 2^-47
// |A||d|, far below the refinement's 1e-6 of |b|), and costs three FP64
// additions per cell where recomputing b - A x64 costs eight FP64
// operations (this GPU's FP64 pipe issues about two per clock per SM).
// Order of the sum: the diagonal, then -x, +x, -y, +y, -z, +z.
template <class T, bool V>
__device__ __forceinline__ void refine_update_pair(const Grid &g, const BLevel<T> &L, const BScene<T> &S, int i, int j,
                                                   int k, long long c, bool second, MaxSumAcc<T> &acc) {
    const long long sy = g.nx, sz = (long long)g.nx * g.ny;
    const Pair<float> zero{0.0f, 0.0f};
    const float *d = reinterpret_cast<const float *>(S.x);
    const float *dh = reinterpret_cast<const float *>(L.diag), *xh = reinterpret_cast<const float *>(L.cx),
                *yh = reinterpret_cast<const float *>(L.cy), *zh = reinterpret_cast<const float *>(L.cz);
    // every load of the pair first
    const Pair<float> dc = ld2<float, V>(d, c, second);
    const float dxm = i > 0 ? __ldg(d + c - 1) : 0.0f, dxp = (second && i + 2 < g.nx) ? __ldg(d + c + 2) : 0.0f;
    const Pair<float> dym = j > 0 ? ld2<float, V>(d, c - sy, second) : zero;
    const Pair<float> dyp = j + 1 < g.ny ? ld2<float, V>(d, c + sy, second) : zero;
    const bool z3 = g.dim == 3;
    const Pair<float> dzm = z3 && k > 0 ? ld2<float, V>(d, c - sz, second) : zero;
    const Pair<float> dzp = z3 && k + 1 < g.nz ? ld2<float, V>(d, c + sz, second) : zero;
    const Pair<float> ddh = ld2<float, V>(dh, c, second), ddl = ld2<float, V>(S.lo.diag, c, second);
    const Pair<float> cxh = ld2<float, V>(xh, c, second), cxl = ld2<float, V>(S.lo.cx, c, second);
    const float cxmh = i > 0 ? __ldg(xh + c - 1) : 0.0f, cxml = i > 0 ? __ldg(S.lo.cx + c - 1) : 0.0f;
    const Pair<float> cymh = j > 0 ? ld2<float, V>(yh, c - sy, second) : zero;
    const Pair<float> cyml = j > 0 ? ld2<float, V>(S.lo.cy, c - sy, second) : zero;
    const Pair<float> cyph = j + 1 < g.ny ? ld2<float, V>(yh, c, second) : zero;
    const Pair<float> cypl = j + 1 < g.ny ? ld2<float, V>(S.lo.cy, c, second) : zero;
    const Pair<float> czmh = z3 && k > 0 ? ld2<float, V>(zh, c - sz, second) : zero;
    const Pair<float> czml = z3 && k > 0 ? ld2<float, V>(S.lo.cz, c - sz, second) : zero;
    const Pair<float> czph = z3 && k + 1 < g.nz ? ld2<float, V>(zh, c, second) : zero;
    const Pair<float> czpl = z3 && k + 1 < g.nz ? ld2<float, V>(S.lo.cz, c, second) : zero;
    const Pair<double> r0 = ld2<double, V>(S.r64, c, second), x0 = ld2<double, V>(S.x64, c, second);
    // c d into the accumulator, negated for the neighbour terms
    auto mac = [](FloatFloat &a, float ch, float cl, float dv, bool neg) {
        float p = __fmul_rn(ch, dv);
        float e = __fadd_rn(__fmaf_rn(ch, dv, -p), __fmul_rn(cl, dv));
        if (neg) {
            p = -p;
            e = -e;
        }
        a.add(p);
        a.add(e);
    };
    FloatFloat t0, t1;
    mac(t0, ddh.a, ddl.a, dc.a, false);
    mac(t1, ddh.b, ddl.b, dc.b, false);
    // x: cell a's -x face (coupling at c - 1), its +x face shared with b
    // (coupling at c), b's +x face (coupling at c + 1)
    mac(t0, cxmh, cxml, dxm, true);
    mac(t0, cxh.a, cxl.a, dc.b, true);
    mac(t1, cxh.a, cxl.a, dc.a, true);
    mac(t1, cxh.b, cxl.b, dxp, true);
    mac(t0, cymh.a, cyml.a, dym.a, true);
    mac(t1, cymh.b, cyml.b, dym.b, true);
    mac(t0, cyph.a, cypl.a, dyp.a, true);
    mac(t1, cyph.b, cypl.b, dyp.b, true);
    mac(t0, czmh.a, czml.a, dzm.a, true);
    mac(t1, czmh.b, czml.b, dzm.b, true);
    mac(t0, czph.a, czpl.a, dzp.a, true);
    mac(t1, czph.b, czpl.b, dzp.b, true);
    // r -= A d and x += d: three FP64 additions per cell
    const Pair<double> rv{r0.a - (widen(t0.hi) + widen(t0.lo)), r0.b - (widen(t1.hi) + widen(t1.lo))};
    const Pair<T> rt{narrow_to<T>(rv.a), narrow_to<T>(rv.b)};
    st2<double, V>(S.r64, c, rv, second);
    st2<T, V>(S.r, c, rt, second);
    st2<double, V>(S.x64, c, Pair<double>{x0.a + widen(dc.a), x0.b + widen(dc.b)}, second);
    acc.add(rv.a, rt.a);
    if (second) acc.add(rv.b, rt.b);
}

// The mixed solver's outer step. initial: r64 = b - A64 prev (FP64; the
// stencil skipped without a warm start, r64 = b), x64 = 0, the threshold,
// |b - A prev|_2 kept. After an inner solve: x64 += d, r64 -= A d
// (refine_update_pair). Either way r_T = r64 for the next inner solve,
// |r64|_inf and |r64|_2, and the scene's last flush applies the stopping rule
// and opens the next inner solve; the last pass's norms are those of the
// returned solution's residual. Four resident blocks per SM (64 registers,
// no spill): the float-pair update keeps many loads in flight per thread,
// and given more registers the compiler takes 125 and halves the warps.
template <class T>
__global__ void __launch_bounds__(BLOCK_THREADS, 4) refine_residual_kernel(
    const BLevel<T> *__restrict__ levels, const BSeg *__restrict__ segs, int nseg, int n,
    const BScene<T> *__restrict__ scenes, double *part, int initial, double residual, int max_iter,
    double inner_rel, int inner_max, BatchCounters *cnt, const int *__restrict__ scene_of) {
    // one thread decides for the block: the launch itself lowers the counter,
    // and a block whose warps disagreed would copy half of a descriptor
    if (!initial && !__syncthreads_or(threadIdx.x == 0 && *(const volatile int *)&cnt->refine > 0)) return;
    __shared__ ItemCtx<T> ctx;
    sum_items<T, MaxSumAcc<T>>(
        segs, nseg, n, part, levels, scenes, initial ? -1 : 2, ctx,
        [&](const BItem &it, MaxSumAcc<T> &acc, T cls) {
            const BLevel<T> L = ctx.L;  // registers: stores through generic pointers would force reloads from shared memory
            const BScene<T> S = ctx.S;
            const Grid &g = L.g;
            const long long sy = g.nx, sz = (long long)g.nx * g.ny;
            const Operator<double> &A = S.A;
            // no unknown: b = 0 and every row of A is 0 there, so r = 0,
            // written by the initial pass (with x64 = 0) and unchanged after
            const bool empty = tile_empty(cls);
            if (empty && !initial) return;
            with_vec(L.vec, [&](auto vt) {
                constexpr bool V = decltype(vt)::value;
                if (empty) {
                    pair_tile(g, it, [&](int, int, int, long long c, bool second) {
                        st2<double, V>(S.r64, c, Pair<double>{0.0, 0.0}, second);
                        st2<T, V>(S.r, c, Pair<T>{T(0), T(0)}, second);
                        st2<double, V>(S.x64, c, Pair<double>{0.0, 0.0}, second);
                    });
                    return;
                }
                auto X2 = [&](long long m, bool sec) {
                    Pair<double> v{0.0, 0.0};
                    if (!initial) v = ld2<double, V>(S.x64, m, sec);
                    if (S.prev) {
                        const Pair<double> pv = ld2<double, V>(S.prev, m, sec);
                        v.a += pv.a;
                        v.b += pv.b;
                    }
                    return v;
                };
                auto X1 = [&](long long m) {
                    double v = initial ? 0.0 : __ldg(S.x64 + m);
                    if (S.prev) v += __ldg(S.prev + m);
                    return v;
                };
                const bool zero_x = initial && S.prev == nullptr;  // r = b exactly
                if constexpr (sizeof(T) == 4) {
                    if (!initial && S.lo.diag != nullptr) {
                        // after an inner solve: x64 += d and r64 -= A d
                        pair_tile(g, it, [&](int i, int j, int k, long long c, bool second) {
                            refine_update_pair<T, V>(g, L, S, i, j, k, c, second, acc);
                        });
                        return;
                    }
                }
                pair_tile(g, it, [&](int i, int j, int k, long long c, bool second) {
                    if (zero_x) {
                        const Pair<double> rv = ld2<double, V>(S.b, c, second);
                        const Pair<T> rt{narrow_to<T>(rv.a), narrow_to<T>(rv.b)};
                        st2<double, V>(S.r64, c, rv, second);
                        st2<T, V>(S.r, c, rt, second);
                        acc.add(rv.a, rt.a);
                        if (second) acc.add(rv.b, rt.b);
                        st2<double, V>(S.x64, c, Pair<double>{0.0, 0.0}, second);
                        return;
                    }
                    const Pair<double> xc = X2(c, second), dg = ld2<double, V>(A.diag, c, second);
                    const Pair<double> cxp = ld2<double, V>(A.cx, c, second);
                    double a0 = dg.a * xc.a, a1 = dg.b * xc.b;
                    if (i > 0) a0 -= __ldg(A.cx + c - 1) * X1(c - 1);
                    if (second) {
                        a0 -= cxp.a * xc.b;
                        a1 -= cxp.a * xc.a;
                        if (i + 2 < g.nx) a1 -= cxp.b * X1(c + 2);
                    }
                    if (j > 0) {
                        const Pair<double> w = ld2<double, V>(A.cy, c - sy, second), v = X2(c - sy, second);
                        a0 -= w.a * v.a;
                        a1 -= w.b * v.b;
                    }
                    if (j + 1 < g.ny) {
                        const Pair<double> w = ld2<double, V>(A.cy, c, second), v = X2(c + sy, second);
                        a0 -= w.a * v.a;
                        a1 -= w.b * v.b;
                    }
                    if (g.dim == 3) {
                        if (k > 0) {
                            const Pair<double> w = ld2<double, V>(A.cz, c - sz, second), v = X2(c - sz, second);
                            a0 -= w.a * v.a;
                            a1 -= w.b * v.b;
                        }
                        if (k + 1 < g.nz) {
                            const Pair<double> w = ld2<double, V>(A.cz, c, second), v = X2(c + sz, second);
                            a0 -= w.a * v.a;
                            a1 -= w.b * v.b;
                        }
                    }
                    const Pair<double> bb = ld2<double, V>(S.b, c, second);
                    const Pair<double> rv{bb.a - a0, bb.b - a1};
                    const Pair<T> rt{narrow_to<T>(rv.a), narrow_to<T>(rv.b)};
                    st2<double, V>(S.r64, c, rv, second);
                    st2<T, V>(S.r, c, rt, second);
                    acc.add(rv.a, rt.a);
                    if (second) acc.add(rv.b, rt.b);
                    if (initial) st2<double, V>(S.x64, c, Pair<double>{0.0, 0.0}, second);
                });
            });
        },
        [&](const BItem &it, int visits, int sums) {
            Scalars *sc = ctx.S.sc;
            if (item_last(&sc->counter[SITE_REFINE], visits)) {
                const double res = max_range(part, it.begin, visits);
                const double ss = sum_range(part + n, it.begin, sums);
                if (threadIdx.x == 0) {
                    sc->aux[0] = res;
                    sc->aux[1] = sqrt(ss);
                    if (initial) sc->aux[2] = sqrt(ss);
                    if (initial) {
                        const double tolf = residual < 1e-30 ? 1e-30 : residual;
                        sc->res0 = res;
                        sc->tol = tolf * res;
                        sc->iter = 0;
                        sc->outer_iter = 0;
                        sc->max_iter = max_iter;
                        sc->inner_max = inner_max;
                        sc->status = 0;
                        sc->done = 0;
                    } else {
                        sc->outer_iter += 1;
                        atomicSub(&cnt->refine, 1);
                    }
                    sc->res = res;
                    int finished = 1;
                    if (res != res) {
                        sc->status = 3;
                    } else if (res <= sc->tol) {
                        sc->status = 1;
                    } else if (sc->iter >= sc->max_iter) {
                        sc->status = 2;
                    } else {
                        finished = 0;
                        sc->inner_done = 0;
                        sc->inner_iter = 0;
                        sc->first = 1;
                        sc->first_update = 1;
                        sc->inner_res0 = res;
                        sc->inner_tol = inner_rel * res;
                    }
                    if (finished) {
                        sc->done = 1;
                        atomicSub(&cnt->remaining, 1);
                    }
                    sc->counter[SITE_REFINE] = 0;
                }
            }
        });
}

// ---- TMA-staged fine-level kernels (FP32) ---------------------------------------------

constexpr int ST_HX = ST_TX + 8, ST_HY = ST_TY + 2, ST_HZ = ST_TZ + 2;
constexpr int ST_HALO = ST_HX * ST_HY * ST_HZ;       // floats of a HALO box
constexpr int ST_OWN = ST_TX * ST_TY * ST_TZ;        // OWN
constexpr int ST_CXN = ST_HX * ST_TY * ST_TZ;        // CX
constexpr int ST_CYN = ST_TX * (ST_TY + 1) * ST_TZ;  // CY
constexpr int ST_CZN = ST_TX * ST_TY * (ST_TZ + 1);  // CZ
constexpr int ST_XCX = 40, ST_XCY = 6, ST_XCZ = 4;
constexpr int ST_XCN = ST_XCX * ST_XCY * ST_XCZ;      // XC
static_assert(ST_HALO % 32 == 0 && ST_OWN % 32 == 0 && ST_CXN % 32 == 0 && ST_CYN % 32 == 0 && ST_CZN % 32 == 0 &&
                  ST_XCN % 32 == 0,
              "every box starts on a 128-byte boundary");

// Box layout of one stage of each kind, in floats: {map, offset, size}.
struct StageBox {
    int map, off, n;
};
template <int KIND> struct StageLayout;
template <> struct StageLayout<STAGE_PRESMOOTH> {
    static constexpr int nbox = 5;
    __host__ __device__ static constexpr StageBox box(int q) {
        return q == 0   ? StageBox{SM_B_HALO, 0, ST_HALO}
               : q == 1 ? StageBox{SM_INV_HALO, ST_HALO, ST_HALO}
               : q == 2 ? StageBox{SM_CX, 2 * ST_HALO, ST_CXN}
               : q == 3 ? StageBox{SM_CY, 2 * ST_HALO + ST_CXN, ST_CYN}
                        : StageBox{SM_CZ, 2 * ST_HALO + ST_CXN + ST_CYN, ST_CZN};
    }
    static constexpr int floats = 2 * ST_HALO + ST_CXN + ST_CYN + ST_CZN;
};
template <> struct StageLayout<STAGE_POST_BLACK> {
    static constexpr int nbox = 7;
    __host__ __device__ static constexpr StageBox box(int q) {
        return q == 0   ? StageBox{SM_X_HALO, 0, ST_HALO}
               : q == 1 ? StageBox{SM_B_OWN, ST_HALO, ST_OWN}
               : q == 2 ? StageBox{SM_INV_OWN, ST_HALO + ST_OWN, ST_OWN}
               : q == 3 ? StageBox{SM_CX, ST_HALO + 2 * ST_OWN, ST_CXN}
               : q == 4 ? StageBox{SM_CY, ST_HALO + 2 * ST_OWN + ST_CXN, ST_CYN}
               : q == 5 ? StageBox{SM_CZ, ST_HALO + 2 * ST_OWN + ST_CXN + ST_CYN, ST_CZN}
                        : StageBox{SM_XC, ST_HALO + 2 * ST_OWN + ST_CXN + ST_CYN + ST_CZN, ST_XCN};
    }
    static constexpr int floats = ST_HALO + 2 * ST_OWN + ST_CXN + ST_CYN + ST_CZN + ST_XCN;
};
template <> struct StageLayout<STAGE_RED_DOT> {
    static constexpr int nbox = 6;
    __host__ __device__ static constexpr StageBox box(int q) {
        return q == 0   ? StageBox{SM_X_HALO, 0, ST_HALO}
               : q == 1 ? StageBox{SM_B_OWN, ST_HALO, ST_OWN}
               : q == 2 ? StageBox{SM_INV_OWN, ST_HALO + ST_OWN, ST_OWN}
               : q == 3 ? StageBox{SM_CX, ST_HALO + 2 * ST_OWN, ST_CXN}
               : q == 4 ? StageBox{SM_CY, ST_HALO + 2 * ST_OWN + ST_CXN, ST_CYN}
                        : StageBox{SM_CZ, ST_HALO + 2 * ST_OWN + ST_CXN + ST_CYN, ST_CZN};
    }
    static constexpr int floats = ST_HALO + 2 * ST_OWN + ST_CXN + ST_CYN + ST_CZN;
};
template <> struct StageLayout<STAGE_SPMV> {
    static constexpr int nbox = 5;
    __host__ __device__ static constexpr StageBox box(int q) {
        return q == 0   ? StageBox{SM_P_HALO, 0, ST_HALO}
               : q == 1 ? StageBox{SM_DIAG_OWN, ST_HALO, ST_OWN}
               : q == 2 ? StageBox{SM_CX, ST_HALO + ST_OWN, ST_CXN}
               : q == 3 ? StageBox{SM_CY, ST_HALO + ST_OWN + ST_CXN, ST_CYN}
                        : StageBox{SM_CZ, ST_HALO + ST_OWN + ST_CXN + ST_CYN, ST_CZN};
    }
    static constexpr int floats = ST_HALO + ST_OWN + ST_CXN + ST_CYN + ST_CZN;
};

__device__ __forceinline__ unsigned smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned long long *b) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(b)));
}
__device__ __forceinline__ void mbar_expect(unsigned long long *b, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(b)), "r"(bytes) : "memory");
}
// Bounded wait for the phase of the given parity (about two seconds at most
// with the default limit of 2^22 polls).
__device__ __forceinline__ bool mbar_wait(unsigned long long *b, unsigned parity, int limit) {
    for (int it = 0; it < limit; ++it) {
        unsigned done;
        asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.b32 %0, 1, 0, p; }"
                     : "=r"(done)
                     : "r"(smem_u32(b)), "r"(parity)
                     : "memory");
        if (done) return true;
    }
    return false;
}
__device__ __forceinline__ void tma_box(float *dst, const CUtensorMap *map, int x, int y, int z,
                                        unsigned long long *b) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
        "[%5];" ::"r"(smem_u32(dst)),
        "l"(map), "r"(x), "r"(y), "r"(z), "r"(smem_u32(b))
        : "memory");
}

// Neighbour sum of cell h (0: i, 1: i+1) of a pair from the staged boxes, in
// the order -x, +x, -y, +y, -z, +z (the arithmetic of pair_nsum): hc is cell
// i's index in a HALO box, cxi / cyi / czi in the CX / CY / CZ boxes, `own`
// the pair's values, val(m, d) the value at HALO index m reached in
// direction d (0..5 for -x, +x, -y, +y, -z, +z). The pair's second cell
// always exists (staged levels have nx % 8 == 0).
template <class VF>
__device__ __forceinline__ float staged_nsum(int h, const Grid &g, int i, int j, int k, int hc, int cxi, int cyi,
                                             int czi, const float *scx, const float *scy, const float *scz,
                                             Pair<float> own, VF val) {
    float s = 0.0f;
    if (h == 0) {
        if (i > 0) s += scx[cxi - 1] * val(hc - 1, 0);
        s += scx[cxi] * own.b;
    } else {
        s += scx[cxi] * own.a;
        if (i + 2 < g.nx) s += scx[cxi + 1] * val(hc + 2, 1);
    }
    const int hh = hc + h;
    if (j > 0) s += scy[cyi + h - ST_TX] * val(hh - ST_HX, 2);
    if (j + 1 < g.ny) s += scy[cyi + h] * val(hh + ST_HX, 3);
    if (k > 0) s += scz[czi + h - ST_TX * ST_TY] * val(hh - ST_HX * ST_HY, 4);
    if (k + 1 < g.nz) s += scz[czi + h] * val(hh + ST_HX * ST_HY, 5);
    return s;
}

// One launch over the staged fine levels of a batch: blocks walk their items
// (one 64 x 8 x 4 tile each) as the other kernels do, with the tiles of the
// next two items in flight: thread 0 issues an item's boxes into a stage
// when the item two back has been consumed, every thread waits on the
// stage's mbarrier (bounded), computes from shared memory, and writes its
// results to global memory. Reductions (red_dot, spmv) flush per scene as
// sum_items does for a single scene. A wait that runs out records cnt->bar_err = 2 and the
// block leaves after letting its other copy land (bounded); the host then
// abandons the solve.
template <int KIND>
__global__ void __launch_bounds__(BLOCK_THREADS, 1)
    staged_kernel(const BLevel<float> *__restrict__ levels, const BSeg *__restrict__ segs, int nseg, int n,
                  const BScene<float> *__restrict__ scenes, int gate, double *part, float alpha, BatchCounters *cnt) {
    using LY = StageLayout<KIND>;
    constexpr bool REDUCE = KIND == STAGE_RED_DOT || KIND == STAGE_SPMV;
    constexpr int STAGE_FLOATS = LY::floats;
    if (batch_idle(cnt)) return;
    extern __shared__ unsigned char st_smem[];
    __shared__ __align__(8) unsigned long long bar[2];
    __shared__ int valid[2];
    __shared__ ItemCtx<float> ctx;
    float *stage0 = reinterpret_cast<float *>(st_smem + ((128u - (smem_u32(st_smem) & 127u)) & 127u));
    const int tid = threadIdx.x, G = gridDim.x;
    if (tid == 0) {
        mbar_init(&bar[0]);
        mbar_init(&bar[1]);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    int issue_seg = 0;
    // thread 0: the boxes of item w into stage s (if its scene is not gated)
    auto issue = [&](int s, int w) {
        const BItem it = item_at(segs, nseg, w, issue_seg);
        const BLevel<float> &L = levels[it.ref];
        const int ok = gate < 0 ? 1 : !gated(scenes[L.scene].sc, gate);
        valid[s] = ok;
        if (!ok) return;
        const Grid &g = L.g;
        const unsigned t = (unsigned)it.tile;
        const unsigned r = fdiv(t, g.ftx2);
        const unsigned tk = fdiv(r, g.fty);
        const int x0 = (int)(t - r * g.ftx2.d) * ST_TX, y0 = (int)(r - tk * (unsigned)g.nty) * ST_TY,
                  z0 = (int)tk * ST_TZ;
        float *dst = stage0 + (size_t)s * STAGE_FLOATS;
        mbar_expect(&bar[s], (unsigned)(LY::floats * 4));
#pragma unroll
        for (int q = 0; q < LY::nbox; ++q) {
            const StageBox bx = LY::box(q);
            int x = x0, y = y0, z = z0;
            if (bx.map == SM_XC) {
                x = x0 / 2 - 4;
                y = y0 / 2 - 1;
                z = z0 / 2 - 1;
            } else if (bx.map <= SM_P_HALO) {
                x = x0 - 4;
                y = y0 - 1;
                z = z0 - 1;
            } else if (bx.map == SM_CX) {
                x = x0 - 4;
            } else if (bx.map == SM_CY) {
                y = y0 - 1;
            } else if (bx.map == SM_CZ) {
                z = z0 - 1;
            }
            tma_box(dst + bx.off, L.tmap + bx.map, x, y, z, &bar[s]);
        }
    };
    const int polls = cnt->test_polls > 0 ? cnt->test_polls : (1 << 22);
    if (tid == 0) {
        if (blockIdx.x < n) {
            if (cnt->test_what == 2 && (int)blockIdx.x == cnt->test_block)
                valid[0] = 1;  // test hook: the first tile is awaited but never copied
            else
                issue(0, blockIdx.x);
        }
        if (blockIdx.x + G < n) issue(1, blockIdx.x + G);
    }
    __syncthreads();
    unsigned phase = 0u;
    int cur = -1, sgc = 0;
    BItem first{};
    DotAcc<float> acc;
    acc.reset();
    auto flush = [&]() {
        const int slot = (int)((((long long)blockIdx.x - first.begin) % G + G) % G);
        acc.store(part, first.begin + slot);
        const int flushes = min(first.count, G);
        Scalars *sc = ctx.S.sc;
        if constexpr (KIND == STAGE_RED_DOT) {
            if (item_last(&sc->counter[SITE_DOT], flushes)) {
                const double rho_new = sum_range(part, first.begin, flushes);
                if (threadIdx.x == 0) {
                    if (sc->first) {
                        sc->beta = 0.0;
                        sc->first = 0;
                    } else {
                        sc->beta = rho_new / sc->rho;
                    }
                    sc->rho = rho_new;
                    if (rho_new != rho_new) {
                        sc->done = 1;
                        sc->status = 3;
                    }
                    sc->counter[SITE_DOT] = 0;
                }
            }
        } else if constexpr (KIND == STAGE_SPMV) {
            if (item_last(&sc->counter[SITE_SPMV], flushes)) {
                const double pq = sum_range(part, first.begin, flushes);
                if (threadIdx.x == 0) {
                    sc->pap = pq;
                    sc->alpha = sc->rho / pq;
                    sc->counter[SITE_SPMV] = 0;
                }
            }
        }
    };
    for (int nn = 0, w = blockIdx.x; w < n; ++nn, w += G) {
        const int s = nn & 1;
        const BItem it = item_at(segs, nseg, w, sgc);
        if (it.ref != cur) {
            if (REDUCE && cur >= 0 && !ctx.skip) flush();
            refresh(ctx, cur, it, levels, scenes, gate);
            first = it;
            acc.reset();
        }
        if (valid[s]) {
            const bool ok = mbar_wait(&bar[s], (phase >> s) & 1u, polls);
            if (__syncthreads_or(!ok)) {
                if (tid == 0) {
                    atomicExch(&cnt->bar_err, 2);
                    if (w + G < n && valid[s ^ 1]) mbar_wait(&bar[s ^ 1], (phase >> (s ^ 1)) & 1u, polls);
                }
                return;
            }
            phase ^= 1u << s;
            const BLevel<float> L = ctx.L;
            const Grid &g = L.g;
            const float *st = stage0 + (size_t)s * STAGE_FLOATS;
            const unsigned t = (unsigned)it.tile;
            const unsigned r = fdiv(t, g.ftx2);
            const unsigned tk = fdiv(r, g.fty);
            const int x0 = (int)(t - r * g.ftx2.d) * ST_TX, y0 = (int)(r - tk * (unsigned)g.nty) * ST_TY,
                      z0 = (int)tk * ST_TZ;
            const int px = tid & 31, qy = tid >> 5;
            const int i = x0 + 2 * px, j = y0 + qy;
            if (i < g.nx && j < g.ny) {
                const float *scx = st + LY::box((KIND == STAGE_PRESMOOTH || KIND == STAGE_SPMV) ? 2 : 3).off;
                const float *scy = scx + ST_CXN, *scz = scy + ST_CYN;
                for (int kk = 0; kk < ST_TZ; ++kk) {
                    const int k = z0 + kk;
                    if (k >= g.nz) break;
                    const int hc = (2 * px + 4) + ST_HX * ((qy + 1) + ST_HY * (kk + 1));
                    const int oc = 2 * px + ST_TX * (qy + ST_TY * kk);
                    const int cxi = (2 * px + 4) + ST_HX * (qy + ST_TY * kk);
                    const int cyi = 2 * px + ST_TX * ((qy + 1) + (ST_TY + 1) * kk);
                    const int czi = 2 * px + ST_TX * (qy + ST_TY * (kk + 1));
                    const long long c = cell_index(g, i, j, k);
                    if constexpr (KIND == STAGE_PRESMOOTH) {
                        const float *sb = st, *si = st + ST_HALO;
                        const Pair<float> b2{sb[hc], sb[hc + 1]}, iv{si[hc], si[hc + 1]};
                        const Pair<float> red{b2.a * iv.a, b2.b * iv.b};
                        auto val = [&](int m, int) { return sb[m] * si[m]; };
                        Pair<float> out = red;
                        if (((i + j + k) & 1) == 0)
                            out.b = (b2.b + staged_nsum(1, g, i, j, k, hc, cxi, cyi, czi, scx, scy, scz, red, val)) *
                                    iv.b;
                        else
                            out.a = (b2.a + staged_nsum(0, g, i, j, k, hc, cxi, cyi, czi, scx, scy, scz, red, val)) *
                                    iv.a;
                        st2<float, true>(L.x, c, out, true);
                    } else if constexpr (KIND == STAGE_POST_BLACK) {
                        const float *sx = st, *sb = st + ST_HALO, *si = sb + ST_OWN, *sxc = scz + ST_CZN;
                        const int h = ((i + j + k) & 1) == 1 ? 0 : 1;
                        // parents in the XC box: own, and the steps to the
                        // parents of the -x, +x, -y, +y, -z, +z neighbours
                        const int P = (px + 4) + ST_XCX * (((qy >> 1) + 1) + ST_XCY * ((kk >> 1) + 1));
                        const int step[6] = {-1, 1, (j & 1) ? 0 : -ST_XCX, (j & 1) ? ST_XCX : 0,
                                             (k & 1) ? 0 : -ST_XCX * ST_XCY, (k & 1) ? ST_XCX * ST_XCY : 0};
                        const float pc = sxc[P];
                        auto val = [&](int m, int d) {
                            const float q = (d >= 2 && step[d] == 0) ? pc : sxc[P + step[d]];
                            return prolong(sx[m], alpha, q);
                        };
                        const Pair<float> own{prolong(sx[hc], alpha, pc), prolong(sx[hc + 1], alpha, pc)};
                        const float sh = staged_nsum(h, g, i, j, k, hc, cxi, cyi, czi, scx, scy, scz, own, val);
                        L.x[c + h] = (sb[oc + h] + sh) * si[oc + h];
                    } else if constexpr (KIND == STAGE_RED_DOT) {
                        const float *sx = st, *sb = st + ST_HALO, *si = sb + ST_OWN;
                        const int hr = ((i + j + k) & 1) == 0 ? 0 : 1;
                        const Pair<float> x2{sx[hc], sx[hc + 1]}, b2{sb[oc], sb[oc + 1]};
                        auto val = [&](int m, int) { return sx[m]; };
                        const float sh = staged_nsum(hr, g, i, j, k, hc, cxi, cyi, czi, scx, scy, scz, x2, val);
                        const float xv = ((hr ? b2.b : b2.a) + sh) * si[oc + hr];
                        Pair<float> out = x2;
                        if (hr) out.b = xv;
                        else out.a = xv;
                        L.x[c + hr] = xv;
                        acc.add(out.a, b2.a);
                        acc.add(out.b, b2.b);
                    } else {
                        const float *sp = st, *sd = st + ST_HALO;
                        const Pair<float> p2{sp[hc], sp[hc + 1]}, d2{sd[oc], sd[oc + 1]};
                        auto val = [&](int m, int) { return sp[m]; };
                        const float sa = staged_nsum(0, g, i, j, k, hc, cxi, cyi, czi, scx, scy, scz, p2, val);
                        const float sb2 = staged_nsum(1, g, i, j, k, hc, cxi, cyi, czi, scx, scy, scz, p2, val);
                        const Pair<float> q2{d2.a * p2.a - sa, d2.b * p2.b - sb2};
                        st2<float, true>(ctx.S.q, c, q2, true);
                        acc.add(p2.a, q2.a);
                        acc.add(p2.b, q2.b);
                    }
                }
            }
        }
        __syncthreads();  // stage s consumed by every thread
        if (tid == 0 && w + 2 * G < n) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            issue(s, w + 2 * G);
        }
    }
    if (REDUCE && cur >= 0 && !ctx.skip) flush();
}

}  // namespace

// Launches kernel<T, OCC> with OCC = L.occ, one of the occupancy variants
// the kernels are compiled for (blocks of 256 threads per SM); 0 selects the
// precision's default.
#define OCC_DISPATCH(L, kernel, T, ARGS)                                                  \
    do {                                                                                  \
        switch ((L).occ ? (L).occ : BatchOcc<T>::blocks) {                                \
        case 4: kernel<T, 4><<<(L).blocks, BLOCK_THREADS, 0, (L).stream>>> ARGS; break;   \
        case 6: kernel<T, 6><<<(L).blocks, BLOCK_THREADS, 0, (L).stream>>> ARGS; break;   \
        default: kernel<T, 5><<<(L).blocks, BLOCK_THREADS, 0, (L).stream>>> ARGS; break;  \
        }                                                                                 \
    } while (0)
// The same for the kernels with a gather-first column form: COL when the
// list holds 4-plane tiles ((L).col), else the plane-by-plane kernel alone.
#define OCC_COL_DISPATCH(L, kernel, T, ARGS)                                                     \
    do {                                                                                         \
        const int occ_ = (L).occ ? (L).occ : BatchOcc<T>::blocks;                                \
        if ((L).col) {                                                                           \
            if (occ_ == 4) kernel<T, 4, true><<<(L).blocks, BLOCK_THREADS, 0, (L).stream>>> ARGS;       \
            else if (occ_ == 6) kernel<T, 6, true><<<(L).blocks, BLOCK_THREADS, 0, (L).stream>>> ARGS;  \
            else kernel<T, 5, true><<<(L).blocks, BLOCK_THREADS, 0, (L).stream>>> ARGS;                 \
        } else {                                                                                 \
            if (occ_ == 4) kernel<T, 4, false><<<(L).blocks, BLOCK_THREADS, 0, (L).stream>>> ARGS;      \
            else if (occ_ == 6) kernel<T, 6, false><<<(L).blocks, BLOCK_THREADS, 0, (L).stream>>> ARGS; \
            else kernel<T, 5, false><<<(L).blocks, BLOCK_THREADS, 0, (L).stream>>> ARGS;                \
        }                                                                                        \
    } while (0)

template <class T>
cudaError_t b_presmooth(const BLaunch &L, const BLevel<T> *levels, const BSeg *segs, int nseg, int n,
                        const BScene<T> *scenes) {
    OCC_COL_DISPATCH(L, presmooth_kernel, T, (levels, segs, nseg, n, scenes, L.gate, L.cnt));
    return cudaGetLastError();
}
template <class T>
cudaError_t b_sweep(const BLaunch &L, const BLevel<T> *levels, const BSeg *segs, int nseg, int n,
                    const BScene<T> *scenes, int color) {
    OCC_DISPATCH(L, sweep_kernel, T, (levels, segs, nseg, n, scenes, L.gate, color, L.cnt));
    return cudaGetLastError();
}
template <class T>
cudaError_t b_restrict(const BLaunch &L, const BLevel<T> *levels, const BSeg *segs, int nseg, int n,
                       const BScene<T> *scenes) {
    OCC_DISPATCH(L, restrict_kernel, T, (levels, segs, nseg, n, scenes, L.gate, L.cnt));
    return cudaGetLastError();
}
template <class T>
cudaError_t b_post_black(const BLaunch &L, const BLevel<T> *levels, const BSeg *segs, int nseg, int n,
                         const BScene<T> *scenes, T alpha) {
    OCC_COL_DISPATCH(L, post_black_kernel, T, (levels, segs, nseg, n, scenes, L.gate, alpha,
                                                                   L.cnt));
    return cudaGetLastError();
}
template <class T>
cudaError_t b_red_dot(const BLaunch &L, const BLevel<T> *levels, const BSeg *segs, int nseg, int n,
                      const BScene<T> *scenes, double *part) {
    OCC_COL_DISPATCH(L, red_dot_kernel, T, (levels, segs, nseg, n, scenes, L.gate, part,
                                                                L.scene_of, L.cnt));
    return cudaGetLastError();
}
template <class T>
cudaError_t b_tail(const BLaunch &L, const BTail<T> *tails, int nscenes, const BScene<T> *scenes, MgSettings ms) {
    tail_kernel<T><<<nscenes, MG_TAIL_THREADS, 0, L.stream>>>(tails, scenes, L.gate, ms, L.cnt);
    return cudaGetLastError();
}
template <class T> cudaError_t b_tail_matrix(cudaStream_t st, const BTail<T> *tails, int nscenes, MgSettings ms) {
    tail_matrix_kernel<T><<<nscenes * TAIL_DENSE, 32, 0, st>>>(tails, ms);
    return cudaGetLastError();
}
template <class T>
cudaError_t b_coarse_descend(const BLaunch &L, const BLevel<T> *levels, const CoarseLists &cl,
                             const BScene<T> *scenes, MgSettings ms) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)L.blocks);
    cfg.blockDim = dim3(BLOCK_THREADS);
    cfg.stream = L.stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (L.occ == 2) return cudaLaunchKernelEx(&cfg, coarse_descend_kernel<T, 2>, levels, cl, scenes, L.gate, ms, L.cnt);
    return cudaLaunchKernelEx(&cfg, coarse_descend_kernel<T, BatchOcc<T>::blocks>, levels, cl, scenes, L.gate, ms,
                              L.cnt);
}
template <class T>
cudaError_t b_coarse_ascend(const BLaunch &L, const BLevel<T> *levels, const CoarseLists &cl,
                            const BScene<T> *scenes, MgSettings ms, T alpha) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)L.blocks);
    cfg.blockDim = dim3(BLOCK_THREADS);
    cfg.stream = L.stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (L.occ == 2)
        return cudaLaunchKernelEx(&cfg, coarse_ascend_kernel<T, 2>, levels, cl, scenes, L.gate, ms, alpha, L.cnt);
    return cudaLaunchKernelEx(&cfg, coarse_ascend_kernel<T, BatchOcc<T>::blocks>, levels, cl, scenes, L.gate, ms,
                              alpha, L.cnt);
}
// resident blocks of the two cooperative kernels on `sms` SMs (the smaller)
template <class T> int b_coarse_capacity(int sms) {
    int a = 0, b = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, coarse_descend_kernel<T, BatchOcc<T>::blocks>,
                                                      BLOCK_THREADS, 0) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, coarse_ascend_kernel<T, BatchOcc<T>::blocks>,
                                                      BLOCK_THREADS, 0) != cudaSuccess)
        return 0;
    return sms * (a < b ? a : b);
}
size_t stage_bytes(int kind) {
    switch (kind) {
    case STAGE_PRESMOOTH: return sizeof(float) * StageLayout<STAGE_PRESMOOTH>::floats;
    case STAGE_POST_BLACK: return sizeof(float) * StageLayout<STAGE_POST_BLACK>::floats;
    case STAGE_RED_DOT: return sizeof(float) * StageLayout<STAGE_RED_DOT>::floats;
    default: return sizeof(float) * StageLayout<STAGE_SPMV>::floats;
    }
}
// two stages and 128 bytes to align them
static size_t staged_smem(int kind) { return 2 * stage_bytes(kind) + 128; }
cudaError_t b_staged_enable() {
    cudaError_t e = cudaFuncSetAttribute(staged_kernel<STAGE_PRESMOOTH>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)staged_smem(STAGE_PRESMOOTH));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(staged_kernel<STAGE_POST_BLACK>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)staged_smem(STAGE_POST_BLACK));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(staged_kernel<STAGE_RED_DOT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)staged_smem(STAGE_RED_DOT));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(staged_kernel<STAGE_SPMV>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)staged_smem(STAGE_SPMV));
    return e;
}
cudaError_t b_staged(int kind, const BLaunch &L, const BLevel<float> *levels, const BSeg *segs, int nseg, int n,
                     const BScene<float> *scenes, double *part, float alpha) {
    const size_t sm = staged_smem(kind);
    switch (kind) {
    case STAGE_PRESMOOTH:
        staged_kernel<STAGE_PRESMOOTH><<<L.blocks, BLOCK_THREADS, sm, L.stream>>>(levels, segs, nseg, n, scenes, L.gate,
                                                                                  part, alpha, L.cnt);
        break;
    case STAGE_POST_BLACK:
        staged_kernel<STAGE_POST_BLACK><<<L.blocks, BLOCK_THREADS, sm, L.stream>>>(levels, segs, nseg, n, scenes,
                                                                                   L.gate, part, alpha, L.cnt);
        break;
    case STAGE_RED_DOT:
        staged_kernel<STAGE_RED_DOT><<<L.blocks, BLOCK_THREADS, sm, L.stream>>>(levels, segs, nseg, n, scenes, L.gate,
                                                                                part, alpha, L.cnt);
        break;
    default:
        staged_kernel<STAGE_SPMV><<<L.blocks, BLOCK_THREADS, sm, L.stream>>>(levels, segs, nseg, n, scenes, L.gate,
                                                                             part, alpha, L.cnt);
    }
    return cudaGetLastError();
}

template <class T>
cudaError_t b_direction(const BLaunch &L, const BLevel<T> *levels, const BSeg *segs, int nseg, int n,
                        const BScene<T> *scenes) {
    OCC_DISPATCH(L, direction_kernel, T, (levels, segs, nseg, n, scenes, L.gate, L.cnt));
    return cudaGetLastError();
}
template <class T>
cudaError_t b_spmv(const BLaunch &L, const BLevel<T> *levels, const BSeg *segs, int nseg, int n,
                   const BScene<T> *scenes, double *part) {
    OCC_COL_DISPATCH(L, spmv_kernel, T, (levels, segs, nseg, n, scenes, L.gate, part, L.scene_of,
                                                             L.cnt));
    return cudaGetLastError();
}
template <class T>
cudaError_t b_direction_spmv(const BLaunch &L, const BLevel<T> *levels, const BSeg *segs, int nseg, int n,
                             const BScene<T> *scenes, double *part) {
    OCC_COL_DISPATCH(L, direction_spmv_kernel, T, (levels, segs, nseg, n, scenes, L.gate, part, L.cnt));
    return cudaGetLastError();
}
template <class T>
cudaError_t b_update(const BLaunch &L, const BLevel<T> *levels, const BSeg *segs, int nseg, int n,
                     const BScene<T> *scenes, double *part, int mode, BatchCounters *cnt) {
    OCC_DISPATCH(L, update_kernel, T, (levels, segs, nseg, n, scenes, L.gate, part, mode, cnt,
                                                               L.scene_of));
    return cudaGetLastError();
}
template <class T>
cudaError_t b_refine_residual(const BLaunch &L, const BLevel<T> *levels, const BSeg *segs, int nseg, int n,
                              const BScene<T> *scenes, double *part, int initial, double residual, int max_iter,
                              double inner_rel, int inner_max, BatchCounters *cnt) {
    refine_residual_kernel<T><<<L.blocks, BLOCK_THREADS, 0, L.stream>>>(
        levels, segs, nseg, n, scenes, part, initial, residual, max_iter, inner_rel, inner_max, cnt, L.scene_of);
    return cudaGetLastError();
}

#define GBP_BATCH_INSTANTIATE(T)                                                                                     \
    template cudaError_t b_presmooth<T>(const BLaunch &, const BLevel<T> *, const BSeg *, int, int,                 \
                                        const BScene<T> *);                                                          \
    template cudaError_t b_sweep<T>(const BLaunch &, const BLevel<T> *, const BSeg *, int, int, const BScene<T> *,  \
                                    int);                                                                            \
    template cudaError_t b_restrict<T>(const BLaunch &, const BLevel<T> *, const BSeg *, int, int,                  \
                                       const BScene<T> *);                                                           \
    template cudaError_t b_post_black<T>(const BLaunch &, const BLevel<T> *, const BSeg *, int, int,                \
                                         const BScene<T> *, T);                                                      \
    template cudaError_t b_red_dot<T>(const BLaunch &, const BLevel<T> *, const BSeg *, int, int,                   \
                                      const BScene<T> *, double *);                                                  \
    template cudaError_t b_tail<T>(const BLaunch &, const BTail<T> *, int, const BScene<T> *, MgSettings);            \
    template cudaError_t b_tail_matrix<T>(cudaStream_t, const BTail<T> *, int, MgSettings);                           \
    template cudaError_t b_coarse_descend<T>(const BLaunch &, const BLevel<T> *, const CoarseLists &,                 \
                                             const BScene<T> *, MgSettings);                                         \
    template cudaError_t b_coarse_ascend<T>(const BLaunch &, const BLevel<T> *, const CoarseLists &,                  \
                                            const BScene<T> *, MgSettings, T);                                       \
    template int b_coarse_capacity<T>(int);                                                                          \
    template cudaError_t b_direction<T>(const BLaunch &, const BLevel<T> *, const BSeg *, int, int,                 \
                                        const BScene<T> *);                                                          \
    template cudaError_t b_spmv<T>(const BLaunch &, const BLevel<T> *, const BSeg *, int, int, const BScene<T> *,   \
                                   double *);                                                                        \
    template cudaError_t b_direction_spmv<T>(const BLaunch &, const BLevel<T> *, const BSeg *, int, int,            \
                                             const BScene<T> *, double *);                                           \
    template cudaError_t b_update<T>(const BLaunch &, const BLevel<T> *, const BSeg *, int, int, const BScene<T> *, \
                                     double *, int, BatchCounters *);                                                \
    template cudaError_t b_refine_residual<T>(const BLaunch &, const BLevel<T> *, const BSeg *, int, int,           \
                                              const BScene<T> *, double *, int, double, int, double, int,            \
                                              BatchCounters *);

GBP_BATCH_INSTANTIATE(double)
GBP_BATCH_INSTANTIATE(float)

}  // namespace gbp
