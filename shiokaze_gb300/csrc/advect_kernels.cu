// advect_kernels.cu -- MacCormack / semi-Lagrangian advection of a cell
// scalar and of the MAC velocity on dense device grids (see advect.h and
// advect_core.cuh). Compiled with --fmad=false: every result equals the
// reference's scalar C++ bit for bit.
//
// A MacCormack step is four launches: scalar forward (forward value and the
// limiter's record per cell), scalar backward (+ the limited correction,
// written in place), velocity forward, velocity backward (in place). The
// backward kernels read the step's input only at their own face or cell, so
// writing the result over it is safe; the forward kernels read neighbours
// and write scratch. One semi-Lagrangian pass is the forward kernel and a
// copy back.
//
// One thread per face (blockIdx.y = component) or cell. Algorithmic DRAM
// bytes per face of a MacCormack velocity step: forward reads u (4; the
// neighbours come from cache) and writes the forward value and the limiter
// record (4 + 8), backward reads them and the input (16) and writes the
// result (4): 32 B. Cell scalar: the same 32 B plus the fluid level set read
// twice (8) and, on the cell passes, the 3 velocity components' two faces
// (counted once, 12). The reference's arithmetic is double precision
// throughout, and in FP64 instructions its trilinear weights and sums kept
// the FP64 pipe 86 % busy; the kernels take each element through the
// float-pair form of advect_fast.cuh, with the FP64 form (advect_core.cuh)
// for the few it leaves undecided, and are bound by FP32 instruction issue
// instead. A 256^3 smoke step (density and velocity): 40.75 ms in FP64,
// 3.51 ms in float pairs; a 1000 x 777 2D step 1.09 ms and 0.19 ms; the same
// bits.
#include <algorithm>
#include <cfloat>
#include <cmath>

#include "advect.h"
#include "advect_core.cuh"
#include "advect_fast.cuh"

namespace gbp {
namespace {

using gba::Dims;
using gba::Fast;
using gba::StepArgs;

constexpr int ADV_THREADS = 256;

// one thread per face, blockIdx.y = component
template <bool MAC>
__global__ void __launch_bounds__(ADV_THREADS) adv_face_forward(const __grid_constant__ StepArgs a,
                                                               const __grid_constant__ Fast k) {
    const unsigned f = blockIdx.x * blockDim.x + threadIdx.x;
    if (blockIdx.y == 0) gba::face_forward_any<0, MAC>(a, k, f);
    else if (blockIdx.y == 1) gba::face_forward_any<1, MAC>(a, k, f);
    else gba::face_forward_any<2, MAC>(a, k, f);
}

__global__ void __launch_bounds__(ADV_THREADS) adv_face_backward(const __grid_constant__ StepArgs a,
                                                                const __grid_constant__ Fast k) {
    const unsigned f = blockIdx.x * blockDim.x + threadIdx.x;
    if (blockIdx.y == 0) gba::face_backward_any<0>(a, k, f);
    else if (blockIdx.y == 1) gba::face_backward_any<1>(a, k, f);
    else gba::face_backward_any<2>(a, k, f);
}

// one thread per cell
template <bool MAC>
__global__ void __launch_bounds__(ADV_THREADS) adv_cell_forward(const __grid_constant__ StepArgs a,
                                                               const __grid_constant__ Fast k) {
    gba::cell_forward_any<MAC>(a, k, blockIdx.x * blockDim.x + threadIdx.x);
}

__global__ void __launch_bounds__(ADV_THREADS) adv_cell_backward(const __grid_constant__ StepArgs a,
                                                                const __grid_constant__ Fast k) {
    gba::cell_backward_any(a, k, blockIdx.x * blockDim.x + threadIdx.x);
}

// the 2D passes: one thread per face (blockIdx.y = component) or cell
template <bool MAC>
__global__ void __launch_bounds__(ADV_THREADS) adv2_face_forward(const __grid_constant__ StepArgs a,
                                                                const __grid_constant__ Fast k) {
    const unsigned f = blockIdx.x * blockDim.x + threadIdx.x;
    if (blockIdx.y == 0) gba::face_forward2_any<0, MAC>(a, k, f);
    else gba::face_forward2_any<1, MAC>(a, k, f);
}

__global__ void __launch_bounds__(ADV_THREADS) adv2_face_backward(const __grid_constant__ StepArgs a,
                                                                 const __grid_constant__ Fast k) {
    const unsigned f = blockIdx.x * blockDim.x + threadIdx.x;
    if (blockIdx.y == 0) gba::face_backward2_any<0>(a, k, f);
    else gba::face_backward2_any<1>(a, k, f);
}

template <bool MAC>
__global__ void __launch_bounds__(ADV_THREADS) adv2_cell_forward(const __grid_constant__ StepArgs a,
                                                                const __grid_constant__ Fast k) {
    gba::cell_forward2_any<MAC>(a, k, blockIdx.x * blockDim.x + threadIdx.x);
}

__global__ void __launch_bounds__(ADV_THREADS) adv2_cell_backward(const __grid_constant__ StepArgs a,
                                                                 const __grid_constant__ Fast k) {
    gba::cell_backward2_any(a, k, blockIdx.x * blockDim.x + threadIdx.x);
}

// The solid constraint in three launches. The faces with lower corner (i, j,
// k) and, at the far walls, the next face, all read the solid at the eight
// nodes of cell (i, j, k): cst_scan looks at those once per cell, sets
// levelset_exist's flag (include/shiokaze/array/array_utility3.h:112-122: any
// negative value) and lists the faces that are not clearly outside the solid;
// cst_solid computes their values from the velocity as it is, a full warp at a
// time however they are scattered; cst_apply writes them and clamps the wall
// faces outside the solid. The velocity is read only where the solid or a wall
// is, and nothing is written before all is read, so no copy of it is kept. One
// thread per face with an FP64 solid branch, reading a saved copy, took 245 us
// on a 150 x 131 x 170 liquid with a solid sphere (0.5 % of the faces), the
// copy included.
struct CstArgs {
    Dims g;
    const float *solid;
    float *vel[3];
    const unsigned char *mask[3];
    unsigned long long *list;  // component << 62 | face
    float *val;
    unsigned *count;  // [0] faces listed, [1] a solid value is negative
    gbp::FastDiv dx, dy, fw[3], fh[3];
};

__device__ __forceinline__ long long cst_face_index(const Dims &g, int d, int i, int j, int k) {
    return gba::at(gba::face_shape(g, d), i, j, k);
}

__global__ void __launch_bounds__(ADV_THREADS) cst_scan(const __grid_constant__ CstArgs a) {
    const unsigned c = blockIdx.x * blockDim.x + threadIdx.x;
    const Dims &g = a.g;
    const gba::Shape ns{g.nx + 1, g.ny + 1, g.nz + 1};
    int side = 1;
    bool neg = false;
    gba::Idx x{0, 0, 0};
    if (c < (unsigned)g.nx * (unsigned)g.ny * (unsigned)g.nz) {
        x = gba::decode_fast(a.dx, a.dy, c);
        side = gba::sign_cell_fast(ns, x.i, x.j, x.k, a.solid);
        neg = side == -1;
        if (side == 2) {
            const float *s = a.solid + gba::at(ns, x.i, x.j, x.k);
            const long long sy = ns.w, sz = (long long)ns.w * ns.h;
#pragma unroll
            for (int n = 0; n < 8; ++n) neg |= s[(n & 1) + ((n & 2) ? sy : 0) + ((n & 4) ? sz : 0)] < 0.0f;
        }
    }
    if (__syncthreads_or(neg) && threadIdx.x == 0) a.count[1] = 1u;
    if (!__any_sync(0xffffffffu, side != 1)) return;
    // this cell's faces: the three at its lower corner, and the far walls'
    const int p[3] = {x.i, x.j, x.k}, n[3] = {g.nx, g.ny, g.nz};
    long long f[6];
    unsigned on = 0;
    if (side != 1) {
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            f[d] = cst_face_index(g, d, x.i, x.j, x.k);
            f[d + 3] = cst_face_index(g, d, x.i + (d == 0), x.j + (d == 1), x.k + (d == 2));
            const unsigned char *m = a.mask[d];
            if (!m || m[f[d]]) on |= 1u << d;
            if (p[d] + 1 == n[d] && (!m || m[f[d + 3]])) on |= 8u << d;
        }
    }
    const unsigned mine = (unsigned)__popc(on);
    unsigned before = mine;
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned t = __shfl_up_sync(0xffffffffu, before, o);
        if (lane >= o) before += t;
    }
    unsigned base = 0;
    if (lane == 31) base = atomicAdd(a.count, before);
    base = __shfl_sync(0xffffffffu, base, 31) + before - mine;
#pragma unroll
    for (int q = 0; q < 6; ++q)
        if (on >> q & 1u) a.list[base++] = (unsigned long long)(q % 3) << 62 | (unsigned long long)f[q];
}

__device__ __forceinline__ gba::Idx cst_decode(const CstArgs &a, unsigned long long e, int &d) {
    d = (int)(e >> 62);
    const unsigned f = (unsigned)e;
    return d == 0 ? gba::decode_fast(a.fw[0], a.fh[0], f)
                  : (d == 1 ? gba::decode_fast(a.fw[1], a.fh[1], f) : gba::decode_fast(a.fw[2], a.fh[2], f));
}

__global__ void __launch_bounds__(ADV_THREADS) cst_solid(const __grid_constant__ CstArgs a) {
    const unsigned n = a.count[0];
    if (!a.count[1]) return;
    const Dims &g = a.g;
    const gba::Shape ns{g.nx + 1, g.ny + 1, g.nz + 1};
    const float *const vel[3] = {a.vel[0], a.vel[1], a.vel[2]};
    for (unsigned q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
        int d;
        const gba::Idx x = cst_decode(a, a.list[q], d);
        const int p2[3] = {2 * x.i + (d != 0), 2 * x.j + (d != 1), 2 * x.k + (d != 2)};
        const int side = gba::sign_corners_fast(ns, p2, a.solid);
        const float in = vel[d][(unsigned)a.list[q]];
        const float val = gba::constrain_solid(g, a.solid, vel, d, x.i, x.j, x.k, in, side);
        a.val[q] = gba::constrain_wall(g, d, d == 0 ? x.i : (d == 1 ? x.j : x.k), val);
    }
}

__global__ void __launch_bounds__(ADV_THREADS) cst_apply(const __grid_constant__ CstArgs a) {
    if (!a.count[1]) return;
    const unsigned n = a.count[0];
    const Dims &g = a.g;
    const gba::Shape ns{g.nx + 1, g.ny + 1, g.nz + 1};
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
    for (unsigned q = t; q < n; q += stride) {
        const unsigned long long e = a.list[q];
        const int d = (int)(e >> 62);
        float *v = d == 0 ? a.vel[0] : (d == 1 ? a.vel[1] : a.vel[2]);
        v[(unsigned)e] = a.val[q];
    }
    // the wall faces that are not listed
    const unsigned area[3] = {(unsigned)g.ny * g.nz, (unsigned)g.nx * g.nz, (unsigned)g.nx * g.ny};
#pragma unroll
    for (int d = 0; d < 3; ++d)
        for (unsigned q = t; q < 2 * area[d]; q += stride) {
            const bool far = q >= area[d];
            const unsigned r = far ? q - area[d] : q;
            const int w = d == 0 ? g.ny : g.nx, hi = (int)(r / (unsigned)w), lo = (int)(r - (unsigned)hi * w);
            const int at = far ? (d == 0 ? g.nx : (d == 1 ? g.ny : g.nz)) : 0;
            const int i = d == 0 ? at : lo, j = d == 1 ? at : (d == 0 ? lo : hi), k = d == 2 ? at : hi;
            const long long f = cst_face_index(g, d, i, j, k);
            if (a.mask[d] && !a.mask[d][f]) continue;
            const float in = a.vel[d][f], val = gba::constrain_wall(g, d, at, in);
            if (val == in || in != in) continue;
            const int p2[3] = {2 * i + (d != 0), 2 * j + (d != 1), 2 * k + (d != 2)};
            if (gba::sign_corners_fast(ns, p2, a.solid) == 1) a.vel[d][f] = val;
        }
}

Dims make_dims(int nx, int ny, int nz, double dx, int trim_narrowband) {
    Dims g{};
    g.nx = nx;
    g.ny = ny;
    g.nz = nz;
    g.dx = dx;
    int e = 0;
    const double m = std::frexp(dx, &e);
    const double inv = 1.0 / dx;
    g.pow2 = (m == 0.5 && std::isfinite(inv) && (double)(float)inv == inv) ? 1 : 0;
    g.inv_dx = inv;
    g.inv_dx_f = (float)inv;
    g.limit = -dx * (double)trim_narrowband;
    return g;
}

unsigned blocks_for(long long n) { return (unsigned)((n + ADV_THREADS - 1) / ADV_THREADS); }

}  // namespace

cudaError_t advect_reserve(AdvectWork &w, long long faces, long long cells) {
    if (faces > w.face_cap) {
        cudaFree(w.v0);
        cudaFree(w.vmm);
        w.v0 = nullptr;
        w.vmm = nullptr;
        w.face_cap = 0;
        cudaError_t e = cudaMalloc(&w.v0, sizeof(float) * (size_t)faces);
        if (e == cudaSuccess) e = cudaMalloc(&w.vmm, sizeof(gba::MinMax) * (size_t)faces);
        if (e != cudaSuccess) return e;
        w.face_cap = faces;
    }
    if (cells > w.cell_cap) {
        cudaFree(w.q0);
        cudaFree(w.qmm);
        w.q0 = nullptr;
        w.qmm = nullptr;
        w.cell_cap = 0;
        cudaError_t e = cudaMalloc(&w.q0, sizeof(float) * (size_t)cells);
        if (e == cudaSuccess) e = cudaMalloc(&w.qmm, sizeof(gba::MinMax) * (size_t)cells);
        if (e != cudaSuccess) return e;
        w.cell_cap = cells;
    }
    return cudaSuccess;
}

void advect_release(AdvectWork &w) {
    cudaFree(w.ext_stamp);
    cudaFree(w.ext_count);
    cudaFree(w.flag);
    cudaFree(w.v0);
    cudaFree(w.vmm);
    cudaFree(w.q0);
    cudaFree(w.qmm);
    w = AdvectWork{};
}

cudaError_t advect_run(AdvectWork &w, const AdvectArgs &a, cudaStream_t st, long long *launches) {
    const long long cells = (long long)a.nx * a.ny * a.nz;
    const long long nf0 = (long long)(a.nx + 1) * a.ny * a.nz, nf1 = (long long)a.nx * (a.ny + 1) * a.nz,
                    nf2 = (long long)a.nx * a.ny * (a.nz + 1);
    long long nfmax = nf0 > nf1 ? nf0 : nf1;
    if (nf2 > nfmax) nfmax = nf2;
    cudaError_t e = advect_reserve(w, a.velocity ? nf0 + nf1 + nf2 : 0, a.q ? cells : 0);
    if (e != cudaSuccess) return e;
    StepArgs s{};
    s.g = make_dims(a.nx, a.ny, a.nz, a.dx, a.trim_narrowband);
    s.dt = a.dt;
    const Fast k = gba::make_fast(s.g, a.dt, true);
    s.u = a.u;
    s.v = a.v;
    s.w = a.w;
    s.fluid = a.fluid;
    s.q = a.q;
    s.mask = a.q_mask;
    s.bg = a.q_bg;
    s.v0 = w.v0;
    s.vmm = w.vmm;
    s.off1 = nf0;
    s.off2 = nf0 + nf1;
    s.q0 = w.q0;
    s.qmm = w.qmm;
    if (a.q) {
        if (a.maccormack) {
            adv_cell_forward<true><<<blocks_for(cells), ADV_THREADS, 0, st>>>(s, k);
            adv_cell_backward<<<blocks_for(cells), ADV_THREADS, 0, st>>>(s, k);
            *launches += 2;
        } else {
            adv_cell_forward<false><<<blocks_for(cells), ADV_THREADS, 0, st>>>(s, k);
            *launches += 1;
            e = cudaMemcpyAsync(a.q, w.q0, sizeof(float) * (size_t)cells, cudaMemcpyDeviceToDevice, st);
            if (e != cudaSuccess) return e;
        }
    }
    if (!a.velocity) return cudaGetLastError();
    const dim3 fgrid(blocks_for(nfmax), 3);
    if (a.maccormack) {
        adv_face_forward<true><<<fgrid, ADV_THREADS, 0, st>>>(s, k);
        adv_face_backward<<<fgrid, ADV_THREADS, 0, st>>>(s, k);
        *launches += 2;
    } else {
        adv_face_forward<false><<<fgrid, ADV_THREADS, 0, st>>>(s, k);
        *launches += 1;
        float *dst[3] = {a.u, a.v, a.w};
        const long long n[3] = {nf0, nf1, nf2}, o[3] = {0, s.off1, s.off2};
        for (int d = 0; d < 3; ++d) {
            e = cudaMemcpyAsync(dst[d], w.v0 + o[d], sizeof(float) * (size_t)n[d], cudaMemcpyDeviceToDevice, st);
            if (e != cudaSuccess) return e;
        }
    }
    return cudaGetLastError();
}

cudaError_t advect_run2(AdvectWork &w, const AdvectArgs &a, cudaStream_t st, long long *launches) {
    const long long cells = (long long)a.nx * a.ny;
    const long long nf0 = (long long)(a.nx + 1) * a.ny, nf1 = (long long)a.nx * (a.ny + 1);
    const long long nfmax = nf0 > nf1 ? nf0 : nf1;
    cudaError_t e = advect_reserve(w, a.velocity ? nf0 + nf1 : 0, a.q ? cells : 0);
    if (e != cudaSuccess) return e;
    StepArgs s{};
    s.g = make_dims(a.nx, a.ny, 1, a.dx, a.trim_narrowband);
    s.dt = a.dt;
    const Fast k = gba::make_fast(s.g, a.dt, false);
    s.u = a.u;
    s.v = a.v;
    s.w = nullptr;
    s.fluid = a.fluid;
    s.q = a.q;
    s.mask = a.q_mask;
    s.bg = a.q_bg;
    s.v0 = w.v0;
    s.vmm = w.vmm;
    s.off1 = nf0;
    s.off2 = 0;
    s.q0 = w.q0;
    s.qmm = w.qmm;
    if (a.q) {
        if (a.maccormack) {
            adv2_cell_forward<true><<<blocks_for(cells), ADV_THREADS, 0, st>>>(s, k);
            adv2_cell_backward<<<blocks_for(cells), ADV_THREADS, 0, st>>>(s, k);
            *launches += 2;
        } else {
            adv2_cell_forward<false><<<blocks_for(cells), ADV_THREADS, 0, st>>>(s, k);
            *launches += 1;
            e = cudaMemcpyAsync(a.q, w.q0, sizeof(float) * (size_t)cells, cudaMemcpyDeviceToDevice, st);
            if (e != cudaSuccess) return e;
        }
    }
    if (!a.velocity) return cudaGetLastError();
    const dim3 fgrid(blocks_for(nfmax), 2);
    if (a.maccormack) {
        adv2_face_forward<true><<<fgrid, ADV_THREADS, 0, st>>>(s, k);
        adv2_face_backward<<<fgrid, ADV_THREADS, 0, st>>>(s, k);
        *launches += 2;
    } else {
        adv2_face_forward<false><<<fgrid, ADV_THREADS, 0, st>>>(s, k);
        *launches += 1;
        e = cudaMemcpyAsync(a.u, w.v0, sizeof(float) * (size_t)nf0, cudaMemcpyDeviceToDevice, st);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(a.v, w.v0 + nf0, sizeof(float) * (size_t)nf1, cudaMemcpyDeviceToDevice, st);
        if (e != cudaSuccess) return e;
    }
    return cudaGetLastError();
}

// The extrapolation's rounds run in place on the values, with a stamp byte per
// cell: 0 inactive, 1 active at the start, g for a cell activated in round
// g - 2. A cell counts as active in round g - 2 if its stamp is below g (and
// not 0), so a round neither reads what it writes nor needs a second copy of
// values and mask, and reads values only beside newly activated cells: one
// byte a cell and round instead of the ten that two dense buffers cost. The
// stamps are padded by a plane on both sides (zeros), so that a thread reads
// its four cells' neighbours as words without a test. Three rounds on each
// component of a 150 x 131 x 170 liquid and the constraint after them: 696 us
// with dense buffers (21 us a round) and the constraint's first form, 321 us
// with these, most of it the calls' own launches and waits.
__global__ void __launch_bounds__(256) ext_stamp(long long n, long long pad, const unsigned char *__restrict__ m,
                                                 unsigned char *stamp, unsigned long long *added) {
    if (blockIdx.x == 0 && threadIdx.x == 0 && added) *added = 0ull;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; 4 * t < n + 2 * pad;
         t += (long long)gridDim.x * blockDim.x) {
        unsigned w = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const long long c = 4 * t + q - pad;
            if (c >= 0 && c < n && m[c]) w |= 1u << (8 * q);
        }
        reinterpret_cast<unsigned *>(stamp)[t] = w;
    }
}

// four bytes at any byte offset from two aligned words
__device__ __forceinline__ unsigned bytes_at(const unsigned char *p) {
    const unsigned long long a = (unsigned long long)p;
    const unsigned *w = reinterpret_cast<const unsigned *>(a & ~3ull);
    const unsigned sh = (unsigned)(a & 3ull) * 8u;
    return sh ? __funnelshift_r(w[0], w[1], sh) : w[0];
}

// One round: stamp points at cell 0 (pad bytes in), g is the stamp of this
// round's cells. `last` also marks every activated cell in the caller's mask.
__global__ void __launch_bounds__(256) ext_round(int W, int H, int D, gbp::FastDiv dw, gbp::FastDiv dh, float *a,
                                                 unsigned char *stamp, unsigned g, unsigned char *m, int last,
                                                 unsigned long long *added) {
    const long long sy = W, sz = (long long)W * H, n = sz * D, words = (n + 3) / 4;
    const unsigned g4 = g * 0x01010101u;
    auto active = [&](unsigned w) { return __vcmpltu4(w, g4) & __vcmpne4(w, 0u); };
    unsigned fresh = 0;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < words;
         t += (long long)gridDim.x * blockDim.x) {
        unsigned char *s = stamp + 4 * t;
        const unsigned own = *reinterpret_cast<const unsigned *>(s);
        unsigned born = 0;  // cells activated now
        if (__vcmpeq4(own, 0u)) {
            const unsigned nb[6] = {active(bytes_at(s + 1)),      active(bytes_at(s - 1)),
                                    active(bytes_at(s + sy)),     active(bytes_at(s - sy)),
                                    active(bytes_at(s - sz)),     active(bytes_at(s + sz))};
            if ((nb[0] | nb[1] | nb[2] | nb[3] | nb[4] | nb[5]) & __vcmpeq4(own, 0u)) {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const long long c = 4 * t + q;
                    if (c >= n || (own >> (8 * q) & 0xffu)) continue;
                    const bool small = n < (1LL << 32);
                    const unsigned r = small ? gbp::fdiv((unsigned)c, dw) : (unsigned)(c / W);
                    const int k = (int)gbp::fdiv(r, dh), j = (int)(r - (unsigned)k * (unsigned)H),
                              i = (int)(c - (long long)r * W);
                    float sum = 0.0f;
                    int weight = 0;
                    auto see = [&](bool in, unsigned on, long long step) {
                        if (in && (on >> (8 * q) & 1u)) {
                            sum += a[c + step];
                            ++weight;
                        }
                    };
                    see(i + 1 < W, nb[0], 1);
                    see(i > 0, nb[1], -1);
                    see(j + 1 < H, nb[2], sy);
                    see(j > 0, nb[3], -sy);
                    see(k > 0, nb[4], -sz);
                    see(k + 1 < D, nb[5], sz);
                    if (weight) {
                        a[c] = sum / (float)weight;
                        s[q] = (unsigned char)g;
                        born |= 1u << (8 * q);
                        ++fresh;
                    }
                }
            }
        }
        if (last && (born || __vcmpgtu4(own, 0x01010101u))) {
            const unsigned grown = __vcmpgtu4(own, 0x01010101u) | born;
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (4 * t + q < n && (grown >> (8 * q) & 1u)) m[4 * t + q] = 1;
        }
    }
    fresh = __reduce_add_sync(0xffffffffu, fresh);
    if ((threadIdx.x & 31) == 0 && fresh) atomicAdd(added, (unsigned long long)fresh);
}

cudaError_t extrapolate_run(AdvectWork &w, int W, int H, int D, float *a, unsigned char *m, int count,
                            cudaStream_t st, long long *launches, unsigned long long *activated_host) {
    const long long n = (long long)W * H * D;
    const long long pad = ((long long)W * H + 16 + 15) / 16 * 16, need = (n + 2 * pad + 15) / 16 * 16;
    cudaError_t e = cudaSuccess;
    if (need > w.ext_cap) {
        cudaFree(w.ext_stamp);
        w.ext_stamp = nullptr;
        w.ext_cap = 0;
        if ((e = cudaMalloc(&w.ext_stamp, (size_t)need)) != cudaSuccess) return e;
        w.ext_cap = need;
    }
    if (!w.ext_count && (e = cudaMalloc(&w.ext_count, sizeof(unsigned long long))) != cudaSuccess) return e;
    const FastDiv dw = make_fastdiv((unsigned)W), dh = make_fastdiv((unsigned)H);
    const int blocks = (int)std::min<long long>((n / 4 + 256) / 256, 152LL * 8);
    // stamps are bytes: rounds go in runs of at most 250, each from fresh stamps
    for (int done = 0; done < count || done == 0;) {
        const int run = std::min(count - done, 250);
        ext_stamp<<<(int)std::min<long long>((need / 4 + 255) / 256, 152LL * 8), 256, 0, st>>>(
            n, pad, m, w.ext_stamp, done == 0 ? w.ext_count : nullptr);
        *launches += 1;
        for (int r = 0; r < run; ++r)
            ext_round<<<blocks, 256, 0, st>>>(W, H, D, dw, dh, a, w.ext_stamp + pad, (unsigned)(r + 2), m,
                                              r + 1 == run ? 1 : 0, w.ext_count);
        *launches += run;
        done += run;
        if (run == 0) break;
    }
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if (activated_host)
        e = cudaMemcpyAsync(activated_host, w.ext_count, sizeof(unsigned long long), cudaMemcpyDeviceToHost, st);
    return e;
}

cudaError_t constrain_run(AdvectWork &w, const ConstrainArgs &a, cudaStream_t st, long long *launches) {
    const long long nf0 = (long long)(a.nx + 1) * a.ny * a.nz, nf1 = (long long)a.nx * (a.ny + 1) * a.nz,
                    nf2 = (long long)a.nx * a.ny * (a.nz + 1);
    long long nfmax = nf0 > nf1 ? nf0 : nf1;
    if (nf2 > nfmax) nfmax = nf2;
    cudaError_t e = advect_reserve(w, nf0 + nf1 + nf2, 0);
    if (e == cudaSuccess && !w.flag) e = cudaMalloc(&w.flag, 2 * sizeof(unsigned));
    if (e != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(w.flag, 0, 2 * sizeof(unsigned), st)) != cudaSuccess) return e;
    CstArgs c{};
    c.g = make_dims(a.nx, a.ny, a.nz, a.dx, 0);
    c.solid = a.solid;
    float *vel[3] = {a.u, a.v, a.w};
    const unsigned char *mask[3] = {a.mu, a.mv, a.mw};
    c.dx = make_fastdiv((unsigned)a.nx);
    c.dy = make_fastdiv((unsigned)a.ny);
    for (int d = 0; d < 3; ++d) {
        c.vel[d] = vel[d];
        c.mask[d] = mask[d];
        c.fw[d] = make_fastdiv((unsigned)(a.nx + (d == 0)));
        c.fh[d] = make_fastdiv((unsigned)(a.ny + (d == 1)));
    }
    c.list = reinterpret_cast<unsigned long long *>(w.vmm);  // 8 bytes a face, as the list needs
    c.val = w.v0;
    c.count = w.flag;
    cst_scan<<<blocks_for((long long)a.nx * a.ny * a.nz), ADV_THREADS, 0, st>>>(c);
    const unsigned nb = (unsigned)std::min<long long>(blocks_for(nfmax), 152LL * 4);
    cst_solid<<<nb, ADV_THREADS, 0, st>>>(c);
    cst_apply<<<nb, ADV_THREADS, 0, st>>>(c);
    *launches += 3;
    return cudaGetLastError();
}

}  // namespace gbp
