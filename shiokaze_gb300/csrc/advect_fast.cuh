// advect_fast.cuh -- the advection passes of advect_core.cuh in float pairs.
//
// The reference traces, weighs and accumulates in double precision, and
// every result must equal its bits. GB300 issues one FP64 warp instruction
// per 16 cycles and SM but four FP32 ones per cycle, so the FP64 form of
// advect_core.cuh keeps the FP64 pipe 86 % busy and DRAM 1 %. Here each
// rounded FP32 result of the reference's double expression is found from an
// unevaluated sum of two floats (about 2^-45 relative) and a bound E on its
// distance to the double value: if value - E and value + E round to the same
// float, that float is the reference's result (rounding is monotonic; Ziv,
// "Fast evaluation of elementary mathematical functions with correctly
// rounded last bit", 1991). An element with any undecided rounding, floor or
// comparison, or an operand outside the ranges the bounds assume (non-finite
// values, magnitudes near the float range's ends), is computed again by the
// FP64 form, out of line: the results are the same bits for every input, and
// about one element in 2^14 takes that way on a moving velocity field.
//
// Pair arithmetic is TwoSum (Knuth) and the FMA product split (Ogita, Rump
// and Oishi 2005). Compiled with --fmad=false: only the fmaf calls fuse.
//
// Measured on one GB300, MacCormack, density and velocity: 256^3 smoke 40.75 ms
// with the FP64 form alone, 3.51 ms here; 1000 x 777 2D 1.09 ms and 0.19 ms.
#pragma once

#include <cmath>
#include <cstring>

#include "advect_core.cuh"
#include "gbp_convert.cuh"
#include "gbp_internal.cuh"

namespace gba {

struct FF {
    float h, l;  // the value h + l
};

// Constants of the float-pair passes of one call (make_fast).
struct Fast {
    int on;            // the bounds below hold for this grid and step; 0: FP64 form throughout
    float dth, dtl;    // dt = dth + dtl within 2^-48
    float dt_e;        // relative half-width of the rounding test of u*dt (0: dt is a float, the product split is exact)
    float ih, il, i_e; // 1/dx alike (a power of two: ih exact, no test)
    // dx = 1/n rounded, n a float (the usual grid): quotients t/dx often lie on
    // or beside the tie of two floats, see trace_ff
    int unit;
    float m0, i_s;
    float ch, cl;      // dt/dx within 2^-46
    double cd;         // dt/dx for a power-of-two dx: u*cd rounds as (u*dt)*(1/dx)
    double dt, dx, inv;  // inv: 1/dx correctly rounded
    int pow2;
    float lim_lo, lim_hi;  // floats just below and above Dims::limit
    gbp::FastDiv fw[3], fh[3], cw, chh;  // face (per component) and cell widths and heights
};

inline void split_pair(double x, float &h, float &l) {
    h = (float)x;
    l = (float)(x - (double)h);
}

// The float-pair constants; `on` only where every bound's assumption holds:
// edges up to 8192 (a position's double spacing is at most 2^-40), element
// numbers within 31 bits, and dt, dx, dt/dx far from the float range's ends.
inline Fast make_fast(const Dims &g, double dt, bool three) {
    Fast f{};
    const int n[3] = {g.nx, g.ny, three ? g.nz : 1};
    const double r = dt / g.dx, a = std::fabs(r), b = std::fabs(dt);
    const long long most = (long long)(n[0] + 1) * (n[1] + 1) * (n[2] + 1);
    f.on = n[0] < 8192 && n[1] < 8192 && n[2] < 8192 && most < (1LL << 31) && a > 0x1p-30 && a < 0x1p30 &&
           b > 0x1p-30 && b < 0x1p30 && g.dx > 0x1p-30 && g.dx < 0x1p30 && std::isfinite(g.limit) &&
           std::fabs(g.limit) < 0x1p30;
    split_pair(dt, f.dth, f.dtl);
    f.dt_e = f.dtl == 0.0f ? 0.0f : 0x1p-44f;
    f.pow2 = g.pow2;
    f.inv = 1.0 / g.dx;
    split_pair(f.inv, f.ih, f.il);
    f.i_e = g.pow2 ? 0.0f : 0x1p-44f;
    const double whole = std::rint(f.inv);
    if (!g.pow2 && whole >= 2.0 && whole <= 16384.0 && 1.0 / whole == g.dx) {
        const double delta = std::fma(g.dx, whole, -1.0);  // dx = (1 + delta)/n
        f.unit = 1;
        f.ih = (float)whole;
        f.m0 = delta == 0.0 ? 4.0f : (float)std::fmin(4.0, 0x1p-53 / std::fabs(delta));
        f.i_s = delta > 0.0 ? -0x1p-44f : 0x1p-44f;
    }
    split_pair(r, f.ch, f.cl);
    f.cd = dt * g.inv_dx;
    f.dt = dt;
    f.dx = g.dx;
    const float lim = (float)g.limit;
    f.lim_lo = std::nextafterf(lim, -INFINITY);
    f.lim_hi = std::nextafterf(lim, INFINITY);
    for (int d = 0; d < 3; ++d) {
        f.fw[d] = gbp::make_fastdiv((unsigned)(g.nx + (d == 0)));
        f.fh[d] = gbp::make_fastdiv((unsigned)(g.ny + (d == 1)));
    }
    f.cw = gbp::make_fastdiv((unsigned)g.nx);
    f.chh = gbp::make_fastdiv((unsigned)g.ny);
    return f;
}

GBA_HD unsigned fbits(float f) {
#ifdef __CUDA_ARCH__
    return __float_as_uint(f);
#else
    unsigned u;
    std::memcpy(&u, &f, sizeof u);
    return u;
#endif
}

GBA_HD FF two_sum(float a, float b) {
    const float s = a + b, t = s - a;
    return FF{s, (a - (s - t)) + (b - t)};
}

GBA_HD FF ff_mul(FF a, FF b) {
    const float h = a.h * b.h;
    float l = fmaf(a.h, b.h, -h);
    l = fmaf(a.h, b.l, l);
    l = fmaf(a.l, b.h, l);
    return FF{h, l};
}

// (float)(sum of four floats, added in double, / 4). The pair sum is exact
// when every nonzero operand is at least 2^-20 of the largest (by bit
// patterns): all partial sums are then multiples of 2^-45 of it (the double
// sums are exact too) and the residuals, at most 2^-21 of it, add without
// rounding. Quotients by 4
// are exact above 2^-100. Otherwise (NaN included) ok turns false.
GBA_HD float mean4(float a, float b, float c, float d, bool &ok) {
    const FF p = two_sum(a, b), q = two_sum(c, d), s = two_sum(p.h, q.h);
    const unsigned ua = fbits(a) & 0x7fffffffu, ub = fbits(b) & 0x7fffffffu, uc = fbits(c) & 0x7fffffffu,
                   ud = fbits(d) & 0x7fffffffu;
    const unsigned m0 = ua > ub ? ua : ub, m1 = uc > ud ? uc : ud, mx = m0 > m1 ? m0 : m1;
    // a zero wraps to the largest number and never is the smallest
    const unsigned n0 = ua - 1 < ub - 1 ? ua - 1 : ub - 1, n1 = uc - 1 < ud - 1 ? uc - 1 : ud - 1,
                   mn = n0 < n1 ? n0 : n1;
    // mn is 0xffffffff for four zeros; else mn + 1 within 20 binades of mx, both in [2^-100, 2^100]
    ok = ok && (mx == 0u || (mn >= (27u << 23) && mx < (227u << 23) && mx - mn <= (20u << 23)));
    return (s.h + ((p.l + q.l) + s.l)) * 0.25f;
}

// (float)((float)((double)u * dt) / dx), the face trace's displacement.
//
// For dx = (1 + delta)/n with a whole n up to 2^14, t/dx is t*n (at most 38
// bits, a double) times 1 - delta, |delta| <= 2^-53: the double quotient is
// t*n where |delta| m <= 2^-53, m in [1, 2) the significand of t*n, else its
// neighbour against delta's sign. Only when t*n is the tie of two floats do
// the two round apart, so a shift of 2^-44 in that direction gives the
// quotient's rounding: t*n's distance from any other tie is 2^-38 at least.
GBA_HD float trace_ff(const Fast &k, float u, bool &ok) {
    float h = u * k.dth;
    float l = fmaf(u, k.dtl, fmaf(u, k.dth, -h));
    float e = fabsf(h) * k.dt_e;
    const float t = h + (l + e);
    ok = ok && t == h + (l - e) && (u == 0.0f || fabsf(h) >= 0x1p-100f);
    if (k.pow2) return t * k.ih;
    h = t * k.ih;
    if (k.unit) {
        l = fmaf(t, k.ih, -h);
        if (l == 0.0f) return h;
        const float m = gbp::d2f_from_bits((fbits(h) & 0x7fffffu) | 0x3f800000u);
        // h's significand stands for t*n's except beside m0 and the binade's ends
        ok = ok && fabsf(m - k.m0) > 0x1p-20f && m > 1.0f + 0x1p-20f && m < 2.0f - 0x1p-20f;
        return h + (m > k.m0 ? fmaf(h, k.i_s, l) : l);
    }
    l = fmaf(t, k.il, fmaf(t, k.ih, -h));
    e = fabsf(h) * k.i_e;
    const float q = h + (l + e);
    ok = ok && q == h + (l - e);
    return q;
}

// One axis of an interpolation: the corner cell and the two weights
struct Axis {
    int i;
    FF w0, w1;
};

// the axis at position c - f, |f| a little over 0.5 at most, clamped to
// [0, w - 1] as Corner is; f nonzero below 2^-40 is left to the FP64 form
// (products of three weights then stay normal floats)
GBA_HD Axis axis_at(int c, FF f, int w, bool &ok) {
    const bool below = f.h > 0.0f;
    const FF g{fabsf(f.h), below ? f.l : -f.l};
    FF r;
    r.h = 1.0f - g.h;
    r.l = ((1.0f - r.h) - g.h) - g.l;
    Axis a;
    a.i = below ? c - 1 : c;
    a.w0 = below ? g : r;
    a.w1 = below ? r : g;
    const bool lo = a.i < 0, hi = a.i > w - 2;
    ok = ok && (lo || hi || g.h == 0.0f || g.h >= 0x1p-40f);
    if (lo || hi) {
        a.i = lo ? 0 : w - 2;
        a.w0 = FF{lo ? 1.0f : 0.0f, 0.0f};
        a.w1 = FF{lo ? 0.0f : 1.0f, 0.0f};
    }
    return a;
}

// (double)ip - (double)t for a displacement below 2^-17: the double position
// may round t to a multiple of its own spacing; the rounded t, exact in float
GBA_HD_OUTLINE float tiny_displacement(int ip, float t) {
    const double p = (double)ip - (double)t;
    return (float)((double)ip - p);
}

GBA_HD float clamp_shift(float t) { return fminf(fmaxf(t, -1e6f), 1e6f); }

// the axis of the face trace ip - t (t a float; the difference in double is
// exact for |t| >= 2^-17, whose lowest bit is at least 2^-40)
GBA_HD Axis face_axis(int ip, float t, int w, bool &ok) {
    ok = ok && fabsf(t) < 1e6f;
    if (fabsf(t) < 0x1p-17f && t != 0.0f) t = tiny_displacement(ip, t);
    t = clamp_shift(t);
    const float r = rintf(t);
    return axis_at(ip - (int)r, FF{t - r, 0.0f}, w, ok);
}

// x / dx correctly rounded, inv = 1/dx correctly rounded: two corrections of
// x*inv by its FMA remainder (Markstein, "Computation of elementary
// functions on the IBM RISC System/6000 processor", 1990; Brisebarre, Muller
// and Raina, "Accelerating correctly rounded floating-point division when
// the divisor is known in advance", 2004). x is 0 or within [2^-180, 2^160].
GBA_HD double div_known(double x, double dx, double inv) {
    double q = x * inv;
    q = fma(fma(-q, dx, x), inv, q);
    return fma(fma(-q, dx, x), inv, q);
}

// a double of magnitude at most 1 as a pair: its top 24 bits and the
// following 29, rounded (2^-48 relative); magnitudes below 2^-100 give +-2^-100
GBA_HD FF pair_of(double f) {
    const unsigned long long b = gbp::d2f_bits_of(f);
    const unsigned hi = (unsigned)(b >> 32), lo = (unsigned)b, e = (hi >> 20) & 0x7ffu, sign = hi & 0x80000000u;
    if ((b << 1) == 0) return FF{0.0f, 0.0f};
    if (e < 1023 - 100) return FF{gbp::d2f_from_bits(sign | (27u << 23)), 0.0f};
    const unsigned m = ((hi & 0x7fffffffu) << 3 | lo >> 29) - (896u << 23);
    const float unit = gbp::d2f_from_bits(sign | ((e - 896u - 52u) << 23));
    return FF{gbp::d2f_from_bits(sign | m), (float)(int)(lo & 0x1fffffffu) * unit};
}

// the axis of the cell trace ip -+ u*dt/dx in double (BACK: +): the product
// (and quotient) and the difference in FP64 as the reference has them, the
// rest in integers and floats
template <bool BACK> GBA_HD Axis cell_axis(const Fast &k, int ip, float u, int w, bool &ok) {
    const float t = clamp_shift(u * k.ch);
    ok = ok && fabsf(u * k.ch) < 1e6f && (u == 0.0f || fabsf(u) > 0x1p-120f);
    const int c = BACK ? ip + (int)rintf(t) : ip - (int)rintf(t);
    const double ud = gbp::f2d_exact(u);
    const double disp = k.pow2 ? ud * k.cd : div_known(ud * k.dt, k.dx, k.inv);
    const double base = gbp::f2d_exact((float)ip);
    const double p = BACK ? base + disp : base - disp;
    return axis_at(c, pair_of(gbp::f2d_exact((float)c) - p), w, ok);
}

// One accumulation of interp: value = (float)((double)value + (double)v*c).
// E covers the weights' error (2^-44 relative), the pair arithmetic's and
// the double expression's own roundings.
GBA_HD void accumulate(float &value, float v, FF c, bool &same) {
    const float ph = v * c.h;
    const float pl = fmaf(v, c.l, fmaf(v, c.h, -ph));
    const FF s = two_sum(value, ph);
    const float t = s.l + pl;
    const float e = fmaf(fabsf(ph), 0x1p-42f, fabsf(s.h) * 0x1p-45f);
    value = s.h + (t + e);
    same = same && value == s.h + (t - e);
}

// What the bounds of accumulate assume of the whole sum: corners below 2^40
// (weights are accurate to 2^-149 absolutely at worst), and a result of at
// least 2^-60, or exactly 0 with every product exactly 0.
template <int N> GBA_HD bool sum_ok(float value, const float (&v)[N], const FF (&c)[N]) {
    float m = 0.0f;
#pragma unroll
    for (int n = 0; n < N; ++n) m = fmaxf(m, fabsf(v[n]));
    if (!(m < 0x1p40f)) return false;
    if (fabsf(value) >= 0x1p-60f) return true;
    bool zero = true;
#pragma unroll
    for (int n = 0; n < N; ++n) zero = zero && (v[n] == 0.0f || c[n].h == 0.0f);
    return zero;
}

// interp from the axes and the eight corners' values
GBA_HD float interp_ff(const Axis &x, const Axis &y, const Axis &z, const float (&v)[8], bool &ok) {
    const FF zx[4] = {ff_mul(z.w0, x.w0), ff_mul(z.w0, x.w1), ff_mul(z.w1, x.w0), ff_mul(z.w1, x.w1)};
    const FF c[8] = {ff_mul(zx[0], y.w0), ff_mul(zx[1], y.w0), ff_mul(zx[0], y.w1), ff_mul(zx[1], y.w1),
                     ff_mul(zx[2], y.w0), ff_mul(zx[3], y.w0), ff_mul(zx[2], y.w1), ff_mul(zx[3], y.w1)};
    float value = 0.0f;
#pragma unroll
    for (int n = 0; n < 8; ++n) accumulate(value, v[n], c[n], ok);
    ok = ok && sum_ok(value, v, c);
    return value;
}

GBA_HD float interp2_ff(const Axis &x, const Axis &y, const float (&v)[4], bool &ok) {
    const FF c[4] = {ff_mul(x.w0, y.w0), ff_mul(x.w1, y.w0), ff_mul(x.w0, y.w1), ff_mul(x.w1, y.w1)};
    float value = 0.0f;
#pragma unroll
    for (int n = 0; n < 4; ++n) accumulate(value, v[n], c[n], ok);
    ok = ok && sum_ok(value, v, c);
    return value;
}

// The corner cell alone and the upper weight to float accuracy, for the
// limiter's corners and the narrow-band test: the trace there subtracts the
// double displacement u*dt/dx, of which the pair D (2^-46 relative) decides
// the floor unless it falls within theta of an integer.
struct Cellf {
    int i;
    float x1;
};

struct Shift {
    float r, f, theta;  // D = r + f, |f| <= 0.5
    bool still;         // D = 0 exactly
};

GBA_HD Shift shift_of(const Fast &k, float u, bool &ok) {
    Shift s;
    const float h = u * k.ch, l = fmaf(u, k.cl, fmaf(u, k.ch, -h));
    ok = ok && fabsf(h) < 1e6f;
    s.r = rintf(clamp_shift(h));
    s.f = (clamp_shift(h) - s.r) + l;
    s.theta = fmaf(fabsf(h), 0x1p-43f, 0x1p-38f);
    s.still = u == 0.0f;
    return s;
}

GBA_HD Cellf clamp_cell(int i, float x1, int w) {
    if (i < 0) return Cellf{0, 0.0f};
    if (i > w - 2) return Cellf{w - 2, 1.0f};
    return Cellf{i, x1};
}

// floor(ip - D)
GBA_HD Cellf cell_of(int ip, const Shift &s, int w, bool &ok) {
    ok = ok && (s.still || fabsf(s.f) >= s.theta);
    const bool below = s.f > 0.0f;
    const int c = ip - (int)s.r;
    return clamp_cell(below ? c - 1 : c, below ? 1.0f - s.f : -s.f, w);
}

// floor(ip - D - 0.5)
GBA_HD Cellf half_cell_of(int ip, const Shift &s, int w, bool &ok) {
    ok = ok && fabsf(s.f) <= 0.5f - s.theta;
    return clamp_cell(ip - (int)s.r - 1, 0.5f - s.f, w);
}

// The narrow-band test above_limit on N corner values: 1 above, 0 not, 2
// undecided. First the corners' range, as compare_interp has it with a wider
// margin, then the interpolant in float (within 2^-19 of the largest corner:
// weights within 2^-23, N roundings) compared outside 2^-18 of it.
template <int N, class W> GBA_HD int above_ff(const Fast &k, const float (&v)[N], W weight) {
    float mn = v[0], mx = v[0], sum = v[0];
#pragma unroll
    for (int n = 1; n < N; ++n) {
        mn = v[n] < mn ? v[n] : mn;
        mx = mx < v[n] ? v[n] : mx;
        sum += v[n];
    }
    if (!(sum - sum == 0.0f)) return 2;
    const float am = (-mn < mx) ? mx : -mn;
    float d = fmaf(am, 0x1p-18f, 1e-30f);
    if (mx + d < k.lim_lo) return 0;
    if (mn - d > k.lim_hi) return 1;
    float x = 0.0f;
#pragma unroll
    for (int n = 0; n < N; ++n) x = fmaf(weight(n), v[n], x);
    if (x + d < k.lim_lo) return 0;
    if (x - d > k.lim_hi) return 1;
    return 2;
}

// The MacCormack value in float: the double sum of a float and half a float
// rounded to float is their float sum (53 >= 2*24 + 2 bits, the double
// rounding is harmless), the clamp is monotonic. Half the difference has to
// be exact.
GBA_HD float maccormack_ff(const MinMax &m, float in, float fwd, float bwd, bool &ok) {
    if (mm_within(m)) return fwd;
    const float diff = in - bwd, half = 0.5f * diff;
    ok = ok && half + half == diff;
    const float s = fwd + half;
    if (s < m.lo) return m.lo;
    if (s > m.hi) return m.hi;
    return s;
}

GBA_HD Idx decode_fast(const gbp::FastDiv &w, const gbp::FastDiv &h, unsigned f) {
    const unsigned t = gbp::fdiv(f, w), k = gbp::fdiv(t, h);
    return Idx{(int)(f - t * w.d), (int)(t - k * h.d), (int)k};
}

// the FP64 forms of a pass, out of line
template <bool MAC> GBA_HD_OUTLINE void face_forward_fp64(const StepArgs &a, int dim, unsigned f) {
    face_forward<MAC>(a, dim, f);
}
GBA_HD_OUTLINE void face_backward_fp64(const StepArgs &a, int dim, unsigned f) { face_backward(a, dim, f); }
template <bool MAC> GBA_HD_OUTLINE void cell_forward_fp64(const StepArgs &a, unsigned c) { cell_forward<MAC>(a, c); }
GBA_HD_OUTLINE void cell_backward_fp64(const StepArgs &a, unsigned c) { cell_backward(a, c); }
template <bool MAC> GBA_HD_OUTLINE void face_forward2_fp64(const StepArgs &a, int dim, unsigned f) {
    face_forward2<MAC>(a, dim, f);
}
GBA_HD_OUTLINE void face_backward2_fp64(const StepArgs &a, int dim, unsigned f) { face_backward2(a, dim, f); }
template <bool MAC> GBA_HD_OUTLINE void cell_forward2_fp64(const StepArgs &a, unsigned c) { cell_forward2<MAC>(a, c); }
GBA_HD_OUTLINE void cell_backward2_fp64(const StepArgs &a, unsigned c) { cell_backward2(a, c); }

// face_full with the means in float pairs; uf[DIM] is the face's own value
template <int DIM>
GBA_HD void face_full_ff(const Dims &g, const float *const comp[3], int i, int j, int k, unsigned f, float (&uf)[3],
                         bool &ok) {
    const int n[3] = {g.nx, g.ny, g.nz};
    const int ip[3] = {i, j, k};
    // the two cells around the face along DIM, clamped
    const int lo = ip[DIM] > 0 ? ip[DIM] - 1 : 0, hi = ip[DIM] < n[DIM] ? ip[DIM] : n[DIM] - 1;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        if (c == DIM) {
            uf[c] = comp[c][f];
            continue;
        }
        const int w = g.nx + (c == 0), h = g.ny + (c == 1);
        const int step[3] = {1, w, w * h};
        int q[3] = {i, j, k};
        q[DIM] = lo;
        const float *p = comp[c] + (q[0] + w * (q[1] + h * q[2]));
        const int up = (hi - lo) * step[DIM];
        uf[c] = mean4(p[0], p[step[c]], p[up], p[up + step[c]], ok);
    }
}

template <int DIM, bool MAC> GBA_HD bool face_forward_try(const StepArgs &a, const Fast &k, unsigned f) {
    const Dims &g = a.g;
    const Idx x = decode_fast(k.fw[DIM], k.fh[DIM], f);
    const int ip[3] = {x.i, x.j, x.k};
    const int nc[3] = {g.nx, g.ny, g.nz};
    const float *const comp[3] = {a.u, a.v, a.w};
    const float *src = comp[DIM];
    const long long o = DIM == 0 ? 0 : (DIM == 1 ? a.off1 : a.off2);
    bool ok = true;
    float uf[3];
    face_full_ff<DIM>(g, comp, x.i, x.j, x.k, f, uf, ok);
    const float own = uf[DIM];
    const bool moving = uf[0] != 0.0f || uf[1] != 0.0f || uf[2] != 0.0f;
    const int w = g.nx + (DIM == 0), wh = w * (g.ny + (DIM == 1));
    Axis ax[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) ax[c] = face_axis(ip[c], trace_ff(k, uf[c], ok), nc[c] + (c == DIM), ok);
    const int base = ax[0].i + w * ax[1].i + wh * ax[2].i;
    float v[8];
#pragma unroll
    for (int n = 0; n < 8; ++n) v[n] = src[base + (n & 1) + ((n & 2) ? w : 0) + ((n & 4) ? wh : 0)];
    float out = interp_ff(ax[0], ax[1], ax[2], v, ok);
    if (!moving) out = own;
    MinMax m;
    if (MAC) {
        // the limiter's corners: the double displacement's cell
        Cellf q[3];
        Cellf band[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const Shift s = shift_of(k, uf[c], ok);
            q[c] = cell_of(ip[c], s, nc[c] + (c == DIM), ok);
            band[c] = c == DIM ? half_cell_of(ip[c], s, nc[c], ok) : q[c];
        }
        const int base2 = q[0].i + w * q[1].i + wh * q[2].i;
        if (base2 != base) {
#pragma unroll
            for (int n = 0; n < 8; ++n) v[n] = src[base2 + (n & 1) + ((n & 2) ? w : 0) + ((n & 4) ? wh : 0)];
        }
        m.lo = INFINITY;
        m.hi = 0.0f;
#pragma unroll
        for (int n = 0; n < 8; ++n) {
            m.lo = (v[n] < m.lo) ? v[n] : m.lo;
            m.hi = (m.hi < v[n]) ? v[n] : m.hi;
        }
        if (!moving) m.lo = m.hi = own;
        const int cw = g.nx, cwh = g.nx * g.ny;
        const float *fl = a.fluid + (band[0].i + cw * band[1].i + cwh * band[2].i);
        float fv[8];
#pragma unroll
        for (int n = 0; n < 8; ++n) fv[n] = fl[(n & 1) + ((n & 2) ? cw : 0) + ((n & 4) ? cwh : 0)];
        const int in = above_ff(k, fv, [&](int n) {
            return ((n & 1) ? band[0].x1 : 1.0f - band[0].x1) * ((n & 2) ? band[1].x1 : 1.0f - band[1].x1) *
                   ((n & 4) ? band[2].x1 : 1.0f - band[2].x1);
        });
        ok = ok && in != 2;
        if (in == 1) m.lo = nan_mark();
    }
    if (!ok) return false;
    a.v0[o + f] = out;
    if (MAC) a.vmm[o + f] = m;
    return true;
}

template <int DIM> GBA_HD bool face_backward_try(const StepArgs &a, const Fast &k, unsigned f) {
    const Dims &g = a.g;
    const Idx x = decode_fast(k.fw[DIM], k.fh[DIM], f);
    const int ip[3] = {x.i, x.j, x.k};
    const int nc[3] = {g.nx, g.ny, g.nz};
    const float *const comp[3] = {a.v0, a.v0 + a.off1, a.v0 + a.off2};
    const float *src = comp[DIM];
    float *io = DIM == 0 ? a.u : (DIM == 1 ? a.v : a.w);
    const long long o = DIM == 0 ? 0 : (DIM == 1 ? a.off1 : a.off2);
    bool ok = true;
    float uf[3];
    const MinMax m = a.vmm[o + f];
    const float in = io[f];
    face_full_ff<DIM>(g, comp, x.i, x.j, x.k, f, uf, ok);
    const float own = uf[DIM];
    const bool moving = uf[0] != 0.0f || uf[1] != 0.0f || uf[2] != 0.0f;
    const int w = g.nx + (DIM == 0), wh = w * (g.ny + (DIM == 1));
    Axis ax[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) ax[c] = face_axis(ip[c], -trace_ff(k, uf[c], ok), nc[c] + (c == DIM), ok);
    const int base = ax[0].i + w * ax[1].i + wh * ax[2].i;
    float v[8];
#pragma unroll
    for (int n = 0; n < 8; ++n) v[n] = src[base + (n & 1) + ((n & 2) ? w : 0) + ((n & 4) ? wh : 0)];
    float bwd = interp_ff(ax[0], ax[1], ax[2], v, ok);
    if (!moving) bwd = own;
    const float out = maccormack_ff(m, in, own, bwd, ok);
    if (!ok) return false;
    io[f] = out;
    return true;
}

// cell_full: the double mean of two floats rounds as the float one
GBA_HD float mean2(float a, float b) { return 0.5f * (a + b); }

template <bool MAC> GBA_HD bool cell_forward_try(const StepArgs &a, const Fast &k, unsigned c) {
    const Dims &g = a.g;
    const unsigned char *mask = a.mask;
    if (mask && !mask[c]) return false;  // the FP64 form writes the background
    const Idx x = decode_fast(k.cw, k.chh, c);
    const int w = g.nx, wh = g.nx * g.ny;
    bool ok = true;
    const float *pu = a.u + (x.i + (g.nx + 1) * (x.j + g.ny * x.k)), *pv = a.v + (x.i + g.nx * (x.j + (g.ny + 1) * x.k)),
                *pw = a.w + c;
    const float u[3] = {mean2(pu[0], pu[1]), mean2(pv[0], pv[w]), mean2(pw[0], pw[wh])};
    const bool moving = u[0] != 0.0f || u[1] != 0.0f || u[2] != 0.0f;
    const Axis ax = cell_axis<false>(k, x.i, u[0], g.nx, ok), ay = cell_axis<false>(k, x.j, u[1], g.ny, ok),
               az = cell_axis<false>(k, x.k, u[2], g.nz, ok);
    const int base = ax.i + w * ay.i + wh * az.i;
    float v[8], fv[8];
#pragma unroll
    for (int n = 0; n < 8; ++n) {
        const int e = base + (n & 1) + ((n & 2) ? w : 0) + ((n & 4) ? wh : 0);
        v[n] = a.q[e];
        if (mask && !mask[e]) v[n] = a.bg;
        if (MAC) fv[n] = a.fluid[e];
    }
    const float own = a.q[c];
    float out = interp_ff(ax, ay, az, v, ok);
    if (!moving) out = own;
    MinMax m;
    if (MAC) {
        m.lo = FLT_MAX;
        m.hi = FLT_MIN;
#pragma unroll
        for (int n = 0; n < 8; ++n) {
            m.lo = (v[n] < m.lo) ? v[n] : m.lo;
            m.hi = (m.hi < v[n]) ? v[n] : m.hi;
        }
        if (!moving) m.lo = m.hi = own;
        const int in = above_ff(k, fv, [&](int n) {
            return ((n & 1) ? ax.w1.h : ax.w0.h) * ((n & 2) ? ay.w1.h : ay.w0.h) * ((n & 4) ? az.w1.h : az.w0.h);
        });
        // a cell at rest compares its own level set: its corner of weight 1
        ok = ok && in != 2;
        if (in == 1) m.lo = nan_mark();
    }
    if (!ok) return false;
    a.q0[c] = out;
    if (MAC) a.qmm[c] = m;
    return true;
}

GBA_HD bool cell_backward_try(const StepArgs &a, const Fast &k, unsigned c) {
    const Dims &g = a.g;
    if (a.mask && !a.mask[c]) return false;
    const Idx x = decode_fast(k.cw, k.chh, c);
    const int w = g.nx, wh = g.nx * g.ny;
    bool ok = true;
    const float *pu = a.u + (x.i + (g.nx + 1) * (x.j + g.ny * x.k)), *pv = a.v + (x.i + g.nx * (x.j + (g.ny + 1) * x.k)),
                *pw = a.w + c;
    const float u[3] = {mean2(pu[0], pu[1]), mean2(pv[0], pv[w]), mean2(pw[0], pw[wh])};
    const bool moving = u[0] != 0.0f || u[1] != 0.0f || u[2] != 0.0f;
    const Axis ax = cell_axis<true>(k, x.i, u[0], g.nx, ok), ay = cell_axis<true>(k, x.j, u[1], g.ny, ok),
               az = cell_axis<true>(k, x.k, u[2], g.nz, ok);
    const int base = ax.i + w * ay.i + wh * az.i;
    float v[8];
#pragma unroll
    for (int n = 0; n < 8; ++n) v[n] = a.q0[base + (n & 1) + ((n & 2) ? w : 0) + ((n & 4) ? wh : 0)];
    const float own = a.q0[c];
    float bwd = interp_ff(ax, ay, az, v, ok);
    if (!moving) bwd = own;
    const float out = maccormack_ff(a.qmm[c], a.q[c], own, bwd, ok);
    if (!ok) return false;
    a.q[c] = out;
    return true;
}

// ---- 2D ------------------------------------------------------------------

template <int DIM>
GBA_HD void face_full2_ff(const Dims &g, const float *const comp[2], int i, int j, unsigned f, float (&uf)[2],
                          bool &ok) {
    constexpr int C = 1 - DIM;
    const int n[2] = {g.nx, g.ny}, ip[2] = {i, j};
    const int lo = ip[DIM] > 0 ? ip[DIM] - 1 : 0, hi = ip[DIM] < n[DIM] ? ip[DIM] : n[DIM] - 1;
    const int w = g.nx + (C == 0), step[2] = {1, w};
    int q[2] = {i, j};
    q[DIM] = lo;
    const float *p = comp[C] + (q[0] + w * q[1]);
    const int up = (hi - lo) * step[DIM];
    uf[DIM] = comp[DIM][f];
    uf[C] = mean4(p[0], p[step[C]], p[up], p[up + step[C]], ok);
}

template <int DIM, bool MAC> GBA_HD bool face_forward2_try(const StepArgs &a, const Fast &k, unsigned f) {
    const Dims &g = a.g;
    const unsigned row = gbp::fdiv(f, k.fw[DIM]);
    const int ip[2] = {(int)(f - row * k.fw[DIM].d), (int)row};
    const int nc[2] = {g.nx, g.ny};
    const float *const comp[2] = {a.u, a.v};
    const float *src = comp[DIM];
    const long long o = DIM == 0 ? 0 : a.off1;
    bool ok = true;
    float uf[2];
    face_full2_ff<DIM>(g, comp, ip[0], ip[1], f, uf, ok);
    const float own = uf[DIM];
    const bool moving = uf[0] != 0.0f || uf[1] != 0.0f;
    const int w = g.nx + (DIM == 0);
    const Axis ax = face_axis(ip[0], trace_ff(k, uf[0], ok), nc[0] + (DIM == 0), ok),
               ay = face_axis(ip[1], trace_ff(k, uf[1], ok), nc[1] + (DIM == 1), ok);
    const int base = ax.i + w * ay.i;
    float v[4] = {src[base], src[base + 1], src[base + w], src[base + w + 1]};
    float out = interp2_ff(ax, ay, v, ok);
    if (!moving) out = own;
    MinMax m;
    if (MAC) {
        Cellf q[2], band[2];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const Shift s = shift_of(k, uf[c], ok);
            q[c] = cell_of(ip[c], s, nc[c] + (c == DIM), ok);
            band[c] = c == DIM ? half_cell_of(ip[c], s, nc[c], ok) : q[c];
        }
        const int base2 = q[0].i + w * q[1].i;
        if (base2 != base) {
            v[0] = src[base2];
            v[1] = src[base2 + 1];
            v[2] = src[base2 + w];
            v[3] = src[base2 + w + 1];
        }
        m.lo = INFINITY;
        m.hi = 0.0f;
#pragma unroll
        for (int n = 0; n < 4; ++n) {
            m.lo = (v[n] < m.lo) ? v[n] : m.lo;
            m.hi = (m.hi < v[n]) ? v[n] : m.hi;
        }
        if (!moving) m.lo = m.hi = own;
        const float *fl = a.fluid + (band[0].i + g.nx * band[1].i);
        const float fv[4] = {fl[0], fl[1], fl[g.nx], fl[g.nx + 1]};
        const int in = above_ff(k, fv, [&](int n) {
            return ((n & 1) ? band[0].x1 : 1.0f - band[0].x1) * ((n & 2) ? band[1].x1 : 1.0f - band[1].x1);
        });
        ok = ok && in != 2;
        if (in == 1) m.lo = nan_mark();
    }
    if (!ok) return false;
    a.v0[o + f] = out;
    if (MAC) a.vmm[o + f] = m;
    return true;
}

template <int DIM> GBA_HD bool face_backward2_try(const StepArgs &a, const Fast &k, unsigned f) {
    const Dims &g = a.g;
    const unsigned row = gbp::fdiv(f, k.fw[DIM]);
    const int ip[2] = {(int)(f - row * k.fw[DIM].d), (int)row};
    const int nc[2] = {g.nx, g.ny};
    const float *const comp[2] = {a.v0, a.v0 + a.off1};
    const float *src = comp[DIM];
    float *io = DIM == 0 ? a.u : a.v;
    const long long o = DIM == 0 ? 0 : a.off1;
    bool ok = true;
    float uf[2];
    face_full2_ff<DIM>(g, comp, ip[0], ip[1], f, uf, ok);
    const float own = uf[DIM];
    const bool moving = uf[0] != 0.0f || uf[1] != 0.0f;
    const int w = g.nx + (DIM == 0);
    const Axis ax = face_axis(ip[0], -trace_ff(k, uf[0], ok), nc[0] + (DIM == 0), ok),
               ay = face_axis(ip[1], -trace_ff(k, uf[1], ok), nc[1] + (DIM == 1), ok);
    const int base = ax.i + w * ay.i;
    const float v[4] = {src[base], src[base + 1], src[base + w], src[base + w + 1]};
    float bwd = interp2_ff(ax, ay, v, ok);
    if (!moving) bwd = own;
    const float out = maccormack_ff(a.vmm[o + f], io[f], own, bwd, ok);
    if (!ok) return false;
    io[f] = out;
    return true;
}

template <bool MAC> GBA_HD bool cell_forward2_try(const StepArgs &a, const Fast &k, unsigned c) {
    const Dims &g = a.g;
    const unsigned char *mask = a.mask;
    if (mask && !mask[c]) return false;
    const unsigned row = gbp::fdiv(c, k.cw);
    const int i = (int)(c - row * k.cw.d), j = (int)row, w = g.nx;
    bool ok = true;
    const float *pu = a.u + (i + (g.nx + 1) * j), *pv = a.v + c;
    const float u[2] = {mean2(pu[0], pu[1]), mean2(pv[0], pv[w])};
    const bool moving = u[0] != 0.0f || u[1] != 0.0f;
    const Axis ax = cell_axis<false>(k, i, u[0], g.nx, ok), ay = cell_axis<false>(k, j, u[1], g.ny, ok);
    const int base = ax.i + w * ay.i;
    float v[4], fv[4];
#pragma unroll
    for (int n = 0; n < 4; ++n) {
        const int e = base + (n & 1) + ((n & 2) ? w : 0);
        v[n] = a.q[e];
        if (mask && !mask[e]) v[n] = a.bg;
        if (MAC) fv[n] = a.fluid[e];
    }
    const float own = a.q[c];
    float out = interp2_ff(ax, ay, v, ok);
    if (!moving) out = own;
    MinMax m;
    if (MAC) {
        m.lo = FLT_MAX;
        m.hi = FLT_MIN;
#pragma unroll
        for (int n = 0; n < 4; ++n) {
            m.lo = (v[n] < m.lo) ? v[n] : m.lo;
            m.hi = (m.hi < v[n]) ? v[n] : m.hi;
        }
        if (!moving) m.lo = m.hi = own;
        const int in = above_ff(k, fv, [&](int n) { return ((n & 1) ? ax.w1.h : ax.w0.h) * ((n & 2) ? ay.w1.h : ay.w0.h); });
        ok = ok && in != 2;
        if (in == 1) m.lo = nan_mark();
    }
    if (!ok) return false;
    a.q0[c] = out;
    if (MAC) a.qmm[c] = m;
    return true;
}

GBA_HD bool cell_backward2_try(const StepArgs &a, const Fast &k, unsigned c) {
    const Dims &g = a.g;
    if (a.mask && !a.mask[c]) return false;
    const unsigned row = gbp::fdiv(c, k.cw);
    const int i = (int)(c - row * k.cw.d), j = (int)row, w = g.nx;
    bool ok = true;
    const float *pu = a.u + (i + (g.nx + 1) * j), *pv = a.v + c;
    const float u[2] = {mean2(pu[0], pu[1]), mean2(pv[0], pv[w])};
    const bool moving = u[0] != 0.0f || u[1] != 0.0f;
    const Axis ax = cell_axis<true>(k, i, u[0], g.nx, ok), ay = cell_axis<true>(k, j, u[1], g.ny, ok);
    const int base = ax.i + w * ay.i;
    const float v[4] = {a.q0[base], a.q0[base + 1], a.q0[base + w], a.q0[base + w + 1]};
    const float own = a.q0[c];
    float bwd = interp2_ff(ax, ay, v, ok);
    if (!moving) bwd = own;
    const float out = maccormack_ff(a.qmm[c], a.q[c], own, bwd, ok);
    if (!ok) return false;
    a.q[c] = out;
    return true;
}

// ---- one element: the float-pair form, the FP64 form where it is undecided

template <int DIM, bool MAC> GBA_HD void face_forward_any(const StepArgs &a, const Fast &k, unsigned f) {
    if (f >= count(face_shape(a.g, DIM))) return;
    if (!k.on || !face_forward_try<DIM, MAC>(a, k, f)) face_forward_fp64<MAC>(a, DIM, f);
}
template <int DIM> GBA_HD void face_backward_any(const StepArgs &a, const Fast &k, unsigned f) {
    if (f >= count(face_shape(a.g, DIM))) return;
    if (!k.on || !face_backward_try<DIM>(a, k, f)) face_backward_fp64(a, DIM, f);
}
template <bool MAC> GBA_HD void cell_forward_any(const StepArgs &a, const Fast &k, unsigned c) {
    if (c >= count(Shape{a.g.nx, a.g.ny, a.g.nz})) return;
    if (!k.on || !cell_forward_try<MAC>(a, k, c)) cell_forward_fp64<MAC>(a, c);
}
GBA_HD void cell_backward_any(const StepArgs &a, const Fast &k, unsigned c) {
    if (c >= count(Shape{a.g.nx, a.g.ny, a.g.nz})) return;
    if (!k.on || !cell_backward_try(a, k, c)) cell_backward_fp64(a, c);
}
template <int DIM, bool MAC> GBA_HD void face_forward2_any(const StepArgs &a, const Fast &k, unsigned f) {
    if (f >= count2(face_shape2(a.g, DIM))) return;
    if (!k.on || !face_forward2_try<DIM, MAC>(a, k, f)) face_forward2_fp64<MAC>(a, DIM, f);
}
template <int DIM> GBA_HD void face_backward2_any(const StepArgs &a, const Fast &k, unsigned f) {
    if (f >= count2(face_shape2(a.g, DIM))) return;
    if (!k.on || !face_backward2_try<DIM>(a, k, f)) face_backward2_fp64(a, DIM, f);
}
template <bool MAC> GBA_HD void cell_forward2_any(const StepArgs &a, const Fast &k, unsigned c) {
    if (c >= count2(Shape2{a.g.nx, a.g.ny})) return;
    if (!k.on || !cell_forward2_try<MAC>(a, k, c)) cell_forward2_fp64<MAC>(a, c);
}
GBA_HD void cell_backward2_any(const StepArgs &a, const Fast &k, unsigned c) {
    if (c >= count2(Shape2{a.g.nx, a.g.ny})) return;
    if (!k.on || !cell_backward2_try(a, k, c)) cell_backward2_fp64(a, c);
}

}  // namespace gba
