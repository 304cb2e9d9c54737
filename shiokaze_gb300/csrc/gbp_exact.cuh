// gbp_exact.cuh -- FP64 results of the setup's arithmetic without FP64
// operations, or with few.
//
// On this GPU the FP64 pipe issues about two operations per clock per SM (a
// sixty-fourth of the integer rate). The functions here produce the
// bit-identical double (or float) and return true, or return false, and the
// caller evaluates the FP64 expression.
//
// * exact_sum: the sequential FP64 sum 0 + t_0 + t_1 + ... of terms
//   t_i = f_i 2^k (floats f_i, one power of two). If every partial sum is a
//   double, no addition rounds and the result is the exact sum, which a
//   64-bit integer holds when the terms' exponents span at most 36 binary
//   orders. Both conditions are checked. (The assembly's right-hand side no
//   longer takes it: six FP64 additions run beside the integer instructions
//   that bound that pass.)
// * mul_round: fl32(fl64(a f) 2^s) for a double a fixed per launch (dt) and
//   a float f (a pressure difference): the 77-bit product of the
//   significands rounded to 53 bits and then to 24, each to nearest with
//   ties to even, as the two hardware roundings do; results outside the
//   normal ranges take the FP64 path.
// * quot_round: the same float, and that of a f / rho, from a float pair and
//   a rounding test; div_round: x / d for a constant d in four operations.
//
// The same source compiles for the host (tests/test_kernel_host.py and
// tests/test_setup_quotients.py check the functions against the compiler's
// FP64 arithmetic).
#pragma once

#include <cstring>

namespace gbp {

__host__ __device__ __forceinline__ unsigned ex_bits(float f) {
#ifdef __CUDA_ARCH__
    return __float_as_uint(f);
#else
    unsigned u;
    std::memcpy(&u, &f, sizeof u);
    return u;
#endif
}
__host__ __device__ __forceinline__ float ex_float(unsigned u) {
#ifdef __CUDA_ARCH__
    return __uint_as_float(u);
#else
    float f;
    std::memcpy(&f, &u, sizeof f);
    return f;
#endif
}
__host__ __device__ __forceinline__ double ex_double(unsigned long long u) {
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)u);
#else
    double d;
    std::memcpy(&d, &u, sizeof d);
    return d;
#endif
}
__host__ __device__ __forceinline__ int ex_clz64(unsigned long long a) {
#ifdef __CUDA_ARCH__
    return __clzll((long long)a);
#else
    return a ? __builtin_clzll(a) : 64;
#endif
}
__host__ __device__ __forceinline__ int ex_ctz64(unsigned long long a) {
#ifdef __CUDA_ARCH__
    return __ffsll((long long)a) - 1;
#else
    return a ? __builtin_ctzll(a) : 64;
#endif
}
__host__ __device__ __forceinline__ unsigned long long ex_mulhi(unsigned long long a, unsigned long long b) {
#ifdef __CUDA_ARCH__
    return __umul64hi(a, b);
#else
    return (unsigned long long)(((unsigned __int128)a * b) >> 64);
#endif
}

// Sequential FP64 sum of n terms sgn_i f_i 2^k, sgn_i = -1 where bit i of
// neg is set; false if an addition could round or a value leaves the normal
// ranges (subnormal, infinite or NaN f_i included).
__host__ __device__ __forceinline__ bool exact_sum(const float *f, int n, unsigned neg, int k, double &out) {
    int emin = 1 << 20, emax = -(1 << 20);
#pragma unroll
    for (int i = 0; i < n; ++i) {
        const unsigned b = ex_bits(f[i]) & 0x7fffffffu;
        if (!b) continue;
        const int ex = (int)(b >> 23);
        if (ex == 0 || ex == 255) return false;
        const int e = ex - 150;  // f = m 2^e, m the 24-bit significand
        emin = e < emin ? e : emin;
        emax = e > emax ? e : emax;
    }
    if (emax < emin) {  // every term is +-0: 0 + (+-0) + ... = +0
        out = 0.0;
        return true;
    }
    if (emax - emin > 36 || emin + k < -1000 || emax + k > 1000) return false;
    // within 26 binades every term is below 2^50 in units of 2^emin, so a
    // partial sum of at most 7 terms stays below 2^53: none can round
    const bool spread = emax - emin > 26;
    long long s = 0;
#pragma unroll
    for (int i = 0; i < n; ++i) {
        const unsigned b = ex_bits(f[i]);
        const unsigned a = b & 0x7fffffffu;
        if (!a) continue;
        const long long m = (long long)((a & 0x7fffffu) | 0x800000u) << ((int)(a >> 23) - 150 - emin);
        // the term's sign: the float's, flipped where neg says
        s += (((b >> 31) ^ (neg >> i)) & 1u) ? -m : m;
        const unsigned long long mag = (unsigned long long)(s < 0 ? -s : s);
        if (spread && (mag >> 53) && ((mag >> ex_ctz64(mag)) >> 53)) return false;  // this partial sum would round
    }
    if (!s) {  // x + (-x) = +0 in round to nearest
        out = 0.0;
        return true;
    }
    const unsigned long long sign = s < 0 ? 1ull << 63 : 0ull;
    unsigned long long mag = (unsigned long long)(s < 0 ? -s : s);
    const int len = 64 - ex_clz64(mag);
    // exact: at most 53 significant bits (checked above)
    mag = len <= 53 ? mag << (53 - len) : mag >> (len - 53);
    const int e = emin + k + len - 1;  // unbiased exponent of the sum
    out = ex_double(sign | ((unsigned long long)(e + 1023) << 52) | (mag & 0xfffffffffffffull));
    return true;
}

// a = m 2^e (m with its hidden bit), prepared on the host for mul_round.
struct MulConst {
    unsigned long long m;
    int e;       // a's exponent with the significand as an integer (unbiased - 52)
    int s;       // the power of two applied after the FP64 rounding
    unsigned sign;  // a's sign in bit 31
    int ok;      // a is a normal double (else every call takes the FP64 path)
};

inline MulConst make_mul_const(double a, int s) {
    unsigned long long b;
    std::memcpy(&b, &a, sizeof b);
    MulConst c{};
    const int ex = (int)((b >> 52) & 0x7ff);
    c.ok = ex != 0 && ex != 0x7ff;
    c.m = (b & 0xfffffffffffffull) | (1ull << 52);
    c.e = ex - 1075;
    c.s = s;
    c.sign = (unsigned)(b >> 63) << 31;
    return c;
}

// fl32(fl64(a f) 2^s), false where the FP64 path must decide.
__host__ __device__ __forceinline__ bool mul_round(const MulConst c, float f, float &out) {
    const unsigned fb = ex_bits(f);
    const unsigned sign = (fb & 0x80000000u) ^ c.sign;
    const unsigned fa = fb & 0x7fffffffu;
    if (!c.ok) return false;
    if (!fa) {  // +-0 * a = +-0, exactly
        out = ex_float(sign);
        return true;
    }
    const int fe = (int)(fa >> 23);
    if (fe == 0 || fe == 255) return false;
    const unsigned long long mf = (fa & 0x7fffffu) | 0x800000u;
    // P = mf c.m in [2^75, 2^77): hi holds bits 64..76
    const unsigned long long lo = mf * c.m, hi = ex_mulhi(mf, c.m);
    const int sh = (hi >> 12) ? 24 : 23;  // bits dropped to keep 53
    unsigned long long q = (hi << (64 - sh)) | (lo >> sh);
    const unsigned long long rem = lo & ((1ull << sh) - 1), half = 1ull << (sh - 1);
    q += (rem > half || (rem == half && (q & 1ull))) ? 1ull : 0ull;
    int e = (fe - 150) + c.e + sh;  // fl64(a f) = q 2^e
    if (q >> 53) {
        q >>= 1;
        e += 1;
    }
    // fl64(a f) and its scaled value must be normal doubles
    const int e64 = e + 52;
    if (e64 < -1022 || e64 > 1023 || e64 + c.s < -1022 || e64 + c.s > 1023) return false;
    int e32 = e64 + c.s;
    if (e32 < -126 || e32 > 127) return false;
    const unsigned long long r29 = q & 0x1fffffffull, h29 = 0x10000000ull;
    unsigned long long r = q >> 29;
    r += (r29 > h29 || (r29 == h29 && (r & 1ull))) ? 1ull : 0ull;
    if (r >> 24) {
        r >>= 1;
        e32 += 1;
        if (e32 > 127) return false;  // rounds to infinity: the FP64 path says so
    }
    out = ex_float(sign | ((unsigned)(e32 + 127) << 23) | ((unsigned)r & 0x7fffffu));
    return true;
}

// A double constant as a pair of floats (within 2^-48 of it) for quot_round;
// hi = 0 where the pair's products could leave the normal floats.
struct PairConst {
    float hi, lo;
};
inline PairConst make_pair_const(double a) {
    const double m = a < 0 ? -a : a;
    if (!(m >= 9.1e-13 && m <= 1.0e12)) return PairConst{0.0f, 0.0f};
    const float hi = (float)a;
    return PairConst{hi, (float)(a - (double)hi)};
}
__host__ __device__ __forceinline__ float ex_fmaf(float a, float b, float c) {
#ifdef __CUDA_ARCH__
    return __fmaf_rn(a, b, c);
#else
    return __builtin_fmaf(a, b, c);
#endif
}
__host__ __device__ __forceinline__ float ex_divf(float a, float b) {
#ifdef __CUDA_ARCH__
    return __fdiv_rn(a, b);
#else
    return a / b;
#endif
}

// The float nearest a f / rho for a constant a (dt / dx), where the FP64
// evaluation of it (a few roundings of 2^-53) must round alike: the float pair
// v + t is within 2^-45 of the real value (f hi exactly by an FMA, 2^-48 each
// for lo, the sums and the quotient's correction), and the test moves it by
// 2^-43 either way. False if the two differ (about 2^-19 of all f; up to half
// of them where a is nearly a fraction like 3/4, whose products are ties) or a
// value leaves the ranges; the caller then evaluates in FP64. No contraction is
// meant here: the sources that include this are built without it.
__host__ __device__ __forceinline__ bool quot_round(const PairConst c, float f, float rho, float &out) {
    float v = f * c.hi;
    if (f == 0.0f && c.hi != 0.0f) {  // a signed zero
        out = v;
        return true;
    }
    float t = ex_fmaf(f, c.lo, ex_fmaf(f, c.hi, -v));
    float m = ex_float(ex_bits(v) & 0x7fffffffu);
    if (!(m >= 8.7e-19f && m <= 1.1e18f)) return false;
    if (rho != 1.0f) {
        if (!(rho >= 9.0e-13f && rho <= 1.0f)) return false;
        const float q = ex_divf(v, rho);
        t = ex_divf(ex_fmaf(-q, rho, v) + t, rho);
        v = q;
        m = ex_float(ex_bits(v) & 0x7fffffffu);
    }
    const float w = m * 1.1368684e-13f;  // 2^-43
    const float lo = v + (t - w), hi = v + (t + w);
    out = hi;
    return lo == hi;
}

// 1/d as a pair of doubles, r the nearest double to 1/d, for div_round.
struct RecipConst {
    double d, r, rlo;
};
// The double nearest x / d: a quotient q0 within less than one unit in the
// last place (the reciprocal pair), its exact remainder, and one correction by
// the nearest double to 1/d, which by Markstein's theorem (Computation of
// elementary functions on the IBM RISC System/6000, IBM J. Res. Dev. 34, 1990)
// rounds the quotient correctly. Four operations of the FP64 pipe where a
// division takes several times that. For finite x with |x| 0 or in
// [2^-300, 2^300] and d in [2^-500, 2^500]; a quotient of -0 may come as +0.
__host__ __device__ __forceinline__ double div_round(const RecipConst c, double x) {
#ifdef __CUDA_ARCH__
    const double q0 = __fma_rn(x, c.r, __dmul_rn(x, c.rlo));
    return __fma_rn(__fma_rn(-q0, c.d, x), c.r, q0);
#else
    const double q0 = __builtin_fma(x, c.r, x * c.rlo);
    return __builtin_fma(__builtin_fma(-q0, c.d, x), c.r, q0);
#endif
}
inline RecipConst make_recip_const(double d) {
    const double r = 1.0 / d;
    return RecipConst{d, r, __builtin_fma(-r, d, 1.0) * r};
}

}  // namespace gbp
