// TEST INFRASTRUCTURE: the setup kernels' float-pair quotient and rounded FP64
// division (shiokaze_gb300/csrc/gbp_exact.cuh) compiled for the host beside the
// FP64 expressions they stand for.
#define __host__
#define __device__
#define __forceinline__ inline
#include "gbp_exact.cuh"

// Values where quot_round decides and differs from (float)(dt f / (rho dx)); undecided ones counted in *left.
extern "C" long long host_quot(double dt, double dx, const float *f, const float *rho, long long n, long long *left) {
    const gbp::PairConst c = gbp::make_pair_const(dt / dx);
    long long bad = 0;
    for (long long i = 0; i < n; ++i) {
        float out;
        if (!gbp::quot_round(c, f[i], rho[i], out)) {
            ++*left;
            continue;
        }
        const float want = (float)(rho[i] == 1.0f ? dt * (double)f[i] / dx : dt * (double)f[i] / ((double)rho[i] * dx));
        bad += gbp::ex_bits(out) != gbp::ex_bits(want);
    }
    return bad;
}

// Values where div_round differs from the division (-0 and +0 alike).
extern "C" long long host_div(double d, const float *x, long long n) {
    const gbp::RecipConst c = gbp::make_recip_const(d);
    long long bad = 0;
    for (long long i = 0; i < n; ++i) bad += !(gbp::div_round(c, (double)x[i]) == (double)x[i] / d);
    return bad;
}
