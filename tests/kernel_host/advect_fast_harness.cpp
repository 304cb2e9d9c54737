// advect_fast_harness.cpp -- TEST INFRASTRUCTURE: the float-pair forms of the
// advection passes (shiokaze_gb300/csrc/advect_fast.cuh) compiled for the host
// and compared element by element with the FP64 forms (advect_core.cuh) they
// stand for. Each pass runs in both forms from the same state; counts[0] is
// the number of values that differ, counts[1] the elements the float-pair
// form left to the FP64 form, counts[2] all elements. Not part of the library.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "advect_fast.cuh"
using namespace gba;

namespace {

struct Both {
    std::vector<float> v[3], q, v0, q0;
    std::vector<MinMax> vmm, qmm;
};

template <class T> long long differ(const std::vector<T> &a, const std::vector<T> &b) {
    long long n = 0;
    for (size_t i = 0; i < a.size(); ++i) n += std::memcmp(&a[i], &b[i], sizeof(T)) != 0;
    return n;
}

StepArgs args_of(Both &s, const Dims &g, double dt, const float *fluid, const unsigned char *mask, float bg, bool three,
                 bool scalar) {
    StepArgs a{};
    a.g = g;
    a.dt = dt;
    a.u = s.v[0].data();
    a.v = s.v[1].data();
    a.w = three ? s.v[2].data() : nullptr;
    a.fluid = fluid;
    a.q = scalar ? s.q.data() : nullptr;
    a.mask = mask;
    a.bg = bg;
    a.v0 = s.v0.data();
    a.vmm = s.vmm.data();
    a.off1 = (long long)s.v[0].size();
    a.off2 = three ? (long long)(s.v[0].size() + s.v[1].size()) : 0;
    a.q0 = s.q0.data();
    a.qmm = s.qmm.data();
    return a;
}

Dims dims_of(int nx, int ny, int nz, double dx, int trim) {
    Dims g{};
    g.nx = nx;
    g.ny = ny;
    g.nz = nz;
    g.dx = dx;
    int e = 0;
    const double m = std::frexp(dx, &e), inv = 1.0 / dx;
    g.pow2 = (m == 0.5 && std::isfinite(inv) && (double)(float)inv == inv) ? 1 : 0;
    g.inv_dx = inv;
    g.inv_dx_f = (float)inv;
    g.limit = -dx * (double)trim;
    return g;
}

}  // namespace

extern "C" int pairs_advect(int dim, int nx, int ny, int nz, double dx, double dt, int mac, int trim, const float *u,
                            const float *v, const float *w, const float *fluid, const float *q,
                            const unsigned char *mask, float bg, long long *counts) {
    const bool three = dim == 3;
    const Dims g = dims_of(nx, ny, three ? nz : 1, dx, trim);
    const Fast k = make_fast(g, dt, three);
    const long long nzz = three ? nz : 1, cells = (long long)nx * ny * nzz;
    const long long nf[3] = {(nx + 1) * ny * nzz, nx * (ny + 1) * nzz, three ? (long long)nx * ny * (nz + 1) : 0};
    Both s;
    const float *src[3] = {u, v, w};
    for (int d = 0; d < dim; ++d) s.v[d].assign(src[d], src[d] + nf[d]);
    s.q.assign(q, q + cells);
    s.v0.assign(nf[0] + nf[1] + nf[2], 0.0f);
    s.vmm.assign(nf[0] + nf[1] + nf[2], MinMax{0.0f, 0.0f});
    s.q0.assign(cells, 0.0f);
    s.qmm.assign(cells, MinMax{0.0f, 0.0f});
    counts[0] = counts[1] = counts[2] = 0;
    // one pass in both forms from the state s; the FP64 form's result goes on
    auto pass = [&](auto pairs, auto fp64, auto tried, long long n) {
        Both t = s;
        StepArgs a = args_of(t, g, dt, fluid, mask, bg, three, true), b = args_of(s, g, dt, fluid, mask, bg, three, true);
        for (long long f = 0; f < n; ++f) {
            counts[1] += !tried(a, (unsigned)f);
            pairs(a, (unsigned)f);
        }
        for (long long f = 0; f < n; ++f) fp64(b, (unsigned)f);
        counts[2] += n;
        for (int d = 0; d < 3; ++d) counts[0] += differ(s.v[d], t.v[d]);
        counts[0] += differ(s.q, t.q) + differ(s.v0, t.v0) + differ(s.q0, t.q0) + differ(s.vmm, t.vmm) +
                     differ(s.qmm, t.qmm);
    };
    if (three) {
        if (mac) {
            pass([&](auto &a, unsigned f) { cell_forward_any<true>(a, k, f); },
                 [&](auto &a, unsigned f) { cell_forward<true>(a, f); },
                 [&](auto &a, unsigned f) { return cell_forward_try<true>(a, k, f) || (mask && !mask[f]); }, cells);
            // the tried call of a backward pass would write the result before the pairs call reads its input
            pass([&](auto &a, unsigned f) { cell_backward_any(a, k, f); },
                 [&](auto &a, unsigned f) { cell_backward(a, f); }, [&](auto &, unsigned) { return true; }, cells);
            pass([&](auto &a, unsigned f) { face_forward_any<0, true>(a, k, f); },
                 [&](auto &a, unsigned f) { face_forward<true>(a, 0, f); },
                 [&](auto &a, unsigned f) { return face_forward_try<0, true>(a, k, f); }, nf[0]);
            pass([&](auto &a, unsigned f) { face_forward_any<1, true>(a, k, f); },
                 [&](auto &a, unsigned f) { face_forward<true>(a, 1, f); },
                 [&](auto &a, unsigned f) { return face_forward_try<1, true>(a, k, f); }, nf[1]);
            pass([&](auto &a, unsigned f) { face_forward_any<2, true>(a, k, f); },
                 [&](auto &a, unsigned f) { face_forward<true>(a, 2, f); },
                 [&](auto &a, unsigned f) { return face_forward_try<2, true>(a, k, f); }, nf[2]);
            pass([&](auto &a, unsigned f) { face_backward_any<0>(a, k, f); },
                 [&](auto &a, unsigned f) { face_backward(a, 0, f); }, [&](auto &, unsigned) { return true; }, nf[0]);
            pass([&](auto &a, unsigned f) { face_backward_any<1>(a, k, f); },
                 [&](auto &a, unsigned f) { face_backward(a, 1, f); }, [&](auto &, unsigned) { return true; }, nf[1]);
            pass([&](auto &a, unsigned f) { face_backward_any<2>(a, k, f); },
                 [&](auto &a, unsigned f) { face_backward(a, 2, f); }, [&](auto &, unsigned) { return true; }, nf[2]);
        } else {
            pass([&](auto &a, unsigned f) { cell_forward_any<false>(a, k, f); },
                 [&](auto &a, unsigned f) { cell_forward<false>(a, f); },
                 [&](auto &a, unsigned f) { return cell_forward_try<false>(a, k, f) || (mask && !mask[f]); }, cells);
            pass([&](auto &a, unsigned f) { face_forward_any<0, false>(a, k, f); },
                 [&](auto &a, unsigned f) { face_forward<false>(a, 0, f); },
                 [&](auto &a, unsigned f) { return face_forward_try<0, false>(a, k, f); }, nf[0]);
            pass([&](auto &a, unsigned f) { face_forward_any<1, false>(a, k, f); },
                 [&](auto &a, unsigned f) { face_forward<false>(a, 1, f); },
                 [&](auto &a, unsigned f) { return face_forward_try<1, false>(a, k, f); }, nf[1]);
            pass([&](auto &a, unsigned f) { face_forward_any<2, false>(a, k, f); },
                 [&](auto &a, unsigned f) { face_forward<false>(a, 2, f); },
                 [&](auto &a, unsigned f) { return face_forward_try<2, false>(a, k, f); }, nf[2]);
        }
    } else {
        if (mac) {
            pass([&](auto &a, unsigned f) { cell_forward2_any<true>(a, k, f); },
                 [&](auto &a, unsigned f) { cell_forward2<true>(a, f); },
                 [&](auto &a, unsigned f) { return cell_forward2_try<true>(a, k, f) || (mask && !mask[f]); }, cells);
            pass([&](auto &a, unsigned f) { cell_backward2_any(a, k, f); },
                 [&](auto &a, unsigned f) { cell_backward2(a, f); }, [&](auto &, unsigned) { return true; }, cells);
            pass([&](auto &a, unsigned f) { face_forward2_any<0, true>(a, k, f); },
                 [&](auto &a, unsigned f) { face_forward2<true>(a, 0, f); },
                 [&](auto &a, unsigned f) { return face_forward2_try<0, true>(a, k, f); }, nf[0]);
            pass([&](auto &a, unsigned f) { face_forward2_any<1, true>(a, k, f); },
                 [&](auto &a, unsigned f) { face_forward2<true>(a, 1, f); },
                 [&](auto &a, unsigned f) { return face_forward2_try<1, true>(a, k, f); }, nf[1]);
            pass([&](auto &a, unsigned f) { face_backward2_any<0>(a, k, f); },
                 [&](auto &a, unsigned f) { face_backward2(a, 0, f); }, [&](auto &, unsigned) { return true; }, nf[0]);
            pass([&](auto &a, unsigned f) { face_backward2_any<1>(a, k, f); },
                 [&](auto &a, unsigned f) { face_backward2(a, 1, f); }, [&](auto &, unsigned) { return true; }, nf[1]);
        } else {
            pass([&](auto &a, unsigned f) { cell_forward2_any<false>(a, k, f); },
                 [&](auto &a, unsigned f) { cell_forward2<false>(a, f); },
                 [&](auto &a, unsigned f) { return cell_forward2_try<false>(a, k, f) || (mask && !mask[f]); }, cells);
            pass([&](auto &a, unsigned f) { face_forward2_any<0, false>(a, k, f); },
                 [&](auto &a, unsigned f) { face_forward2<false>(a, 0, f); },
                 [&](auto &a, unsigned f) { return face_forward2_try<0, false>(a, k, f); }, nf[0]);
            pass([&](auto &a, unsigned f) { face_forward2_any<1, false>(a, k, f); },
                 [&](auto &a, unsigned f) { face_forward2<false>(a, 1, f); },
                 [&](auto &a, unsigned f) { return face_forward2_try<1, false>(a, k, f); }, nf[1]);
        }
    }
    return k.on;
}

// x/dx by div_known against the division, n seeded operands; returns the number that differ
extern "C" long long pairs_division(double dx, long long n, const double *x) {
    const double inv = 1.0 / dx;
    long long bad = 0;
    for (long long i = 0; i < n; ++i) bad += div_known(x[i], dx, inv) != x[i] / dx;
    return bad;
}
