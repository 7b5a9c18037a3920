// boris32_common.cuh -- what the FP32C push kernels share: the termination
// predicate on compensated positions and the saver.
#pragma once

#include "fp32c_common.cuh"
#include "tp_device.cuh"
#include "tp_launch.h"

namespace tpb {

namespace {

template <int FK>
__device__ __forceinline__ bool outside32(const BorisArgs& a, const CPos& p, const typename Vel32<FK>::V& v,
                                          double t) {
    const DevTerm& T = a.term;
    int f = T.flags;
    if (f & TP_TERM_NAN)
        if (isnan(p.hi[0]) || isnan(p.hi[1]) || isnan(p.hi[2]) || Vel32<FK>::has_nan(v)) return true;
    if (f & (TP_TERM_SHELL | TP_TERM_BOX)) {
        // in float on hi + lo: no axis wraps when a spatial predicate is set,
        // and the float-side position already differs from the float64 one
        // by more than the float rounding of the test (no float64 sqrt)
        const float x = p.hi[0] + p.lo[0], y = p.hi[1] + p.lo[1], z = p.hi[2] + p.lo[2];
        if (f & TP_TERM_SHELL) {
            const float r2 = fmaf(x, x, fmaf(y, y, z * z));
            if (r2 < T.smin32 || r2 > T.smax32) return true;
        }
        if (f & TP_TERM_BOX) {
            if (x < T.lo32[0] || x > T.hi32[0] || y < T.lo32[1] || y > T.hi32[1] || z < T.lo32[2] || z > T.hi32[2])
                return true;
        }
    }
    if (f & TP_TERM_TIME)
        if (t > T.tmax) return true;
    return false;
}

template <int FK>
struct Saver32 {
    using P = Vel32<FK>;
    const BorisArgs& a;
    int W;
    // slot width: the state, E and B (float evaluation, as the push sees
    // them) when save_fields, and four work-rate columns when save_work that
    // a post-pass over the saved states fills (keeps that float64 code out
    // of this kernel's registers)
    __device__ Saver32(const BorisArgs& a_)
        : a(a_), W(6 + (a_.save_fields ? 6 : 0) + (a_.save_work ? 4 : 0)) {}
    __device__ __forceinline__ void save(int64_t i, int64_t k, const CPos& p, const typename P::V& v,
                                         double t) const {
        if (k >= a.nslots) {
            set_status(a.status, TP_E_OVERFLOW);
            return;
        }
        const int64_t n = a.n;
        a.t_out[k * n + i] = t;
        double* u = a.u_out + (k * W) * n + i;
        u[0 * n] = cpos_value(a, p, 0);
        u[1 * n] = cpos_value(a, p, 1);
        u[2 * n] = cpos_value(a, p, 2);
        u[3 * n] = P::comp(v, 0);
        u[4 * n] = P::comp(v, 1);
        u[5 * n] = P::comp(v, 2);
        if (a.save_fields) {
            typename P::Fv E, B;
            P::fields(a.f, p, t, E, B);
            u[6 * n] = E.x;
            u[7 * n] = E.y;
            u[8 * n] = E.z;
            u[9 * n] = B.x;
            u[10 * n] = B.y;
            u[11 * n] = B.z;
        }
    }
};

// save slot 0: u0 itself, and the fields as the push sees them
template <int FK>
__device__ __forceinline__ void save_first32(const BorisArgs& a, int64_t i, const CPos& p) {
    if (a.nslots < 1) {
        set_status(a.status, TP_E_OVERFLOW);
        return;
    }
    a.t_out[i] = a.t0;
    const double* u0 = a.u0 + 6 * i;
    double* u = a.u_out + i;
    for (int c = 0; c < 6; ++c) u[c * a.n] = u0[c];
    if (a.save_fields) {
        typename Vel32<FK>::Fv E, B;
        Vel32<FK>::fields(a.f, p, a.t0, E, B);
        u[6 * a.n] = E.x; u[7 * a.n] = E.y; u[8 * a.n] = E.z;
        u[9 * a.n] = B.x; u[10 * a.n] = B.y; u[11 * a.n] = B.z;
    }
}

}  // namespace

}  // namespace tpb
