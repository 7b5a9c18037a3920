// boris64_common.cuh -- what the float64 push kernels share: the saver and the
// schedules.  Included by translation units compiled with -fmad=false.
#pragma once

#include "fields64.cuh"
#include "tp_launch.h"

namespace tpb {

namespace {

template <int FK>
struct Saver64 {
    const BorisArgs& a;
    int W;
    __device__ Saver64(const BorisArgs& a_)
        : a(a_), W(6 + (a_.save_fields ? 6 : 0) + (a_.save_work ? 4 : 0)) {}
    // slot k of particle i: state, then E and B at (r, t) when save_fields
    // (_prepare_saved_data, boris.jl:405-440); the four work-rate columns of
    // save_work are filled by a post-pass over the saved states
    __device__ __forceinline__ void save(int64_t i, int64_t k, D3 r, D3 v, double t) const {
        if (k >= a.nslots) {
            set_status(a.status, TP_E_OVERFLOW);
            return;
        }
        const int64_t n = a.n;
        a.t_out[k * n + i] = t;
        double* u = a.u_out + (k * W) * n + i;
        u[0 * n] = r.x;
        u[1 * n] = r.y;
        u[2 * n] = r.z;
        u[3 * n] = v.x;
        u[4 * n] = v.y;
        u[5 * n] = v.z;
        if (a.save_fields) {
            D3 E, B;
            eval_EB64t<FK>(a.f, r, t, E, B);
            u[6 * n] = E.x;
            u[7 * n] = E.y;
            u[8 * n] = E.z;
            u[9 * n] = B.x;
            u[10 * n] = B.y;
            u[11 * n] = B.z;
        }
    }
};

template <bool QUEUE>
__device__ __forceinline__ int64_t next_particle(const BorisArgs& a, int64_t& first) {
    if (!QUEUE) {
        int64_t g = first;
        first = a.n;  // static: one particle per thread
        return take_particle(a, g);
    }
    return take_particle(a, (int64_t)atomicAdd(a.queue, 1ULL));
}

}  // namespace

}  // namespace tpb
