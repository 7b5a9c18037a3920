// boris_seg64.cu -- float64 fixed-step push in the two analytic field
// configurations that have kernels of their own (compiled with -fmad=false):
// E zero and B a dipole, or both fields uniform.
//
// k_fixed64 decides after every step whether a save, the end, the time budget
// or a refill is due, and evaluates whatever field kind it finds.  With E zero
// and B a dipole, or both fields uniform, k_seg64 takes its place: the warp
// agrees on a number of steps in which nothing but a step (and its termination
// test) can happen, at most kSegSteps, and runs them in a loop that holds the
// step alone.  Steps that save, and steps the fast functions refuse, are taken
// outside that loop, so it holds no call and spills nothing (with the calls
// inside, 30 local-memory instructions per step made the dipole kernel 40 %
// slower).  A lane that terminates inside a segment waits for its end, which
// kSegSteps bounds.
//
// Measured on the device, against k_fixed64: dipole, MultistepBoris4(2), 1e6
// protons x 1000 steps 31.7 -> 16.9 ms (443 instead of 733 warp instructions
// per step, 243 instead of 358 of them on the float64 pipe, which is 71 %
// busy: that pipe is the bound); uniform field, Boris, 1000 protons x 1e4
// steps 13.5 -> 0.85 ms (one warp per sub-partition: the bound is the chain
// of dependent operations, 166 cycles per step).
#include "boris64_common.cuh"

namespace tpb {

// one update of length dt at (r, v) through the general functions: the half
// steps at the start, the saves and the end, and out-of-range denominators
template <bool MULTI>
static __device__ __noinline__ D3 kick_general64(const BorisArgs& a, D3 r, D3 v, double dt) {
    const D3 E = analytic_eval64(a.f.E, r, 0.0), B = analytic_eval64(a.f.B, r, 0.0);
    return vel_update64<MULTI>(v, E, B, a.q2m, dt, a.order, a.nsub);
}

template <bool MULTI, int ORD>
struct DipolePush64 {
    // register cap: 640 threads (96 registers, five 128-thread blocks per SM)
    // 16.9 ms on the ensemble above; 512: 17.6, 768: 17.1, 1024: 17.1
    static constexpr int kBound = 640;
    double h;
    __device__ __forceinline__ void start(const BorisArgs& a, double dt) {
        h = MULTI ? a.q2m * dt / (double)(2 * a.nsub) : a.q2m * 0.5 * dt;
    }
    __device__ __forceinline__ bool kick(const BorisArgs& a, D3 r, D3 v, D3& out) const {
        D3 B;
        return dipole_fast64(a.f.B, r, B) &&
               (MULTI ? multistep_fast64<ORD>(v, B, h, a.nsub, out) : boris_fast64(v, B, h, out));
    }
};

// In uniform fields the rotation of a step depends on dt alone, so it is
// formed once per particle.  A step is then a chain of 8 dependent float64
// operations (Boris), without a division.
template <bool MULTI>
struct UniformPush64;

template <>
struct UniformPush64<false> {
    static constexpr int kBound = TPB_MAXT(FK_ANALYTIC);
    D3 t, s, he;
    __device__ __forceinline__ void start(const BorisArgs& a, double dt) {
        const D3 z{0.0, 0.0, 0.0};
        const double h = a.q2m * 0.5 * dt;
        t = h * analytic_eval64(a.f.B, z, 0.0);
        s = (2.0 * t) / (1.0 + abs2sum(t));
        he = h * analytic_eval64(a.f.E, z, 0.0);
    }
    __device__ __forceinline__ bool kick(const BorisArgs&, D3, D3 v, D3& out) const {
        const D3 vm = v + he;
        const D3 vp = vm + cross(vm, t);
        out = (vm + cross(vp, s)) + he;
        return true;
    }
};

template <>
struct UniformPush64<true> {
    static constexpr int kBound = TPB_MAXT(FK_ANALYTIC);
    MultistepRot64 m;
    D3 e1, e2, e3;  // the three terms of E
    __device__ __forceinline__ void start(const BorisArgs& a, double dt) {
        const D3 z{0.0, 0.0, 0.0};
        m = multistep_rotation64(analytic_eval64(a.f.E, z, 0.0), analytic_eval64(a.f.B, z, 0.0), a.q2m, dt, a.order,
                                 a.nsub);
        e1 = m.c2 * m.e;
        e2 = m.c3 * cross(m.e, m.t);
        e3 = (m.c6 * dot(m.e, m.t)) * m.t;
    }
    __device__ __forceinline__ bool kick(const BorisArgs&, D3, D3 v, D3& out) const {
        out = m.c1 * v + m.c2 * cross(v, m.t);
        out = out + (m.c3 * dot(v, m.t)) * m.t;
        out = ((out + e1) + e2) + e3;
        return true;
    }
};

constexpr int kSegSteps = 64;

template <bool MULTI, bool QUEUE, class PUSH>
__global__ void __launch_bounds__(PUSH::kBound, 1) k_seg64(const __grid_constant__ BorisArgs a) {
    const Saver64<FK_ANALYTIC> S(a);
    const uint64_t t_start = globaltimer_ns();
    int64_t first = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    bool more = true, slow = false;

    int64_t i = -1;  // the lane's particle
    D3 r{0, 0, 0}, v{0, 0, 0};
    PUSH push{};
    double dt = 0, t = 0, t1 = 0, t_last = 0;
    int64_t it = 1, nt = 0, csave = 0;  // csave = (it - 1) % ssi
    int32_t nout = 0, iout = 0, segs = 0;

    for (;;) {
        if (i < 0 && more) {
            // ---- set-up: _boris_single (boris.jl:480-514)
            i = next_particle<QUEUE>(a, first);
            if (i >= a.n) {
                more = false;
                i = -1;
            } else {
                dt = a.dt_i ? a.dt_i[i] : a.dt;
                t1 = a.tend_i ? a.tend_i[i] : a.t1;
                const bool small = fabs(dt) < 10.0 * 2.220446049250313e-16;
                nt = small ? 0 : jl_round((t1 - a.t0) / dt);
                if (nt < 0) nt = -nt;
                if (small || nt > a.maxiters) {
                    set_status(a.status, TP_E_ARG);
                    a.nsaved[i] = 0;
                    a.retcode[i] = TP_RET_DEFAULT;
                    a.nsteps[i] = 0;
                    particle_done(a, i);
                    i = -1;
                } else {
                    nout = (int32_t)calc_nout(nt, a.ssi, a.save_start, a.save_end, a.save_everystep);
                    const double* u0 = a.u0 + 6 * i;
                    r = {u0[0], u0[1], u0[2]};
                    v = {u0[3], u0[4], u0[5]};
                    iout = 0;
                    if (a.save_start) {
                        S.save(i, 0, r, v, a.t0);
                        t_last = a.t0;
                        iout = 1;
                    }
                    push.start(a, dt);
                    v = kick_general64<MULTI>(a, r, v, -0.5 * dt);
                    it = 1;
                    t = a.t0 - 0.5 * dt;
                    csave = 0;
                }
            }
        }
        bool done = i >= 0 && it > nt;
        // ---- a step that saves, or that the fast functions refused
        if (i >= 0 && !done && (slow || (a.save_everystep && it > 1 && csave == 0))) {
            slow = false;
            const double tn = t + dt;
            D3 vn;
            if (!push.kick(a, r, v, vn)) vn = kick_general64<MULTI>(a, r, v, dt);
            const D3 rn = r + vn * dt;
            if (a.term.flags && outside64(a.term, rn, vn, tn + 0.5 * dt)) {
                done = true;
            } else {
                if (a.save_everystep && it > 1 && csave == 0) {
                    iout += 1;
                    if (iout <= nout) {
                        t_last = tn - 0.5 * dt;
                        S.save(i, iout - 1, r, kick_general64<MULTI>(a, r, v, 0.5 * dt), t_last);
                    }
                }
                r = rn;
                v = vn;
                t = tn;
                it += 1;
                csave = csave + 1 == a.ssi ? 0 : csave + 1;
                done = it > nt;
            }
        }
        // ---- the steps before any lane has something else to do: the next
        // save step is it + k with csave + k = ssi
        bool go = i >= 0 && !done && !(a.save_everystep && it > 1 && csave == 0);
        int len = kSegSteps;
        if (go) {
            int64_t left = nt - it + 1;
            if (a.save_everystep && a.ssi - csave < left) left = a.ssi - csave;
            if (left < len) len = (int)left;
        } else if (i >= 0) {
            len = 0;
        }
        len = __reduce_min_sync(0xffffffffu, len);
        if (!__any_sync(0xffffffffu, i >= 0)) {
            if (!__any_sync(0xffffffffu, more)) break;
            continue;
        }
        // ---- steps of _boris_loop! (boris.jl:452-476); v stays the pre-step
        // velocity (the reference's v_prev) until the step is accepted, which
        // serves the termination rollback
        int taken = 0;
        for (int k = 0; k < len; ++k) {
            if (!go) continue;
            const double tn = t + dt;
            D3 vn;
            if (!push.kick(a, r, v, vn)) {
                slow = true;
                go = false;
                continue;
            }
            const D3 rn = r + vn * dt;
            if (a.term.flags && outside64(a.term, rn, vn, tn + 0.5 * dt)) {
                done = true;
                go = false;
                continue;
            }
            r = rn;
            v = vn;
            t = tn;
            taken = k + 1;
        }
        it += taken;
        csave += taken;
        if (csave == a.ssi) csave = 0;
        if (i >= 0 && it > nt) done = true;
        if (i >= 0 && (++segs & 15) == 0 && globaltimer_ns() - t_start > a.budget_ns) {
            set_status(a.status, TP_E_TIMEOUT);
            done = true;
        }
        if (done) {
            // ---- final save and retcode (boris.jl:522-551)
            const int64_t final_step = it - 1;
            const bool save_final = a.save_end || (a.save_everystep && final_step > 0 && final_step % a.ssi == 0);
            if (iout < nout && save_final) {
                const double t_final = (final_step == nt) ? t1 : fma((double)final_step, dt, a.t0);
                if (iout == 0 || t_last < t_final) {
                    const double dt_final = t_final - fma((double)final_step - 0.5, dt, a.t0);
                    S.save(i, iout, r, kick_general64<MULTI>(a, r, v, dt_final), t_final);
                    iout += 1;
                }
            }
            a.nsaved[i] = (int32_t)iout;
            a.retcode[i] = (int8_t)((iout < nout) ? TP_RET_TERMINATED : TP_RET_SUCCESS);
            a.nsteps[i] = final_step;
            particle_done(a, i);
            i = -1;
        }
    }
}

template <bool MULTI, bool QUEUE>
static const void* seg_ptr64(const BorisArgs& a) {
    if (kernel_config_of(a.f) == FK_UNIFORM) return (const void*)k_seg64<MULTI, QUEUE, UniformPush64<MULTI>>;
    if constexpr (MULTI) {
        if (a.order == 4) return (const void*)k_seg64<true, QUEUE, DipolePush64<true, 4>>;
        if (a.order == 6) return (const void*)k_seg64<true, QUEUE, DipolePush64<true, 6>>;
    }
    return (const void*)k_seg64<MULTI, QUEUE, DipolePush64<MULTI, 2>>;
}

const void* seg_kernel64(const BorisArgs& a, bool queue) {
    if (a.alg == TP_ALG_MULTISTEP) return queue ? seg_ptr64<true, true>(a) : seg_ptr64<true, false>(a);
    return queue ? seg_ptr64<false, true>(a) : seg_ptr64<false, false>(a);
}

}  // namespace tpb
