// seg_common.cuh -- the fixed-step and adaptive drivers of the field
// configurations that have kernels of their own: E zero and B a dipole, both
// fields uniform, and (fixed steps) E and B on one trilinear grid.  Instantiated
// by boris_seg64.cu (float64) and boris_seg32.cu (FP32C) with the arithmetic as a
// policy.
//
// The general kernels (k_fixed*, k_adaptive*) decide after every step whether a
// save, the end, the time budget or a refill is due, and evaluate whatever
// field kind they find.  Here the warp agrees on a number of steps in which
// nothing but a step and its termination test can happen, at most kSegSteps,
// and runs them in a loop that holds the step alone.  Steps that save, and
// steps the policy's fast functions refuse, are taken outside that loop, so it
// holds no call and spills nothing (with the calls inside, 30 local-memory
// instructions per step made the float64 dipole kernel 40 % slower).  A lane
// that terminates inside a segment waits for its end, which kSegSteps bounds.
//
// A policy PUSH has
//   Pos, V, Saver, kBound          state, saver and register cap (threads)
//   init(a, p, v, u0)              state of a particle
//   save_first(a, S, i, p, v)      save slot 0 (the initial state)
//   start(a, dt)                   per-particle constants of a step of length dt
//   F, fields(a, p)                what a lane evaluates alone at p (may be empty)
//   kWarp, gather(a, p)            or what the whole warp evaluates together
//   kick(a, p, v, F, out)          velocity after that step; false: refused
//   update(a, p, v, F, x, half)    one update of length x with those fields; `half`: x is
//                                  half of start's dt
//   refused(a, p, v, F, dt)        the update of a step that kick refused
//   kJoin                          saves make theirs together with the lanes that start or
//                                  end: cheaper where update is long (uniform fields, FP32C
//                                  Multistep, 500000 protons with uneven ends, saves every
//                                  20: 2.37 -> 1.97 ms) and 9 % slower where it is short
//   advance(a, p, v, dt)           position after the step
//   outside(a, p, v, t)            termination predicate
// and, for the adaptive driver,
//   Bv, field(a, p, B), kick_dt(a, v, B, dt, out), length(C, B, dt) (false: refused),
//   field_general(a, p), length_general(C, B), general(a, p, v, dt).
#pragma once

#include "tp_device.cuh"

namespace tpb {

template <bool QUEUE>
__device__ __forceinline__ int64_t seg_next(const BorisArgs& a, int64_t& first) {
    if (QUEUE) return take_particle(a, (int64_t)atomicAdd(a.queue, 1ULL));
    const int64_t g = first;
    first = a.n;  // static: one particle per thread
    return take_particle(a, g);
}

constexpr int kSegSteps = 64;

// TERM = false: the run has no termination predicate
template <bool QUEUE, class PUSH, bool TERM = true>
__global__ void __launch_bounds__(PUSH::kBound, 1) k_seg(const __grid_constant__ BorisArgs a) {
    const typename PUSH::Saver S(a);
    const uint64_t t_start = globaltimer_ns();
    const unsigned full = 0xffffffffu;
    int64_t first = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    bool more = true, slow = false, done = false;

    int64_t i = -1;  // the lane's particle
    typename PUSH::Pos r{};
    typename PUSH::V v{};
    PUSH push{};
    double dt = 0, t = 0, t1 = 0, t_last = 0;
    int64_t it = 1, nt = 0, csave = 0;  // csave = (it - 1) % ssi
    int32_t nout = 0, iout = 0, segs = 0;

    for (;;) {
        if (i >= 0 && (++segs & 15) == 0 && globaltimer_ns() - t_start > a.budget_ns) {
            set_status(a.status, TP_E_TIMEOUT);
            done = true;
        }
        bool start = false;
        if (i < 0 && more) {
            // ---- set-up: _boris_single (boris.jl:480-514)
            i = seg_next<QUEUE>(a, first);
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
                    PUSH::init(a, r, v, a.u0 + 6 * i);
                    iout = 0;
                    if (a.save_start) {
                        PUSH::save_first(a, S, i, r, v);
                        t_last = a.t0;
                        iout = 1;
                    }
                    push.start(a, dt);
                    it = 1;
                    t = a.t0 - 0.5 * dt;
                    csave = 0;
                    slow = false;
                    done = nt < 1;
                    start = true;
                }
            }
        }
        // ---- the pass of everything but a plain step: the first half step, a save, the
        // final save, a step that the fast functions refused.  The lanes that need none
        // of it take a step in the same pass, so that lanes out of phase (refilled by the
        // queue) do not wait for one another.  Measured with ends at different steps, 400000
        // protons x 200 steps on an E/B grid, MultistepBoris4(2), saves every 20: float64
        // k_fixed64 12.5 ms, with the other lanes idle in this pass 15.0, so 5.7; FP32C
        // 5.6, 6.3 and 4.1.
        const bool save = i >= 0 && !done && a.save_everystep && it > 1 && csave == 0;
        if (__any_sync(full, start || save || slow || done)) {
            typename PUSH::F f;
            if constexpr (PUSH::kWarp) f = PUSH::gather(a, r);
            if (i >= 0) {
                if constexpr (!PUSH::kWarp) f = PUSH::fields(a, r);
                typename PUSH::V vx = v;
                if (start || done || (PUSH::kJoin && save)) {
                    double x = 0.5 * dt, t_final = 0.0;
                    bool last = false;
                    const int64_t final_step = it - 1;
                    if (start) {
                        x = -0.5 * dt;
                    } else if (done && iout < nout &&
                               (a.save_end || (a.save_everystep && final_step > 0 && final_step % a.ssi == 0))) {
                        // final save (boris.jl:522-551)
                        t_final = (final_step == nt) ? t1 : fma((double)final_step, dt, a.t0);
                        last = iout == 0 || t_last < t_final;
                        x = t_final - fma((double)final_step - 0.5, dt, a.t0);
                    }
                    if (start || last || (PUSH::kJoin && save)) vx = push.update(a, r, v, f, x, PUSH::kJoin && save);
                    if (start) {
                        v = vx;
                    } else if (done) {
                        if (last) {
                            S.save(i, iout, r, vx, t_final);
                            iout += 1;
                        }
                        a.nsaved[i] = (int32_t)iout;
                        a.retcode[i] = (int8_t)((iout < nout) ? TP_RET_TERMINATED : TP_RET_SUCCESS);
                        a.nsteps[i] = final_step;
                        particle_done(a, i);
                        i = -1;
                        done = false;
                    }
                }
                if (i >= 0 && !done) {
                    const double tn = t + dt;
                    typename PUSH::V vn;
                    if (!push.kick(a, r, v, f, vn)) vn = PUSH::refused(a, r, v, f, dt);
                    const typename PUSH::Pos rn = push.advance(a, r, vn, dt);
                    if (TERM && a.term.flags && PUSH::outside(a, rn, vn, tn + 0.5 * dt)) {
                        done = true;
                    } else {
                        if (save) {
                            iout += 1;
                            if (iout <= nout) {
                                t_last = tn - 0.5 * dt;
                                if (!PUSH::kJoin) vx = push.update(a, r, v, f, 0.5 * dt, true);
                                S.save(i, iout - 1, r, vx, t_last);
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
                slow = false;
            }
        }
        const bool again = i >= 0 ? done || (a.save_everystep && it > 1 && csave == 0) : more;
        if (__any_sync(full, again)) continue;
        // ---- the steps before any lane has something else to do: the next
        // save step is it + k with csave + k = ssi
        bool go = i >= 0;
        int len = kSegSteps;
        if (go) {
            int64_t left = nt - it + 1;
            if (a.save_everystep && a.ssi - csave < left) left = a.ssi - csave;
            if (left < len) len = (int)left;
        }
        len = __reduce_min_sync(full, len);
        if (!__any_sync(full, go)) break;
        // ---- steps of _boris_loop! (boris.jl:452-476); v stays the pre-step
        // velocity (the reference's v_prev) until the step is accepted, which
        // serves the termination rollback
        int taken = 0;
        for (int k = 0; k < len; ++k) {
            typename PUSH::F f;
            if constexpr (PUSH::kWarp) f = PUSH::gather(a, r);
            if (!go) continue;
            if constexpr (!PUSH::kWarp) f = PUSH::fields(a, r);
            const double tn = t + dt;
            typename PUSH::V vn;
            if (!push.kick(a, r, v, f, vn)) {
                slow = true;
                go = false;
                continue;
            }
            const typename PUSH::Pos rn = push.advance(a, r, vn, dt);
            if (TERM && a.term.flags && PUSH::outside(a, rn, vn, tn + 0.5 * dt)) {
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
    }
}

// _adaptive_boris_single (adaptive_boris.jl:145-266).  `fresh`: the state was
// reached by a step (or is the first), so clipping and saving are still due;
// a step taken inside a segment that makes either due ends the lane's segment.
template <bool QUEUE, class PUSH>
__global__ void __launch_bounds__(PUSH::kAdaptiveBound, 1) k_aseg(const __grid_constant__ BorisArgs a) {
    const typename PUSH::Saver S(a);
    const uint64_t t_start = globaltimer_ns();
    int64_t first = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const double twopi = 6.283185307179586;
    bool more = true, slow = false, fresh = false, ssf = false;

    int64_t i = -1;
    typename PUSH::Pos r{};
    typename PUSH::V v{};
    typename PUSH::Bv B{};
    double t = 0, t1 = 0, dt = 0, C = 0, ttotal = 0, t_last = 0;
    int64_t steps = 0, csave = 0, iout = 0;  // csave = steps % ssi
    int32_t segs = 0;
    int ret = TP_RET_SUCCESS;

    for (;;) {
        if (i < 0 && more) {
            // ---- set-up (adaptive_boris.jl:149-196)
            i = seg_next<QUEUE>(a, first);
            if (i >= a.n) {
                more = false;
                i = -1;
            } else {
                t1 = a.tend_i ? a.tend_i[i] : a.t1;
                ttotal = t1 - a.t0;
                const double sgn = ttotal > 0 ? 1.0 : (ttotal < 0 ? -1.0 : 0.0);
                C = (twopi * a.safety * sgn) / fabs(a.q2m);
                PUSH::init(a, r, v, a.u0 + 6 * i);
                t = a.t0;
                iout = 0;
                if (a.save_start) {
                    PUSH::save_first(a, S, i, r, v);
                    t_last = t;
                    iout = 1;
                }
                B = PUSH::field_general(a, r);
                dt = PUSH::length_general(C, B);
                v = PUSH::general(a, r, v, -0.5 * dt);
                steps = csave = 0;
                fresh = true;
                slow = false;
                ssf = a.save_end;
                ret = TP_RET_SUCCESS;
            }
        }
        bool done = false;
        if (i >= 0) {
            done = !(fabs(t - a.t0) < fabs(ttotal));
            if (!done && a.step_cap > 0 && steps >= a.step_cap) {
                ret = TP_RET_MAXITERS;
                done = true;
            }
            if (!done && fresh) {
                fresh = false;
                if (fabs(t + dt - a.t0) > fabs(ttotal)) {
                    const double dt_step = t1 - t;
                    v = PUSH::general(a, r, v, 0.5 * dt);
                    v = PUSH::general(a, r, v, -0.5 * dt_step);
                    dt = dt_step;
                }
                if (a.save_everystep && steps > 0 && csave == 0) {
                    typename PUSH::V vs;
                    if (!PUSH::kick_dt(a, v, B, 0.5 * dt, vs)) vs = PUSH::general(a, r, v, 0.5 * dt);
                    S.save(i, iout, r, vs, t);
                    t_last = t;
                    iout += 1;
                }
            }
            // ---- a step that the fast functions refused
            if (!done && slow) {
                slow = false;
                typename PUSH::V vn = PUSH::general(a, r, v, dt);
                const typename PUSH::Pos rn = PUSH::advance(a, r, vn, dt);
                if (a.term.flags && PUSH::outside(a, rn, vn, t + dt)) {
                    ssf = true;
                    ret = TP_RET_TERMINATED;
                    done = true;
                } else {
                    r = rn;
                    t = t + dt;
                    B = PUSH::field_general(a, r);
                    const double dt_new = PUSH::length_general(C, B);
                    vn = PUSH::general(a, r, vn, 0.5 * dt);
                    v = PUSH::general(a, r, vn, -0.5 * dt_new);
                    dt = dt_new;
                    steps += 1;
                    csave = csave + 1 == a.ssi ? 0 : csave + 1;
                    if (a.save_everystep && csave == 0) ssf = true;
                    fresh = true;
                }
            }
        }
        bool go = i >= 0 && !done && !fresh;
        int len = kSegSteps;
        if (go) {
            int64_t left = len;
            if (a.step_cap > 0 && a.step_cap - steps < left) left = a.step_cap - steps;
            if (a.save_everystep && a.ssi - csave < left) left = a.ssi - csave;
            len = (int)left;
        } else if (i >= 0) {
            len = 0;
        }
        len = __reduce_min_sync(0xffffffffu, len);
        if (!__any_sync(0xffffffffu, i >= 0)) {
            if (!__any_sync(0xffffffffu, more)) break;
            continue;
        }
        // ---- iterations of the while loop (adaptive_boris.jl:197-248)
        int taken = 0;
        for (int k = 0; k < len; ++k) {
            if (!go) continue;
            typename PUSH::V vn, vh;
            if (!PUSH::kick_dt(a, v, B, dt, vn)) {
                slow = true;
                go = false;
                continue;
            }
            const typename PUSH::Pos rn = PUSH::advance(a, r, vn, dt);
            const double tn = t + dt;
            if (a.term.flags && PUSH::outside(a, rn, vn, tn)) {
                ssf = true;
                ret = TP_RET_TERMINATED;
                done = true;
                go = false;
                continue;
            }
            typename PUSH::Bv Bn;
            double dt_new;
            if (!(PUSH::field(a, rn, Bn) && PUSH::length(C, Bn, dt_new) && PUSH::kick_dt(a, vn, Bn, 0.5 * dt, vh) &&
                  PUSH::kick_dt(a, vh, Bn, -0.5 * dt_new, vn))) {
                slow = true;
                go = false;
                continue;
            }
            r = rn;
            v = vn;
            B = Bn;
            t = tn;
            dt = dt_new;
            taken = k + 1;
            fresh = true;
            // at its end, or the next step is clipped to it
            if (!(fabs(t - a.t0) < fabs(ttotal)) || fabs(t + dt - a.t0) > fabs(ttotal)) go = false;
        }
        steps += taken;
        csave += taken;
        if (csave == a.ssi) csave = 0;
        if (a.save_everystep && taken > 0 && csave == 0) ssf = true;
        if (i >= 0 && !done && (++segs & 15) == 0 && globaltimer_ns() - t_start > a.budget_ns) {
            set_status(a.status, TP_E_TIMEOUT);
            ret = TP_RET_DEFAULT;
            done = true;
        }
        if (done) {
            // ---- final save (adaptive_boris.jl:250-259)
            if (ssf && (iout == 0 || t_last != t)) {
                S.save(i, iout, r, PUSH::general(a, r, v, 0.5 * dt), t);
                iout += 1;
            }
            a.nsaved[i] = (int32_t)iout;
            a.retcode[i] = (int8_t)ret;
            a.nsteps[i] = steps;
            particle_done(a, i);
            i = -1;
        }
    }
}

}  // namespace tpb
