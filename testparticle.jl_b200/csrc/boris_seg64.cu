// boris_seg64.cu -- float64 push in the two analytic field configurations that
// have kernels of their own (seg_common.cuh), compiled with -fmad=false: E zero
// and B a dipole (fixed steps, and adaptive steps with the plain Boris update),
// or both fields uniform (fixed steps).
//
// Measured on the device, against k_fixed64: dipole, MultistepBoris4(2), 1e6
// protons x 1000 steps 31.7 -> 16.9 ms (447 instead of 733 warp instructions
// per step, 244 instead of 358 of them on the float64 pipe, which is 72 %
// busy: that pipe is the bound); uniform field, Boris, 1000 protons x 1e4
// steps 13.5 -> 0.85 ms (one warp per sub-partition: the bound is the chain
// of dependent operations, 166 cycles per step); dipole, AdaptiveBoris(0.1), 300001 protons
// of at most 1000 steps 7.53 -> 4.25 ms.
#include "boris64_common.cuh"
#include "seg_common.cuh"

namespace tpb {

// one update of length dt at (r, v) through the general functions: the half
// steps at the start, the saves and the end, and out-of-range denominators
template <bool MULTI>
static __device__ __noinline__ D3 kick_general64(const BorisArgs& a, D3 r, D3 v, double dt) {
    const D3 E = analytic_eval64(a.f.E, r, 0.0), B = analytic_eval64(a.f.B, r, 0.0);
    return vel_update64<MULTI>(v, E, B, a.q2m, dt, a.order, a.nsub);
}

template <bool MULTI>
struct Push64 {
    using Pos = D3;
    using V = D3;
    using Saver = Saver64<FK_ANALYTIC>;
    static __device__ __forceinline__ void init(const BorisArgs&, D3& r, D3& v, const double* u0) {
        r = {u0[0], u0[1], u0[2]};
        v = {u0[3], u0[4], u0[5]};
    }
    static __device__ __forceinline__ void save_first(const BorisArgs& a, const Saver& S, int64_t i, D3 r, D3 v) {
        S.save(i, 0, r, v, a.t0);
    }
    static __device__ __forceinline__ D3 general(const BorisArgs& a, D3 r, D3 v, double dt) {
        return kick_general64<MULTI>(a, r, v, dt);
    }
    template <class F>
    static __device__ __forceinline__ D3 refused(const BorisArgs& a, D3 r, D3 v, const F&, double dt) {
        return kick_general64<MULTI>(a, r, v, dt);
    }
    struct F {};
    static constexpr bool kWarp = false, kJoin = MULTI;
    static __device__ __forceinline__ F fields(const BorisArgs&, D3) { return {}; }
    static __device__ __forceinline__ D3 advance(const BorisArgs&, D3 r, D3 v, double dt) { return r + v * dt; }
    static __device__ __forceinline__ bool outside(const BorisArgs& a, D3 r, D3 v, double t) {
        return outside64(a.term, r, v, t);
    }
};

template <bool MULTI, int ORD>
struct DipolePush64 : Push64<MULTI> {
    // register cap: 640 threads (96 registers, five 128-thread blocks per SM)
    // 16.9 ms on the ensemble above; 512: 17.6, 768: 17.1, 1024: 17.1
    static constexpr int kBound = 640;
    // adaptive, 300001 protons, at most 1000 steps: 512 4.27 ms, 640 4.33, 768 4.55
    static constexpr int kAdaptiveBound = 512;
    double h;
    __device__ __forceinline__ void start(const BorisArgs& a, double dt) {
        h = MULTI ? a.q2m * dt / (double)(2 * a.nsub) : a.q2m * 0.5 * dt;
    }
    struct F {
        D3 B;
        bool ok;
    };
    static __device__ __forceinline__ F fields(const BorisArgs& a, D3 r) {
        F f;
        f.ok = dipole_fast64(a.f.B, r, f.B);
        return f;
    }
    __device__ __forceinline__ bool fast(const BorisArgs& a, D3 v, const F& f, double hh, D3& out) const {
        return f.ok && (MULTI ? multistep_fast64<ORD>(v, f.B, hh, a.nsub, out) : boris_fast64(v, f.B, hh, out));
    }
    __device__ __forceinline__ bool kick(const BorisArgs& a, D3, D3 v, const F& f, D3& out) const {
        return fast(a, v, f, h, out);
    }
    // half the factor is the factor of half the step, exactly
    __device__ __forceinline__ D3 update(const BorisArgs& a, D3 r, D3 v, const F& f, double x, bool half) const {
        D3 out;
        double hh = 0.5 * h;
        if (!half) hh = MULTI ? a.q2m * x / (double)(2 * a.nsub) : a.q2m * 0.5 * x;
        return fast(a, v, f, hh, out) ? out : kick_general64<MULTI>(a, r, v, x);
    }
    // adaptive steps
    using Bv = D3;
    static __device__ __forceinline__ bool field(const BorisArgs& a, D3 r, D3& B) { return dipole_fast64(a.f.B, r, B); }
    static __device__ __forceinline__ D3 field_general(const BorisArgs& a, D3 r) {
        return analytic_eval64(a.f.B, r, 0.0);
    }
    static __device__ __forceinline__ bool kick_dt(const BorisArgs& a, D3 v, D3 B, double dt, D3& out) {
        return boris_fast64(v, B, a.q2m * 0.5 * dt, out);
    }
    // C / |B|
    static __device__ __forceinline__ bool length(double C, D3 B, double& dt) {
        const double b2 = abs2sum(B);
        if (!in_range64(b2)) return false;
        const double y = rsqrt64(b2);
        dt = quot64(C, rec64(sqrt64(b2, y), y));
        return true;
    }
    static __device__ __forceinline__ double length_general(double C, D3 B) { return C / norm(B); }
};

// In uniform fields the rotation of a step depends on dt alone, so it is
// formed once per particle.  A step is then a chain of 8 dependent float64
// operations (Boris), without a division.
template <bool MULTI>
struct UniformPush64;

template <>
struct UniformPush64<false> : Push64<false> {
    static constexpr int kBound = TPB_MAXT(FK_ANALYTIC);
    D3 t, s, he;
    D3 s2;  // s of half a step, whose t and he are half of these
    __device__ __forceinline__ void start(const BorisArgs& a, double dt) {
        const D3 z{0.0, 0.0, 0.0};
        const double h = a.q2m * 0.5 * dt;
        t = h * analytic_eval64(a.f.B, z, 0.0);
        s = (2.0 * t) / (1.0 + abs2sum(t));
        s2 = t / (1.0 + abs2sum(0.5 * t));
        he = h * analytic_eval64(a.f.E, z, 0.0);
    }
    __device__ __forceinline__ bool kick(const BorisArgs&, D3, D3 v, F, D3& out) const {
        out = rotate(v, t, s, he);
        return true;
    }
    __device__ __forceinline__ D3 update(const BorisArgs& a, D3 r, D3 v, F, double x, bool half) const {
        return half ? rotate(v, 0.5 * t, s2, 0.5 * he) : kick_general64<false>(a, r, v, x);
    }
    static __device__ __forceinline__ D3 rotate(D3 v, D3 t, D3 s, D3 he) {
        const D3 vm = v + he;
        const D3 vp = vm + cross(vm, t);
        return (vm + cross(vp, s)) + he;
    }
};

template <>
struct UniformPush64<true> : Push64<true> {
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
    static __device__ __forceinline__ D3 update(const BorisArgs& a, D3 r, D3 v, F, double x, bool) {
        return kick_general64<true>(a, r, v, x);
    }
    __device__ __forceinline__ bool kick(const BorisArgs&, D3, D3 v, F, D3& out) const {
        out = m.c1 * v + m.c2 * cross(v, m.t);
        out = out + (m.c3 * dot(v, m.t)) * m.t;
        out = ((out + e1) + e2) + e3;
        return true;
    }
};

template <bool MULTI, bool QUEUE>
static const void* seg_ptr64(const BorisArgs& a) {
    if (kernel_config_of(a.f) == FK_UNIFORM) return (const void*)k_seg<QUEUE, UniformPush64<MULTI>>;
    if constexpr (MULTI) {
        if (a.order == 4) return (const void*)k_seg<QUEUE, DipolePush64<true, 4>>;
        if (a.order == 6) return (const void*)k_seg<QUEUE, DipolePush64<true, 6>>;
    }
    return (const void*)k_seg<QUEUE, DipolePush64<MULTI, 2>>;
}

const void* seg_kernel64(const BorisArgs& a, bool queue) {
    if (a.alg == TP_ALG_ADAPTIVE)
        return queue ? (const void*)k_aseg<true, DipolePush64<false, 2>> : (const void*)k_aseg<false, DipolePush64<false, 2>>;
    if (a.alg == TP_ALG_MULTISTEP) return queue ? seg_ptr64<true, true>(a) : seg_ptr64<true, false>(a);
    return queue ? seg_ptr64<false, true>(a) : seg_ptr64<false, false>(a);
}

}  // namespace tpb
