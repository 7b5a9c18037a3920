// boris_seg32.cu -- FP32C push in the two analytic field configurations that
// have kernels of their own (seg_common.cuh): E zero and B a dipole (fixed steps,
// and adaptive steps with the plain Boris update), or both fields uniform (fixed
// steps).  The arithmetic is that of Vel32<FK_ANALYTIC> (fp32c_common.cuh), with
// the field kind, the Multistep order and the absence of E known at compile time.
//
// Measured on the device against the general kernels, dipole, 1e6 protons x 1000
// steps: MultistepBoris4(2) 12.44 -> 9.03 ms, Boris 10.93 -> 7.73 ms; 300001
// protons with AdaptiveBoris(0.1) of at most 1000 steps 4.81 -> 4.04 ms.  A
// Multistep step is 253 warp instructions (341 before): 88 on the float64 pipe,
// 70 FMA, 43 ALU, 24 XU (float <-> float64 conversions); issue is 69 % busy,
// the float64 and XU pipes about half, so issue and latency bound it.
#include "boris32_common.cuh"
#include "seg_common.cuh"

namespace tpb {

// one update of length dt at (p, v) through the general functions
template <bool MULTI>
static __device__ __noinline__ D3 kick_general32(const BorisArgs& a, CPos p, D3 v, double dt) {
    const D3 E = analytic_eval_mixed(a.f.E, p, 0.0), B = analytic_eval_mixed(a.f.B, p, 0.0);
    return vel_mixed<MULTI>(v, E, B, a, dt);
}

template <bool MULTI>
struct Push32 {
    using Pos = CPos;
    using V = D3;
    using Saver = Saver32<FK_ANALYTIC>;
    static __device__ __forceinline__ void init(const BorisArgs& a, CPos& p, D3& v, const double* u0) {
        cpos_init(a, p, u0);
        v = {u0[3], u0[4], u0[5]};
    }
    static __device__ __forceinline__ void save_first(const BorisArgs& a, const Saver&, int64_t i, const CPos& p, D3) {
        save_first32<FK_ANALYTIC>(a, i, p);
    }
    static __device__ __forceinline__ D3 general(const BorisArgs& a, const CPos& p, D3 v, double dt) {
        return kick_general32<MULTI>(a, p, v, dt);
    }
    template <class F>
    static __device__ __forceinline__ D3 refused(const BorisArgs&, const CPos&, D3 v, const F&, double) { return v; }  // kick never refuses
    struct F {};
    static constexpr bool kWarp = false, kJoin = MULTI;
    static __device__ __forceinline__ F fields(const BorisArgs&, const CPos&) { return {}; }
    static __device__ __forceinline__ CPos advance(const BorisArgs& a, CPos p, D3 v, double dt) {
        cpos_push_d(a, p, v, dt);
        return p;
    }
    static __device__ __forceinline__ bool outside(const BorisArgs& a, const CPos& p, D3 v, double t) {
        return outside32<FK_ANALYTIC>(a, p, v, t);
    }
};

template <bool MULTI, int ORD>
struct DipolePush32 : Push32<MULTI> {
    // register caps (threads), on the ensembles above.  Multistep: 640 9.55 ms, 768 9.30,
    // 896 9.03, 1024 9.24; Boris: 512 8.67, 640 8.14, 768 8.05, 1024 7.73; adaptive:
    // 512 4.06, 640 4.04, 768 4.38, 1024 4.30
    static constexpr int kBound = MULTI ? 896 : 1024;
    static constexpr int kAdaptiveBound = 640;
    double h;
    __device__ __forceinline__ void start(const BorisArgs& a, double dt) {
        h = MULTI ? a.q2m * dt / (double)(2 * a.nsub) : a.q2m * 0.5 * dt;
    }
    using F = D3;  // B
    static __device__ __forceinline__ D3 fields(const BorisArgs& a, const CPos& p) { return dipole_mixed(a.f.B, p); }
    __device__ __forceinline__ D3 rotate(const BorisArgs& a, D3 v, D3 B, double hh) const {
        return rot_mixed(v, D3{0.0, 0.0, 0.0}, B, hh, ORD, MULTI ? a.nsub : 1, false);
    }
    __device__ __forceinline__ bool kick(const BorisArgs& a, const CPos&, D3 v, D3 B, D3& out) const {
        out = rotate(a, v, B, h);
        return true;
    }
    // half the factor is the factor of half the step, exactly
    __device__ __forceinline__ D3 update(const BorisArgs& a, const CPos& p, D3 v, D3 B, double x, bool half) const {
        return half ? rotate(a, v, B, 0.5 * h) : kick_general32<MULTI>(a, p, v, x);
    }
    // adaptive steps
    using Bv = D3;
    static __device__ __forceinline__ bool field(const BorisArgs& a, const CPos& p, D3& B) {
        B = dipole_mixed(a.f.B, p);
        return true;
    }
    static __device__ __forceinline__ D3 field_general(const BorisArgs& a, const CPos& p) { return dipole_mixed(a.f.B, p); }
    static __device__ __forceinline__ bool kick_dt(const BorisArgs& a, D3 v, D3 B, double dt, D3& out) {
        out = rot_mixed(v, D3{0.0, 0.0, 0.0}, B, a.q2m * 0.5 * dt, 2, 1, false);
        return true;
    }
    // C / |B|
    static __device__ __forceinline__ bool length(double C, D3 B, double& dt) {
        const double b2 = dot(B, B);
        if (!in_range64(b2)) return false;
        const double y = rsqrt64(b2);
        dt = quot64(C, rec64(sqrt64(b2, y), y));
        return true;
    }
    static __device__ __forceinline__ double length_general(double C, D3 B) { return C / sqrt(dot(B, B)); }
};

// in uniform fields the rotation of a step depends on dt alone
template <bool MULTI>
struct UniformPush32 : Push32<MULTI> {
    static constexpr bool kJoin = true;
    static constexpr int kBound = TPB_MAXT(FK_ANALYTIC);
    RotMixed m;
    __device__ __forceinline__ void start(const BorisArgs& a, double dt) {
        const CPos z{};
        const bool hasE = a.f.E.kind != TP_FIELD_ZERO;
        const D3 E = analytic_eval_mixed(a.f.E, z, 0.0), B = analytic_eval_mixed(a.f.B, z, 0.0);
        m = MULTI ? rotation_mixed(E, B, a.q2m * dt / (double)(2 * a.nsub), a.order, a.nsub, hasE)
                  : rotation_mixed(E, B, a.q2m * 0.5 * dt, 2, 1, hasE);
    }
    __device__ __forceinline__ bool kick(const BorisArgs& a, const CPos&, D3 v, typename Push32<MULTI>::F, D3& out) const {
        out = rotate_mixed(v, m, a.f.E.kind != TP_FIELD_ZERO);
        return true;
    }
    static __device__ __forceinline__ D3 update(const BorisArgs& a, const CPos& p, D3 v, typename Push32<MULTI>::F, double x, bool) {
        return kick_general32<MULTI>(a, p, v, x);
    }
};

template <bool MULTI, bool QUEUE>
static const void* seg_ptr32(const BorisArgs& a) {
    if (kernel_config_of(a.f) == FK_UNIFORM) return (const void*)k_seg<QUEUE, UniformPush32<MULTI>>;
    if constexpr (MULTI) {
        if (a.order == 4) return (const void*)k_seg<QUEUE, DipolePush32<true, 4>>;
        if (a.order == 6) return (const void*)k_seg<QUEUE, DipolePush32<true, 6>>;
    }
    return (const void*)k_seg<QUEUE, DipolePush32<MULTI, 2>>;
}

const void* seg_kernel32(const BorisArgs& a, bool queue) {
    if (a.alg == TP_ALG_ADAPTIVE)
        return queue ? (const void*)k_aseg<true, DipolePush32<false, 2>> : (const void*)k_aseg<false, DipolePush32<false, 2>>;
    if (a.alg == TP_ALG_MULTISTEP) return queue ? seg_ptr32<true, true>(a) : seg_ptr32<true, false>(a);
    return queue ? seg_ptr32<false, true>(a) : seg_ptr32<false, false>(a);
}

}  // namespace tpb
