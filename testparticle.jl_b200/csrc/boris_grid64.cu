// boris_grid64.cu -- float64 fixed-step push with E and B float grids on one
// geometry (trilinear), or with E zero and B alone on a grid, in the segments of
// seg_common.cuh with the stencils gathered by pairs of lanes (pair_gather.cuh).
// Compiled with -fmad=false; the results equal those of eb_eval64_f32, tri64 and
// vel_update64 bit for bit.
//
// Measured on the device, 400009 protons x 250 steps on a 120 x 100 x 91 grid:
// Boris 4.72 -> 2.51 ms, MultistepBoris4(2) 6.42 -> 4.07 ms (Boris 2.79 while the
// particles were still sorted by cell first).  A Boris step is 474 warp
// instructions, 206 on the float64 pipe and 58 on the XU (float to float64
// conversions); L1 is 71 % busy with 5 line look-ups per particle.
//
// B alone, float64 data, 61 x 53 x 47 nodes, 250 steps between absorbing walls:
// 200003 protons, Boris 2.89 -> 1.01 ms, MultistepBoris4(2) 8.81 -> 1.65;
// 400000, Boris 6.33 -> 1.89; 20000 0.47 -> 0.38.  k_fixed64 read a stencil with
// 16 loads of 32 lines each and decided on the field kinds in every step.
#include "boris64_common.cuh"
#include "pair_gather.cuh"
#include "seg_common.cuh"

namespace tpb {

// the axes of the stencil; false outside a grid that is filled with NaN
template <bool PERIODIC>
static __device__ __forceinline__ bool grid_axes_bc(const DevField& g, D3 r, Ax& ax, Ax& ay, Ax& az) {
    if (!PERIODIC) return grid_axes64(g, r, ax, ay, az);
    grid_axis_periodic(g, 0, r.x, ax);
    grid_axis_periodic(g, 1, r.y, ay);
    grid_axis_periodic(g, 2, r.z, az);
    return true;
}

template <bool MULTI, bool PERIODIC>
struct GridPush64 {
    // register cap (threads), 250 Boris steps of the ensemble above, sorted: 384 3.42 ms,
    // 512 3.00, 640 (96 registers) 2.79, 768 3.49, 1024 4.59 (spills in the loop)
    static constexpr int kBound = 640;
    using Pos = D3;
    using V = D3;
    using Saver = Saver64<FK_EBGRID>;
    struct F {
        D3 E, B;
    };
    static constexpr bool kWarp = true, kJoin = MULTI;
    double h;
    static __device__ __forceinline__ void init(const BorisArgs&, D3& r, D3& v, const double* u0) {
        r = {u0[0], u0[1], u0[2]};
        v = {u0[3], u0[4], u0[5]};
    }
    static __device__ __forceinline__ void save_first(const BorisArgs& a, const Saver& S, int64_t i, D3 r, D3 v) {
        S.save(i, 0, r, v, a.t0);
    }
    // Boris: q2m * 0.5 * dt; Multistep: dt itself (the update forms its factor)
    __device__ __forceinline__ void start(const BorisArgs& a, double dt) { h = MULTI ? dt : a.q2m * 0.5 * dt; }
    // eb_eval64_f32 with the stencils of the warp gathered by pairs of lanes
    static __device__ __forceinline__ F gather(const BorisArgs& a, D3 r) {
        const DevField& g = a.f.B;
        Ax ax, ay, az;
        const bool ok = grid_axes_bc<PERIODIC>(g, r, ax, ay, az);
        double c0[6], c1[6];
        pair_planes<double>(a.f.eb32, ok ? eb_node(g, ax.i0, ay.i0, az.i0) : 0, ok ? (ax.i1 - ax.i0) * g.n[1] * g.n[2] : 0,
                            ok ? (ay.i1 - ay.i0) * g.n[2] : 0, ok ? az.i1 - az.i0 : 0, ax.f, ay.f, c0, c1);
        F f;
        f.E = {lerp64(c0[0], c1[0], az.f), lerp64(c0[1], c1[1], az.f), lerp64(c0[2], c1[2], az.f)};
        f.B = {lerp64(c0[3], c1[3], az.f), lerp64(c0[4], c1[4], az.f), lerp64(c0[5], c1[5], az.f)};
        if (!ok) f.E = f.B = nan3();
        return f;
    }
    __device__ __forceinline__ bool kick(const BorisArgs& a, D3, D3 v, const F& f, D3& out) const {
        if (!MULTI) return boris_fast64(v, f.E, f.B, h, out);
        out = multistep_rot64(v, f.E, f.B, a.q2m, h, a.order, a.nsub);
        return true;
    }
    static __device__ __forceinline__ D3 update(const BorisArgs& a, D3, D3 v, const F& f, double x, bool) {
        return vel_update64<MULTI>(v, f.E, f.B, a.q2m, x, a.order, a.nsub);
    }
    static __device__ __forceinline__ D3 refused(const BorisArgs& a, D3 r, D3 v, const F& f, double dt) {
        return update(a, r, v, f, dt, false);
    }
    static __device__ __forceinline__ D3 advance(const BorisArgs&, D3 r, D3 v, double dt) { return r + v * dt; }
    static __device__ __forceinline__ bool outside(const BorisArgs& a, D3 r, D3 v, double t) {
        return outside64(a.term, r, v, t);
    }
};

// E zero, B alone on a grid.  ORD 0: Boris, else the order of the multistep
template <int ORD, bool PERIODIC, class NODE>
struct GridBPush64 : GridPush64<ORD != 0, PERIODIC> {
    static constexpr bool MULTI = ORD != 0;
    // register cap (threads), 400000 protons, 250 Boris steps on a 61 x 53 x 47 float64
    // grid: 384 1.95 ms, 512 1.89, 640 1.99, 768 2.13
    static constexpr int kBound = 512;
    using Saver = Saver64<FK_GENERIC>;
    struct F {
        D3 B;
    };
    double h;
    static __device__ __forceinline__ void save_first(const BorisArgs& a, const Saver& S, int64_t i, D3 r, D3 v) {
        S.save(i, 0, r, v, a.t0);
    }
    __device__ __forceinline__ void start(const BorisArgs& a, double dt) {
        h = MULTI ? a.q2m * dt / (double)(2 * a.nsub) : a.q2m * 0.5 * dt;
    }
    static __device__ __forceinline__ F gather(const BorisArgs& a, D3 r) {
        const DevField& g = a.f.B;
        Ax ax, ay, az;
        const bool ok = grid_axes_bc<PERIODIC>(g, r, ax, ay, az);
        double c0[3], c1[3];
        pair_planes<double, NODE>(g.tab, ok ? eb_node(g, ax.i0, ay.i0, az.i0) : 0, ok ? (ax.i1 - ax.i0) * g.n[1] * g.n[2] : 0,
                                  ok ? (ay.i1 - ay.i0) * g.n[2] : 0, ok ? az.i1 - az.i0 : 0, ax.f, ay.f, c0, c1);
        F f;
        f.B = {lerp64(c0[0], c1[0], az.f), lerp64(c0[1], c1[1], az.f), lerp64(c0[2], c1[2], az.f)};
        if (!ok) f.B = nan3();
        return f;
    }
    __device__ __forceinline__ bool fast(const BorisArgs& a, D3 v, const F& f, double hh, D3& out) const {
        if constexpr (MULTI) return multistep_fast64<ORD>(v, f.B, hh, a.nsub, out);
        else return boris_fast64(v, f.B, hh, out);
    }
    __device__ __forceinline__ bool kick(const BorisArgs& a, D3, D3 v, const F& f, D3& out) const {
        return fast(a, v, f, h, out);
    }
    // half the factor is the factor of half the step, exactly
    __device__ __forceinline__ D3 update(const BorisArgs& a, D3 r, D3 v, const F& f, double x, bool half) const {
        D3 out;
        double hh = 0.5 * h;
        if (!half) hh = MULTI ? a.q2m * x / (double)(2 * a.nsub) : a.q2m * 0.5 * x;
        if (fast(a, v, f, hh, out)) return out;
        return refused(a, r, v, f, x);
    }
    static __device__ __forceinline__ D3 refused(const BorisArgs& a, D3, D3 v, const F& f, double x) {
        return vel_update64<MULTI>(v, {0.0, 0.0, 0.0}, f.B, a.q2m, x, a.order, a.nsub);
    }
};

template <class P>
static const void* seg_ptr(bool queue) {
    return queue ? (const void*)k_seg<true, P> : (const void*)k_seg<false, P>;
}

template <int ORD, class NODE>
static const void* gridb_ptr64(const BorisArgs& a, bool queue) {
    if (a.f.B.bc == TP_BC_PERIODIC) return seg_ptr<GridBPush64<ORD, true, NODE>>(queue);
    return seg_ptr<GridBPush64<ORD, false, NODE>>(queue);
}

template <int ORD>
static const void* gridb_ptr64(const BorisArgs& a, bool queue) {
    return a.f.B.f64 ? gridb_ptr64<ORD, Node64>(a, queue) : gridb_ptr64<ORD, Node32>(a, queue);
}

const void* gridb_kernel64(const BorisArgs& a, bool queue) {
    if (a.alg != TP_ALG_MULTISTEP) return gridb_ptr64<0>(a, queue);
    if (a.order == 4) return gridb_ptr64<4>(a, queue);
    return a.order == 6 ? gridb_ptr64<6>(a, queue) : gridb_ptr64<2>(a, queue);
}

template <bool MULTI, bool PERIODIC>
static const void* grid_ptr64(bool queue) {
    return seg_ptr<GridPush64<MULTI, PERIODIC>>(queue);
}

const void* grid_kernel64(const BorisArgs& a, bool queue) {
    const bool multi = a.alg == TP_ALG_MULTISTEP;
    if (a.f.B.bc == TP_BC_PERIODIC) return multi ? grid_ptr64<true, true>(queue) : grid_ptr64<false, true>(queue);
    return multi ? grid_ptr64<true, false>(queue) : grid_ptr64<false, false>(queue);
}

}  // namespace tpb
