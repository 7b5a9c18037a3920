// boris_grid32.cu -- FP32C fixed-step push with E and B on one trilinear grid, in
// the segments of seg_common.cuh with the stencils gathered by pairs of lanes
// (pair_gather.cuh).  The arithmetic is that of Vel32<FK_EBGRID>.
//
// Measured on the 128^3 turbulent field, 1e6 protons, device time: 250 steps 8.43
// -> 5.37 ms (4.7e10 particle-steps/s), 5.71 while the particles were still sorted by
// cell first.  What bounds it
// is the L1 cache (88 % busy): 5 line look-ups per particle and step, 11 shuffles
// per warp, and the 8 sectors that come from L2.
#include "boris32_common.cuh"
#include "seg_common.cuh"

namespace tpb {

// the contraction of |t|^2 (dot_fma) in the steps, and in the first half step and the
// saves, as k_fixed32c had it: a float rounding that differs in a step or at the
// start grows 1000-fold in 250 steps of the turbulent field
constexpr int kStep = 1, kSave = 2;

template <bool MULTI, bool PERIODIC>
struct GridPush32 {
    // register cap (threads), 250 steps of the ensemble above, sorted: 384 (165 registers)
    // 7.17 ms, 512 6.40, 640 5.99, 768 (80) 5.72, 896 5.78
    static constexpr int kBound = 768;
    using Pos = CPos;
    using V = CV;
    using Saver = Saver32<FK_EBGRID>;
    struct F {
        F3 E, B;
    };
    static constexpr bool kWarp = true;
    float h, dth, dtl;
    static __device__ __forceinline__ void init(const BorisArgs& a, CPos& p, CV& v, const double* u0) {
        cpos_init(a, p, u0);
        v = cv_from(u0 + 3);
    }
    static __device__ __forceinline__ void save_first(const BorisArgs& a, const Saver&, int64_t i, const CPos& p, const CV&) {
        save_first32<FK_EBGRID>(a, i, p);
    }
    __device__ __forceinline__ void start(const BorisArgs& a, double dt) {
        h = vfac<MULTI>(a, dt);
        dth = (float)dt;
        dtl = (float)(dt - (double)dth);
    }
    static __device__ __forceinline__ F gather(const BorisArgs& a, const CPos& p) {
        F f;
        eb_pair_gather32<PERIODIC>(a.f, p, f.E, f.B);
        return f;
    }
    __device__ __forceinline__ bool kick(const BorisArgs& a, const CPos&, const CV& v, const F& f, CV& out) const {
        out = vel32h<MULTI, kStep>(v, f.E, f.B, a, h);
        return true;
    }
    __device__ __forceinline__ CV half(const BorisArgs& a, const CPos&, const CV& v, const F& f, double dt) const {
        return vel32<MULTI, kSave>(v, f.E, f.B, a, 0.5 * dt);
    }
    // one update of length dt at (p, v) by the lane alone
    static __device__ __forceinline__ CV general(const BorisArgs& a, const CPos& p, const CV& v, double dt) {
        AxF ax, ay, az;
        F3 E = nanf3(), B = nanf3();
        if (eb_axes32<PERIODIC>(a.f.B, p, ax, ay, az)) eb_gather32(a.f, ax, ay, az, E, B);
        return vel32<MULTI, kSave>(v, E, B, a, dt);
    }
    __device__ __forceinline__ CPos advance(const BorisArgs& a, CPos p, const CV& v, double) const {
        cpos_push_cv(a, p, v, dth, dtl);
        return p;
    }
    static __device__ __forceinline__ bool outside(const BorisArgs& a, const CPos& p, const CV& v, double t) {
        return outside32<FK_EBGRID>(a, p, v, t);
    }
};

template <bool MULTI, bool PERIODIC>
static const void* grid_ptr32(bool queue) {
    using P = GridPush32<MULTI, PERIODIC>;
    return queue ? (const void*)k_seg<true, P> : (const void*)k_seg<false, P>;
}

const void* grid_kernel32(const BorisArgs& a, bool queue) {
    const bool multi = a.alg == TP_ALG_MULTISTEP;
    if (a.f.B.bc == TP_BC_PERIODIC) return multi ? grid_ptr32<true, true>(queue) : grid_ptr32<false, true>(queue);
    return multi ? grid_ptr32<true, false>(queue) : grid_ptr32<false, false>(queue);
}

}  // namespace tpb
