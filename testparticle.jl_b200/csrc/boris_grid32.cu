// boris_grid32.cu -- FP32C fixed-step push with E and B on one trilinear grid, in
// the segments of seg_common.cuh with the stencils gathered by pairs of lanes
// (pair_gather.cuh).  The arithmetic is that of Vel32<FK_EBGRID>.
//
// Measured on the 128^3 turbulent field, 1e6 protons, device time: 250 steps 8.43
// -> 5.29 ms (4.7e10 particle-steps/s).  What bounds it is the L1 cache (88 % busy): 5 line
// look-ups per particle and step, 11 shuffles per warp, and the 8 sectors that come from L2.
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
    static constexpr bool kWarp = true, kJoin = MULTI;
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
    static __device__ __forceinline__ CV update(const BorisArgs& a, const CPos&, const CV& v, const F& f, double x, bool) {
        return vel32<MULTI, kSave>(v, f.E, f.B, a, x);
    }
    static __device__ __forceinline__ CV refused(const BorisArgs&, const CPos&, const CV& v, const F&, double) { return v; }
    __device__ __forceinline__ CPos advance(const BorisArgs& a, CPos p, const CV& v, double) const {
        cpos_push_cv(a, p, v, dth, dtl);
        return p;
    }
    static __device__ __forceinline__ bool outside(const BorisArgs& a, const CPos& p, const CV& v, double t) {
        return outside32<FK_EBGRID>(a, p, v, t);
    }
};

// Without a predicate no state is kept for a rollback, which takes copies in every step:
// 1e6 protons x 250 steps 5.95 -> 5.29 ms, with ends at different steps 2.85 -> 2.34 (400000
// x 200; unrolling the loop twice instead: 5.41 and 3.38, instruction cache misses)
template <bool MULTI, bool PERIODIC>
static const void* grid_ptr32(bool queue, bool term) {
    using P = GridPush32<MULTI, PERIODIC>;
    if (!queue && !term) return (const void*)k_seg<false, P, false>;
    return queue ? (const void*)k_seg<true, P> : (const void*)k_seg<false, P>;
}

const void* grid_kernel32(const BorisArgs& a, bool queue) {
    const bool multi = a.alg == TP_ALG_MULTISTEP, term = a.term.flags != 0;
    if (a.f.B.bc == TP_BC_PERIODIC) return multi ? grid_ptr32<true, true>(queue, term) : grid_ptr32<false, true>(queue, term);
    return multi ? grid_ptr32<true, false>(queue, term) : grid_ptr32<false, false>(queue, term);
}

}  // namespace tpb
