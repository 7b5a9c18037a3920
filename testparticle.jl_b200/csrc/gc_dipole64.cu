// gc_dipole64.cu -- float64 guiding centres with E zero and B a dipole (compiled
// with -fmad=false): the right-hand side of RHS64 in the same operations, so the
// same bits, but
//   * quotients of one denominator share its reciprocal (fdiv64.cuh): 15
//     divisions and 2 square roots of a right-hand side become 9 reciprocals,
//     the per-particle one of q/m formed once;
//   * the sums of the Jacobian that are symmetric are formed once (the products
//     d_i d_j / r^7 are not: their rounding depends on the order);
//   * AXIAL: a moment along z (every planetary dipole in its own frame) leaves
//     out the products with its zero components;
//   * the zero E is left out.
// What bounds it is the float64 pipe.  Measured on the device, 262144 electrons and
// protons over one bounce period: RK4 (200 steps) 7.21 -> 3.36 ms, RK45 (rtol 1e-6)
// 4.47 -> 2.45 ms.
#include "gc_common.cuh"

namespace tpb {

template <bool AXIAL>
struct RHSDipole {
    // register caps (threads), on the ensemble below: RK4 256 (132 registers)
    // 3.58 ms, 512 3.39, 640 3.36, 768 3.42; RK45 384 2.50, 512 2.45, 640 2.51
    static constexpr int kGM = GM_ANALYTIC, kRk4Bound = 640, kRk45Bound = 512;
    static constexpr bool kFast = true;
    bool ok, par_ok;
    Rec64 rq2m;   // 1 / (q/m)
    double muq;   // mu / q
    __device__ __forceinline__ void start(const GCPar& p) {
        muq = p.mu / p.q;
        rq2m = rec64(p.q2m, 1.0 / p.q2m);
        par_ok = in_range64(fabs(p.q2m));
        ok = true;
    }
    __device__ __forceinline__ G4 operator()(const DevFields& F, const G4& s, const GCPar& p, double) {
        const DevField& g = F.B;
        const D3 d = D3{s.y[0], s.y[1], s.y[2]} - D3{g.c[0], g.c[1], g.c[2]};
        const double d2 = abs2sum(d);
        if (!par_ok || !in_range64(d2)) {
            ok = false;
            return s;
        }
        // B (analytic_eval64)
        const double y = rsqrt64(d2);
        const double dm = sqrt64(d2, y);
        const Rec64 rm = rec64(dm, y);
        const D3 rh{quot64(d.x, rm), quot64(d.y, rm), quot64(d.z, rm)};
        const double mr = AXIAL ? g.m[2] * rh.z : dot(D3{g.m[0], g.m[1], g.m[2]}, rh);
        const double y2 = y * y;
        const Rec64 r3 = rec64((dm * dm) * dm, y2 * y);
        const double mr3 = 3.0 * mr;
        const D3 w{AXIAL ? mr3 * rh.x : mr3 * rh.x - g.m[0], AXIAL ? mr3 * rh.y : mr3 * rh.y - g.m[1], mr3 * rh.z - g.m[2]};
        const D3 B{quot64(g.coef * w.x, r3), quot64(g.coef * w.y, r3), quot64(g.coef * w.z, r3)};
        // its Jacobian (field_jac64)
        const double inv5 = quot64(1.0, rec64((d2 * d2) * dm, (y2 * y2) * y));
        const double inv7 = quot64(inv5, rec64(d2, y2));
        double md, sxx, sxy, sxz, syy, syz, szz;
        const double pzz = g.m[2] * d.z;
        if (AXIAL) {
            md = pzz;
            sxx = syy = md;
            sxy = 0.0;
            sxz = g.m[2] * d.x;
            syz = g.m[2] * d.y;
        } else {
            const double pxx = g.m[0] * d.x, pyy = g.m[1] * d.y;
            md = (pxx + pyy) + pzz;
            sxx = (pxx + md) + pxx;
            syy = (pyy + md) + pyy;
            sxy = g.m[1] * d.x + g.m[0] * d.y;
            sxz = g.m[2] * d.x + g.m[0] * d.z;
            syz = g.m[2] * d.y + g.m[1] * d.z;
        }
        szz = (pzz + md) + pzz;
        const double txx = 3.0 * sxx * inv5, tyy = AXIAL ? txx : 3.0 * syy * inv5, tzz = 3.0 * szz * inv5;
        const double txy = AXIAL ? 0.0 : 3.0 * sxy * inv5, txz = 3.0 * sxz * inv5, tyz = 3.0 * syz * inv5;
        const double md15 = 15.0 * md;
        const D3 e{md15 * d.x, md15 * d.y, md15 * d.z};
        const double J0 = g.coef * (txx - e.x * d.x * inv7), J1 = g.coef * (txy - e.x * d.y * inv7),
                     J2 = g.coef * (txz - e.x * d.z * inv7), J3 = g.coef * (txy - e.y * d.x * inv7),
                     J4 = g.coef * (tyy - e.y * d.y * inv7), J5 = g.coef * (tyz - e.y * d.z * inv7),
                     J6 = g.coef * (txz - e.z * d.x * inv7), J7 = g.coef * (tyz - e.z * d.y * inv7),
                     J8 = g.coef * (tzz - e.z * d.z * inv7);
        // the drift equations (RHS64)
        const double b2 = abs2sum(B);
        if (!in_range64(b2)) {
            ok = false;
            return s;
        }
        const double yb = rsqrt64(b2);
        const Rec64 rb = rec64(sqrt64(b2, yb), yb);
        const D3 bh{quot64(B.x, rb), quot64(B.y, rb), quot64(B.z, rb)};
        const D3 gB{(J0 * bh.x + J3 * bh.y) + J6 * bh.z, (J1 * bh.x + J4 * bh.y) + J7 * bh.z,
                    (J2 * bh.x + J5 * bh.y) + J8 * bh.z};
        const D3 q = D3{J7 - J5, J2 - J6, J3 - J1} + cross(bh, gB);
        const D3 curlb{quot64(q.x, rb), quot64(q.y, rb), quot64(q.z, rb)};
        const D3 Bs = B + quot64(s.y[3], rq2m) * curlb;
        const D3 Es = D3{0.0, 0.0, 0.0} - muq * gB;
        const double bp = dot(bh, Bs);
        if (!in_range64(fabs(bp))) {
            ok = false;
            return s;
        }
        const double ib = quot64(1.0, rec64(bp, rcp64(bp)));
        const D3 v = (s.y[3] * Bs + cross(Es, bh)) * ib;
        return {{v.x, v.y, v.z, dot((p.q2m * ib) * Bs, Es)}};
    }
};

template <bool AXIAL>
static const void* dipole_ptr(bool rk4, bool queue) {
    using R = RHSDipole<AXIAL>;
    if (rk4) return queue ? (const void*)k_rk4<R, true> : (const void*)k_rk4<R, false>;
    return queue ? (const void*)k_rk45<R, true> : (const void*)k_rk45<R, false>;
}

// E zero and B a dipole, else null
const void* gc_dipole_kernel64(const GCArgs& a, bool queue) {
    if (a.f.E.kind != TP_FIELD_ZERO || a.f.B.kind != TP_FIELD_DIPOLE) return nullptr;
    const bool rk4 = a.alg == TP_GC_RK4;
    return a.f.B.m[0] == 0.0 && a.f.B.m[1] == 0.0 ? dipole_ptr<true>(rk4, queue) : dipole_ptr<false>(rk4, queue);
}

}  // namespace tpb
