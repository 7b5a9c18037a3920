// pair_gather.cuh -- trilinear stencils gathered by pairs of lanes.
//
// A node of the interleaved table (E xyz0, B xyz0) or of one float64 field is 32
// bytes, z is the tables' fastest axis, and a 128-byte line holds four nodes that are
// neighbours along z.  When
// every lane loads the 8 corners of its own particle, the 32 lanes of a load
// instruction touch 32 different lines, and the L1 cache, which looks up one
// line per clock, needs 8 x 32 clocks per warp and step: that bounded the
// gridded pushes.  Here the lanes 2k and 2k + 1 load the two z-neighbours of
// one particle in the same instruction, first the even lane's particle, then
// the odd lane's: the neighbours share a line three times out of four, so a
// load instruction touches 16 x 1.25 lines, 5 instead of 8 clocks per particle
// and step.  Each lane then interpolates its z-plane of both particles along x
// and y (the order of tri3 and tri64, so the same bits) and the pair exchanges
// the six values that the other's last interpolation, along z, needs.  (With x
// fastest, the exchange must come before the first interpolation: 24 shuffles
// and 48 selects, which cost what the fewer lines saved.)
//
// All 32 lanes of the warp must call this together; a lane that has no particle
// passes valid node offsets (0) and ignores the result.
#pragma once

#include <cstdint>

namespace tpb {

__device__ __forceinline__ float pair_lerp(float a, float b, float f) { return fmaf(f, b - a, a); }
// in units compiled with -fmad=false: lerp64
__device__ __forceinline__ double pair_lerp(double a, double b, double f) { return a + f * (b - a); }

// one 32-byte, 32-byte-aligned node record in a single 256-bit read-only load
__device__ __forceinline__ void ldg_words8(const float4* p, float w[8]) {
    asm("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=f"(w[0]), "=f"(w[1]), "=f"(w[2]), "=f"(w[3]), "=f"(w[4]), "=f"(w[5]), "=f"(w[6]), "=f"(w[7])
        : "l"(p));
}

// node records: NC values of type W from the table at node `i`
struct NodeEB {  // interleaved float table
    static constexpr int NC = 6;
    using W = float;
    static __device__ __forceinline__ void load(const void* T, int i, W w[NC]) {
        float r[8];
        ldg_words8(static_cast<const float4*>(T) + 2 * (int64_t)i, r);
#pragma unroll
        for (int c = 0; c < 6; ++c) w[c] = r[c < 3 ? c : c + 1];
    }
};
struct Node32 {  // float table of one field
    static constexpr int NC = 3;
    using W = float;
    static __device__ __forceinline__ void load(const void* T, int i, W w[NC]) {
        const float4 q = __ldg(static_cast<const float4*>(T) + i);
        w[0] = q.x;
        w[1] = q.y;
        w[2] = q.z;
    }
};
struct Node64 {  // float64 table of one field
    static constexpr int NC = 3;
    using W = double;
    static __device__ __forceinline__ void load(const void* T, int i, W w[NC]) {
        double r[4];
        asm("ld.global.nc.v4.f64 {%0,%1,%2,%3}, [%4];"
            : "=d"(r[0]), "=d"(r[1]), "=d"(r[2]), "=d"(r[3])
            : "l"(static_cast<const double*>(T) + 4 * (int64_t)i));
        w[0] = r[0];
        w[1] = r[1];
        w[2] = r[2];
    }
};

// The node's values (E xyz, B xyz, or one field) at the stencil's lower (c0) and
// upper (c1) z-plane, interpolated along x and y.  `base` is the node of the
// lower corner, dx, dy, dz the node offsets to the neighbours; fx, fy the fractions.
template <class R, class NODE = NodeEB>
__device__ __forceinline__ void pair_planes(const void* T, int base, int dx, int dy, int dz, R fx, R fy, R c0[NODE::NC],
                                            R c1[NODE::NC]) {
    constexpr int NC = NODE::NC;
    const unsigned full = 0xffffffffu;
    const bool odd = threadIdx.x & 1;
    const int pb = __shfl_xor_sync(full, base + dz, 1);
    const int pdx = __shfl_xor_sync(full, dx, 1), pdy = __shfl_xor_sync(full, dy, 1);
    // A: the even lane's particle, B: the odd lane's; a particle's owner loads
    // its lower plane, the partner its upper plane
    const int ab = odd ? pb : base, adx = odd ? pdx : dx, ady = odd ? pdy : dy;
    const int bb = odd ? base : pb, bdx = odd ? dx : pdx, bdy = odd ? dy : pdy;
    typename NODE::W A[4][NC], B[4][NC];  // corners (x, y) = 00, 10, 01, 11
    NODE::load(T, ab, A[0]);
    NODE::load(T, ab + adx, A[1]);
    NODE::load(T, ab + ady, A[2]);
    NODE::load(T, ab + adx + ady, A[3]);
    NODE::load(T, bb, B[0]);
    NODE::load(T, bb + bdx, B[1]);
    NODE::load(T, bb + bdy, B[2]);
    NODE::load(T, bb + bdx + bdy, B[3]);
    const R pfx = __shfl_xor_sync(full, fx, 1), pfy = __shfl_xor_sync(full, fy, 1);
    const R ax = odd ? pfx : fx, ay = odd ? pfy : fy, bx = odd ? fx : pfx, by = odd ? fy : pfy;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        const R va = pair_lerp(pair_lerp((R)A[0][c], (R)A[1][c], ax), pair_lerp((R)A[2][c], (R)A[3][c], ax), ay);
        const R vb = pair_lerp(pair_lerp((R)B[0][c], (R)B[1][c], bx), pair_lerp((R)B[2][c], (R)B[3][c], bx), by);
        c0[c] = odd ? vb : va;
        c1[c] = __shfl_xor_sync(full, odd ? va : vb, 1);
    }
}

}  // namespace tpb
