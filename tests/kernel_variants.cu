// prints kernel_variant of runs that take different kernels (test_kernel_variants.py)
#include <cstdio>

#include "tp_device.cuh"

using namespace tpb;

static BorisArgs run(int alg, int E, int B, int64_t n = 100000) {
    BorisArgs a{};
    a.alg = alg;
    a.n = n;
    a.save_everystep = 1;
    a.ssi = 2;
    a.f.E.kind = E;
    a.f.B.kind = B;
    return a;
}

int main() {
    const float4 table{};
    for (int fp32c = 0; fp32c < 2; ++fp32c) {
        BorisArgs large = run(TP_ALG_BORIS, TP_FIELD_GRID, TP_FIELD_GRID), cubic = large;
        large.f.eb32 = &table;
        BorisArgs small = large;
        small.n = 1000;
        cubic.f.E.general = cubic.f.B.general = 1;
        BorisArgs coop = cubic;
        coop.f.ebc32 = &table;
        const BorisArgs list[] = {run(TP_ALG_BORIS, TP_FIELD_ZERO, TP_FIELD_DIPOLE), run(TP_ALG_BORIS, TP_FIELD_ZERO, TP_FIELD_UNIFORM),
                                  run(TP_ALG_BORIS, TP_FIELD_ZERO, TP_FIELD_AFFINE), run(TP_ALG_BORIS, TP_FIELD_ZERO, TP_FIELD_GRID),
                                  run(TP_ALG_BORIS, TP_FIELD_UNIFORM, TP_FIELD_GRID), large, small, cubic, coop};
        for (const BorisArgs& a : list) std::printf("%d ", kernel_variant(a, fp32c != 0));
        std::printf("\n");
    }
    return 0;
}
