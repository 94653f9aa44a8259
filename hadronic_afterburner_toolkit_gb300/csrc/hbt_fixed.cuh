// Fixed-point particle columns and the values of a binned same-event pair
// computed from them (FP64 form).
//
// GB300 issues an FP64 instruction in 64 times the slots of an integer one,
// and the pair values need differences and products of nearby numbers, which
// integers give exactly.  Each column of a same-event list is kept as a
// 60-bit integer in two signed limbs, value = (h 2^30 + l) / scale with l in
// [-2^29, 2^29):
//   momenta    scale 2^56 / GeV (h in 2^-26 GeV): exact for |p| >= 2^-4 GeV,
//              within 2^-57 GeV below;
//   positions  times 512 / (2 pi hbarC), scale 2^41 (h in 2^-11 table steps
//              per GeV): q.dx comes out in steps of the cos table's 512
//              points per period.  x, y and z are stored negated, so that
//              q.dx = q_E dt - q_x dx - q_y dy - q_z dz is a sum of four
//              products.
// Differences of limbs stay below 2^30 (l) and, for |p| < 8 GeV and
// positions within 2^18 steps per GeV (634 fm), below 2^30 (h), so the four
// products' high, cross and low parts accumulate in 64 bits without
// overflow: 16 multiply-adds of 32 x 32 -> 64 bits for the phase, whose
// rounding is that of the two stored values alone (2^-42 |q| + 2^-57 |dx|
// steps: about 1e-15 rad for |q| = 0.2 GeV, dx = 50 fm; the FP64 sum of
// four rounded products has about 5e-15).  Whole periods drop out as high
// bits, the table point and the remainder are bit fields, and the remainder
// enters the table's polynomials as an exact FP64 integer.  A particle
// outside those ranges (or not finite) carries kFar, and its pairs take the
// FP64 values (values64).
//
// Of the FP64 pipe a binned pair then takes 9 instructions for the cosine
// and one addition per q component, where the FP64 differences, phase and
// table reduction took 29 (with the undecided pairs' chain 13.7 against 31.3
// measured).  Same-event kernel, central group (150k pions): 109 -> 60.8 ms,
// FP64 pipe 73 % busy instead of 84 %; 45k-particle group 10.96 -> 5.52 ms.
// The numerator's distance from the 64-bit sums is unchanged on that group
// (4.7e-15) and halves on small ones (2.3e-15 -> 1.2e-15), where rounding
// averages less.
#pragma once

#include "hbt_engine.cuh"

namespace hbt {
namespace tile {

constexpr int kFar = (int)0x80000000;  // h limb of E: not representable

// hi + lo (|hi| < 2^31, in units of h) as limbs.
__device__ __forceinline__ int2 to_limbs(double hi, double lo) {
    const double t = hi + 6755399441055744.0;  // 1.5 2^52: low word = rint
    const double r = (hi - (t - 6755399441055744.0)) + lo;
    const double s = __fma_rn(r, 1073741824.0, 6755399441055744.0);
    return make_int2(__double2loint(t), min(__double2loint(s), (1 << 29) - 1));
}

// The eight columns of a same-event particle, two to an entry: (px, py),
// (pz, E), (-x, -y), (-z, t), each (h, l).
struct FixedCols {
    int4 c[4];
};

__device__ __forceinline__ FixedCols fixed_cols(const Grid &g, const double *v) {
    int2 q[8];
    bool near = true;
#pragma unroll
    for (int f = 0; f < 8; f++) {
        double hi, lo = 0.0;
        if (f < 4) {
            near = near && fabs(v[f]) < 8.0;
            hi = v[f] * 67108864.0;
        } else {
            const double x = f < 7 ? -v[f] : v[f];
            hi = x * g.pos_h;
            lo = __fma_rn(x, g.pos_h, -hi) + x * g.pos_l;
            near = near && fabs(hi) < 536870912.0;  // 2^18 2^11
        }
        q[f] = to_limbs(hi, lo);
    }
    if (!near) q[3].x = kFar;
    FixedCols r;
#pragma unroll
    for (int k = 0; k < 4; k++)
        r.c[k] = make_int4(q[2 * k].x, q[2 * k].y, q[2 * k + 1].x, q[2 * k + 1].y);
    return r;
}

}  // namespace tile
}  // namespace hbt
