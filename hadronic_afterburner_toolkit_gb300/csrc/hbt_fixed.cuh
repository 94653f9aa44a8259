// Fixed-point particle columns and the values of a binned same-event pair
// computed from them (FP64 form).
//
// GB300 issues an FP64 instruction in 64 times the slots of an integer one,
// and the pair values need differences and products of nearby numbers, which
// integers give exactly.  Each column of a same-event list is kept as a
// 60-bit integer in two signed limbs, value = (h 2^30 + l) / scale with l in
// [-2^29, 2^29):
//   p_x, p_y, m = E - p_z, p = E + p_z   scale 2^56 / GeV (h in 2^-26 GeV):
//              exact for p_x, p_y of 2^-4 GeV and more, within 2^-57 GeV;
//   -x, -y, v = (t + z) / 2, u = (t - z) / 2   times 512 / (2 pi hbarC),
//              scale 2^41 (h in 2^-11 steps of a 512-point cos table, per
//              GeV).
// In these, with d the difference of a column over the pair,
//   q.dx = d(p_x) d(-x) + d(p_y) d(-y) + d(m) d(v) + d(p) d(u)
// is a sum of four products, and q_long = (s(m) d(p) - s(p) d(m)) /
// (2 sqrt(s(m) s(p))) needs no sums of E and p_z (s: sums over the pair).
// (q_out as the difference of p_x^2 + p_y^2 over |s_T| loses its digits for
// small |s_T|: it is formed from the differences and sums.)  Differences of
// limbs stay below 2^30 (l) and, for |p_x|, |p_y|, E < 8 GeV and positions within
// 2^18 steps per GeV (634 fm), below 2^30 (h), so the products' high, cross and
// low parts accumulate in 64 bits without overflow: 16 multiply-adds of 32 x 32 -> 64 bits for the
// phase, whose rounding is that of the stored values alone (2^-42 |q| +
// 2^-57 |dx| steps: about 1e-15 rad for |q| = 0.2 GeV, dx = 50 fm; the FP64
// sum of four rounded products has about 5e-15).  Whole periods drop out as
// high bits, the table point and the remainder are bit fields, and the
// remainder enters the cosine as an exact FP64 integer.
//
// A particle outside those ranges (or not finite) carries kFar in v, and in m
// where its momentum is outside; its pairs take the FP64 phase, or all values in
// FP64 (far_values).  On grids with bins below 2^-11 GeV the momenta's 2^-57 GeV
// would exceed the 2^-46 of a q value that double-float keeps: there no momentum
// is taken (Grid::fixed_p).
//
// Of the FP64 pipe a binned pair takes 8 instructions, 5 for the cosine and an
// addition for each of the three q values (9 to 10 counted, with the undecided
// pairs' chains), where the FP64 differences, phase, table reduction and sums
// took 29.
#pragma once

#include "hbt_engine.cuh"

namespace hbt {
namespace tile {

constexpr int kFar = (int)0x80000000;  // h limb of m or v: not representable

// hi + lo (|hi| < 2^31, in units of h) as limbs.
__device__ __forceinline__ int2 to_limbs(double hi, double lo) {
    const double t = hi + 6755399441055744.0;  // 1.5 2^52: low word = rint
    const double r = (hi - (t - 6755399441055744.0)) + lo;
    const double s = __fma_rn(r, 1073741824.0, 6755399441055744.0);
    return make_int2(__double2loint(t), min(__double2loint(s), (1 << 29) - 1));
}

// Limbs as one integer, and back.
__device__ __forceinline__ long long join_limbs(int2 a) {
    return (long long)a.x * (1 << 30) + a.y;
}
__device__ __forceinline__ int2 split_limbs(long long v) {
    const long long h = (v + (1 << 29)) >> 30;
    return make_int2((int)h, (int)(v - h * (1 << 30)));
}

// The columns of a same-event particle, two to an entry, each (h, l):
// (px, py), (m, p), (-x, -y), (v, u).
constexpr int kFixedCols = 4;
struct FixedCols {
    int4 c[kFixedCols];
};

// v: px py pz E x y z t; fixed_p: may the momenta be taken (Grid::fixed_p)?
__device__ __forceinline__ FixedCols fixed_cols(const Grid &g, bool fixed_p, const double *v) {
    int2 q[8];
    bool near_p = fixed_p, near_x = true;
#pragma unroll
    for (int f = 0; f < 8; f++) {
        double hi, lo = 0.0;
        if (f < 4) {
            near_p = near_p && fabs(v[f]) < 8.0;
            hi = v[f] * 67108864.0;  // 2^26
        } else {
            hi = v[f] * g.pos_h;
            lo = __fma_rn(v[f], g.pos_h, -hi) + v[f] * g.pos_l;
            near_x = near_x && fabs(hi) < 536870912.0;  // 2^18 2^11
        }
        q[f] = to_limbs(hi, lo);
    }
    // E > |p_z|: m and p positive, their sums below 2^31 as unsigned h
    near_p = near_p && v[3] > fabs(v[2]);
    const long long E = join_limbs(q[3]), z = join_limbs(q[2]);
    const long long T = join_limbs(q[7]), Z = join_limbs(q[6]);
    const int2 m = split_limbs(E - z), p = split_limbs(E + z);
    const int2 vv = split_limbs((T + Z) >> 1), uu = split_limbs((T - Z) >> 1);
    const int2 X = split_limbs(-join_limbs(q[4])), Y = split_limbs(-join_limbs(q[5]));
    FixedCols r;
    r.c[0] = make_int4(q[0].x, q[0].y, q[1].x, q[1].y);
    r.c[1] = make_int4(near_p ? m.x : kFar, m.y, p.x, p.y);
    r.c[2] = make_int4(X.x, X.y, Y.x, Y.y);
    r.c[3] = make_int4(near_p && near_x ? vv.x : kFar, vv.y, uu.x, uu.y);
    return r;
}

// The FP32 value of the leading 24 bits of a normal FP64 one within FP32's
// exponent range.
__device__ __forceinline__ float f64_top_bits(double x) {
    const unsigned h = (unsigned)__double2hiint(x), l = (unsigned)__double2loint(x);
    return __uint_as_float(__funnelshift_l(l, h - (896u << 20), 3) & 0x7fffffffu | h & 0x80000000u);
}

// cos of a phase given as hh 2^-37 + (low 30 bits of hl) 2^-67 steps of
// 2 pi / 512.  In steps of 2 pi / 2048 (hh counts 2^-35): the nearest table
// point j, of which the quarter period gives signs and the roles of U = cos
// and V = sin of its place, and the remainder d, |d| <= pi / 2048:
//   cos(j + d) = U - V d - U d^2 / 2 + V d^3 / 6 + U d^4 / 24,
// the first three terms in FP64 (d exact but for one rounding), the last
// two, below 6e-10, in FP32 (the next, V d^5 / 120, is below 7e-17).  Error
// below 4e-16.
__device__ __forceinline__ double cos_fixed(const Grid &g, const double *t, long long hh,
                                            unsigned hl) {
    const unsigned fl = (unsigned)hh, low = hl << 2;
    const int top = (int)(hh >> 32) + 4;  // + half a step
    const int r = (top & 7) - 4;          // remainder: r, fl, low as one signed number
    const int j = top >> 3, odd = j & 512, idx = j & 511;
    const int iu = odd ? 512 - idx : idx;
    const double U = t[iu], tv = t[512 - iu];
    const unsigned sv = (unsigned)odd << 22;              // V's sign, as a sign bit
    const unsigned sr = (unsigned)((j + 512) & 1024) << 21;  // the result's
    const double V = __hiloint2double(__double2hiint(tv) ^ (int)sv, __double2loint(tv));
    // 52-bit signed integer remainder (2^-52 steps) as FP64
    const double z = __hiloint2double(0x43380000 + (int)__funnelshift_r(fl, (unsigned)r, 15),
                                      (int)__funnelshift_l(low, fl, 17)) -
                     6755399441055744.0;
    const double hd = z * g.cfx_half;  // d / 2
    const double d = __hiloint2double(__double2hiint(hd) + (1 << 20), __double2loint(hd));
    const double main = __fma_rn(-d, __fma_rn(hd, U, V), U);
    const float x = __int2float_rn((int)__funnelshift_r(fl, (unsigned)r, 3)) *
                    (float)(6.283185307179586 / 2048.0 / 4294967296.0);
    const float x2 = x * x;
    // d^3 V / 6 + d^4 U / 24
    const float b = (x2 * (1.0f / 6.0f)) *
                    __fmaf_rn(x, f64_top_bits(V), 0.25f * (x2 * f64_top_bits(U)));
    // b as FP64 through its bits (a zero becomes a number below 1e-38)
    const int bi = __float_as_int(b);
    const double bd = __hiloint2double(((bi >> 3) & (int)0x8fffffff) + (896 << 20), bi << 29);
    const double w = main + bd;
    return __hiloint2double(__double2hiint(w) ^ (int)sr, __double2loint(w));
}

}  // namespace tile
}  // namespace hbt
