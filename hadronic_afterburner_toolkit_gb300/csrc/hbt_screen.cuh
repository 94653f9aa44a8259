// FP32 screen of the pair binning: decides, for every pair of two tiles of
// 128 particles, whether it is certainly outside the q window, certainly in
// one q bin, or undecided (the FP64 reference chain of hbt_chain.cuh then
// decides it).  GB300 runs FP64 at 1/58 of its FP32 rate, and most pairs are
// rejected, so this loop must cost as few issue slots per pair as it can; it
// is bound by instruction issue.
//
// Terms.  Each particle brings six FP32 numbers, rounded once from FP64:
// p_x, p_y, r2 = p_x^2 + p_y^2 and, with the longitudinal boost, the
// light-cone momenta m = E - p_z, p = E + p_z and t2 = m p.  With a the
// first and b the second particle of a pair, the LCMS components are
//   q_out  = (r2_a - r2_b) / k,           k^2 = |a_T + b_T|^2,
//   q_side = 2 (a_y b_x - a_x b_y) / k,
//   q_long = (p_a m_b - p_b m_a) / sqrt(M2),
//   M2     = p_a m_b + p_b m_a + t2_a + t2_b,
// the reference's expressions (src/HBT_correlation.cpp:366-393) in real
// arithmetic: sums of positive terms and one difference each, about half
// the operations of forming the momentum sums and differences, and with
// error bounds that depend on s2 = r2_a + r2_b, 1/k and M2 alone.  Without
// the boost q_long = z_a - z_b (the m and p places hold z and |z|).
//
// Packed arithmetic.  The j-tile is stored two particles side by side, so
// that one f32x2 instruction works on two pairs: 35 packed operations and
// two scalar reciprocal roots per pair decide a pair's three bins, where the
// scalar screen before (a prefilter, a queue, a window test with per-pair
// bounds on each component, then the bins) took about 50 instructions for
// every pair and 375 for every pair past its prefilter.
//
// Bounds (u = 2^-24; every term is an FP64 value rounded once).  With
// s2 = r2_a + r2_b, |a_x b_x| + |a_y b_y| <= s2 / 2 and |a_y b_x| +
// |a_x b_y| <= s2 / 2, each FP32 operation adding u of its result:
//   k2 (two FMAs on s2)                  8.3 u s2
//   r2_a - r2_b                          2.1 u s2
//   2 (a_y b_x - a_x b_y)                4.1 u s2
//   1/k (rsqrt.approx, 2^-22.9)          0.53 (8.3 u s2 / k^2) + 4.5 u, relative
//   D = p_a m_b - p_b m_a                4.1 u S, S = p_a m_b + p_b m_a
//   1/sqrt(M2)                           7.1 u relative
// so for a pair whose components lie within Q = max(|lo|, |hi|)
//   |dq_out|, |dq_side| <= 4.1 u w + Q (4.4 u w / k + 5.6 u), w = s2 / k,
//   |dq_long|           <= 4.1 u S / sqrt(M2) + 8.3 u Q.
// In units of the bin width, doubled, plus the rounding of the conversion
// to bins and the distance of the window's bounds from the outer bin edges
// (1e-8 GeV), this is the one margin et of a pair's three bins.  The
// reference's own FP64 rounding is 2^-29 times smaller but for that of q_long,
// which cancels from E and p_z: some 20 2^-53 gamma^2 of Q, at p = 2^28 m
// (rapidity 9.7) a third of this bound.  Particles beyond get a NaN t2,
// unphysical ones NaN for all longitudinal terms: their pairs that pass the
// transverse test are undecided (with NaN for all terms from rapidity 6.6 on,
// 30,000 particles spread to 8 took 28.6 ms in the place of 1.0).  A pair is
// outside when a bin coordinate
// lies beyond the grid by more than et, decided when all three lie farther
// than et from a bin edge, undecided otherwise; a NaN or infinite margin
// (k = 0, an overflow) leaves it undecided.  The coefficient of w / k is at
// least 10 bins per unit of relative error of k^2, so that a pair whose k is
// lost to cancellation cannot be decided.
//
// The first test of a pair, before the rest, is on its transverse momentum
// difference alone: q_out^2 + q_side^2 = |a_T - b_T|^2 = 2 s2 - k^2 <= 2 Q^2
// for a binned pair.  A warp skips the rest when none of its 64 pairs of
// two steps passes it.
#pragma once

#include "hbt_engine.cuh"

namespace hbt {
namespace tile {

constexpr int FT = 128;  // tile edge (particles) for both lists

// Two FP32 numbers in one 64-bit register pair.
typedef unsigned long long f2;
__device__ __forceinline__ f2 pack2(float a, float b) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ f2 both(float a) { return pack2(a, a); }
__device__ __forceinline__ void unpack2(f2 v, float &a, float &b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// 1 / sqrt(x): the special-function unit's estimate (relative error
// 2^-22.9), +inf for zero and subnormals, NaN below zero.
__device__ __forceinline__ float rsqrt_approx(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
// 1 / x, relative error 1 ulp (as 1 / sqrt(x): no subnormals).
__device__ __forceinline__ float rcp_approx(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ f2 rsqrt2(f2 v) {
    float a, b;
    unpack2(v, a, b);
    return pack2(rsqrt_approx(a), rsqrt_approx(b));
}

// A particle's screen terms: light-cone (LC: with the boost or the q_inv
// histograms) m = E - p_z, p = E + p_z, t2 = m p; otherwise m = p_z, p =
// |p_z|, t2 = 0.
struct Terms {
    float x, y, m, p, r2, t2;
};

// FP32 terms of a particle from its FP64 momentum.
template <bool LC>
__device__ __forceinline__ Terms screen_terms(double px, double py, double pz, double E) {
    Terms t;
    t.x = (float)px;
    t.y = (float)py;
    t.r2 = (float)(px * px + py * py);
    if (LC) {
        const double m = E - pz, p = E + pz;
        t.m = (float)m;
        t.p = (float)p;
        t.t2 = (float)(m * p);
        const float nan = __int_as_float(0x7fffffff);
        if (!(t.m * 0x1p28f > t.p && t.p * 0x1p28f > t.m)) t.t2 = nan;  // rapidity past 9.7
        if (!(t.m > 0.0f && t.p > 0.0f)) t.m = t.p = nan;               // E <= |p_z|, NaN
    } else {
        t.m = (float)pz;
        t.p = fabsf(t.m);
        t.t2 = 0.0f;
    }
    return t;
}
// Rows past the end of a list: far from every particle, so that the
// transverse test rejects their pairs.
__device__ __forceinline__ Terms pad_terms(float x) { return Terms{x, 0.f, 1.f, 1.f, x * x, 1.f}; }

// j-tile terms, two particles side by side.
struct __align__(16) TermsPair {
    float x[2], y[2], m[2], p[2], r2[2], t2[2];
};
__device__ __forceinline__ void put_terms(TermsPair *b, int k, const Terms &t) {
    TermsPair &d = b[k >> 1];
    const int h = k & 1;
    d.x[h] = t.x;
    d.y[h] = t.y;
    d.m[h] = t.m;
    d.p[h] = t.p;
    d.r2[h] = t.r2;
    d.t2[h] = t.t2;
}

// round to nearest by addition: 1.5 2^23, the integer in the low bits
constexpr float kRound = 12582912.0f;
constexpr unsigned kRoundBits = 0x4b400000u;

// What the screen says about two pairs, the row a against particles 2 jp and
// 2 jp + 1 of the j-tile: take[h] false when pair h is certainly outside,
// bin[h] its q bin, und[h] when only the reference chain can tell.
// With q_inv histograms takeq, undq and kq say the same of the q_inv bin.
struct Screened {
    bool take[2], und[2];
    unsigned bin[2];
    bool takeq[2], undq[2];
    unsigned kq[2];
};

// The row of one lane, in packed form (both halves alike).
struct Row {
    f2 x2, y2, nx2, m, nm, p, r2, t2;  // x2 = 2 p_x, nx2 = -2 p_x, nm = -m
};
__device__ __forceinline__ Row row_of(const Terms &a) {
    return Row{both(2.0f * a.x), both(2.0f * a.y), both(-2.0f * a.x), both(a.m),
               both(-a.m),       both(a.p),        both(a.r2),        both(a.t2)};
}

// The q_inv bin of two pairs (src/HBT_correlation.cpp:331-356, :595-607):
// q_inv^2 = |a_T - b_T|^2 - (m_a - m_b)(p_a - p_b).  With w = s2 / k >=
// sqrt(s2 / 2), each difference within 2.01 u of its operands' sum:
//   transverse part      8.1 u (|d_x| + |d_y|) w
//   longitudinal part    2.1 u (s_m |d_p| + s_p |d_m|)
//   roundings            4 u (|d_T|^2 + |d_m d_p|)
//   the reference's q_E^2 - q_z^2 in FP64
//                        2^-51 (d_m^2 + d_p^2) = 2.1 u (2^-28 d_m^2 + 2^-28 d_p^2)
// and, T not negative, |sqrt(t) - sqrt(T)| <= |t - T| / sqrt(t), plus 4 u of it
// for the reciprocal root and the product.  q_inv^2 certainly negative: no
// event (the reference's NaN fails both bounds); its sign not certain (within
// twice the bound of zero): undecided, as a T below zero has no root to be near
// to.
__device__ __forceinline__ void screen_qinv(const Screen &S, const Row &a, const f2 *v, f2 w,
                                            Screened &r) {
    const f2 dx = fma2(v[0], both(-2.0f), a.x2), dy = fma2(v[1], both(-2.0f), a.y2);  // twice
    const f2 qt = fma2(dx, dx, mul2(dy, dy));                                        // 4 times
    const f2 dm = add2(v[2], a.nm), dp = fma2(v[3], both(-1.0f), a.p);               // -d_m, d_p
    const f2 lg = mul2(dm, dp);
    const f2 sm = add2(v[2], a.m), sp = add2(v[3], a.p);
    const f2 t2 = fma2(qt, both(0.25f), lg);
    float x[2], y[2], m[2], p[2], g[2], t[2], q[2], M[2], P[2], W[2];
    unpack2(dx, x[0], x[1]);
    unpack2(dy, y[0], y[1]);
    unpack2(dm, m[0], m[1]);
    unpack2(dp, p[0], p[1]);
    unpack2(lg, g[0], g[1]);
    unpack2(t2, t[0], t[1]);
    unpack2(qt, q[0], q[1]);
    unpack2(sm, M[0], M[1]);
    unpack2(sp, P[0], P[1]);
    unpack2(w, W[0], W[1]);
    constexpr float U = 5.9604645e-8f;
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const float Mp = __fmaf_rn(0x1p-28f, fabsf(p[k]), M[k]);
        const float Pm = __fmaf_rn(0x1p-28f, fabsf(m[k]), P[k]);
        const float e = U * __fmaf_rn(4.1f * (fabsf(x[k]) + fabsf(y[k])), W[k],
                                      __fmaf_rn(2.1f, __fmaf_rn(Mp, fabsf(p[k]), Pm * fabsf(m[k])),
                                                q[k] + 4.0f * fabsf(g[k])));
        const float rs = rsqrt_approx(t[k]), qi = t[k] * rs;
        const float h = __fmaf_rn(__fmaf_rn(e, rs, 4.0f * U * qi), S.sc_nkq, S.sc_h0);
        const float tq = __fmaf_rn(qi, S.inv_dq, S.sc_c0);
        const float kr = tq + kRound;
        r.takeq[k] = !(t[k] + 2.0f * e < 0.0f) && !(tq > S.sc_top - h) && !(tq < S.sc_bot + h);
        r.undq[k] = !(t[k] > 2.0f * e) || !(fabsf(tq - (kr - kRound)) < h);
        r.kq[k] = __float_as_uint(kr) - kRoundBits;
    }
}

// Screens two pairs.  `inv_dq`: 1 / bin width for each pair, negative when b
// is the pair's first particle in the caller's order (every component of q
// then changes sign).  False when neither pair of any lane passes the
// transverse test (warp-uniform; never with q_inv histograms, whose window
// that test does not cover).
template <bool BOOST, bool QINV>
__device__ __forceinline__ bool screen_two(const Screen &S, const Row &a, const TermsPair &b,
                                           f2 inv_dq, Screened &r) {
    const f2 *v = reinterpret_cast<const f2 *>(&b);
    const f2 bx = v[0], by = v[1], bm = v[2], bp = v[3];
    const f2 s2 = add2(a.r2, v[4]);
    const f2 k2 = fma2(a.y2, by, fma2(a.x2, bx, s2));
    // reject: 2 s2 - k2 > 2 Q^2 by more than 14 u s2
    const f2 thr = fma2(s2, both(2.0f - 0x1p-20f), both(-S.pqt2));
    float ka, kb, ta, tb;
    unpack2(k2, ka, kb);
    unpack2(thr, ta, tb);
    r.take[0] = !(ka < ta);
    r.take[1] = !(kb < tb);
    if (!QINV && !__any_sync(0xffffffffu, r.take[0] || r.take[1])) return false;
    const f2 inv = pack2(rsqrt_approx(ka), rsqrt_approx(kb));
    const f2 w = mul2(s2, inv);
    const f2 qo = mul2(fma2(v[4], both(-1.0f), a.r2), inv);
    const f2 qs = mul2(fma2(a.y2, bx, mul2(a.nx2, by)), inv);
    f2 ql, el;
    if (BOOST) {
        const f2 P = mul2(a.p, bm);
        const f2 D = fma2(bp, a.nm, P), sum = fma2(bp, a.m, P);
        const f2 rl = rsqrt2(add2(sum, add2(a.t2, v[5])));
        ql = mul2(D, rl);
        el = mul2(sum, rl);
    } else if (QINV) {
        // z = (p - m) / 2, the sums E in the place of |z|
        ql = mul2(both(0.5f), fma2(fma2(bp, both(-1.0f), a.p), both(1.0f), add2(bm, a.nm)));
        el = mul2(both(0.5f), add2(add2(a.m, bm), add2(a.p, bp)));
    } else {
        ql = fma2(bm, both(-1.0f), a.m);
        el = add2(a.p, bp);
    }
    if (QINV) screen_qinv(S, a, v, w, r);
    // h = 0.5 - et
    const f2 h = fma2(w, fma2(inv, both(S.sc_nk1), both(S.sc_nk2)),
                      fma2(el, both(S.sc_nk3), both(S.sc_h0)));
    const f2 c0 = both(S.sc_c0), rnd = both(kRound), nrnd = both(-kRound);
    // bin coordinates shifted by half a bin (rint is the bin), their rint
    // and their distance to it
    const f2 to = fma2(qo, inv_dq, c0), ts = fma2(qs, inv_dq, c0), tl = fma2(ql, inv_dq, c0);
    const f2 ko = add2(to, rnd), ks = add2(ts, rnd), kl = add2(tl, rnd);
    const f2 minus = both(-1.0f);
    const f2 fo = fma2(add2(ko, nrnd), minus, to), fs = fma2(add2(ks, nrnd), minus, ts),
             fl = fma2(add2(kl, nrnd), minus, tl);
    // beyond the grid: a coordinate above n - 0.5 + et or below -0.5 - et
    // (each limit a little inside et, fill_tile_screen)
    const f2 top = fma2(h, minus, both(S.sc_top)), bot = add2(h, both(S.sc_bot));
    float o[2], s[2], l[2], df[3][2], hh[2], up[2], dn[2], io[2], is[2], il[2];
    unpack2(to, o[0], o[1]);
    unpack2(ts, s[0], s[1]);
    unpack2(tl, l[0], l[1]);
    unpack2(fo, df[0][0], df[0][1]);
    unpack2(fs, df[1][0], df[1][1]);
    unpack2(fl, df[2][0], df[2][1]);
    unpack2(h, hh[0], hh[1]);
    unpack2(top, up[0], up[1]);
    unpack2(bot, dn[0], dn[1]);
    unpack2(ko, io[0], io[1]);
    unpack2(ks, is[0], is[1]);
    unpack2(kl, il[0], il[1]);
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const float hi = fmaxf(fmaxf(o[k], s[k]), l[k]), lo = fminf(fminf(o[k], s[k]), l[k]);
        const float far = fmaxf(fmaxf(fabsf(df[0][k]), fabsf(df[1][k])), fabsf(df[2][k]));
        r.take[k] = r.take[k] && !(hi > up[k]) && !(lo < dn[k]);
        r.und[k] = !(far < hh[k]);
        r.bin[k] = __float_as_uint(io[k]) * S.sc_n2 + __float_as_uint(is[k]) * (unsigned)S.qnpts +
                   __float_as_uint(il[k]) - S.sc_bin0;
    }
    return true;
}

// 3-D slot (K_T bin, or K_T x K_phi bin) of a pair from its particles' FP32
// p_x, p_y: >= 0 certain, -1 undecided, -2 certainly outside the K_T window.
// K_T = |s| / 2 with s = a + b: each component within 2.01 u (|a| + |b|) of
// the exact sum, |s| within 2.01 u A of it, A the sum of the four
// magnitudes, and 8 u of itself for the square, the reciprocal root and the
// products.  K_phi: s turned by -psi (the sine and cosine of psi rounded to
// FP32), then the angle of (c_x, c_y) in bins: the arctangent of the smaller
// over the larger magnitude by an odd polynomial of degree 11 fitted on
// [0, 1] (1.7e-6, 2e-6 with its FP32 evaluation), and the octant's
// reflections; the angle of s is within 2.01 u A / |s| of the exact one.
// Bin edges are at multiples of the bin width from psi, the wrap included,
// so one test of the distance to the rint covers them all.  All bounds are
// doubled.
// iK: the K_T bin, valid when the result is >= 0.
template <bool AZ>
__device__ __forceinline__ int slot_of(const Screen &S, float ax, float ay, float bx, float by,
                                       int &iK) {
    const float sx = ax + bx, sy = ay + by;
    const float A = (fabsf(ax) + fabsf(ay)) + (fabsf(bx) + fabsf(by));
    const float k2 = __fmaf_rn(sx, sx, sy * sy);
    const float inv = rsqrt_approx(k2);
    const float k = k2 * inv;
    const float t = __fmaf_rn(k, S.sk_half_inv, S.sk_c0);
    const float h = __fmaf_rn(A, S.sk_nkA, __fmaf_rn(k, S.sk_nkk, S.sk_h0));
    if (t > S.sk_top - h || t < h + S.sc_bot) return -2;
    const float kr = t + kRound;
    bool sure = fabsf(t - (kr - kRound)) < h;
    int slot = (int)(__float_as_uint(kr) - kRoundBits);
    iK = slot;
    if (AZ) {
        const float cx = __fmaf_rn(sy, S.sp_sin, sx * S.sp_cos);
        const float cy = __fmaf_rn(sy, S.sp_cos, -(sx * S.sp_sin));
        const float ux = fabsf(cx), uy = fabsf(cy);
        const float z = fminf(ux, uy) * rcp_approx(fmaxf(ux, uy));
        const float z2 = z * z;
        // arctan z / z, times n_Kphi / (2 pi) at the end
        const float pl = __fmaf_rn(
            z2,
            __fmaf_rn(z2,
                      __fmaf_rn(z2,
                                __fmaf_rn(z2, __fmaf_rn(z2, -0.01171914f, 0.05264735f),
                                          -0.11642648f),
                                0.19354038f),
                      -0.33262283f),
            0.99997722f);
        float r = z * pl * S.sp_scale;
        if (uy > ux) r = S.sp_quarter - r;
        if (cx < 0.0f) r = 2.0f * S.sp_quarter - r;
        if (cy < 0.0f) r = 4.0f * S.sp_quarter - r;
        const float tp = r - 0.5f;
        const float kp = tp + kRound;
        const float hp = __fmaf_rn(A * inv, S.sp_nkA, S.sp_h0);
        sure = sure && fabsf(tp - (kp - kRound)) < hp;
        slot = slot * S.n_Kphi + (int)(__float_as_uint(kp) - kRoundBits);
    }
    return sure ? slot : -1;
}

}  // namespace tile
}  // namespace hbt
