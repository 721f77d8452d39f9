// The EOS evaluation in integers (see block_fixed.cuh for the products).
//
// One evaluation (lulesh.cc:1692-1871) is a chain of some 45 dependent double
// operations, 4 of them square roots and reciprocals: with 64 cycles to each
// step of the FP64 pipe, 8,600 cycles for a lone warp and, on a busy SM, a
// pipe that takes 5,000 per pass. Here energies are integers in one unit and
// pressures (p, q and their sums) in another, both chosen per evaluation
// from the exponents of its inputs so that nothing can grow out of 60 bits:
// sums are integer adds, products 3 mul.wide and a shift. Reciprocals and
// square roots start from the float unit's approximation and take one
// third-order step.
//
// Precision. Energies keep about 2^-57 of the larger of the old energy and the
// work done, those before the viscosity enters (the predictor) of the old
// energy and the work of the old pressures alone: at a shock front the work of
// the viscosity is 2^20 to 2^35 times a cold element's energy, whose root is a
// factor of the viscosity. The pressure and the viscosity that come out are
// formed from the energy's and the root's own mantissas, not from the shared
// unit. Worst relative errors against extended precision, here and in plain
// double (e; 4,000 states each): front of du = 100, e = 1e-6, delv = -0.1:
// 1.6e-16, 7.9e-16 (in one unit 1.6e-13); bulk of e = 1000, delv = -0.01:
// 1.1e-16, 2.8e-16; opening by 0.1: 1.2e-16, 2.8e-16.
#pragma once

#include "block_fixed.cuh"

namespace lulesh {
namespace bf {

#ifdef __CUDACC__
LULESH_BF float seed_rcp(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
LULESH_BF float seed_rsqrt(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
LULESH_BF int lead_zeros64(int64_t v) { return __clzll(v); }
#else
LULESH_BF float seed_rcp(float x) { return 1.0f / x; }
LULESH_BF float seed_rsqrt(float x) { return 1.0f / sqrtf(x); }
LULESH_BF int lead_zeros64(int64_t v) { return v ? __builtin_clzll(uint64_t(v)) : 64; }
#endif

LULESH_BF int64_t mul(int64_t a, int64_t b) { return mul(limb(a), limb(b)); }

// 2^115 / m for m in [2^57, 2^58): a 24-bit approximation r of 2^81 / m, the
// exact remainder D = 2^81 - m r (below 2^60, so its low 64 bits are all of
// it) and 1 / (1 - d) = 1 + d + d^2 + ..., d = D / 2^81.
LULESH_BF int64_t reciprocal(int64_t m) {
    const int32_t r = int32_t(seed_rcp(float(int32_t(m >> 34))) * 140737488355328.0f);  // 2^47
    const Limb l = limb(m);
    const int64_t D = -(wide(l.l, r, 0) + int64_t(uint64_t(wide(l.h, r, 0)) << kLow));
    const int32_t dh = int32_t(D >> kLow);
    const Limb c = limb(D + (wide(dh, dh, 0) >> 23));
    return (int64_t(r) << 34) + (wide(r, c.h, wide(r, c.l, 0) >> kLow) >> 18);
}

// sqrt(m 2^58) for m in [2^56, 2^58): y, an approximation of 2^53 / sqrt(m)
// to 23 bits, d = 1 - m y^2 / 2^106, and m y (1 + d / 2 + 3 d^2 / 8).
LULESH_BF int64_t root(int64_t m) {
    const int32_t y = int32_t(seed_rsqrt(float(int32_t(m >> 34))) * 68719476736.0f);  // 2^36
    const Limb l = limb(m);
    const int64_t w = wide(y, y, 0);  // below 2^51
    const int32_t wh = int32_t(w >> 25), wl = int32_t(w) & 0x1ffffff;
    const int64_t D = (int64_t(1) << 58) - (wide(l.h, wh, 0) << 6) -
                      (wide(l.l, wh, (wide(l.h, wl, 0) << 4) + (wide(l.l, wl, 0) >> 25)) >> 23);
    const int32_t dq = int32_t(D >> 8);
    const int64_t C = (D >> 1) + ((3 * wide(dq, dq, 0)) >> 45);
    const int64_t s = (wide(l.h, y, 0) << 5) + (wide(l.l, y, 0) >> 24);
    return s + mul(s, C);
}

constexpr double kCold = 1e-30;  // energies above have more than the least sound speed, .3333333e-18

// The parameters the integer path depends on: it needs pmin = 0, a unit
// reference density and cutoffs that hide what it flushes to zero.
struct EosCuts {
    int64_t e_cut, p_cut;  // 58-bit mantissas
    int ue, up;            // and units
    int emin;              // the exponent of -emin
    bool ok;
};

LULESH_BF int exponent(double x) { return (high_word(x) >> 20) & 0x7ff; }
// The mantissa of x in [2^57, 2^58) with x's sign, in unit exponent(x) - 1080;
// 0 for zero and subnormals.
LULESH_BF int64_t mantissa(double x) {
    const int64_t b = bits_of(x);
    const int64_t m = ((b & 0xfffffffffffffll) | 0x10000000000000ll) << 5;
    return exponent(x) == 0 ? 0 : b < 0 ? -m : m;
}

LULESH_BF EosCuts eos_cuts(double e_cut, double p_cut, double q_cut, double pmin, double emin, double refdens) {
    EosCuts c;
    c.e_cut = mantissa(e_cut);
    c.p_cut = mantissa(p_cut);
    c.ue = exponent(e_cut) - 1080;
    c.up = exponent(p_cut) - 1080;
    c.emin = exponent(emin);
    // cutoffs in [2^-300, 2^300], as far from the flushed 2^-1022 as from overflow;
    // that of energies above those that have the least sound speed
    auto sane = [](double x) { return bits_of(x) >= bits_of(4.9e-91) && bits_of(x) <= bits_of(2.0e90); };
    c.ok = sane(e_cut) && bits_of(e_cut) >= bits_of(kCold) && sane(p_cut) && sane(q_cut) && bits_of(pmin) << 1 == 0 &&
           bits_of(emin) < 0 && bits_of(emin) << 1 != 0 &&
           uint64_t(bits_of(emin)) <= 0xfff0000000000000ull && bits_of(refdens) == bits_of(1.0);
    return c;
}

// A cutoff in units of 2^unit (at most 2^62).
LULESH_BF int64_t cut_in(int64_t m, int u, int unit) {
    const int n = unit - u;
    return n >= 0 ? m >> clamp63(n) : n >= -4 ? m << -n : int64_t(1) << 62;
}

constexpr int64_t kTwoThirds = 192153584101141162ll;   // 2/3 2^58
constexpr int64_t kThird = 96076792050570581ll;        // 1/3 2^58
// sqrt(10/9) 2^57 and sqrt(2/3) 2^57: the sound speed is the root of
// 2/3 (e + v p), where v p is 2/3 e unless the pressure was cut to zero
constexpr int64_t kRootFull = 151910746581081142ll;
constexpr int64_t kRootCut = 117669558323692511ll;

// sqrt(e) of an energy 0 < e < 2^60 in unit ue: a mantissa in [2^57, 2^58)
// and its unit. (Of e <= 0: some number; the callers drop it.)
LULESH_BF int64_t energy_root(int64_t e, int ue, int& us) {
    int n = lead_zeros64(e) - 6;  // to [2^57, 2^58), or half of it so that the unit is even
    n -= (ue - n) & 1;
    us = ((ue - n) >> 1) - 29;
    return root((e << (n + 3)) >> 3);
}

// One evaluation, and the sound speed of the state it ends with. False where
// the double path has to do it.
LULESH_BF bool eos_pass(double e_old, double p_old, double q_old, double ql, double qq, double delv, double v,
                        const EosCuts& cut, double& e_new, double& p_new, double& q_new, double& ss) {
    // opening: no viscosity, and qq and ql set no unit either
    const bool opening = bits_of(delv) > 0;
    ql = opening ? 0.0 : ql;
    qq = opening ? 0.0 : qq;
    const int xe = exponent(e_old), xp = exponent(p_old), xq = exponent(q_old), xl = exponent(ql), xqq = exponent(qq),
              xd = exponent(delv), xv = exponent(v);
    // everything normal or zero, of sane magnitude; v positive and |delv| below v / 2
    bool ok = max3(max3(xe, xp, xq), xl, xqq) < 1800 && xd + 2 <= xv && uint32_t((high_word(v) >> 20) - 701) < 699u;
    // |x| < 2^(exponent - 1022): tops of the pressures (tp) and energies (te),
    // which their sums pass by a factor 3 at most
    const int tb = opening ? 1024 - xv : 1023 - xv;  // of 2/3 / v and 2/3 / vhalf
    const int th = xd - 1023;                        // of delv / 2
    // before the viscosity enters: p + q of the old state, predicted energy
    const int tp0 = (xp > xq ? xp : xq) - 1021;
    int te = th + tp0 + 1 > xe - 1022 ? th + tp0 + 1 : xe - 1022;
    const int up0 = tp0 - 57, ue0 = te - 58;
    // and with it
    int tp = xqq - 1022 > tp0 ? xqq - 1022 : tp0;
    tp = te + tb > tp ? te + tb : tp;
    te = th + tp + 2 > te ? th + tp + 2 : te;
    const int tl = xl - 1022 + ((te + 3) >> 1);  // of the linear viscosity
    tp = te + tb > tp ? te + tb : tp;
    ok &= tl <= tp + 1;  // else the corrector's own sets a unit too coarse for the pressures it comes from
    tp = tl > tp ? tl : tp;
    te = th + tp + 2 > te ? th + tp + 2 : te;
    const int up = tp - 57, ue = te - 58;
    // no result below emin, infinite or subnormal
    ok &= cut.emin - 1023 > te + 3 && tp < 1000 && uint32_t(xl - 1) >= 200u;
    // Without energy the linear viscosity is .3333333e-18 ql, left out below:
    // less than half a last place of qq unless ql is above 2^7 qq, and of no
    // account while all energies are below the cutoff with and without it
    const int tc = cut.ue + 56;  // of half the cutoff
    ok &= xl <= xqq + 7 || (te < tc && xl - 1079 + th <= tc) || (high_word(e_old) > high_word(kCold) && xl < 1053);
    const int64_t po = mantissa(p_old) >> clamp63(up0 - (xp - 1080)), qo = mantissa(q_old) >> clamp63(up0 - (xq - 1080)),
                  qb = mantissa(qq) >> clamp63(up - (xqq - 1080)), ec = cut_in(cut.e_cut, cut.ue, ue);
    // volumes: 2/3 over the half-step one and the new one
    const int64_t mv = mantissa(v), md = mantissa(delv);
    int64_t mh = mv - (md >> clamp63(xv - xd + 1));  // in (2^56, 1.25 2^58)
    const int nh = lead_zeros(uint32_t(mh >> 32)) - 5;
    mh = (mh << nh) >> 1;
    const int uh = xv - 1080 + 1 - nh;
    const Limb bh = limb(mul(reciprocal(mh), kTwoThirds)), bv = limb(mul(reciprocal(mv), kTwoThirds));
    // pressures of an energy, in units of the energy's own precision: there the
    // cutoff is tested, which may be far below the unit of their sums
    const int uph = ue0 + 58 - 115 - uh, upv = ue + 58 - 115 - (xv - 1080);
    const int64_t pch = cut_in(cut.p_cut, cut.up, uph), pcv = cut_in(cut.p_cut, cut.up, upv);
    const int nph = up - uph, npv = up - upv;
    // work factors: delv / 2 in a unit that takes it to 2^59, delv / 6 in half of it.
    // (By the bounds te and tp: nph, npv >= 1, nw0 >= 0, nw >= 2, |pqh| below 2.7 2^57.)
    const Limb hd = limb(2 * md), d6 = limb(mul(md, 4 * kThird));
    const int nw0 = ue0 - (xd - 1082 + up0 + 58), nw = ue - (xd - 1082 + up + 58);
    const int sph = clamp63(nph), spv = clamp63(npv), sw2 = clamp63(nw - 2);
    const Limb lf = limb(mul(mantissa(ql), kRootFull)), lc = limb(mul(mantissa(ql), kRootCut));
    const int ul = xl - 1080 + 1, ql_unit = up - (ul + 58);
    // the viscosity of an energy, whose pressure may have been cut
    auto viscosity = [&](int64_t e, int unit, bool off) {
        int us;
        const int64_t s = energy_root(e, unit, us);
        const int n = ql_unit - us;
        const int64_t lin = mul(limb(s), off ? lc : lf) >> (n < 0 ? 0 : clamp63(n));
        ok &= n >= 0 || e <= 0;
        return (e > 0 ? lin : 0) + qb;
    };
    const int64_t kBig = int64_t(1) << 59;
    // predictor, in the units of what it is made of: those of the rest of the
    // evaluation follow the viscosity, which at a shock front is some 2^30
    // times the cold element's energy, and its root is a part of the result
    int64_t e = (mantissa(e_old) >> clamp63(ue0 - (xe - 1080))) - (mul(hd, limb(po + qo)) >> clamp63(nw0));
    ok &= e >= 0 || xl == 0;  // the unit of the pressures counts a root in
    int64_t p = mul(bh, limb(e));
    bool off = p < pch;
    p = off ? 0 : p >> sph;
    const int64_t pq = (po + qo) >> clamp63(up - up0);
    const int64_t pqh = p + viscosity(e, ue0, off);
    e = (e >> clamp63(ue - ue0)) + (mul(hd, limb((3 * pq - 4 * pqh) >> 2)) >> sw2);
    e = e < ec && e > -ec ? 0 : e;
    ok &= e < 2 * kBig && e > -2 * kBig;
    // corrector
    p = mul(bv, limb(e));
    off = p < pcv;
    p = off ? 0 : p >> spv;
    const int64_t pqt = p + viscosity(e, ue, off);
    ok &= pqt < kBig && pqt > -kBig;
    e -= mul(d6, limb((7 * pq - 8 * pqh + pqt) >> 3)) >> sw2;
    e = e < ec && e > -ec ? 0 : e;
    ok &= e < 2 * kBig && e > -2 * kBig;
    // the pressure, the viscosity and the sound speed from the energy's own
    // mantissa and root
    off = mul(bv, limb(e)) < pcv;
    const bool warm = e > 0;
    int us;
    const int64_t s = energy_root(e, ue, us);
    const int n = lead_zeros64(e) - 6;
    const int64_t m = (e << (n + 3)) >> 3;
    e_new = scaled(e, ue);
    p_new = warm && !off ? scaled(mul(bv, limb(m)), ue - n - 115 - (xv - 1080) + 58) : 0.0;
    const double lin = scaled(mul(limb(s), off ? lc : lf), us + ul + 58);
    q_new = (warm ? lin : .3333333e-18 * ql) + qq;
    ss = warm ? scaled(mul(s, off ? kRootCut : kRootFull), us + 1) : .3333333e-18;
    return ok;
}

// --- monotonic Q ------------------------------------------------------------

constexpr int64_t kOne = int64_t(1) << 57;  // 1 as a limiter

// The limiter phi = min((m + p) / 2, 2 m, 2 p) of one direction, cut to
// [0, 1], in units of 2^-57 (lulesh.cc:1464-1531): m and p are the
// neighbours' gradients dm and dp over self + 1e-36. A neighbour's gradient
// of more than 4 times self enters as 4 times self, which gives the same phi.
LULESH_BF bool limiter_fixed(double self, double dm, double dp, int64_t& phi) {
    const double s = self + 1.e-36;
    const int xs = exponent(s);
    auto part = [&](double d) {
        const int n = xs - exponent(d);
        const int64_t a = mantissa(d), big = a < 0 ? -(int64_t(1) << 60) : int64_t(1) << 60;
        return n >= 0 ? a >> clamp63(n) : n >= -2 ? a << -n : big;
    };
    const int64_t ms = mantissa(s), flip = ms >> 63;  // -1 for a negative self
    const int64_t am = (part(dm) ^ flip) - flip, ap = (part(dp) ^ flip) - flip, as = (ms ^ flip) - flip;
    int64_t c = (am + ap) >> 1;
    const int64_t lo = am < ap ? am : ap;
    c = 2 * lo < c ? 2 * lo : c;
    c = c < 0 ? 0 : c;
    const bool full = c >= as;  // then exactly 1
    phi = full ? kOne : mul(c, reciprocal(as));
    return xs != 0 && xs != 0x7ff && exponent(dm) != 0x7ff && exponent(dp) != 0x7ff;
}

// The linear and quadratic viscosity coefficients (lulesh.cc:1600-1656):
// ql = -qlc rho sum dxi (1 - phi), qq = qqc rho sum dxi^2 (1 - phi^2) with
// dxi = min(0, delv delx) of each direction; subnormal gradients count as
// zero. False where the double path has to do it.
LULESH_BF bool q_sums(const double dv[3], const double dm[3], const double dp[3], const double dx[3], double& lin,
                      double& quad) {
    bool ok = true;
    lin = quad = 0.0;
    LULESH_UNROLL
    for (int d = 0; d < 3; ++d) {
        int64_t phi;
        ok &= limiter_fixed(dv[d], dm[d], dp[d], phi);
        const int xv = exponent(dv[d]), xx = exponent(dx[d]);
        ok &= uint32_t(xx - 501) < 999u;
        const int64_t t = mul(mantissa(dv[d]), mantissa(dx[d]));  // delv delx, up to 2^58
        // delv delx, its square and 2^-57 of that are normal numbers
        ok &= t >= 0 || uint32_t(xv + xx - (2046 - 480)) < 960u;
        const bool push = t < 0;
        const int u = xv + xx - 2160 + 58;
        // 1 - phi at full width, and with it 1 - phi^2 = (1 - phi) (1 + phi)
        const int64_t rest = kOne - phi;
        const int n = lead_zeros64(rest) - 6;
        const Limb l = limb(t), w = limb(rest << n), w2 = limb(mul(w, limb((kOne + phi) >> 1)));
        lin += push ? scaled(mul(neg(l), w), u + 1 - n) : 0.0;
        quad += push ? scaled(mul(limb(mul(l, l)), w2), 2 * u + 61 - n) : 0.0;
    }
    return ok;
}

}  // namespace bf
}  // namespace lulesh
