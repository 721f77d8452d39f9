// Block fixed point: sums and products of doubles on the integer pipes.
//
// GB300's FP64 pipe takes 62 cycles for a warp's double multiply-add and 73
// for an add (per SM quarter); a 64-bit integer add takes 2 and a 32 x 32 bit
// product of 64 bits (mul.wide) 3. The element kernels' vector arithmetic,
// sums of corner values and products of such sums, therefore runs in
// 64-bit integers that share one power-of-two unit per block of values:
//
//   * fix8 turns 8 doubles into integers up to 2^54 (or 2^55) in a unit set
//     by the largest of them. Corners within a factor 2 (4) of it are exact
//     (53 bits), so sums of corners are exact where a double sum would round.
//   * a value splits into limbs h * 2^29 + l; a product adds h h' to one
//     64-bit sum and h l' + l h' to another (3 mul.wide), and their value, in
//     units of 2^58 of the product, is off by about one unit: some 2^-56 of
//     the block's largest product, against 2^-53 of each product and each
//     sum in double.
//   * values are shifted up to a block's full width before they are
//     multiplied again, so no leading zeros are carried along.
//
// Bounds. One factor of a product stays below 2^58 and the other below 2^60,
// with at most 6 products to a sum: h h' <= 2^60 and h l' + l h' <= 1.25 2^60
// each, so the sums fit 64 bits. The comments give each value's bound.
//
// Units are tracked as plain integers. Inputs that do not fit (infinite,
// NaN, above 2^53 or all below 2^-959) make the callers take their double
// path instead.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#include "fp64_emu.cuh"
#endif

#ifdef __CUDACC__
#define LULESH_BF static __device__ __forceinline__
#define LULESH_UNROLL _Pragma("unroll")
#else  // the host build of the accuracy checks
#include <math.h>
#include <string.h>
#define LULESH_BF static inline
#define LULESH_UNROLL
#endif

namespace lulesh {
namespace bf {

constexpr int kLow = 29;         // bits of the low limb
constexpr int kUnit = 2 * kLow;  // a product's value is in units of 2^kUnit
constexpr int kBias = 1019;      // + width: exponent field of the largest value whose fix8 unit is 1
constexpr int kLeast = 64;       // exponent field of the largest value of a fix8 block that is not zero, at least

struct Limb {
    int32_t h, l;
};
struct Acc {
    int64_t hh, mid;
};

#ifdef __CUDACC__
LULESH_BF int64_t bits_of(double x) { return __double_as_longlong(x); }
// The bits for a test of the whole of them: seen as a double's, the compiler
// would make it an FP64 compare (dmul_bits). Not for every use: the opaque
// move keeps it from sharing work too (the EOS and Q terms, which use none,
// take 0.628 ms at s=150, with it 0.644).
LULESH_BF int64_t tested_bits(double x) { return static_cast<int64_t>(dmul_bits(x)); }
LULESH_BF double of_bits(int64_t b) { return __longlong_as_double(b); }
LULESH_BF int32_t high_word(double x) { return int32_t(bits_of(x) >> 32); }
// x times 2^k through the exponent field (x normal; of 0 and subnormals up to 2^(k - 1022))
LULESH_BF double up_exponent(double x, int k) { return __hiloint2double(__double2hiint(x) + (k << 20), __double2loint(x)); }
LULESH_BF int64_t round_to_int(double x) { return __double2ll_rn(x); }
LULESH_BF double to_double(int64_t v) { return __ll2double_rn(v); }
LULESH_BF int lead_zeros(uint32_t v) { return __clz(int(v)); }
// Product and sum apart: a multiply-add with a 64-bit addend takes 6.2 cycles
// of its pipe, the product alone 3.3 and the addition, two to three of which
// go together, runs on others (s=150: forces 0.90 -> 0.78 ms, kinematics
// 0.69 -> 0.65, material 0.66 -> 0.63).
LULESH_BF int64_t wide(int32_t a, int32_t b, int64_t c) {
    int64_t r;
    asm("mul.wide.s32 %0, %1, %2;" : "=l"(r) : "r"(a), "r"(b));
    return r + c;
}
// v << s as limbs for 0 <= s < 29
LULESH_BF Limb limb_up(int64_t v, int s) {
    return {int32_t(__funnelshift_r(uint32_t(v), uint32_t(v >> 32), kLow - s)),
            int32_t((uint32_t(v) << s) & ((1u << kLow) - 1u))};
}
#else
LULESH_BF int64_t bits_of(double x) { int64_t b; memcpy(&b, &x, 8); return b; }
LULESH_BF int64_t tested_bits(double x) { return bits_of(x); }
LULESH_BF double of_bits(int64_t b) { double x; memcpy(&x, &b, 8); return x; }
LULESH_BF int32_t high_word(double x) { return int32_t(bits_of(x) >> 32); }
LULESH_BF double up_exponent(double x, int k) { return of_bits(bits_of(x) + int64_t(uint64_t(int64_t(k)) << 52)); }
LULESH_BF int64_t round_to_int(double x) { return llrint(x); }
LULESH_BF double to_double(int64_t v) { return double(v); }
LULESH_BF int lead_zeros(uint32_t v) { return v ? __builtin_clz(v) : 32; }
LULESH_BF int64_t wide(int32_t a, int32_t b, int64_t c) { return int64_t(a) * b + c; }
LULESH_BF Limb limb_up(int64_t v, int s) {
    const int64_t w = int64_t(uint64_t(v) << s);
    return {int32_t(w >> kLow), int32_t(w) & ((1 << kLow) - 1)};
}
#endif

LULESH_BF Limb limb(int64_t v) { return {int32_t(v >> kLow), int32_t(v) & ((1 << kLow) - 1)}; }
LULESH_BF Limb neg(Limb a) { return {-a.h, -a.l}; }
LULESH_BF Acc product(Limb a, Limb b) {
    return {wide(a.h, b.h, 0), wide(a.l, b.h, wide(a.h, b.l, int64_t(1) << (kLow - 1)))};
}
LULESH_BF void mac(Acc& s, Limb a, Limb b) {
    s.hh = wide(a.h, b.h, s.hh);
    s.mid = wide(a.l, b.h, wide(a.h, b.l, s.mid));
}
LULESH_BF Acc self_product(Limb a) { return {wide(a.h, a.h, 0), wide(a.l, 2 * a.h, int64_t(1) << (kLow - 1))}; }
LULESH_BF void mac_self(Acc& s, Limb a) {
    s.hh = wide(a.h, a.h, s.hh);
    s.mid = wide(a.l, 2 * a.h, s.mid);
}
LULESH_BF int64_t value(Acc s) { return s.hh + (s.mid >> kLow); }
LULESH_BF int64_t mul(Limb a, Limb b) { return value(product(a, b)); }
// The same with the middle products' sum cut at its high word: off by up to 4
// units (some 2^-54 of the block's largest product, still below what double
// sums of them lose), for two instructions in place of four.
LULESH_BF int64_t near(Acc s) { return wide(int32_t((s.mid + (int64_t(1) << 31)) >> 32), 8, s.hh); }
LULESH_BF int64_t mul_near(Limb a, Limb b) { return near(product(a, b)); }

// The width of a block: the largest high word of its values or of their
// complements, two values to an instruction.
#ifdef __CUDACC__
LULESH_BF int32_t max3(int32_t a, int32_t b, int32_t c) { return __vimax3_s32(a, b, c); }
LULESH_BF int32_t min3(int32_t a, int32_t b, int32_t c) { return __vimin3_s32(a, b, c); }
#else
LULESH_BF int32_t max3(int32_t a, int32_t b, int32_t c) { return a > b ? (a > c ? a : c) : (b > c ? b : c); }
LULESH_BF int32_t min3(int32_t a, int32_t b, int32_t c) { return a < b ? (a < c ? a : c) : (b < c ? b : c); }
#endif
struct Top {
    int32_t hi = 0, lo = 0;
#ifdef __CUDACC__
    __device__ __forceinline__
#endif
    void add(int64_t v, int64_t w) {
        hi = max3(hi, int32_t(v >> 32), int32_t(w >> 32));
        lo = min3(lo, int32_t(v >> 32), int32_t(w >> 32));
    }
#ifdef __CUDACC__
    __device__ __forceinline__
#endif
    void add(int64_t v) { add(v, v); }
};
LULESH_BF uint32_t top_bits(Top t) { return uint32_t(t.hi > ~t.lo ? t.hi : ~t.lo); }
// Left shift that brings a block of values below 2^top to at least 2^(top - 1)
// (or by top - 32, when all are below 2^32).
LULESH_BF int room(Top m, int top) { return lead_zeros(top_bits(m)) - (64 - top); }
LULESH_BF int64_t down(int64_t v, int s) { return v >> s; }
LULESH_BF int clamp63(int s) { return s < 63 ? s : 63; }

// 8 doubles as integers up to 2^(WIDTH - 3), so that their signed sums stay
// below 2^WIDTH, times 2^unit. False where they do not fit, as where all are
// below 2^-959 but not all zero. CVT: a block of zeros, of either sign, is all
// zero. Else its values are +-2^(WIDTH - 4) by their signs, in a unit below
// kUnitMin: the callers send it to their double path unless all sums cancel.
template <int WIDTH, bool CVT>
LULESH_BF bool fix8(const double v[8], int64_t q[8], int& unit) {
    int32_t top = 0, low = 0;
    LULESH_UNROLL
    for (int k = 0; k < 8; ++k) {
        const int32_t m = high_word(v[k]) & 0x7fffffff;
        top = m > top ? m : top;
        low |= int32_t(bits_of(v[k]));
    }
    const int e = top >> 20;
    // all that fit but zeros have e >= kLeast; the exponent of these then
    // becomes that of 2^-11 or less
    const int up = kBias + WIDTH - (e > kLeast ? e : kLeast);
    unit = e - (kBias + WIDTH);
    // CVT: by the FP64 pipe's conversion, 62 cycles. Else the significand is
    // shifted into place by 15 integer instructions. The kernels take what
    // balances their pipes: kinematics, with 80 FP64 instructions of other
    // kinds, the latter (s=150: 0.717 -> 0.633 ms), forces the former for the
    // velocities only (0.780; 0.790 with integers for all, 0.819 with
    // conversions for all, 0.803 the other way round).
    LULESH_UNROLL
    for (int k = 0; k < 8; ++k) {
        if (CVT) {
            q[k] = round_to_int(up_exponent(v[k], up));
            continue;
        }
        const int64_t b = bits_of(v[k]);
        const int n = e - (int(b >> 52) & 0x7ff);
        const uint64_t m = uint64_t((b & 0xfffffffffffffll) | 0x10000000000000ll) << (WIDTH - 56);
        const int64_t a = int64_t(m >> clamp63(n)), s = b >> 63;
        q[k] = (a ^ s) - s;
    }
    return (CVT ? top | low : top) == 0 || (e >= kLeast && e <= kBias + WIDTH);
}

// A normal double as limbs (below 2^58) and unit; false for 0, subnormals,
// infinities and NaN.
LULESH_BF bool fix1(double x, Limb& v, int& unit) {
    const int64_t b = bits_of(x);
    const int e = int(b >> 52) & 0x7ff;
    unit = e - (1023 + kUnit - 1);
    const int64_t m = ((b & 0xfffffffffffffll) | 0x10000000000000ll) << (kUnit - 53);
    v = limb(b < 0 ? -m : m);
    return e != 0 && e != 0x7ff;
}

// v * 2^unit as a double (correctly rounded while the result is normal).
LULESH_BF double scaled(int64_t v, int unit) {
    const double d = to_double(v);
    return v == 0 ? 0.0 : up_exponent(d, unit);
}

// The non-constant coefficients of the Walsh-Hadamard transform over the
// corners' (xi, eta, zeta) signs: d along xi, eta, zeta; h the modes eta
// zeta, zeta xi, xi eta, xi eta zeta. Exact.
LULESH_BF void walsh(const int64_t v[8], int64_t d[3], int64_t h[4]) {
    const int64_t p00 = v[1] + v[0], m00 = v[1] - v[0], p10 = v[2] + v[3], m10 = v[2] - v[3];
    const int64_t p01 = v[5] + v[4], m01 = v[5] - v[4], p11 = v[6] + v[7], m11 = v[6] - v[7];
    const int64_t pp0 = p10 + p00, pm0 = p10 - p00, mp0 = m10 + m00, mm0 = m10 - m00;
    const int64_t pp1 = p11 + p01, pm1 = p11 - p01, mp1 = m11 + m01, mm1 = m11 - m01;
    d[0] = mp1 + mp0;
    d[1] = pm1 + pm0;
    d[2] = pp1 - pp0;
    h[0] = pm1 - pm0;
    h[1] = mp1 - mp0;
    h[2] = mm1 + mm0;
    h[3] = mm1 - mm0;
}
// Its inverse without the constant and the factor 1/8: corner values of the
// coefficients d and h.
LULESH_BF void walsh_corners(const int64_t d[3], const int64_t h[4], int64_t v[8]) {
    LULESH_UNROLL
    for (int t = 0; t < 2; ++t) {  // zeta = -1 (corners 0..3), +1 (corners 4..7)
        // x: multiplies xi, y: eta, c: constant, e: xi eta
        const int64_t x = t ? d[0] + h[1] : d[0] - h[1], y = t ? d[1] + h[0] : d[1] - h[0];
        const int64_t c = t ? d[2] : -d[2], e = t ? h[2] + h[3] : h[2] - h[3];
        const int64_t p = x + y, q = x - y, ce = c + e, cm = c - e;
        v[4 * t + 0] = ce - p;
        v[4 * t + 1] = cm + q;
        v[4 * t + 2] = ce + p;
        v[4 * t + 3] = cm - q;
    }
}

// Component a of u x v, and of u x v + w x z.
LULESH_BF Acc cross(const Limb u[3], const Limb v[3], int a) {
    const int b = (a + 1) % 3, c = (a + 2) % 3;
    Acc s = product(u[b], v[c]);
    mac(s, neg(u[c]), v[b]);
    return s;
}
LULESH_BF Acc cross2(const Limb u[3], const Limb v[3], const Limb w[3], const Limb z[3], int a) {
    const int b = (a + 1) % 3, c = (a + 2) % 3;
    Acc s = cross(u, v, a);
    mac(s, w[b], z[c]);
    mac(s, neg(w[c]), z[b]);
    return s;
}

// Units outside this range (coordinates below 2^-195) take the double path,
// so that products of three of them stay normal doubles.
constexpr int kUnitMin = -250;

// The body-diagonal sums A_d (d = xi, eta, zeta) and mode sums H_m of the
// corner coordinates, each axis a in its own unit 2^unit[a] at full width.
struct Sums {
    Limb A[3][3], H[4][3];  // [direction or mode][axis]
    int unit[3];
};

template <int WIDTH, bool CVT>
LULESH_BF bool axis_sums(const double x[8], int a, Sums& s) {
    int64_t q[8], d[3], h[4];
    const bool ok = fix8<WIDTH, CVT>(x, q, s.unit[a]);
    walsh(q, d, h);
    Top m;
    m.add(d[0], d[1]);
    m.add(d[2], h[0]);
    m.add(h[1], h[2]);
    m.add(h[3]);
    const int up = room(m, WIDTH);
    s.unit[a] -= up;
    LULESH_UNROLL
    for (int k = 0; k < 3; ++k) s.A[k][a] = limb_up(d[k], up);
    LULESH_UNROLL
    for (int k = 0; k < 4; ++k) s.H[k][a] = limb_up(h[k], up);
    return ok && s.unit[a] > kUnitMin;
}

// --- corner forces (from sums of width 57) ----------------------------------
//
// Everything is kept in the Walsh basis of the corners' signs, where the
// geometry is a few cross products of the sums:
//   c_d = A_{d+1} x A_{d+2}, e_d = H_{d+2} x H_{d+1} (modes eta zeta, zeta xi, xi eta)
//   face area vectors summed per corner: sum_d sign_d (c_d + e_d) / 8 (the
//     terms linear in H cancel over the closed surface)
//   192 dV/dx: g_d = 3 c_d + e_d along d and H_{d+2} x A_{d+1} + A_{d+2} x H_{d+1}
//     along mode d (the trilinear hexahedron's volume, as volume_gradient)
// and the hourglass force (lulesh.cc:965-1063) with the shape vectors
// gamma_m - (g . H_m) / (192 V) is, per velocity component,
//   T = g . V^,  amp_m = W_m - H_m . T sc,  U = sum_m H_m amp_m sc,
//   force = coefficient (sum_m gamma_m amp_m - g . U),
// V^ and W the velocity's transform, sc = 1 / (192 volo v): no 8 x 4 shape
// vectors, 252 products where the corner form takes 330 and 190 sums.

struct ForceGeo {
    Limb g[6][3], H[4][3];  // g below 2^58, H below 2^57
    int64_t n[3][3];        // c_d + e_d [d][axis], unit 2^(58 + cross - unit[axis]), up to 2^58
    int unit[3];
    int cross;              // sum of the axes' units
    int gshift;             // g is shifted left by this
};

// False when the double path must decide: a centre Jacobian determinant at
// or near zero.
LULESH_BF bool force_geometry(const Sums& s, ForceGeo& o) {
    int64_t g[6][3];
    Top m;
    bool ok = true;
    LULESH_UNROLL
    for (int d = 0; d < 3; ++d) {
        const int i = (d + 1) % 3, j = (d + 2) % 3;
        Acc det;
        LULESH_UNROLL
        for (int a = 0; a < 3; ++a) {
            const int64_t c = value(cross(s.A[i], s.A[j], a));  // up to 2^57
            const int64_t e = value(cross(s.H[j], s.H[i], a));
            o.n[d][a] = c + e;
            g[d][a] = (o.n[d][a] + 2 * c) >> 1;  // up to 2^58
            g[3 + d][a] = value(cross2(s.H[j], s.A[i], s.A[j], s.H[i], a)) >> 1;
            m.add(g[d][a], g[3 + d][a]);
            if (d == 0) {
                if (a == 0) det = product(s.A[0][a], limb(c));
                else mac(det, s.A[0][a], limb(c));
            }
        }
        if (d == 0) {
            const int64_t v = value(det);
            ok = v > 64 || v < -64;
        }
    }
    const int up = room(m, kUnit);
    o.gshift = up - 1;
    LULESH_UNROLL
    for (int a = 0; a < 3; ++a) {
        LULESH_UNROLL
        for (int j = 0; j < 6; ++j) o.g[j][a] = limb_up(g[j][a], up);
        LULESH_UNROLL
        for (int k = 0; k < 4; ++k) o.H[k][a] = s.H[k][a];
        o.unit[a] = s.unit[a];
    }
    o.cross = s.unit[0] + s.unit[1] + s.unit[2];
    return ok;
}

// The scalars of an element's force as limbs: sc = 1 / (192 volo v), the
// hourglass coefficient and the stress p + q over 64.
LULESH_BF bool is_zero(double x) { return uint64_t(tested_bits(x)) << 1 == 0; }
constexpr int kNone = -20000;  // unit of a part that is zero
struct ForceScale {
    Limb sc, coef, press;
    int kappa;  // exponent of g H sc (as integers) relative to 1
    int ucoef, upress;
};
LULESH_BF bool force_scale(const ForceGeo& o, double sc, double coef, double press, ForceScale& f) {
    int usc;
    bool ok = fix1(sc, f.sc, usc);
    f.kappa = 4 * kUnit - o.gshift + o.cross + usc;
    ok &= fix1(coef, f.coef, f.ucoef) | is_zero(coef);
    ok &= fix1(press, f.press, f.upress) | is_zero(press);
    f.upress += 2 * kUnit + o.cross - 6;
    if (is_zero(coef)) {
        f.coef = {0, 0};
        f.ucoef = kNone;
    }
    if (is_zero(press)) {
        f.press = {0, 0};
        f.upress = kNone;
    }
    return ok;
}

// Corner forces along one axis for the corner velocities vel; n and unit_a
// are the axis' column of ForceGeo::n and its unit.
LULESH_BF bool force_axis(const ForceGeo& o, const ForceScale& f, const int64_t n[3], int unit_a, const double vel[8],
                          double out[8]) {
    int64_t q[8], v[3], amp[4];
    int unit;
    bool ok = fix8<kUnit - 1, true>(vel, q, unit);
    const bool still = unit == -(kBias + kUnit - 1);  // all zero, or none of it fits
    walsh(q, v, amp);
    Top m;
    m.add(v[0], v[1]);
    m.add(v[2], amp[0]);
    m.add(amp[1], amp[2]);
    m.add(amp[3]);
    const int up = room(m, kUnit - 1);
    unit -= up;
    Limb vl[6];  // below 2^57
    LULESH_UNROLL
    for (int d = 0; d < 3; ++d) vl[d] = limb_up(v[d], up);
    LULESH_UNROLL
    for (int k = 0; k < 3; ++k) vl[3 + k] = limb_up(amp[k], up);
    LULESH_UNROLL
    for (int k = 0; k < 4; ++k) amp[k] <<= up;
    // T, up to 6 2^57 / 2
    int64_t t[3];
    LULESH_UNROLL
    for (int a = 0; a < 3; ++a) {
        Acc s = product(o.g[0][a], vl[0]);
        LULESH_UNROLL
        for (int j = 1; j < 6; ++j) mac(s, o.g[j][a], vl[j]);
        t[a] = near(s) >> 1;
    }
    Top mt;
    mt.add(t[0], t[1]);
    mt.add(t[2]);
    const int nt = room(mt, kUnit + 1);
    Limb tl[3];  // below 2^59
    LULESH_UNROLL
    for (int a = 0; a < 3; ++a) tl[a] = limb_up(t[a], nt);
    // H_m . T, up to 3 2^58, then times sc; a correction that does not fit
    // beside W takes the double path
    int64_t r[4];
    LULESH_UNROLL
    for (int k = 0; k < 4; ++k) {
        Acc s = product(o.H[k][0], tl[0]);
        mac(s, o.H[k][1], tl[1]);
        mac(s, o.H[k][2], tl[2]);
        r[k] = near(s);
    }
    Top mp, mr, ma;
    mp.add(r[0], r[1]);
    mp.add(r[2], r[3]);
    const int np = room(mp, kUnit + 2);
    LULESH_UNROLL
    for (int k = 0; k < 4; ++k) r[k] = mul_near(limb_up(r[k], np), f.sc);
    mr.add(r[0], r[1]);
    mr.add(r[2], r[3]);
    int right = nt - 1 + np - f.kappa;
    ok &= right >= 0 && lead_zeros(top_bits(mr)) + right >= 6;  // below 2^58
    right = clamp63(right);
    LULESH_UNROLL
    for (int k = 0; k < 4; ++k) amp[k] -= down(r[k], right);
    ma.add(amp[0], amp[1]);
    ma.add(amp[2], amp[3]);
    const int na = room(ma, kUnit + 1);
    unit -= na;
    Limb al[4];  // below 2^59
    LULESH_UNROLL
    for (int k = 0; k < 4; ++k) {
        al[k] = limb_up(amp[k], na);
        amp[k] <<= na;
    }
    // U, up to 4 2^58, then times sc
    LULESH_UNROLL
    for (int a = 0; a < 3; ++a) {
        Acc s = product(o.H[0][a], al[0]);
        LULESH_UNROLL
        for (int k = 1; k < 4; ++k) mac(s, o.H[k][a], al[k]);
        t[a] = mul_near(limb(near(s)), f.sc);
    }
    Top mu;
    mu.add(t[0], t[1]);
    mu.add(t[2]);
    const int nu = room(mu, kUnit + 2);
    LULESH_UNROLL
    for (int a = 0; a < 3; ++a) tl[a] = limb_up(t[a], nu);
    // coefficients of the force in the Walsh basis
    int64_t w[7];
    right = nu - f.kappa;
    ok &= right >= 0;
    right = clamp63(right);
    Top mc, mw;
    LULESH_UNROLL
    for (int j = 0; j < 6; ++j) {
        Acc s = product(o.g[j][0], tl[0]);
        mac(s, o.g[j][1], tl[1]);
        mac(s, o.g[j][2], tl[2]);
        w[j] = near(s);
    }
    mc.add(w[0], w[1]);
    mc.add(w[2], w[3]);
    mc.add(w[4], w[5]);
    ok &= lead_zeros(top_bits(mc)) + right >= 5;  // below 2^59, so w stays below 2^60
    LULESH_UNROLL
    for (int j = 0; j < 6; ++j) w[j] = (j >= 3 ? amp[j - 3] : 0) - down(w[j], right);
    w[6] = amp[3];
    mw.add(w[0], w[1]);
    mw.add(w[2], w[3]);
    mw.add(w[4], w[5]);
    mw.add(w[6]);
    const int nw = room(mw, kUnit + 2);
    const int u1 = still ? kNone : kUnit + unit + f.ucoef - nw;
    // stress
    Top mn;
    mn.add(n[0], n[1]);
    mn.add(n[2]);
    const int ns = room(mn, kUnit + 2);
    const int u2 = f.upress - unit_a - ns;
    const int u = u1 > u2 ? u1 : u2, s1 = clamp63(u - u1), s2 = clamp63(u - u2);
    int64_t x[3], h[4];  // up to 2 2^60 and 2^60: a quarter of it in the corner sums
    LULESH_UNROLL
    for (int d = 0; d < 3; ++d)
        x[d] = (down(mul(limb_up(w[d], nw), f.coef), s1) + down(mul(limb_up(n[d], ns), f.press), s2)) >> 2;
    LULESH_UNROLL
    for (int k = 0; k < 4; ++k) h[k] = down(mul(limb_up(w[3 + k], nw), f.coef), s1) >> 2;
    walsh_corners(x, h, q);
    LULESH_UNROLL
    for (int k = 0; k < 8; ++k) out[k] = scaled(q[k], u + 2);
    // a unit by kNone: both parts are zero, and so is every q[k]
    return ok && (u < kNone / 2 || (u > -1000 && u < 950));
}

// --- kinematics (from sums of width 58) --------------------------------------
//
// From the same sums: the volume 192 V = sum_d A_d . (c_d + e_d), the largest
// face measure (the area vector of face d = +-1 is (+-(c_d + e_d) + P_{d+1} -
// P_{d+2}) / 8 with P_d = A_d x H_d), the Q gradients' |c_d|^2 and c_d . V_d,
// and det(A - t V) = det A - t sum c_d . V_d + t^2 sum A_d . k_d - t^3 det V
// (k the cofactors of V), whose derivative in t is minus the numerator of the
// velocity gradient's trace.
struct KinGeo {
    double vol192, face2;  // 192 V, the largest |8 x area vector|^2
    double cc[3], det;     // |c_d|^2, det A
    Limb A[3][3], c[3][3];
    int unit[3], cross;
};

// Axes whose units differ by more than this (an element some 8 to 16 times
// longer than wide) take the double path: squares of vectors are summed in
// the coarsest axis' unit, which costs their components that many bits. A
// mesh of nothing but such elements pays for both paths: s=150, 32 times
// wider than high, k_kinematics 2.42 ms in place of 0.64 (the double path by
// itself took 2.09; the forces stay at 0.78).
constexpr int kAspect = 3;

LULESH_BF bool kin_geometry(const Sums& s, KinGeo& o) {
    int lo = s.unit[0], hi = s.unit[0];
    LULESH_UNROLL
    for (int a = 1; a < 3; ++a) {
        lo = s.unit[a] < lo ? s.unit[a] : lo;
        hi = s.unit[a] > hi ? s.unit[a] : hi;
    }
    const bool ok = hi - lo <= kAspect;
    o.cross = s.unit[0] + s.unit[1] + s.unit[2];
    const int square = kUnit + 2 * (kUnit + o.cross - lo);  // unit of a square of vectors in the coarsest unit
    int64_t n[3][3];
    Top mn;
    int coarse[3];
    LULESH_UNROLL
    for (int a = 0; a < 3; ++a) coarse[a] = clamp63(s.unit[a] - lo);
    LULESH_UNROLL
    for (int d = 0; d < 3; ++d) {
        const int i = (d + 1) % 3, j = (d + 2) % 3;
        int64_t cs[3];
        LULESH_UNROLL
        for (int a = 0; a < 3; ++a) {
            const int64_t c = value(cross(s.A[i], s.A[j], a));  // up to 2^59
            n[d][a] = (c + value(cross(s.H[j], s.H[i], a))) >> 2;
            o.c[d][a] = limb(c);
            cs[a] = down(c, clamp63(coarse[a] + 1));
        }
        mn.add(n[d][0], n[d][1]);
        mn.add(n[d][2]);
        Top m;
        m.add(cs[0], cs[1]);
        m.add(cs[2]);
        const int up = room(m, kUnit);
        const Limb l0 = limb_up(cs[0], up), l1 = limb_up(cs[1], up), l2 = limb_up(cs[2], up);
        Acc sq = self_product(l0);
        mac_self(sq, l1);
        mac_self(sq, l2);
        o.cc[d] = scaled(value(sq), square - 2 * (up - 1));
    }
    const int nv = room(mn, kUnit);
    Acc det, vol;
    LULESH_UNROLL
    for (int a = 0; a < 3; ++a) {
        if (a == 0) det = product(s.A[0][a], o.c[0][a]);
        else mac(det, s.A[0][a], o.c[0][a]);
        LULESH_UNROLL
        for (int d = 0; d < 3; ++d) {
            if (a + d == 0) vol = product(s.A[d][a], limb_up(n[d][a], nv));
            else mac(vol, s.A[d][a], limb_up(n[d][a], nv));
        }
    }
    o.det = scaled(value(det), 2 * kUnit + o.cross);
    o.vol192 = scaled(value(vol), 2 * kUnit + o.cross + 2 - nv);
    // faces: an eighth of n and of the differences of P in the coarsest unit, up to 2^57
    int64_t p[3][3];
    Top m;
    LULESH_UNROLL
    for (int a = 0; a < 3; ++a) {
        const int64_t p0 = value(cross(s.A[0], s.H[0], a)), p1 = value(cross(s.A[1], s.H[1], a)),
                      p2 = value(cross(s.A[2], s.H[2], a));
        const int down3 = clamp63(coarse[a] + 3), down1 = clamp63(coarse[a] + 1);
        p[0][a] = down(p1 - p2, down3);
        p[1][a] = down(p2 - p0, down3);
        p[2][a] = down(p0 - p1, down3);
        LULESH_UNROLL
        for (int d = 0; d < 3; ++d) {
            n[d][a] = down(n[d][a], down1);
            m.add(p[d][a], n[d][a]);
        }
    }
    const int nf = room(m, kUnit - 1);
    int64_t top = 0;
    LULESH_UNROLL
    for (int d = 0; d < 3; ++d) {
        Acc plus, minus;
        LULESH_UNROLL
        for (int a = 0; a < 3; ++a) {
            const Limb lp = limb_up(n[d][a] + p[d][a], nf), lm = limb_up(n[d][a] - p[d][a], nf);
            if (a == 0) {
                plus = self_product(lp);
                minus = self_product(lm);
            } else {
                mac_self(plus, lp);
                mac_self(minus, lm);
            }
        }
        const int64_t vp = value(plus), vm = value(minus);
        top = vp > top ? vp : top;
        top = vm > top ? vm : top;
    }
    o.face2 = scaled(top, square - 2 * (nf - 3));
    LULESH_UNROLL
    for (int a = 0; a < 3; ++a) {
        o.unit[a] = s.unit[a];
        LULESH_UNROLL
        for (int d = 0; d < 3; ++d) o.A[d][a] = s.A[d][a];
    }
    return ok;
}

// The body-diagonal sums of the corner velocities along axis a.
struct VelSums {
    Limb V[3][3];  // [direction][axis]
    int unit[3];
};
LULESH_BF bool vel_sums(const double v[8], int a, VelSums& o) {
    int64_t q[8], d[3], h[4];
    int unit;
    const bool ok = fix8<kUnit, false>(v, q, unit);
    walsh(q, d, h);
    Top m;
    m.add(d[0], d[1]);
    m.add(d[2]);
    const int up = room(m, kUnit);
    LULESH_UNROLL
    for (int k = 0; k < 3; ++k) o.V[k][a] = limb_up(d[k], up);
    const bool zero = (d[0] | d[1] | d[2]) == 0;
    o.unit[a] = zero ? 0 : unit - up;
    return ok && o.unit[a] > kUnitMin;
}

struct KinVel {
    double cv[3], ak, detv;  // c_d . V_d, sum A_d . k_d, det V
};
LULESH_BF void kin_velocity(const KinGeo& g, const VelSums& v, KinVel& o) {
    const int all = v.unit[0] + v.unit[1] + v.unit[2];
    Limb k[3][3];
    LULESH_UNROLL
    for (int d = 0; d < 3; ++d) {
        const int i = (d + 1) % 3, j = (d + 2) % 3;
        double cv = 0.0;
        LULESH_UNROLL
        for (int a = 0; a < 3; ++a) {
            k[d][a] = limb(value(cross(v.V[i], v.V[j], a)));
            const double t = scaled(mul(g.c[d][a], v.V[d][a]), 2 * kUnit + g.cross - g.unit[a] + v.unit[a]);
            cv = a == 0 ? t : cv + t;
        }
        o.cv[d] = cv;
    }
    Acc det;
    o.ak = 0.0;
    LULESH_UNROLL
    for (int a = 0; a < 3; ++a) {
        Acc s = product(g.A[0][a], k[0][a]);
        mac(s, g.A[1][a], k[1][a]);
        mac(s, g.A[2][a], k[2][a]);
        const double t = scaled(value(s), 2 * kUnit + g.unit[a] + all - v.unit[a]);
        o.ak = a == 0 ? t : o.ak + t;
        if (a == 0) det = product(v.V[0][a], k[0][a]);
        else mac(det, v.V[0][a], k[0][a]);
    }
    o.detv = scaled(value(det), 2 * kUnit + all);
}

}  // namespace bf
}  // namespace lulesh
