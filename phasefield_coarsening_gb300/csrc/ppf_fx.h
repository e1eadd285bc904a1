// ppf_fx.h -- the cell arithmetic of the float64 step in 64-bit fixed point.
//
// The float64 step is bound by this GPU's FP64 pipe (1/64 of the FP32 and
// integer rates: about 75 FP64 operations per cell-step, 85 % of the pipe
// busy).  Every quantity of the step but the state itself is bounded once
// the state lies in a box (|eta| < 1.75, eta_S^2 + eta_L^2 >= 1/4, |c| below
// twice a power of two above the parabola minima), so it is held here as a
// 64-bit integer with a fixed binary scale ("x@s" is x 2^s).
//
// A fixed scale bounds errors absolutely, so it serves the quantities whose
// float64 arithmetic has an absolute error too: the interpolation h, w and M',
// the fluxes (differences of numbers of the size of the parabola minima), and
// the rates of the phase fields, in which terms of the size of the model's
// constants cancel.  The products' resolution, 2^-56 to 2^-62, is finer than
// float64's rounding of the same values.  A phase field itself falls off by
// orders of magnitude behind an interface, where float64 keeps 53 bits of
// whatever is left, and a fixed scale would lose them.  So a cell's larger
// field, at least 0.35 in the box, takes its increment in fixed point, and the
// smaller one's, rate x eta - kt x Laplacian, is formed in float64, as exact
// relative to a value of 1e-300 as to one of 1.  The new values are as close to
// the exact ones as float64 arithmetic's (root mean square within 0.01 %, each
// relative to its own size).  An increment of a larger field is resolved to
// 2^(eu-62), 1e-19 with the reference's constants, where a bulk phase may change by
// less: sums of squares take it from a formula of its own.
// Integer sums are exact, and a face's flux is the same number with the
// opposite sign seen from its other side.  A product is three 32 x 32 ->
// 64-bit multiply-adds.
//
// Functions are host-callable, so that their accuracy can be measured
// against extended precision without a GPU.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

namespace ppf {
namespace fx {

#ifdef __CUDACC__
#define PPF_FX __host__ __device__ __forceinline__
#else
#define PPF_FX inline
#endif

typedef long long i64;

// the box
constexpr double kEtaMax = 1.75;     // |eta| below
constexpr double kS2Min = 0.25;      // eta_S^2 + eta_L^2 at least

// Coefficients (see Coef in ppf_internal.h), as integers at the scales that
// the products below need, and the scales of the results.
struct FxCoef {
    i64 cL0;       // @59, in units of 2^ec
    i64 dc0;       // @62
    i64 m0, m1;    // A M' = m0 + m1 h: m0@64, m1@65
    i64 k0, k1;    // drive k = k0 + k1 w, in units of 2^eu: k0@62, k1@65
    i64 mt, mtg;   // mt and mt (2 gamma - 1) @68, units of 2^eu
    i64 nkt, nk6;  // -kt @67 and -6 kt @61, units of 2^eu
    i64 g;         // gamma @61
    double su, sc; // 2^(eu-61), 2^(ec-59): increments of eta and c
    double kb;     // -kt in units of su
    i64 mtm, mtgm; // mt and mt (2 gamma - 1) @68 in units of 2^em (finer than 2^eu)
    i64 nktm;      // -kt @67 in units of 2^em
    int um;        // em - eu
    int se;        // -eu (0 to 40)
    int ec, eu;
    unsigned cmax; // high word of the box bound of |c|, 2^(ec+1)
};

PPF_FX int hi32(i64 v) { return (int)(v >> 32); }
PPF_FX unsigned lo32(i64 v) { return (unsigned)v; }
PPF_FX i64 wide(int a, int b) { return (i64)a * (i64)b; }

// a b / 2^64, rounded to nearest (up to the neglected low x low part, a
// quarter of the last unit): the words of an operand are rebalanced so that
// the low one is signed.  |a|, |b| <= 2^62.
PPF_FX i64 mulq(i64 a, i64 b) {
    const int al = (int)lo32(a), bl = (int)lo32(b);
    const int ah = hi32(a) + (int)(lo32(a) >> 31), bh = hi32(b) + (int)(lo32(b) >> 31);
    const i64 cross = wide(ah, bl) + (wide(al, bh) + 0x80000000ll);
    return wide(ah, bh) + (i64)hi32(cross);
}

// The same with X more bits of the product, a b / 2^(64-X): the cross
// products' low bits are kept and the low x low part is added to them.
template <int X>
PPF_FX i64 mulx(i64 a, i64 b) {
    const int al = (int)lo32(a), bl = (int)lo32(b);
    const int ah = hi32(a) + (int)(lo32(a) >> 31), bh = hi32(b) + (int)(lo32(b) >> 31);
    const i64 low = (i64)hi32(wide(al, bl)) + (1ll << (31 - X));
    const i64 cross = wide(ah, bl) + (wide(al, bh) + low);
    return (i64)((unsigned long long)wide(ah, bh) << X) + (cross >> (32 - X));
}

// v 2^(1085 - bias), |v| < 2^(bias - 1022); truncated towards zero.  Exact for values
// whose last bit is a unit or more.
PPF_FX i64 to_fx(int hi, unsigned lo, int bias) {
    const int e = (hi >> 20) & 0x7ff;
    const unsigned mh = ((unsigned)hi & 0xfffffu) | 0x100000u;
    const unsigned long long m = ((unsigned long long)((mh << 10) | (lo >> 22)) << 32) | (lo << 10);
    const int sh = bias - e;
    const i64 a = (i64)(m >> (sh > 63 ? 63 : sh));
    const i64 s = hi >> 31;
    return (a ^ s) - s;
}
PPF_FX i64 to_fx(double v, int bias) {
#ifdef __CUDA_ARCH__
    return to_fx(__double2hiint(v), (unsigned)__double2loint(v), bias);
#else
    uint64_t b;
    std::memcpy(&b, &v, 8);
    return to_fx((int)(uint32_t)(b >> 32), (unsigned)b, bias);
#endif
}
constexpr int kEtaBias = 1085 - 61;            // eta@61
PPF_FX int c_bias(int ec) { return 1085 - 59 + ec; }   // c@59 in units of 2^ec

// 1/s2 @60 for s2@60 in [1/4, 6.2): a 20-bit estimate R0 from the float
// reciprocal of the leading bits, then R0 (1 + e + e^2) with
// e = 1 - s2 R0 exact (the third-order Newton step; the remainder e^3 is
// below 2^-60).
PPF_FX i64 recip(i64 s2) {
    const float f = (float)hi32(s2);           // s2@28
#ifdef __CUDA_ARCH__
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(f));
    const unsigned r0 = __float2uint_rn(y * 1125899906842624.0f);   // 2^50: R0@22
#else
    const unsigned r0 = (unsigned)lrintf(1.0f / f * 1125899906842624.0f);
#endif
    // e@82 = 2^82 - s2 R0, modulo 2^64
    const i64 e = -(i64)((unsigned long long)s2 * (unsigned long long)r0);
    const int eh = hi32(e);                    // @50
    const i64 t = e + (wide(eh, eh) >> 18);    // e + e^2 @82
    // R0 t @104 -> @72 -> @60
    const i64 v = wide((int)r0, hi32(t)) + (i64)(unsigned)(((unsigned long long)r0 * lo32(t)) >> 32);
    return ((i64)r0 << 38) + ((v + (1ll << 11)) >> 12);
}

// v 2^e of a normal number whose product is normal, without FP64 operations
PPF_FX double times_2(double v, int e) {
#ifdef __CUDA_ARCH__
    return __hiloint2double(__double2hiint(v) + (e << 20), __double2loint(v));
#else
    return std::ldexp(v, e);
#endif
}

// v 2^e as a double (|v| < 2^63, the result normal or 0), without FP64 operations:
// a conversion instruction takes the FP64 pipe as long as two or three additions.
// unit60 is the same for v > 0 and e = -60.
PPF_FX double unit60(i64 v) {
#ifdef __CUDA_ARCH__
    const int z = __clzll(v);
    const unsigned long long m = (unsigned long long)v << z;
    // (a carry out of the mantissa goes on into the exponent)
    return __longlong_as_double((i64)(((unsigned long long)(1025 - z) << 52) + (m >> 11) + ((m >> 10) & 1)));
#else
    return std::ldexp((double)v, -60);
#endif
}
PPF_FX double to_double(i64 v, int e) {
#ifdef __CUDA_ARCH__
    const i64 neg = v >> 63;
    const i64 a = (v ^ neg) - neg;
    const double d = times_2(unit60(a), e + 60);
    return a ? __hiloint2double(__double2hiint(d) | (hi32(neg) & (int)0x80000000), __double2loint(d)) : 0.0;
#else
    return std::ldexp((double)v, e);
#endif
}

// what a cell's neighbours need
struct Nb {
    i64 S, L;      // eta @58
    i64 W, M;      // w @59 in units of 2^ec, A M' @64
};
// the cell's rates @61 (units of 2^eu, below 2.1 of them): the increment of
// eta is rate x eta - kt x its Laplacian
struct Own {
    i64 bS, bL;
};

// `rates`: whether the cell's own rates are wanted too
template <bool C_ONLY>
PPF_FX void pass_a(const FxCoef &k, double eS, double eL, double c, int cbias, Nb &n, Own &o, bool rates = true) {
    const i64 S = to_fx(eS, kEtaBias), L = to_fx(eL, kEtaBias);
    const i64 S2 = mulx<2>(S, S), L2 = mulx<2>(L, L);        // @60
    const i64 R = recip(S2 + L2);                            // @60
    const i64 h = mulx<5>(S2, R);                            // @61
    const i64 C = to_fx(c, cbias);                           // @59
    n.W = C - k.cL0 + mulq(k.dc0, h);
    n.M = k.m0 + (mulq(k.m1, h) << 2);
    if (!C_ONLY) {
        n.S = S >> 3;
        n.L = L >> 3;
        if (!rates) return;
        // phasefield.c:360-373 divided by eta:
        //   mt (eta^2 - 1 + 2 gamma other^2) + drive k other^2 / (etaS^2 + etaL^2)^2,
        // the first as mt (etaS^2 + etaL^2 - 1) + mt (2 gamma - 1) other^2, @64;
        // the second with G = k / (etaS^2 + etaL^2) as G (1 - h), -G h, all @61
        const i64 u = mulq(k.mt, S2 + L2 - (1ll << 60)) + 4;
        const i64 G = mulx<3>(k.k0 + mulx<2>(k.k1, n.W), R);
        o.bS = ((u + mulq(k.mtg, L2)) >> 3) + mulx<3>(G, (1ll << 61) - h);
        o.bL = ((u + mulq(k.mtg, S2)) >> 3) - mulx<3>(G, h);
    }
}

// (M' + M)(mu' - mu) of one face, @59
PPF_FX i64 face(i64 Mn, i64 M, i64 Wn, i64 W) { return mulq(Mn + M, Wn - W); }

// The increment of a phase field in units of su, @61 in fixed point (below
// 1.1 of 2^eu: eta other^2 / (etaS^2 + etaL^2)^2 is at most 0.77): from its
// rate, its own value and the sum of its six neighbours', all @58.
PPF_FX i64 eta_inc(const FxCoef &k, i64 rate, i64 v, i64 six) {
    return mulx<3>(v << 3, rate) + mulq(k.nkt, six - 6 * v);
}
PPF_FX void eta_inc(const FxCoef &k, const Own &o, i64 S, i64 L, i64 S6, i64 L6, i64 &dS, i64 &dL) {
    dS = eta_inc(k, o.bS, S, S6);
    dL = eta_inc(k, o.bL, L, L6);
}
// The new value of a cell's larger field, from the value @58 (exact: at least
// 0.35) and its increment: added as integers @60, then rounded once.
PPF_FX double eta_large(const FxCoef &k, i64 v, i64 inc) {
    const i64 n = (v << 2) + ((inc + (1ll << k.se)) >> (k.se + 1));
#ifdef __CUDA_ARCH__
    const double d = (double)n;
    return n ? times_2(d, -60) : 0.0;
#else
    return std::ldexp((double)n, -60);
#endif
}
// The same increment, in units of su, with a relative precision of its own, for
// the sums of squares: the well and Laplacian terms @61 on their own scale, the
// drive with the smaller field's square in float64 (against extended precision at
// least as close as float64 arithmetic, in interfaces ten times).  (Below 2^-62 of the units
// the integer holds nothing, and a bulk phase may change by less.)  v and s are
// the larger and the smaller field, iv and is the same @58, W the cell's w, lap the
// larger field's six neighbours less six times itself @58; `solid`: v is etaS.
PPF_FX double eta_inc_large(const FxCoef &k, double v, double s, i64 iv, i64 is, i64 W, i64 lap, bool solid) {
    const i64 V = iv << 3, V2 = mulx<2>(V, V), s2 = mulx<2>(is << 3, is << 3);                       // @61, @60
    const i64 R = recip(V2 + s2);
    const i64 u = mulq(k.mtm, V2 + s2 - (1ll << 60)) + mulq(k.mtgm, s2);                             // @64
    const i64 e = mulq(V, u) + mulq(k.nktm, lap);                                                    // @61
    const i64 d = mulx<2>(mulx<3>(k.k0 + mulx<2>(k.k1, W), R), R);                                   // @59
    return fma(to_double(solid ? d : -d, 2), s * s * v, to_double(e, k.um));
}
// The increment of the smaller one, in the same units, in float64.  Its six
// neighbours' weight is not in the rate; add it with one rounding,
// fma(increment, su, v).
PPF_FX double eta_inc(const FxCoef &k, i64 rate, double v, double six) {
    return fma(k.kb, six, (double)(rate - k.nk6) * v);
}

// A cell's terms of the observables: c @59 and w @59 (in units of 2^ec), the
// reciprocal of etaS^2 + etaL^2 @60 and the well energy f0 @57 (its constant 1/4
// included).
PPF_FX void observe(const FxCoef &k, double eS, double eL, double c, int cbias, i64 &C, i64 &W, i64 &R, i64 &f0) {
    const i64 S = to_fx(eS, kEtaBias), L = to_fx(eL, kEtaBias);
    const i64 S2 = mulx<2>(S, S), L2 = mulx<2>(L, L);                                                // @60
    R = recip(S2 + L2);
    C = to_fx(c, cbias);
    W = C - k.cL0 + mulq(k.dc0, mulx<5>(S2, R));
    // S2 (S2/4 - 1/2 + gamma L2) + L2 (L2/4 - 1/2) + 1/4, the factors @57
    const i64 xS = (S2 >> 5) - (1ll << 56) + mulq(k.g, L2), xL = (L2 >> 5) - (1ll << 56);
    f0 = mulx<4>(S2, xS) + mulx<4>(L2, xL) + (1ll << 55);
}

// Whether a state cell lies in the box, from the high words alone (a margin
// of 2^-20 relative towards "no"); NaN and infinities do not.
PPF_FX int hi_fx26(unsigned hi) {              // v @26, truncated, for the high word of 0 <= v < 2
    const int e = (int)(hi >> 20), sh = 1023 - e;
    const unsigned m = ((hi & 0xfffffu) | 0x100000u) << 6;
    return (int)(m >> (sh > 31 ? 31 : sh));
}
PPF_FX bool in_box_eta(unsigned hS, unsigned hL) {
    const unsigned m = hS > hL ? hS : hL;
    if (m >= 0x3ffc0000u) return false;        // 1.75
    if (m >= 0x3fe00000u) return true;         // one of them at least 1/2
    const int s = hi_fx26(hS), l = hi_fx26(hL);
    return (i64)s * s + (i64)l * l >= (1ll << 50) + (1ll << 32);   // 1/4 @52
}
PPF_FX bool in_box_c(unsigned hC, unsigned cmax) { return (hC & 0x7fffffffu) < cmax; }

// The coefficients for a parameter set; false when they do not fit (AS !=
// AL, a liquid minimum below 1/16 of the scale of c, a time step above the solute equation's explicit limit, phase-field
// rates so large that their increments would lose resolution): then the
// step stays in float64 arithmetic.  `A` .. `kt` as in Coef<double>.
inline bool make_fxcoef(double AS, double AL, double cL0, double dc0, double Mt0, double Mt1, double dC, double q1,
                        double dm2, double mt, double tg, double kt, FxCoef *out) {
    if (AS != AL) return false;
    const double all[] = {AS, cL0, dc0, Mt0, Mt1, dC, q1, dm2, mt, tg, kt};
    for (double v : all)
        if (!std::isfinite(v)) return false;
    FxCoef f;
    const double cmag = std::fmax(std::fabs(cL0), std::fmax(std::fabs(cL0 - dc0), std::fabs(dc0)));
    int ec = 0;
    if (cmag > 0) {
        std::frexp(cmag, &ec);                 // cmag < 2^ec
    }
    if (ec < -500 || ec > 500) return false;
    // c - cL0 has an absolute error of 2^-54 |cL0| in float64 for any |c| below
    // cL0; with a liquid minimum near zero it has none, and small values of c would
    // lose bits on the fixed scale
    if (std::fabs(cL0) < std::ldexp(1.0, ec - 4)) return false;
    // (products of coefficients in extended precision: rounded once, here)
    typedef long double ld;
    const ld m0 = (ld)AS * Mt0, m1 = (ld)AS * Mt1;
    if (!(m0 >= 0 && m0 <= 1.0 / 12 && m0 + m1 >= 0 && m0 + m1 <= 1.0 / 12)) return false;
    if (!(std::fabs(tg) < 4)) return false;
    // drive of tmp1 dmu: dm2 (dC - q1 mu) = k0 + k1 w, w in units of 2^ec
    const ld k0 = (ld)dm2 * dC, k1 = -(ld)dm2 * q1 * AS * std::ldexp(1.0, ec);
    const double a0 = std::fabs((double)k0), a1 = std::fabs((double)k1);
    const double need = std::fmax(std::fmax(8.0 * a1, 2.0 * (a0 + 3.5 * a1)),
                                  std::fmax(1024.0 * std::fabs(mt), 32.0 * std::fabs(kt)));
    // the same for the well and the Laplacian alone
    const double need_m = std::fmax(1024.0 * std::fabs(mt), 32.0 * std::fabs(kt));
    int em = 0;
    if (need_m > 0) std::frexp(need_m, &em);
    if (need_m > 0 && em < -500) em = -500;
    int eu = -40;
    if (need > 0) {
        int e;
        std::frexp(need, &e);                  // need < 2^e
        if (e > eu) eu = e;
    }
    if (eu > 0) return false;                  // rates coarser than 2^-61
    auto q = [](ld v, int s) { return (i64)std::llrint(std::ldexp(v, s)); };
    f.cL0 = q(cL0, 59 - ec);
    f.dc0 = q(dc0, 62 - ec);
    f.m0 = q(m0, 64);
    f.m1 = q(m1, 65);
    f.k0 = q(k0, 62 - eu);
    f.k1 = q(k1, 65 - eu);
    f.mt = q(mt, 68 - eu);
    f.mtg = q((ld)mt * ((ld)tg - 1), 68 - eu);
    f.nkt = q(-kt, 67 - eu);
    f.nk6 = q(-6 * (ld)kt, 61 - eu);
    f.se = -eu;
    f.mtm = q(mt, 68 - em);
    f.mtgm = q((ld)mt * ((ld)tg - 1), 68 - em);
    f.nktm = q(-kt, 67 - em);
    f.um = em - eu;
    f.g = q(0.5 * tg, 61);
    f.su = std::ldexp(1.0, eu - 61);
    f.sc = std::ldexp(1.0, ec - 59);
    f.kb = std::ldexp(-kt, 61 - eu);
    f.ec = ec;
    f.eu = eu;
    f.cmax = (unsigned)(1023 + ec + 1) << 20;
    *out = f;
    return true;
}

}  // namespace fx
}  // namespace ppf
