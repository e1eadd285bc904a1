// One explicit step of a small box on the host, for tests: in the fixed-point
// arithmetic of csrc/ppf_fx.h, in float64 and in extended precision (the
// last two in the general kernel's formulas).
#include <cmath>
#include <cstdint>
#include <vector>

#include "ppf_fx.h"

using ppf::fx::i64;

namespace {

struct K {   // Coef<double>'s fields
    double A, cL0, dc0, Mt0, Mt1, dC, q1, dm2, mt, tg, kt;
};

struct Grid {
    int nz, ny, nx, bc;
    int at(int z, int y, int x) const {
        auto f = [&](int i, int n) { return bc == 0 ? (i + n) % n : i < 0 ? 0 : i >= n ? n - 1 : i; };
        return (f(z, nz) * ny + f(y, ny)) * nx + f(x, nx);
    }
    void nb(int i, int (&o)[6]) const {
        const int x = i % nx, y = i / nx % ny, z = i / (nx * ny);
        o[0] = at(z + 1, y, x); o[1] = at(z - 1, y, x); o[2] = at(z, y + 1, x);
        o[3] = at(z, y - 1, x); o[4] = at(z, y, x + 1); o[5] = at(z, y, x - 1);
    }
};

template <typename T>
void step_t(const Grid &g, const K &k, const T *S, const T *L, const T *c, T *S1, T *L1, T *c1) {
    const int n = g.nz * g.ny * g.nx;
    std::vector<T> mu(n), M(n), d(n);
    for (int i = 0; i < n; ++i) {
        const T S2 = S[i] * S[i], s2 = std::fma(L[i], L[i], S2), rs = T(1) / s2, h = S2 * rs;
        mu[i] = T(k.A) * std::fma(h, T(k.dc0), c[i] - T(k.cL0));
        M[i] = std::fma(h, T(k.Mt1), T(k.Mt0));
        d[i] = T(k.dm2) * (S[i] * L[i]) * (rs * rs) * std::fma(mu[i], T(-k.q1), T(k.dC));
    }
    for (int i = 0; i < n; ++i) {
        int b[6];
        g.nb(i, b);
        T fl = 0, S6 = 0, L6 = 0;
        for (int q = 0; q < 6; ++q) {
            fl = std::fma(M[b[q]] + M[i], mu[b[q]] - mu[i], fl);
            S6 += S[b[q]];
            L6 += L[b[q]];
        }
        const T S2 = S[i] * S[i], L2 = L[i] * L[i];
        const T lS = std::fma(T(-6), S[i], S6), lL = std::fma(T(-6), L[i], L6);
        S1[i] = S[i] + std::fma(T(k.mt) * S[i], std::fma(T(k.tg), L2, S2 - 1), std::fma(T(-k.kt), lS, L[i] * d[i]));
        L1[i] = L[i] + std::fma(T(k.mt) * L[i], std::fma(T(k.tg), S2, L2 - 1), std::fma(T(-k.kt), lL, -(S[i] * d[i])));
        c1[i] = c[i] + fl;
    }
}

}  // namespace

extern "C" {

// k: A, cL0, dc0, Mt0, Mt1, dC, q1, dm2, mt, tg, kt.  Returns 0 when the
// parameters do not fit the fixed-point step, else 1; units: 2^ec, 2^eu.
int fx_units(double AS, double AL, const double *k, double *units) {
    ppf::fx::FxCoef f;
    if (!ppf::fx::make_fxcoef(AS, AL, k[1], k[2], k[3], k[4], k[5], k[6], k[7], k[8], k[9], k[10], &f)) return 0;
    units[0] = std::ldexp(1.0, f.ec);
    units[1] = std::ldexp(1.0, f.eu);
    return 1;
}

// in: etaS, etaL, c after one another.  diff[0..2]: largest absolute error
// of the fixed-point step's increments, before they are rounded and added;
// rms[0..2], rms[3..5]: root-mean-square errors of the fixed-point and the
// float64 step; drift: sum of c after the fixed-point step minus before, in
// extended precision.  Returns the number of cells outside the box.
int fx_step_errors(int nz, int ny, int nx, int bc, const double *kk, const double *in, double *diff, double *rms,
                   double *drift) {
    const Grid g = {nz, ny, nx, bc};
    const K k = {kk[0], kk[1], kk[2], kk[3], kk[4], kk[5], kk[6], kk[7], kk[8], kk[9], kk[10]};
    const int n = nz * ny * nx;
    ppf::fx::FxCoef f;
    if (!ppf::fx::make_fxcoef(k.A, k.A, k.cL0, k.dc0, k.Mt0, k.Mt1, k.dC, k.q1, k.dm2, k.mt, k.tg, k.kt, &f)) return -1;
    const double *S = in, *L = in + n, *c = in + 2 * n;
    std::vector<ppf::fx::Nb> nb(n);
    std::vector<ppf::fx::Own> own(n);
    std::vector<double> r(3 * n), d(3 * n);
    std::vector<long double> inc(3 * n);
    int out = 0;
    for (int i = 0; i < n; ++i) {
        ppf::fx::pass_a<false>(f, S[i], L[i], c[i], ppf::fx::c_bias(f.ec), nb[i], own[i]);
        uint64_t w[3];
        std::memcpy(&w[0], S + i, 8);
        std::memcpy(&w[1], L + i, 8);
        std::memcpy(&w[2], c + i, 8);
        out += !ppf::fx::in_box_eta((w[0] >> 32) & 0x7fffffffu, (w[1] >> 32) & 0x7fffffffu) ||
               !ppf::fx::in_box_c(w[2] >> 32, f.cmax);
    }
    long double sum0 = 0, sum1 = 0;
    for (int i = 0; i < n; ++i) {
        int b[6];
        g.nb(i, b);
        i64 fl = 0, S6 = 0, L6 = 0, dS, dL;
        for (int q = 0; q < 6; ++q) {
            // low to high, as the kernel orients faces
            fl += q & 1 ? -ppf::fx::face(nb[i].M, nb[b[q]].M, nb[i].W, nb[b[q]].W)
                        : ppf::fx::face(nb[b[q]].M, nb[i].M, nb[b[q]].W, nb[i].W);
            S6 += nb[b[q]].S;
            L6 += nb[b[q]].L;
        }
        ppf::fx::eta_inc(f, own[i], nb[i].S, nb[i].L, S6, L6, dS, dL);
        inc[i] = (long double)dS * f.su;
        inc[n + i] = (long double)dL * f.su;
        inc[2 * n + i] = (long double)fl * f.sc;
        r[i] = std::fma((double)dS, f.su, S[i]);
        r[n + i] = std::fma((double)dL, f.su, L[i]);
        r[2 * n + i] = std::fma((double)fl, f.sc, c[i]);
        sum0 += c[i];
        sum1 += (long double)c[i] + (long double)fl * f.sc;
    }
    *drift = (double)(sum1 - sum0);
    step_t<double>(g, k, S, L, c, d.data(), d.data() + n, d.data() + 2 * n);
    std::vector<long double> e(3 * n), x(in, in + 3 * n);
    step_t<long double>(g, k, x.data(), x.data() + n, x.data() + 2 * n, e.data(), e.data() + n, e.data() + 2 * n);
    for (int q = 0; q < 3; ++q) {
        long double mx = 0, s = 0, sd = 0;
        for (int i = q * n; i < (q + 1) * n; ++i) {
            const long double er = std::fabs((long double)r[i] - e[i]), ed = (long double)d[i] - e[i];
            const long double ei = std::fabs(inc[i] - (e[i] - x[i]));
            if (ei > mx) mx = ei;
            s += er * er;
            sd += ed * ed;
        }
        diff[q] = (double)mx;
        rms[q] = (double)std::sqrt(s / n);
        rms[3 + q] = (double)std::sqrt(sd / n);
    }
    return out;
}

// largest relative error of the reciprocal over s2 in [1/4, 6.2)
double fx_recip_error(int n) {
    long double worst = 0;
    for (int i = 0; i < n; ++i) {
        const double v = 0.25 + 5.95 * (i + 0.37) / n;
        const i64 s2 = (i64)std::ldexp(v, 60);
        const long double p = std::ldexp((long double)ppf::fx::recip(s2), -60) * std::ldexp((long double)s2, -60);
        if (std::fabs(p - 1) > worst) worst = std::fabs(p - 1);
    }
    return (double)worst;
}

}  // extern "C"
