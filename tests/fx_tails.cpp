// One explicit step of the two phase fields on the host, for tests of small
// values: with the arithmetic of csrc/ppf_fx.h (a cell's larger field in fixed
// point, the smaller one's increment in float64), as the step kernel takes it,
// in float64 and in extended precision throughout.
#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector>

#include "ppf_fx.h"

using ppf::fx::i64;

namespace {

struct K {
    double A, cL0, dc0, Mt0, Mt1, dC, q1, dm2, mt, tg, kt;
};

template <typename T>
void step_t(const K &k, int n, const int *nb, const double *S, const double *L, const double *c, T *S1, T *L1) {
    for (int i = 0; i < n; ++i) {
        const T s = S[i], l = L[i], S2 = s * s, L2 = l * l, s2 = std::fma(l, l, S2), rs = T(1) / s2, h = S2 * rs;
        const T mu = T(k.A) * std::fma(h, T(k.dc0), T(c[i]) - T(k.cL0));
        const T d = T(k.dm2) * (s * l) * (rs * rs) * std::fma(mu, T(-k.q1), T(k.dC));
        T S6 = 0, L6 = 0;
        for (int q = 0; q < 6; ++q) {
            S6 += T(S[nb[6 * i + q]]);
            L6 += T(L[nb[6 * i + q]]);
        }
        const T lS = std::fma(T(-6), s, S6), lL = std::fma(T(-6), l, L6);
        S1[i] = s + std::fma(T(k.mt) * s, std::fma(T(k.tg), L2, S2 - 1), std::fma(T(-k.kt), lS, l * d));
        L1[i] = l + std::fma(T(k.mt) * l, std::fma(T(k.tg), S2, L2 - 1), std::fma(T(-k.kt), lL, -(s * d)));
    }
}

}  // namespace

// nb: six neighbours of every cell.  err[0..2n): the new etaS and etaL of the
// step kernel's arithmetic minus the exact ones, err[2n..4n): those of float64,
// each relative to the largest of the cell's own value and its neighbours'
// (0 where all are 0).
extern "C" int fx_tail_errors(int n, const int *nb, const double *kk, const double *in, double *err) {
    const K k = {kk[0], kk[1], kk[2], kk[3], kk[4], kk[5], kk[6], kk[7], kk[8], kk[9], kk[10]};
    ppf::fx::FxCoef f;
    if (!ppf::fx::make_fxcoef(k.A, k.A, k.cL0, k.dc0, k.Mt0, k.Mt1, k.dC, k.q1, k.dm2, k.mt, k.tg, k.kt, &f)) return 0;
    const double *S = in, *L = in + n, *c = in + 2 * n;
    std::vector<double> d(2 * n);
    std::vector<long double> e(2 * n);
    step_t<double>(k, n, nb, S, L, c, d.data(), d.data() + n);
    step_t<long double>(k, n, nb, S, L, c, e.data(), e.data() + n);
    std::vector<ppf::fx::Nb> m(n);
    std::vector<ppf::fx::Own> o(n);
    for (int i = 0; i < n; ++i) ppf::fx::pass_a<false>(f, S[i], L[i], c[i], ppf::fx::c_bias(f.ec), m[i], o[i]);
    for (int i = 0; i < n; ++i) {
        const int *b = nb + 6 * i;
        for (int q = 0; q < 2; ++q) {
            const double *u = q ? L : S;
            const i64 rate = q ? o[i].bL : o[i].bS;
            const bool small = q == (std::fabs(L[i]) < std::fabs(S[i]));
            double got;
            if (small) {
                const double six = (u[b[4]] + u[b[5]]) + (u[b[2]] + u[b[3]]) + (u[b[0]] + u[b[1]]);
                got = std::fma(ppf::fx::eta_inc(f, rate, u[i], six), f.su, u[i]);
            } else {
                i64 six = 0;
                for (int j = 0; j < 6; ++j) six += q ? m[b[j]].L : m[b[j]].S;
                const i64 v = q ? m[i].L : m[i].S;
                got = ppf::fx::eta_large(f, v, ppf::fx::eta_inc(f, rate, v, six));
            }
            double size = std::fabs(u[i]);
            for (int j = 0; j < 6; ++j) size = std::fmax(size, std::fabs(u[b[j]]));
            const long double x = e[q * n + i], s = size > 0 ? size : 1;
            err[q * n + i] = (double)((got - x) / s);
            err[2 * n + q * n + i] = (double)((d[q * n + i] - x) / s);
        }
    }
    return 1;
}
