// The fixed-point pair sum of csrc/gmi_pairs_fx.cuh on the host, for
// test_pairs_fx_cpu.py: the pack and pair kernels' arithmetic, one target
// after another.  Returns 0, 1 (radii not held) or 2 (a value out of range).
#include <algorithm>
#include <vector>

#include "gmi_pairs_fx.cuh"

using namespace gmi;

template <int KIND>
static int sum(int nt, const double *xt, int ns, const double *xs, const double *f, double as, double ab, double mu,
               double *out)
{
    constexpr bool torque = KIND == kFxSS || KIND == kFxBS;
    constexpr int nf = torque ? 6 : 3, nout = (KIND == kFxSS || KIND == kFxSB) ? 6 : 3, tile = 512;
    FxConsts K;
    if (!fx_consts(KIND, as, ab, mu, &K)) return 1;
    std::vector<FxSource> src(ns);
    std::vector<char> wide(ns);
    std::vector<int> e(ns), te(ns), E((ns + tile - 1) / tile, kFxNoLoad);
    FxOrigin origin[3];
    for (int c = 0; c < 3; ++c) origin[c] = fx_origin(xs[c], K);
    for (int j = 0; j < ns; ++j) {
        for (int c = 0; c < 3; ++c)
            if (!fx_position(xs[3 * j + c], K, origin[c], &src[j].X[c])) return 2;
        e[j] = te[j] = kFxNoLoad;
        for (int c = 0; c < 3; ++c) e[j] = std::max(e[j], fx_exponent(f[nf * j + c], 0));
        for (int c = 3; c < nf; ++c) te[j] = std::max(te[j], fx_exponent(f[nf * j + c], K.unit_exp));
        if (!fx_exponent_held(std::max(e[j], te[j]))) return 2;
        E[j / tile] = std::max(E[j / tile], std::max(e[j], te[j]));
    }
    for (int j = 0; j < ns; ++j) {
        const int Ej = E[j / tile] == kFxNoLoad ? 0 : E[j / tile];
        const FxHeld h = fx_held<KIND>(e[j], te[j], Ej);
        const int used = Ej - h.gap, tused = Ej - h.tgap;
        src[j].gap = h.gap;
        src[j].tgap = h.tgap;
        wide[j] = h.wide;
        for (int c = 0; c < 3; ++c) {
            long long v;
            fx_fixed(f[nf * j + c], 62 - used, &v);
            src[j].F[c] = fx_split(v);
            src[j].T[c] = 0;
            if (torque) fx_fixed(f[nf * j + nf - 3 + c], 62 - tused - K.unit_exp, &src[j].T[c]);
        }
    }
    for (int i = 0; i < nt; ++i) {
        long long X[3];
        double tot[6] = {0, 0, 0, 0, 0, 0};
        for (int c = 0; c < 3; ++c)
            if (!fx_position(xt[3 * i + c], K, origin[c], &X[c])) return 2;
        for (int j0 = 0; j0 < ns; j0 += kFxFold) {
            FxAcc<nout> acc;
            fx_clear(acc);
            for (int j = j0; j < std::min(ns, j0 + kFxFold); ++j) {
                unsigned close = 0;
                if (wide[j])
                    fx_pair<KIND, true>(X, src[j], K, acc, close, 1);
                else
                    fx_pair<KIND, false>(X, src[j], K, acc, close, 1);
                if constexpr (KIND == kFxSS) {
                    if (close != 0 && wide[j])
                        fx_close_cross<true>(X, src[j], K, acc);
                    else if (close != 0)
                        fx_close_cross<false>(X, src[j], K, acc);
                }
                if ((j - j0) % kFxSettle[KIND] == kFxSettle[KIND] - 1) fx_settle(acc);
            }
            fx_settle(acc);
            const int Ej = E[j0 / tile] == kFxNoLoad ? 0 : E[j0 / tile];
            for (int c = 0; c < nout; ++c)
                tot[c] += fx_value(fx_total(acc, c), Ej, c < 3 ? K.vscale : K.wscale, c < 3 ? K.vfix : K.wfix);
        }
        for (int c = 0; c < nout; ++c) out[nout * i + c] = tot[c];
    }
    return 0;
}

extern "C" int fx_host_sum(int kind, int nt, const double *xt, int ns, const double *xs, const double *f, double as,
                           double ab, double mu, double *out)
{
    return kind == 0 ? sum<kFxSS>(nt, xt, ns, xs, f, as, ab, mu, out)
         : kind == 2 ? sum<kFxBB>(nt, xt, ns, xs, f, as, ab, mu, out)
         : kind == 3 ? sum<kFxSB>(nt, xt, ns, xs, f, as, ab, mu, out)
                     : sum<kFxBS>(nt, xt, ns, xs, f, as, ab, mu, out);
}

extern "C" int fx_host_fixed(double v, int s, long long *r) { return fx_fixed(v, s, r) ? 1 : 0; }
extern "C" double fx_host_value(long long a, long long b, int E) { return fx_value(FxTotal{a, b}, E, 1.0, 0.0); }
extern "C" int fx_host_chunk(int groups, int n_src, int sm_count, int most) { return fx_chunk(groups, n_src, sm_count, most); }
