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
    std::vector<int> e(ns), E((ns + tile - 1) / tile, kFxNoLoad);
    double origin[3];
    for (int c = 0; c < 3; ++c) origin[c] = fx_origin(xs[c], K.pos_scale);
    for (int j = 0; j < ns; ++j) {
        double mx = 0;
        for (int c = 0; c < 3; ++c)
            if (!fx_position(xs[3 * j + c], K.pos_scale, origin[c], &src[j].X[c])) return 2;
        for (int c = 0; c < nf; ++c) {
            const double v = fabs(f[nf * j + c]) * (c < 3 ? 1.0 : K.inv_unit);
            mx = v > mx || v != v ? v : mx;  // a NaN stays
        }
        if (!fx_load_exponent(mx, &e[j])) return 2;
        E[j / tile] = std::max(E[j / tile], e[j]);
    }
    for (int j = 0; j < ns; ++j) {
        src[j].gap = e[j] == kFxNoLoad ? 0 : std::min(E[j / tile] - e[j], kFxMaxGap);
        const double s = fx_exp2(e[j] == kFxNoLoad ? 0 : -(E[j / tile] - src[j].gap));
        for (int c = 0; c < 3; ++c) {
            src[j].F[c] = fx_from_double(f[nf * j + c] * s);
            src[j].T[c] = torque ? fx_rint(f[nf * j + nf - 3 + c] * K.inv_unit * s * 4611686018427387904.0) : 0;
        }
    }
    for (int i = 0; i < nt; ++i) {
        long long X[3];
        double tot[6] = {0, 0, 0, 0, 0, 0};
        for (int c = 0; c < 3; ++c)
            if (!fx_position(xt[3 * i + c], K.pos_scale, origin[c], &X[c])) return 2;
        for (int j0 = 0; j0 < ns; j0 += kFxFold) {
            FxAcc<nout> acc;
            fx_clear(acc);
            for (int j = j0; j < std::min(ns, j0 + kFxFold); ++j) {
                fx_pair<KIND>(X, src[j], K, acc);
                if ((j - j0) % kFxSettle[KIND] == kFxSettle[KIND] - 1) fx_settle(acc);
            }
            fx_settle(acc);
            const double s = fx_exp2(E[j0 / tile] == kFxNoLoad ? 0 : E[j0 / tile]);
            for (int c = 0; c < nout; ++c) tot[c] += fx_fold(acc, c, (c < 3 ? K.vscale : K.wscale) * s, K.vscale_fix);
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
