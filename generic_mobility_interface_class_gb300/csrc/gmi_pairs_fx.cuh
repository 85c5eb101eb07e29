// gmi_pairs_fx.cuh -- the RPY pair sums in the fixed-point arithmetic of
// gmi_fx.cuh: FP64-grade results on the integer and FP32 pipes.
//
// Units.  U is the largest power of two not above the smaller radius.
// Positions are 64-bit integers of 2^-51 U relative to an origin near the
// first source; a separation is exact.  It is normalised by a shift to
// d' = d / (2^k U) with its largest component in [1, 2), so r' = r / (2^k U)
// lies in [1, 3.47).  A source's loads share one exponent: force components
// and torque components over U are fractions of 2^e.  Sums are formed in
// units of 2^e / (8 pi mu U) (velocity) and 2^e / (8 pi mu U^2) (angular
// velocity), with the unit vector e' = d' / r' and T'' = 2^-k T:
//   far:  v = 2^-k  [ A F + B (e'.F) e' + C T'' x e' ]
//         w = 2^-2k [ Ar T'' + Br (e'.T'') e' + C F x e' ]
//         A = (1 + t)/r', B = (1 - 3t)/r', t = (as^2 + ab^2)/(3 r^2),
//         C = 1/r'^2, Ar = -1/(2 r'^3), Br = 3/(2 r'^3)
//   near: the same without the powers of two, with the near-field scalars.
// The formulas are those of gmi_pairs.cuh, which cites the reference kernels.
// d' has scale 29, everything after it is below 2 and has scale 30, and every
// term of v and w scale 60.
//
// Accumulation.  A term's integer part enters by its two words times
// 2^(24 - s), s the term's shift (k or 2k plus the source's exponent gap, at
// most 24): two integer multiply-adds instead of a variable shift and a
// three-word add.  Its FP32 part enters an FP32 sum, which fx_settle adds to a
// compensated one every kFxSettle terms.  |term| < 8, so 128 terms keep the
// 64-bit accumulators in range; the caller folds them into FP64 by then.
//
// Wide sources.  A term is rounded at about 2^-55 of its operands' ranges
// before its shift, so a product must be as large as its range to have FP64's
// relative error.  Two things break that: a torque so much larger than the force (or
// the reverse) that the shared exponent leaves the smaller load too few bits where
// it decides a target's sum (T'' = 2^-k T loses k more), and a source far below its
// block's largest load.  Such a source (fx_held) is held with an exponent for its
// force and one for its torque, and its terms enter apart, T's with the shift 2k or
// 3k in the term in place of T'', and integer parts shifted down beyond 24 (one
// of the two enters times 2^-3 at most, a near pair's cross products times 2^-1, so
// the low words' sum of 128 sources stays below 2^64).  With the block's largest
// load at distance 2^10 U its own w is still above 2^-30 of the unit, 54 bits above
// the accumulators' last place.  All targets of a warp meet the same source, so
// nothing diverges.  Worst target of two groups 300 radii apart, torques only, the
// one group's 1e-6 of the other's: error of w 3.6e-12 with one exponent, 6.8e-16
// with two (FP64 formulas: 1.6e-15).  Where a target's terms cancel (a lone force
// nearly along the separation, and its w) the error is a few 2^-55 of the terms,
// up to five times that of the FP64 formulas.
#pragma once

#include <math.h>

#include "gmi_fx.cuh"

namespace gmi {

constexpr int kFxTile = 128;       // sources per tile of the pair kernel: one stage
constexpr int kFxPosBits = 51;     // position quantum 2^-51 U
constexpr int kFxAccBits = 24;     // a term without shift enters times 2^24
// Exponent gap of a source within its block: with one exponent for force and
// torque (shifts up to k = 9 for v and 18 for w stay within 24), and at all, by
// which a source is below what rounds away.
constexpr int kFxEvenGap[5] = {6, 0, 15, 6, 15};  // by FxKind
constexpr int kFxMaxGap = 40;
// A torque may exceed the force of its source by 2^kFxTorqueOver, or stay
// below it by 2^kFxTorqueUnder, and share its exponent: 1.3 % of sources with
// normally distributed loads are wide (8 % with 1 and 3, whose error is no smaller).
constexpr int kFxTorqueOver = 2, kFxTorqueUnder = 3;
constexpr int kFxFold = 128;       // terms between folds
// Terms between fx_settle: the running FP32 parts are a quarter of the error
// of a few hundred particles' sum; every 4 instead of 8 takes 1.3 % longer.
// The blobs' sum over segments has the largest terms next to its total.
constexpr int kFxSettle[5] = {4, 4, 4, 4, 2};  // by FxKind
constexpr double kFxPosLimit = 1152921504606845952.0;  // 2^60 - 2^10: |position| stays below

enum FxKind : int { kFxSS = 0, kFxBB = 2, kFxSB = 3, kFxBS = 4 };  // as PairKind

struct FxConsts {
    int pos_shift, unit_exp;   // 2^pos_shift = 2^51 / U, 2^unit_exp = U
    double pos_scale, unit;    // 2^51 / U, U
    double vscale, vfix;       // 1/(8 pi mu U), and what its rounding leaves out
    double wscale, wfix;       // 1/(8 pi mu U^2)
    double as, ab;             // radii (equal kinds: both the one radius)
    double a0, ar0;            // near field: 4U/(3a) (unequal: 4U/(3 as ab)), (U/a)^3
    int turn;                  // Ar and Br of the near field carry 2^turn, with which (U/a)^3 exceeds 1/2
    double ar0_turn;           // (U/a)^3 2^turn
    fxop k3;                   // far field: (as^2 + ab^2) / (3 U^2)
    unsigned long long t4;     // near up to r^2 = t4 U^2 (2^-58): (as + ab)^2 < 36 U^2, so more than 63 bits
    fxop a_zero, ar_zero;      // at r = 0: A = 4U / (3 max(as, ab)), Ar = (U/a)^3 2^turn
    fxop bb_b;                 // blob-blob near field: (U/a)^2, an eighth of it at scale 33
};

struct FxSource {
    long long X[3];
    fxop F[3];
    long long T[3];  // torques over U, 2^-62
    int gap, tgap;   // the block's exponent less the source's, of F and (wide) of T
};

// How a source is held whose forces are below 2^f and torques (over U) below
// 2^t (kFxNoLoad: none), in a block of exponent E: wide, or with one exponent.
struct FxHeld {
    int gap, tgap;
    bool wide;
};

// One target's accumulators, in 2^(-60 - 24) of the block's unit: H 2^32 + L,
// and the FP32 parts x, settled into xh + xl.
template <int N> struct FxAcc {
    long long H[N];
    unsigned long long L[N];
    float x[N], xh[N], xl[N];
};

GMI_FX_HD long long fx_rint(double v)
{
#ifdef __CUDA_ARCH__
    return __double2ll_rn(v);
#else
    return (long long)llrint(v);
#endif
}

// v (|v| < 2) as a value of scale 30
GMI_FX_HD fxop fx_from_double(double v) { return fx_split(fx_rint(v * 4611686018427387904.0)); }

GMI_FX_HD double fx_exp2(int e)  // 2^e, -1022 <= e <= 1023
{
    union {
        unsigned long long u;
        double d;
    } c;
    c.u = (unsigned long long)(unsigned)(e + 1023) << 52;
    return c.d;
}

// The scalars of one pair: A of F, B of (e'.F) e', C of the cross products, Ar
// of T'', Br of (e'.T'') e'.
struct FxScalars {
    fxop A, B, C, Ar, Br;
    int up;  // near field: C carries 2^up
};

// C times 2^up, up >= 1, in [1/2, 1): C is below 0.4 (largest at 4/3 of the radius), and
// vanishes with r and next to r = ab - as.
GMI_FX_HD void fx_normalised(double C, FxScalars &s)
{
    union {
        double d;
        unsigned long long u;
    } c;
    c.d = C;
    const int up = 1022 - ((int)(c.u >> 52) & 2047);
    s.up = up < 1 ? 1 : up > 64 ? 64 : up;
    s.C = fx_from_double(C * fx_exp2(s.up));
}

// Near-field scalars of the segment kinds in FP64 (few pairs get here), at r = ru U.
template <int KIND>
#ifdef __CUDACC__
__host__ __device__ __noinline__
#endif
FxScalars fx_near_scalars(double ru, const FxConsts &K)
{
    const fxop none{0, 0.0f, 0.0f};
    FxScalars s;
    if (KIND == kFxSS) {
        const double rho = ru * K.unit / K.as, q = rho * (1.0 / 32.0), rho3 = rho * rho * rho;
        s.A = fx_from_double(K.a0 - K.a0 * 9.0 * q);
        s.B = fx_from_double(K.a0 * 3.0 * q);
        s.Ar = fx_from_double(K.ar0_turn * fma(5.0 / 64.0, rho3, fma(-27.0, q, 1.0)));
        s.Br = fx_from_double(K.ar0_turn * fma(-3.0 / 64.0, rho3, 9.0 * q));
        fx_normalised(0.5 * K.ar0 * ru * (1.0 - 12.0 * q), s);
        return s;
    }
    s.Ar = s.Br = none;
    const double r = ru * K.unit, dm = K.as - K.ab;
    if (r > fabs(dm)) {
        const double i3 = 1.0 / (32.0 * r * r * r), dm2 = dm * dm, r2d = r * r;
        const double t = dm2 + 3.0 * r2d, b = dm2 - r2d, u = dm + r;
        const double p = K.ab * K.ab + 2.0 * K.ab * (r + K.as) - 3.0 * (K.as - r) * (K.as - r);
        s.A = fx_from_double(K.a0 * (0.5 * (K.as + K.ab) - t * t * i3));
        s.B = fx_from_double(K.a0 * 3.0 * b * b * i3);
        fx_normalised(K.unit * K.unit * u * u * p / (16.0 * K.ab * K.as * K.as * K.as * r2d), s);
    } else {
        s.A = K.a_zero;
        s.B = none;
        fx_normalised(K.as > K.ab ? K.unit * K.unit * r / (K.as * K.as * K.as) : 0.0, s);
    }
    return s;
}

// (h, x) 2^k, by shifts (k <= 1)
GMI_FX_HD fxsum fx_scale(fxsum s, int k)
{
    const int dn = k < -62 ? 62 : -k;
    s.h = k > 0 ? (long long)((unsigned long long)s.h << k) : s.h >> dn;
    s.x *= fx_as_float((127 + (k < -126 ? -126 : k)) << 23);
    return s;
}

// The factors by which a term of shift s enters the accumulators, and (kWide) its
// shift beyond them.
struct FxEnter {
    int m, down;
    float f;
};
template <bool kWide> GMI_FX_HD FxEnter fx_enter(int s)
{
    FxEnter n;
    n.down = kWide && s > kFxAccBits ? s - kFxAccBits : 0;
    n.m = 1 << (kFxAccBits - s + n.down);
    n.f = fx_as_float((127 + kFxAccBits - 32 - s) << 23);
    return n;
}
template <bool kWide, int N> GMI_FX_HD void fx_add_term(FxAcc<N> &acc, int c, const fxsum &q, const FxEnter &n)
{
    const long long h = kWide ? q.h >> (n.down < 63 ? n.down : 63) : q.h;
    acc.H[c] = fx_madw((int)(h >> 32), n.m, acc.H[c]);
    acc.L[c] = fx_madw_u((unsigned)h, (unsigned)n.m, acc.L[c]);
    acc.x[c] = fmaf(q.x, n.f, acc.x[c]);
}

// The separation of a target and a source, as fx_pair has it in place: d' (scale 29),
// r'^2 (58), 1/r' (30), and k.
struct FxSeparation {
    fxop d[3], ir;
    fxsum s;
    int k;
    bool zero;
};
GMI_FX_HD FxSeparation fx_separation(const long long *X, const FxSource &S)
{
    FxSeparation p;
    long long D[3] = {X[0] - S.X[0], X[1] - S.X[1], X[2] - S.X[2]};  // |D| < 2^61
    int m;
    {
        const int h0 = (int)(D[0] >> 32), h1 = (int)(D[1] >> 32), h2 = (int)(D[2] >> 32);
        const int a0 = h0 ^ (h0 >> 31), a1 = h1 ^ (h1 >> 31), a2 = h2 ^ (h2 >> 31);
        m = a0 > a1 ? a0 : a1;
        m = m > a2 ? m : a2;
    }
    int sl;
    p.zero = false;
    if (m == 0) {  // closer than 2^-19 U: the leading bit is in the low words
        unsigned long long mx = 0;
        for (int c = 0; c < 3; ++c) {
            const unsigned long long a = (unsigned long long)(D[c] < 0 ? -D[c] : D[c]);
            mx = a > mx ? a : mx;
        }
        p.zero = mx == 0;
        if (p.zero) D[0] = 1;
        sl = p.zero ? 61 : fx_clzll(mx) - 2;
    } else {
        sl = fx_clz((unsigned)m) - 2;  // the leading bit moves to 2^61 (one place off for a negative power of two)
    }
    p.k = 61 - kFxPosBits - sl;
    for (int c = 0; c < 3; ++c) p.d[c] = fx_split((long long)((unsigned long long)D[c] << sl));  // scale 29
    p.s = fxsum{0, 0.0f};
    for (int c = 0; c < 3; ++c) {
        p.s.h = fx_madw(p.d[c].h, p.d[c].h, p.s.h);
        p.s.x = fmaf(p.d[c].hf, p.d[c].lf, p.s.x);
    }
    p.s.x *= 2.0f;
    p.ir = fx_rsqrt(p.s.h, p.s.x);
    return p;
}

// r / U in FP64
GMI_FX_HD double fx_distance(const fxsum &s, const fxop &ir, int k)
{
    const double ird = ((double)ir.h + (double)ir.lf * (1.0 / 4294967296.0)) * (1.0 / 1073741824.0);
    const double r2 = ((double)s.h + (double)s.x * (1.0 / 4294967296.0)) * (1.0 / 288230376151711744.0);
    return r2 * ird * fx_exp2(k);
}

// The cross products' terms of a near pair, with C times 2^up and the shift up in the
// term: C can be small, and these terms can be all of a target's sum (two
// segments 1e-4 radii apart, torques alone: error of v 3e-12 with C at the others'
// scale, 3e-16 so).
template <int KIND, bool kWide, int N>
GMI_FX_HD void fx_cross_terms(const fxop *e, const fxop &C, int up, const FxSource &S, FxAcc<N> &acc)
{
    const FxEnter nv = fx_enter<true>((kWide ? S.tgap : S.gap) + up), nw = fx_enter<true>(S.gap + up);
    fxop cp[3];
    for (int c = 0; c < 3; ++c) cp[c] = fx_product<30>(e[c], C);
    for (int c = 0; c < 3; ++c) {
        const int c1 = (c + 1) % 3, c2 = (c + 2) % 3, o = N == 6 ? 3 + c : c;
        if (KIND == kFxSS || KIND == kFxBS) {
            fxsum q = fx_mul(fx_split(S.T[c1]), cp[c2]);
            fx_mac(q, fx_split(S.T[c2]), fx_neg(cp[c1]));
            fx_add_term<true>(acc, c, q, nv);
        }
        if (KIND == kFxSS || KIND == kFxSB) {
            fxsum q = fx_mul(S.F[c1], cp[c2]);
            fx_mac(q, S.F[c2], fx_neg(cp[c1]));
            fx_add_term<true>(acc, o, q, nw);
        }
    }
}

// One source's contribution to one target's accumulators.  M_ss leaves out the cross
// products of a near pair and sets `bit` in `close` (fx_close_cross adds them in a
// loop of its own: in this function they cost it 2 % of its time; the other kinds
// lose 1 % by such a loop and 0.1 % by a branch here).
template <int KIND, bool kWide, int N>
GMI_FX_HD void fx_pair(const long long *X, const FxSource &S, const FxConsts &K, FxAcc<N> &acc, unsigned &close,
                       unsigned bit)
{
    constexpr bool kTorque = KIND == kFxSS || KIND == kFxBS;  // sources carry torques
    constexpr bool kAngular = KIND == kFxSS || KIND == kFxSB; // targets turn
    constexpr bool kCross = kTorque || kAngular, kShared = KIND == kFxSS && !kWide;
    long long D[3] = {X[0] - S.X[0], X[1] - S.X[1], X[2] - S.X[2]};  // |D| < 2^61
    int m;
    {
        const int h0 = (int)(D[0] >> 32), h1 = (int)(D[1] >> 32), h2 = (int)(D[2] >> 32);
        const int a0 = h0 ^ (h0 >> 31), a1 = h1 ^ (h1 >> 31), a2 = h2 ^ (h2 >> 31);
        m = a0 > a1 ? a0 : a1;
        m = m > a2 ? m : a2;
    }
    int sl;
    bool zero = false;
    if (m == 0) {  // closer than 2^-19 U: the leading bit is in the low words
        unsigned long long mx = 0;
        for (int c = 0; c < 3; ++c) {
            const unsigned long long a = (unsigned long long)(D[c] < 0 ? -D[c] : D[c]);
            mx = a > mx ? a : mx;
        }
        zero = mx == 0;
        if (zero) D[0] = 1;
        sl = zero ? 61 : fx_clzll(mx) - 2;
    } else {
        sl = fx_clz((unsigned)m) - 2;  // the leading bit moves to 2^61 (one place off for a negative power of two)
    }
    const int k = 61 - kFxPosBits - sl;
    fxop d[3];
    for (int c = 0; c < 3; ++c) d[c] = fx_split((long long)((unsigned long long)D[c] << sl));  // scale 29
    fxsum s{0, 0.0f};  // r'^2, scale 58
    for (int c = 0; c < 3; ++c) {
        s.h = fx_madw(d[c].h, d[c].h, s.h);
        s.x = fmaf(d[c].hf, d[c].lf, s.x);
    }
    s.x *= 2.0f;
    const fxop ir = fx_rsqrt(s.h, s.x);  // 30
    const bool near = k < 0 || (k <= 2 && (unsigned long long)s.h <= (K.t4 >> (2 * k)));

    fxop e[3];
    for (int c = 0; c < 3; ++c) e[c] = fx_product<29>(d[c], ir);

    FxScalars g;  // far field
    int kk = k, kw = 2 * k;
    {
        const fxop ir2 = fx_close<30>(fx_madw(ir.h, ir.h, 0), 2.0f * (ir.hf * ir.lf));
        const fxsum u = fx_mul(K.k3, ir2);  // 28 + 30
        const int k2 = near ? 0 : 2 * k;
        const fxop t = fx_close<28>(u.h >> k2, u.x * fx_as_float((127 - k2) << 23));
        const fxop p = fx_product_low<30>(ir, t);
        g.A = fx_add(ir, 1, p);
        g.B = fx_add(ir, -3, p);
        g.C = ir2;
        if (KIND == kFxSS) {
            const fxop c3 = fx_product<31>(ir, ir2);  // r'^-3 of scale 29, so half of it of scale 30
            g.Ar = fx_neg(c3);
            g.Br = fx_add(fxop{0, 0.0f, 0.0f}, 3, c3);
        }
    }
    if (near) {
        kk = 0;
        kw = KIND == kFxSS ? K.turn : 0;
        if (zero) {  // r -> 0
            g.A = K.a_zero;
            g.B = g.Br = g.C = fxop{0, 0.0f, 0.0f};
            g.Ar = K.ar_zero;
        } else if (KIND == kFxBB) {
            // B = (U/a)^2 r / (8 U), A = 4U/(3a) - 3 B
            fxop r2 = fx_split(s.h);  // 26
            r2.lf = fmaf(s.x, 1.0f / 4294967296.0f, r2.lf);
            const fxop rp = fx_product<28>(r2, ir);           // r', 28
            const fxsum u = fx_scale(fx_mul(K.bb_b, rp), k);  // 33 + 28
            g.B = fx_close<31>(u.h, u.x);
            g.A = fx_add(K.a_zero, -3, g.B);
        } else {
            g = fx_near_scalars<KIND>(fx_distance(s, ir, k), K);
            if (KIND == kFxSS)
                close |= bit;
            else
                fx_cross_terms<KIND, kWide>(e, g.C, g.up, S, acc);
            g.C = fxop{0, 0.0f, 0.0f};
        }
    }

    // dot products and loads
    fxsum q{0, 0.0f};
    for (int c = 0; c < 3; ++c) fx_mac(q, e[c], S.F[c]);
    const fxop Bt = fx_product<30>(g.B, fx_close<30>(q.h, q.x));
    // a cross product is the load's with C e, where v and w share that in the loop
    // that counts, else C times the load's with e, which spares the rounding of C e at
    // the scale of e: error of M_sb's w 1.03 -> 0.83 of the FP64 kernel's, no longer
    fxop T[3], cp[3], cn[3], Br;
    if (kCross)
        for (int c = 0; c < 3; ++c) {
            cp[c] = kShared ? fx_product<30>(e[c], g.C) : e[c];
            cn[c] = fx_neg(cp[c]);
        }
    if (kTorque)
        for (int c = 0; c < 3; ++c) T[c] = fx_split(kWide ? S.T[c] : S.T[c] >> kk);
    if (KIND == kFxSS) {
        q = fxsum{0, 0.0f};
        for (int c = 0; c < 3; ++c) fx_mac(q, e[c], T[c]);
        Br = fx_product<30>(g.Br, fx_close<30>(q.h, q.x));
    }
    const FxEnter nv = fx_enter<kWide>(S.gap + kk), nw = fx_enter<kWide>(S.gap + kw);
    FxEnter tv = nv, tw = nw;  // of the torque's terms
    if (kWide) {
        tv = fx_enter<true>(S.tgap + 2 * kk);
        tw = fx_enter<true>(S.tgap + kk + kw);
    }
    for (int c = 0; c < 3; ++c) {
        const int c1 = (c + 1) % 3, c2 = (c + 2) % 3;
        q = fx_mul(g.A, S.F[c]);
        fx_mac(q, Bt, e[c]);
        if (kTorque) {
            if (kWide) {
                fx_add_term<true>(acc, c, q, nv);
                q = fxsum{0, 0.0f};
            }
            if (kShared) {
                fx_mac(q, T[c1], cp[c2]);
                fx_mac(q, T[c2], cn[c1]);
            } else {
                fxsum x = fx_mul(T[c1], cp[c2]);
                fx_mac(x, T[c2], cn[c1]);
                fx_mac(q, fx_close<30>(x.h, x.x), g.C);
            }
        }
        fx_add_term<kWide>(acc, c, q, kTorque ? tv : nv);
    }
    if (kAngular)
        for (int c = 0; c < 3; ++c) {
            const int c1 = (c + 1) % 3, c2 = (c + 2) % 3, o = N == 6 ? 3 + c : c;
            q = fx_mul(S.F[c1], cp[c2]);
            fx_mac(q, S.F[c2], cn[c1]);
            if (!kShared) q = fx_mul(fx_close<30>(q.h, q.x), g.C);
            if (KIND == kFxSS) {
                if (kWide) {
                    fx_add_term<true>(acc, o, q, nw);
                    q = fxsum{0, 0.0f};
                }
                fx_mac(q, g.Ar, T[c]);
                fx_mac(q, Br, e[c]);
            }
            fx_add_term<kWide>(acc, o, q, KIND == kFxSS ? tw : nw);
        }
}

// The cross products of a near pair of segments that fx_pair marked.
template <bool kWide, int N>
GMI_FX_HD void fx_close_cross(const long long *X, const FxSource &S, const FxConsts &K, FxAcc<N> &acc)
{
    const FxSeparation p = fx_separation(X, S);
    fxop e[3];
    for (int c = 0; c < 3; ++c) e[c] = fx_product<29>(p.d[c], p.ir);
    const FxScalars g = fx_near_scalars<kFxSS>(fx_distance(p.s, p.ir, p.k), K);
    fx_cross_terms<kFxSS, kWide>(e, g.C, g.up, S, acc);
}

template <int N> GMI_FX_HD void fx_clear(FxAcc<N> &a)
{
    for (int c = 0; c < N; ++c) {
        a.H[c] = 0;
        a.L[c] = 0;
        a.x[c] = a.xh[c] = a.xl[c] = 0.0f;
    }
}

// Knuth's two-sum of the running FP32 parts into the settled ones
template <int N> GMI_FX_HD void fx_settle(FxAcc<N> &a)
{
    for (int c = 0; c < N; ++c) {
        const float s = a.xh[c] + a.x[c], b = s - a.xh[c];
        a.xl[c] += (a.xh[c] - (s - b)) + (a.x[c] - b);
        a.xh[c] = s;
        a.x[c] = 0.0f;
    }
}

GMI_FX_HD long long fx_rintf(float v)
{
#ifdef __CUDA_ARCH__
    return __float2ll_rn(v);
#else
    return (long long)llrintf(v);
#endif
}

// A sum as an integer a 2^32 + b in 2^-84 of the block's unit; sums add part
// by part.
struct FxTotal {
    long long a, b;
};

// One settled accumulator.  Its FP32 parts lie below 2^65.
template <int N> GMI_FX_HD FxTotal fx_total(const FxAcc<N> &acc, int c)
{
    const float top = rintf(acc.xh[c] * (1.0f / 4294967296.0f));
    const long long low = (long long)(acc.L[c] & 0xffffffffull) + fx_rintf(acc.xh[c] - top * 4294967296.0f) +
                          fx_rintf(acc.xl[c]);
    return FxTotal{acc.H[c] + (long long)(acc.L[c] >> 32) + fx_rintf(top) + (low >> 32), low & 0xffffffffll};
}

// A sum in FP64, times 2^E (scale + fix): the integer is rounded once, to 53
// bits, by integer instructions (a conversion holds the FP64 unit longer than
// an addition does).
GMI_FX_HD double fx_value(const FxTotal &t, int E, double scale, double fix)
{
    const long long a = t.a + (t.b >> 32);
    const unsigned b = (unsigned)t.b;
    const bool neg = a < 0;
    // |a 2^32 + b| as the 128-bit number (hi, lo) 2^-32
    unsigned long long hi = neg ? ~(unsigned long long)a + (b == 0) : (unsigned long long)a;
    unsigned long long lo = (unsigned long long)(neg ? 0u - b : b) << 32;
    int e = 32 + 11;  // of the 53-bit significand's last place, before the shift
    if (hi == 0) {
        hi = lo;
        lo = 0;
        e -= 64;
    }
    if (hi == 0) return 0.0;
    const int z = fx_clzll(hi);
    if (z > 0) {
        hi = (hi << z) | (lo >> (64 - z));
        lo <<= z;
    }
    e -= z;
    const unsigned rest = ((unsigned)hi & 2047u) * 2u + (lo != 0);
    const unsigned long long m = hi >> 11;  // 2^52 <= m < 2^53
    union {
        unsigned long long u;
        double d;
    } c;
    c.u = ((unsigned long long)(unsigned)(1023 + 52 - 60 - kFxAccBits + e + E - 1) << 52) + m +
          (rest > 2048u || (rest == 2048u && (m & 1)));
    const double v = neg ? -c.d : c.d;
    return fma(v, scale, v * fix);
}

// The constants of one kind; false where the formats do not hold them: the
// radii's ratio keeps (as^2 + ab^2) / (3 U^2) below 8.
inline bool fx_consts(int kind, double as, double ab, double mu, FxConsts *K)
{
    const bool equal = kind == kFxSS || kind == kFxBB;
    const double amin = as < ab ? as : ab, amax = as < ab ? ab : as;
    if (!(amin > 1e-60 && amax < 1e60 && mu > 1e-60 && mu < 1e60) || amax > 2.0 * amin) return false;
    int e;
    frexp(amin, &e);
    const double U = ldexp(1.0, e - 1);
    // 8 pi mu in two parts: the one rounding that every velocity shares
    const double pi = 3.14159265358979323846264338327950288, pi_low = 1.2246467991473532e-16;
    const double d8 = 8.0 * pi * mu, d8_low = fma(8.0 * pi, mu, -d8) + 8.0 * pi_low * mu, f8 = 1.0 / d8;
    const double fix = fma(-f8, d8, 1.0) - f8 * d8_low;
    K->unit = U;
    K->unit_exp = e - 1;
    K->pos_shift = kFxPosBits - (e - 1);
    K->pos_scale = ldexp(1.0, kFxPosBits) / U;
    K->vscale = f8 / U;
    K->vfix = K->vscale * fix;
    K->wscale = f8 / (U * U);
    K->wfix = K->wscale * fix;
    K->as = as;
    K->ab = ab;
    K->a0 = equal ? 4.0 * U / (3.0 * as) : 4.0 * U / (3.0 * as * ab);
    // (U/a)^3 in two parts: all rotation of near pairs and a target's own shares its error
    const double a2 = as * as, a3c = a2 * as, a3_low = fma(a2, as, -a3c) + fma(as, as, -a2) * as, U3 = U * U * U;
    const double q3 = U3 / a3c, q3_low = (fma(-q3, a3c, U3) - q3 * a3_low) / a3c;
    K->ar0 = q3 + q3_low;
    K->turn = 0;
    while (equal && ldexp(K->ar0, K->turn) <= 0.5) ++K->turn;
    K->ar0_turn = ldexp(K->ar0, K->turn);
    K->k3 = fx_split(fx_rint((as * as + ab * ab) / (3.0 * U * U) * 1152921504606846976.0));  // 28
    K->t4 = (unsigned long long)((as + ab) * (as + ab) / (U * U) * 288230376151711744.0);  // a whole number
    // the self term is the largest of most sums: the quotient's remainder too
    const double a3 = 3.0 * amax, a_zero = 4.0 * U / a3;
    K->a_zero = fx_from_double(a_zero);
    K->a_zero.lf += (float)((fma(-a_zero, a3, 4.0 * U) - a_zero * fma(3.0, amax, -a3)) / a3 * 4611686018427387904.0);
    K->ar_zero = fx_from_double(ldexp(q3, K->turn));
    K->ar_zero.lf += (float)(ldexp(q3_low, K->turn) * 4611686018427387904.0);
    K->bb_b = fx_from_double(U * U / (as * as));
    return true;
}

// v 2^s to the nearest integer, ties to even, by integer instructions; false
// (and 0) when that reaches 2^62 or v is not finite.  Denormals are zeros.
GMI_FX_HD bool fx_fixed(double v, int s, long long *r)
{
    union {
        double d;
        unsigned long long u;
    } c;
    c.d = v;
    const int be = (int)(c.u >> 52) & 2047, sh = be - 1075 + s;
    *r = 0;
    if (be == 2047) return false;
    if (be == 0 || sh < -54) return true;
    if (sh > 9) return false;
    long long m = (long long)((c.u & 0xfffffffffffffull) | 0x10000000000000ull);
    if (sh >= 0)
        m <<= sh;
    else
        m = (m + ((1ll << (-sh - 1)) - 1) + ((m >> -sh) & 1)) >> -sh;
    *r = (long long)c.u < 0 ? -m : m;
    return true;
}

// Where positions are counted from, in quanta: a multiple of 2^59 next to the
// first source; in FP64 (d) when that is 2^62 quanta from zero or further.
struct FxOrigin {
    long long i;
    double d;
    bool far;
};
GMI_FX_HD FxOrigin fx_origin(double x0, const FxConsts &K)
{
    FxOrigin o;
    long long t;
    o.far = !fx_fixed(x0, K.pos_shift, &t);
    o.i = ((t + (1ll << 58)) >> 59) << 59;
    o.d = o.far ? rint(x0 * K.pos_scale * (1.0 / 576460752303423488.0)) * 576460752303423488.0 : 0.0;
    return o;
}

// A position in quanta relative to the origin; false when it is out of range
// or not finite.  Past 2^62 quanta the FP64 difference is exact.
GMI_FX_HD bool fx_position(double x, const FxConsts &K, const FxOrigin &o, long long *X)
{
    long long t;
    if (!o.far && fx_fixed(x, K.pos_shift, &t)) {
        t -= o.i;
    } else {
        const double rel = x * K.pos_scale - (o.far ? o.d : (double)o.i);
        t = fabs(rel) < kFxPosLimit ? fx_rint(rel) : (long long)kFxPosLimit;
    }
    const bool ok = t < (long long)kFxPosLimit && t > -(long long)kFxPosLimit;
    *X = ok ? t : 0;
    return ok;
}

// The exponent e that makes v 2^-unit_exp a fraction (below 2^e): kFxNoLoad for
// a zero, out of the range +-kFxMaxExp for what the formats do not hold.
constexpr int kFxNoLoad = -100000;
constexpr int kFxMaxExp = 900;
GMI_FX_HD int fx_exponent(double v, int unit_exp)
{
    union {
        double d;
        unsigned long long u;
    } c;
    c.d = v;
    const int be = (int)(c.u >> 52) & 2047;
    if (be == 0) return (c.u << 1) == 0 ? kFxNoLoad : -5000;
    return be == 2047 ? 5000 : be - 1022 - unit_exp;
}
GMI_FX_HD int fx_gap(int e, int E, int most) { return e == kFxNoLoad ? 0 : E - e < most ? E - e : most; }
template <int KIND> GMI_FX_HD FxHeld fx_held(int f, int t, int E)
{
    constexpr int kEven = kFxEvenGap[KIND];
    const int e = f > t ? f : t;
    FxHeld h;
    h.wide = (t != kFxNoLoad && (t > f + kFxTorqueOver || t < f - kFxTorqueUnder)) ||
             (KIND != kFxBB && e != kFxNoLoad && E - e > kEven);
    h.gap = fx_gap(h.wide ? f : e, E, h.wide ? kFxMaxGap : kEven);
    h.tgap = h.wide ? fx_gap(t, E, kFxMaxGap) : h.gap;
    return h;
}
// The exponent of a source is its components' largest.
GMI_FX_HD bool fx_exponent_held(int e) { return e == kFxNoLoad || (e <= kFxMaxExp && e >= -kFxMaxExp); }

// Sources per split, a power of two.  Measured on M_ss and M_bb of 200 to
// 12,800 particles (152 SMs): with work enough, the largest split that still
// gives 24 CTAs per SM, so that the last CTAs to finish idle the chip for
// little of the launch (4096 segments: 128 sources 325 us, 1024 403; 12,800:
// 1024 sources 2.82 ms, 128 2.87, 2048 2.84); below that a tile, down to 1.5
// CTAs per SM (1669 segments: 128 72 us, 64 78, 32 82); then parts of a tile,
// whose CTAs have less to do than to set up (642: 32 20.6 us, 64 24.7, 128
// 30.8), and 16 or 8 while the CTAs still find an SM each (60: 8 12.4 us, 16
// 14.4, 32 16.5; 320: 32 17.7 us, 16 and 8 16.5).
inline int fx_chunk(int groups, int n_src, int sm_count, int most_splits)
{
    const auto splits = [&](long long chunk) { return ((long long)n_src + chunk - 1) / chunk; };
    const auto ctas = [&](long long chunk) { return (double)groups * (double)splits(chunk) / sm_count; };
    long long chunk = kFxTile;
    while (chunk < n_src && ctas(2 * chunk) >= 24.0) chunk *= 2;
    if (ctas(kFxTile) < 1.5) chunk = ctas(64) >= 2.0 ? 64 : ctas(8) <= 0.5 ? 8 : ctas(16) <= 1.0 ? 16 : 32;
    while (splits(chunk) > (most_splits < 65535 ? most_splits : 65535)) chunk *= 2;
    return (int)(chunk < 1 << 30 ? chunk : 1 << 30);
}

}  // namespace gmi
