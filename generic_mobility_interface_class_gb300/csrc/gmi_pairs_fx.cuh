// gmi_pairs_fx.cuh -- the RPY pair sums in the fixed-point arithmetic of
// gmi_fx.cuh: FP64-grade results (a term is rounded at 2^-56 of its source's
// load) on the integer multiply pipe.
//
// Units.  U is the largest power of two not above the smaller radius.
// Positions are 64-bit integers of 2^-51 U relative to an origin near the
// first source; a separation is exact.  It is normalised by a shift to
// d' = d / (2^k U) with its largest component in [1, 2), so r' = r / (2^k U)
// lies in [1, 3.47).  A source's loads share one exponent: force components
// and torque components over U are fractions of 2^e.  Sums are formed in
// units of 2^e / (8 pi mu U) (velocity) and 2^e / (8 pi mu U^2) (angular
// velocity):
//   far:  v = 2^-k  [ A F + B (d'.F) d' + C T''x d' ]
//         w = 2^-2k [ -C/2 T'' + Br (d'.T'') d' + C F x d' ],   T'' = 2^-k T
//   near: the same without the powers of two, with the near-field scalars.
// The formulas are those of gmi_pairs.cuh, which cites the reference kernels.
//
// Accumulation.  A term P (2^-56) enters as its limbs times 2^(26 - s), s the
// term's shift (k or 2k plus the source's exponent gap, at most 26): two
// integer multiply-adds instead of a variable shift and a three-word add,
// and nothing is rounded.  |P| < 8, so 32 terms keep both 64-bit
// accumulators below 2^62; the caller folds them into FP64 by then.
#pragma once

#include <math.h>

#include "gmi_fx.cuh"

namespace gmi {

constexpr int kFxPosBits = 51;     // position quantum 2^-51 U
constexpr int kFxAccBits = 26;     // a term without shift enters times 2^26
constexpr int kFxMaxGap = 8;       // exponent gap of a source within its tile
constexpr int kFxFold = 32;        // terms between folds
constexpr double kFxPosLimit = 1152921504606845952.0;  // 2^60 - 2^10: |position| stays below

enum FxKind : int { kFxSS = 0, kFxBB = 2, kFxSB = 3, kFxBS = 4 };  // as PairKind

struct FxConsts {
    double pos_scale;          // 2^51 / U
    double unit, inv_unit;     // U, 1/U
    double vscale, wscale;     // 1/(8 pi mu U), 1/(8 pi mu U^2)
    double as, ab, inv_as;     // radii (equal kinds: both the one radius)
    double a0, ar0;            // near field: 4U/(3a) (unequal: 4U/(3 as ab)), (U/a)^3
    fx k3;                     // far field: (as^2 + ab^2) / (3 U^2)
    long long t4;              // near up to r^2 = t4 U^2 (2^-56): (as + ab)^2
    long long a_zero;          // A at r = 0: 4U / (3 max(as, ab))
    long long bb_b;            // blob-blob near field: (U/a)^2 / 8
    fx bb_a1;                  // and 3 (U/a)^2 / 8
};

struct FxSource {
    long long X[3];
    fx F[3];
    long long T[3];  // torques over U, 2^-60
    int gap;         // the tile's exponent less the source's, <= kFxMaxGap
};

GMI_FX_HD long long fx_from_double(double v)  // 2^-60, |v| < 8
{
#ifdef __CUDA_ARCH__
    return __double2ll_rn(v * 1152921504606846976.0);
#else
    return (long long)llrint(v * 1152921504606846976.0);
#endif
}

GMI_FX_HD double fx_exp2(int e)  // 2^e, -1022 <= e <= 1023
{
    union {
        unsigned long long u;
        double d;
    } c;
    c.u = (unsigned long long)(unsigned)(e + 1023) << 52;
    return c.d;
}

// The scalars of one pair in 2^-60: A of F, B of (d'.F) d', C of the cross
// products, Ar of T'', Br of (d'.T'') d'.
struct FxScalars {
    long long A, B, C, Ar, Br;
};

// Near-field scalars of the segment kinds in FP64 (few pairs get here):
// r' and 1/r'^2 from the fixed-point separation, 2^k U the separation's unit.
template <int KIND>
#ifdef __CUDACC__
__host__ __device__ __noinline__
#endif
FxScalars fx_near_scalars(long long r2, long long ir, int k, const FxConsts &K)
{
    const double ird = (double)ir * (1.0 / 1152921504606846976.0);
    const double rp = (double)r2 * (1.0 / 72057594037927936.0) * ird;  // r'
    const double ru = rp * fx_exp2(k);             // r / U
    const double ir2 = ird * ird;
    FxScalars s;
    if (KIND == kFxSS) {
        const double rho = ru * K.unit * K.inv_as, q = rho * (1.0 / 32.0), rho3 = rho * rho * rho;
        s.A = fx_from_double(K.a0 - K.a0 * 9.0 * q);
        s.B = fx_from_double(K.a0 * 3.0 * q * ir2);
        s.Ar = fx_from_double(K.ar0 * (1.0 - 27.0 * q + (5.0 / 64.0) * rho3));
        s.Br = fx_from_double(K.ar0 * (9.0 * q - (3.0 / 64.0) * rho3) * ir2);
        s.C = fx_from_double(0.5 * K.ar0 * ru * (1.0 - 12.0 * q) * ird);
        return s;
    }
    s.Ar = s.Br = 0;
    const double r = ru * K.unit, dm = K.as - K.ab;
    if (r > fabs(dm)) {
        const double i3 = 1.0 / (32.0 * r * r * r), dm2 = dm * dm, r2d = r * r;
        const double t = dm2 + 3.0 * r2d, b = dm2 - r2d, u = dm + r;
        const double p = K.ab * K.ab + 2.0 * K.ab * (r + K.as) - 3.0 * (K.as - r) * (K.as - r);
        s.A = fx_from_double(K.a0 * (0.5 * (K.as + K.ab) - t * t * i3));
        s.B = fx_from_double(K.a0 * 3.0 * b * b * i3 * ir2);
        s.C = fx_from_double(K.unit * K.unit * u * u * p / (16.0 * K.ab * K.as * K.as * K.as * r2d) * ird);
    } else {
        const double amax = K.as > K.ab ? K.as : K.ab;
        s.A = fx_from_double(K.unit * 4.0 / (3.0 * amax));
        s.B = 0;
        s.C = K.as > K.ab ? fx_from_double(K.unit * K.unit * r / (K.as * K.as * K.as) * ird) : 0;
    }
    return s;
}

// One source's contribution to one target's accumulators (H: 2^32, L: 1, both
// times 2^(-56 - 26) of the tile's unit).
template <int KIND>
GMI_FX_HD void fx_pair(const long long *X, const FxSource &S, const FxConsts &K, long long *H, long long *L)
{
    constexpr bool kTorque = KIND == kFxSS || KIND == kFxBS;  // sources carry torques
    constexpr bool kAngular = KIND == kFxSS || KIND == kFxSB; // targets turn
    constexpr bool kCross = kTorque || kAngular;
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
        sl = zero ? 60 : fx_clzll(mx) - 3;
    } else {
        sl = fx_clz((unsigned)m) - 3;  // the leading bit moves to 2^60 (one place off for a negative power of two)
    }
    const int k = 60 - kFxPosBits - sl;
    fx d[3];
    for (int c = 0; c < 3; ++c) d[c] = fx_split((long long)((unsigned long long)D[c] << sl));
    // r'^2 in 2^-56
    fxacc s{0, 0};
    for (int c = 0; c < 3; ++c) {
        s.h = fx_madw(d[c].hi, d[c].hi, s.h);
        s.x = fx_madw(d[c].hi, d[c].lo, s.x);
    }
    const long long r2 = s.h + (s.x >> 31);
    const long long irq = fx_rsqrt(r2);
    const fx ir = fx_split(irq);

    FxScalars g;
    int kk = k;
    const bool near = k < 0 || (k <= 2 && r2 <= (K.t4 >> (2 * k)));
    // far field: A = (1 + t)/r', B = (1 - 3t)/r'^3, t = (as^2 + ab^2)/(3 r^2)
    {
        s = fxacc{fx_madw(ir.hi, ir.hi, 0), fx_madw(ir.hi, ir.lo, 0)};
        const fx ir2 = fx_split((s.h << 4) + (s.x >> 27));
        const long long c3 = fx_mul60(ir, ir2);
        const int k2 = near ? 0 : 2 * k;
        const fx t = fx_split(fx_mul60(K.k3, ir2) >> k2);
        const fx c3f = fx_split(c3);
        g.A = irq + fx_mul60(ir, t);
        g.B = c3 - 3 * fx_mul60(c3f, t);
        g.C = c3;
        if (KIND == kFxSS) {
            const long long c5 = fx_mul60(c3f, ir2);
            g.Ar = -(c3 >> 1);
            g.Br = c5 + (c5 >> 1);
        }
    }
    if (near) {
        kk = 0;
        if (zero) {  // r -> 0
            g.A = K.a_zero;
            g.B = g.Br = g.C = 0;
            g.Ar = KIND == kFxSS ? fx_from_double(K.ar0) : 0;
        } else if (KIND == kFxBB) {
            // A = 4U/(3a) (1 - 9r/(32a)), B = (U/a)^2 2^k / (8 r')
            const int rh = (int)(r2 >> 32);  // 2^-24
            const long long rx = (long long)ir.lo * rh + (long long)((unsigned long long)(unsigned)r2 * (unsigned)ir.hi);
            const long long rp = (((long long)ir.hi * rh) << 8) + (rx >> 24);  // r' = r'^2 / r'
            const int dn = k < 0 ? (k < -62 ? 62 : -k) : 0, up = k < 0 ? 0 : k;
            const fx ru = fx_split((rp << up) >> dn);  // r / U < 4
            g.A = K.a_zero - fx_mul60(K.bb_a1, ru);
            g.B = (fx_mul60(fx_split(K.bb_b), ir) << up) >> dn;
        } else {
            g = fx_near_scalars<KIND>(r2, irq, k, K);
        }
    }

    // dot products and loads
    fxacc q{0, 0};
    for (int c = 0; c < 3; ++c) fx_mac(q, d[c], S.F[c]);
    const fx dF = fx_split(fx_q60(q));
    const fx A = fx_split(g.A), Bt = fx_split(fx_mul60(fx_split(g.B), dF));
    fx T[3], cp[3], cn[3], Ar, Br;
    if (kCross) {
        const fx C = fx_split(g.C);
        for (int c = 0; c < 3; ++c) {
            cp[c] = fx_split(fx_mul60(C, d[c]));
            cn[c] = fx{-cp[c].hi, ~cp[c].lo};  // -cp but for one unit of 2^-60 (and no -2^31 to negate)
        }
    }
    if (kTorque)
        for (int c = 0; c < 3; ++c) T[c] = fx_split(S.T[c] >> kk);
    if (KIND == kFxSS) {
        q = fxacc{0, 0};
        for (int c = 0; c < 3; ++c) fx_mac(q, d[c], T[c]);
        Ar = fx_split(g.Ar);
        Br = fx_split(fx_mul60(fx_split(g.Br), fx_split(fx_q60(q))));
    }
    const int mv = 1 << (kFxAccBits - S.gap - kk);
    const int mw = 1 << (kFxAccBits - S.gap - 2 * kk);
    constexpr long long kRoundP = 1ll << 31;  // of x's shift, and of the split of P
    for (int c = 0; c < 3; ++c) {
        const int c1 = (c + 1) % 3, c2 = (c + 2) % 3;
        q = fxacc{kRoundP, kRoundP};
        fx_mac(q, A, S.F[c]);
        fx_mac(q, Bt, d[c]);
        if (kTorque) {
            fx_mac(q, T[c1], cp[c2]);
            fx_mac(q, T[c2], cn[c1]);
        }
        const long long P = q.h + (q.x >> 32);
        H[c] = fx_madw((int)(P >> 32), mv, H[c]);
        L[c] = fx_madw((int)((unsigned)P ^ 0x80000000u), mv, L[c]);
    }
    if (kAngular)
        for (int c = 0; c < 3; ++c) {
            const int c1 = (c + 1) % 3, c2 = (c + 2) % 3;
            q = fxacc{kRoundP, kRoundP};
            if (KIND == kFxSS) {
                fx_mac(q, Ar, T[c]);
                fx_mac(q, Br, d[c]);
            }
            fx_mac(q, S.F[c1], cp[c2]);
            fx_mac(q, S.F[c2], cn[c1]);
            const long long P = q.h + (q.x >> 32);
            H[3 + c] = fx_madw((int)(P >> 32), mw, H[3 + c]);
            L[3 + c] = fx_madw((int)((unsigned)P ^ 0x80000000u), mw, L[3 + c]);
        }
}

// Accumulators to FP64 in final units: scale = vscale or wscale times the
// tile's 2^E.
GMI_FX_HD double fx_fold(long long H, long long L, double scale)
{
    const double s = scale * (1.0 / 72057594037927936.0) * (1.0 / (double)(1 << kFxAccBits));
    return (double)H * (s * 4294967296.0) + (double)L * s;
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
    const double U = ldexp(1.0, e - 1), f8 = 1.0 / (8.0 * 3.14159265358979323846264338327950288 * mu);
    const double one = 1152921504606846976.0;  // 2^60
    K->unit = U;
    K->inv_unit = 1.0 / U;
    K->pos_scale = ldexp(1.0, kFxPosBits) / U;
    K->vscale = f8 / U;
    K->wscale = f8 / (U * U);
    K->as = as;
    K->ab = ab;
    K->inv_as = 1.0 / as;
    K->a0 = equal ? 4.0 * U / (3.0 * as) : 4.0 * U / (3.0 * as * ab);
    K->ar0 = (U / as) * (U / as) * (U / as);
    K->k3 = fx_split((long long)llrint((as * as + ab * ab) / (3.0 * U * U) * one));
    K->t4 = (long long)llrint((as + ab) * (as + ab) / (U * U) * 72057594037927936.0);
    K->a_zero = (long long)llrint(4.0 * U / (3.0 * amax) * one);
    K->bb_b = (long long)llrint(U * U / (8.0 * as * as) * one);
    K->bb_a1 = fx_split((long long)llrint(3.0 * U * U / (8.0 * as * as) * one));
    return true;
}

// A position in quanta relative to `origin` (a multiple of 2^59 quanta, in
// quanta).  False when it is out of range or not finite.  Below 2^62 quanta
// the subtraction is done in integers; above, the FP64 difference is exact.
GMI_FX_HD bool fx_position(double x, double pos_scale, double origin, long long *X)
{
    const double t = x * pos_scale, rel = t - origin;
    if (!(fabs(rel) < kFxPosLimit)) {
        *X = 0;
        return false;
    }
#ifdef __CUDA_ARCH__
    *X = fabs(t) < 4611686018427387904.0 ? __double2ll_rn(t) - (long long)origin : __double2ll_rn(rel);
#else
    *X = fabs(t) < 4611686018427387904.0 ? (long long)llrint(t) - (long long)origin : (long long)llrint(rel);
#endif
    return true;
}

GMI_FX_HD double fx_origin(double x0, double pos_scale)
{
    return rint(x0 * pos_scale * (1.0 / 576460752303423488.0)) * 576460752303423488.0;
}

// The exponent that makes the loads fractions (every |load| < 2^e), or
// kFxNoLoad when all are zero; false when not finite or out of range.
constexpr int kFxNoLoad = -100000;
constexpr int kFxMaxExp = 900;
GMI_FX_HD bool fx_load_exponent(double largest, int *e)
{
    union {
        double d;
        unsigned long long u;
    } c;
    c.d = largest;
    const int be = (int)(c.u >> 52);  // largest >= 0
    if (largest == 0.0) {
        *e = kFxNoLoad;
        return true;
    }
    *e = be - 1022;
    return be != 2047 && *e <= kFxMaxExp && *e >= -kFxMaxExp;
}

}  // namespace gmi
