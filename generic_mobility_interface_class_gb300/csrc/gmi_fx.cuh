// gmi_fx.cuh -- fixed-point arithmetic for the FP64-grade pair sums.
//
// This GPU retires one FP64 warp instruction per ~19 cycles and SM, against
// four FP32 or two integer ones per cycle.  The pair formulas are sums of
// products of numbers whose sizes are known once the separation is
// normalised, so they need FP64's 53 bits but not its exponents.  A value
// here is an integer limb and a float for what is below it,
//     h 2^-s + lf 2^-(s + 32),      |lf| <= 2^31 but for rounding,
// with the scale s of each quantity fixed in the formulas.  A product's high
// part is exact, one 32x32 -> 64-bit multiply-add; the cross parts, 2^-30 of
// it, are two FP32 multiply-adds, which leaves about 2^-55 of the operands'
// ranges; the low part (2^-60) is left out:
//     S.h += a.h b.h  (2^-(sa + sb))      S.x += a.hf b.lf + a.lf b.hf  (2^-(sa + sb + 32))
// with hf = (float)h.  The first form of this kept both limbs as integers and
// took three wide products and twice the integer instructions (an integer
// multiply-add holds up the integer pipe too: measured): M_bb 1.9 times longer.
//
// Everything here and in gmi_pairs_fx.cuh compiles for the host too, where
// the tests compare it with the oracle.
#pragma once

#include <math.h>
#include <stdint.h>

#ifdef __CUDACC__
#include <cuda_runtime.h>
#define GMI_FX_HD __host__ __device__ __forceinline__
#else
#define GMI_FX_HD inline
#endif

namespace gmi {

struct fxop {
    int h;
    float hf, lf;
};

struct fxsum {
    long long h;
    float x;
};

// a b + c, 32 x 32 -> 64 bits, as one instruction (the compiler would
// reassociate chains of these into separate products and 64-bit sums)
GMI_FX_HD long long fx_madw(int a, int b, long long c)
{
#ifdef __CUDA_ARCH__
    long long r;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
    return r;
#else
    return c + (long long)a * b;
#endif
}
GMI_FX_HD unsigned long long fx_madw_u(unsigned a, unsigned b, unsigned long long c)
{
#ifdef __CUDA_ARCH__
    unsigned long long r;
    asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
    return r;
#else
    return c + (unsigned long long)a * b;
#endif
}

GMI_FX_HD void fx_mac(fxsum &s, const fxop &a, const fxop &b)
{
    s.h = fx_madw(a.h, b.h, s.h);
    s.x = fmaf(a.hf, b.lf, s.x);
    s.x = fmaf(a.lf, b.hf, s.x);
}

GMI_FX_HD fxsum fx_mul(const fxop &a, const fxop &b)
{
    return fxsum{fx_madw(a.h, b.h, 0), fmaf(a.lf, b.hf, a.hf * b.lf)};
}

// A sum of scale sa + sb as a value of scale sa + sb - T, without hf.  h is
// rounded so that lf is small: the cross parts' FP32 rounding scales with it.
template <int T> GMI_FX_HD fxop fx_close_low(long long h, float x)
{
    static_assert(T > 0 && T < 32, "the remainder is the low word's");
    const unsigned r = (unsigned)h << (32 - T);
    fxop v;
    v.h = (int)(h >> T) + (int)(r >> 31);
    v.lf = fmaf(x, 1.0f / (float)(1u << T), (float)(int)r);
    v.hf = 0.0f;
    return v;
}
template <int T> GMI_FX_HD fxop fx_close(long long h, float x)
{
    fxop r = fx_close_low<T>(h, x);
    r.hf = (float)r.h;
    return r;
}
// a b, closed (hf needs no more than the factors' FP32 product)
template <int T> GMI_FX_HD fxop fx_product_low(const fxop &a, const fxop &b)
{
    const fxsum s = fx_mul(a, b);
    return fx_close_low<T>(s.h, s.x);
}
template <int T> GMI_FX_HD fxop fx_product(const fxop &a, const fxop &b)
{
    fxop r = fx_product_low<T>(a, b);
    r.hf = a.hf * (b.hf * (1.0f / (float)(1u << T)));
    return r;
}

// a 64-bit number of scale s + 32 as a value of scale s
GMI_FX_HD fxop fx_split(long long q)
{
    const int h = (int)(q >> 32) + (int)((unsigned)q >> 31);
    return fxop{h, (float)h, (float)(int)q};
}

// a + m b on the parts of a value (the sums of the unused branch of a
// formula may wrap)
GMI_FX_HD fxop fx_add(const fxop &a, int m, const fxop &b)
{
    fxop r;
    r.h = (int)((unsigned)a.h + (unsigned)m * (unsigned)b.h);
    r.hf = (float)r.h;
    r.lf = fmaf((float)m, b.lf, a.lf);
    return r;
}

GMI_FX_HD fxop fx_neg(const fxop &a) { return fxop{-a.h, -a.hf, -a.lf}; }

GMI_FX_HD int fx_clz(unsigned v)
{
#ifdef __CUDA_ARCH__
    return __clz((int)v);
#else
    return v ? __builtin_clz(v) : 32;
#endif
}

GMI_FX_HD int fx_clzll(unsigned long long v)
{
#ifdef __CUDA_ARCH__
    return __clzll((long long)v);
#else
    return v ? __builtin_clzll(v) : 64;
#endif
}

GMI_FX_HD float fx_as_float(int bits)
{
    union {
        int i;
        float f;
    } c;
    c.i = bits;
    return c.f;
}

// 2^28 / sqrt(v 2^-26) for v > 0, rounded to an integer (relative error below 2^-21)
GMI_FX_HD int fx_rsqrt_seed(int v)
{
#ifdef __CUDA_ARCH__
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__int2float_rn(v)));
    return __float2int_rn(y * 2199023255552.0f);
#else
    return (int)lrintf((1.0f / sqrtf((float)v)) * 2199023255552.0f);
#endif
}

// 1/sqrt(r2) of scale 30, for r2 = h 2^-58 + x 2^-90 in [1, 13).
// y: the FP32 estimate, in 2^-28.  e = 1 - r2 y^2 (below 2^-20): the part of h
// comes from the product's bits 2^-18..2^-82 in modular arithmetic, the part
// of x in FP32.  The result is y (1 + e/2 + 3 e^2 / 8), the binomial series
// of (1 - e)^(-1/2); its next term is below 2^-61.
GMI_FX_HD fxop fx_rsqrt(long long h, float x)
{
    const unsigned rh = (unsigned)((unsigned long long)h >> 32), rl = (unsigned)h;
    const int y = fx_rsqrt_seed((int)rh);
    const unsigned long long yy = fx_madw_u((unsigned)y, (unsigned)y, 0);  // 2^-56
    const unsigned yh = (unsigned)(yy >> 32), yl = (unsigned)yy;
    unsigned long long p = fx_madw_u(rl, yl, 0) >> 32;  // h y^2 in 2^-82, modulo 2^64
    p = fx_madw_u(rh, yl, p);
    p = fx_madw_u(rl, yh, p);
    p += (unsigned long long)(rh * yh) << 32;
    const long long e = (long long)(0ull - p);
    const int eh = (int)(e >> 32);           // 2^-50
    const long long t = fx_madw(y, eh, 0);  // y e, high part, in 2^-78
    const float yf = (float)y * (1.0f / 268435456.0f);
    const float ex = -(x * 8.0779356694631609e-28f) * (yf * yf);  // -x 2^-90 y^2
    const float el = fmaf((float)(unsigned)e, 2.0679515313825692e-25f, ex);  // and the low word's 2^-82
    const float E = fmaf((float)eh, 8.8817841970012523e-16f, ex);
    const float f = yf * fmaf(0.375f * E, E, 0.5f * el);
    // y 2^-28 + t 2^-79 + f in h 2^-30 + lf 2^-62
    fxop r;
    const unsigned rest = (unsigned)(t >> 17);
    r.h = (y << 2) + (int)(t >> 49) + (int)(rest >> 31);
    r.hf = (float)r.h;
    r.lf = fmaf(f, 4611686018427387904.0f, (float)(int)rest);
    return r;
}

}  // namespace gmi
