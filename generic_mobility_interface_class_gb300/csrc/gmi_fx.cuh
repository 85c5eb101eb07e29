// gmi_fx.cuh -- 64-bit fixed-point arithmetic for the FP64-grade pair sums.
//
// This GPU retires one FP64 warp instruction per ~19 cycles and SM, against
// four FP32 or two 32x32 -> 64-bit integer multiply-adds per cycle.  The pair
// formulas are sums of products of numbers whose sizes are known once the
// separation is normalised, so they need FP64's 53 bits but not its
// exponents.  A value here is a pair of signed 32-bit limbs,
//     (hi 2^32 + lo) 2^-60,   |value| < 8,   -2^31 <= lo < 2^31,
// and a product is three 32x32 multiply-adds into two 64-bit accumulators:
//     h += a.hi b.hi   (2^-56)      x += a.hi b.lo + a.lo b.hi   (2^-88)
// (lo lo, below 2^-58, is left out), so that a sum of products rounds once.
// The operands' sizes (each bound is at its use) keep x below 2^63.
//
// Everything here and in gmi_pairs_fx.cuh compiles for the host too, where
// the tests compare it with the oracle.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#include <cuda_runtime.h>
#define GMI_FX_HD __host__ __device__ __forceinline__
#else
#include <math.h>
#define GMI_FX_HD inline
#endif

namespace gmi {

struct fx {
    int hi, lo;
};

struct fxacc {
    long long h, x;
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

// limbs of the 2^-60 fixed-point number q
GMI_FX_HD fx fx_split(long long q) { return fx{(int)((q + 0x80000000ll) >> 32), (int)q}; }

GMI_FX_HD void fx_mac(fxacc &s, fx a, fx b)
{
    s.h = fx_madw(a.hi, b.hi, s.h);
    s.x = fx_madw(a.hi, b.lo, s.x);
    s.x = fx_madw(a.lo, b.hi, s.x);
}

// the sum as a 2^-60 number (|sum| < 8), rounded down
GMI_FX_HD long long fx_q60(const fxacc &s) { return (long long)((unsigned long long)s.h << 4) + (s.x >> 28); }

GMI_FX_HD long long fx_mul60(fx a, fx b)
{
    fxacc s{0, 0};
    fx_mac(s, a, b);
    return fx_q60(s);
}

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

// FP32 estimate of 2^40 / sqrt(v), v > 0, as an integer (relative error below 2^-21)
GMI_FX_HD int fx_rsqrt_seed(int v)
{
#ifdef __CUDA_ARCH__
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__int2float_rn(v)));
    return __float2int_rn(y * 1099511627776.0f);
#else
    return (int)lrintf((1.0f / sqrtf((float)v)) * 1099511627776.0f);
#endif
}

// 1/sqrt(r2) in 2^-60, for r2 in [1, 13) in 2^-56.
// y: the FP32 estimate, in 2^-28.  e = 1 - r2 y^2 (below 2^-20) comes from
// the product's bits 2^-16..2^-80 in modular arithmetic, and the result is
// y (1 + e/2 + 3 e^2 / 8), the binomial series of (1 - e)^(-1/2); its next
// term is below 2^-61.
GMI_FX_HD long long fx_rsqrt(long long r2)
{
    const unsigned rh = (unsigned)((unsigned long long)r2 >> 32), rl = (unsigned)r2;
    const int y = fx_rsqrt_seed((int)rh);
    const unsigned long long yy = fx_madw_u((unsigned)y, (unsigned)y, 0);  // 2^-56
    const unsigned yh = (unsigned)(yy >> 32), yl = (unsigned)yy;
    unsigned long long p = fx_madw_u(rl, yl, 0) >> 32;  // r2 y^2 in 2^-80, modulo 2^64
    p = fx_madw_u(rh, yl, p);
    p = fx_madw_u(rl, yh, p);
    p += (unsigned long long)(rh * yh) << 32;
    const long long e = (long long)(0ull - p);  // 1 - r2 y^2 in 2^-80
    const int eh = (int)(e >> 32);              // 2^-48
    const long long t = fx_madw(y, eh, (long long)(fx_madw_u((unsigned)y, (unsigned)e, 0) >> 32));
    const int th = (int)(t >> 32);              // y e in 2^-44
    return ((long long)y << 32) + (t >> 17) + ((3 * fx_madw(th, eh, 0)) >> 35);
}

}  // namespace gmi
