// gmi_wall_kernel.cu -- M_ss above a no-slip wall in FP64
// (cuda_functions.cu:10-242), arranged for this GPU's FP64 pipe.
//
// The sum is bound by that pipe: a warp instruction takes it 19 cycles per
// SM, and everything else (loads, integer work, waiting) hides behind it.  So
// the pair formula is written for the fewest FP64 instructions.  The free
// and the image part act on the same loads along the same x and y
// separations, so their coefficients are added up first and applied once: 24
// multiply-adds where the two parts apart take 63.  Roots and the quotient
// start from the hardware's estimates and take one third-order step.  About
// 150 FP64 instructions a pair, from 227.
//
// A CTA owns 32 targets, one per lane; its four warps take a quarter each of
// a slice of the sources ("split"), sized so that every SM gets the same
// number of CTAs to within a few per cent; reduce_splits_tree adds the splits.
// 1280 segments: 1287 us (two targets per warp, 160 CTAs on 152 SMs, so 8 of
// them set the time) -> 480 us, at the pipe's rate for these instructions.
#include <algorithm>

#include "gmi_pair_kernels.hpp"
#include "gmi_wall_kernel.hpp"

namespace gmi {

constexpr int kWallTpb = 128;
constexpr int kWallWarps = kWallTpb / 32;
constexpr int kWallTile = 128;  // sources staged at a time

// 1/sqrt(x): the hardware estimate y (measured within 2^-20) and the
// binomial series of (1 - e)^(-1/2), e = 1 - x y^2, to e^2: the next term,
// 5/16 e^3, is below 2^-58.  By integer instructions a square that overflows counts
// as the largest number (particles that far apart do not reach each other, while
// 0 in place of y would make e a NaN) and one below 1e-120 as that, whose powers to
// y^5 are finite: a source without loads in a target's place adds zeros.
__device__ __forceinline__ double wall_rsqrt(double x)
{
    x = __hiloint2double(max(min(__double2hiint(x), 0x7fefffff), 0x2704a872), __double2loint(x));
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x * y, y, 1.0);
    return fma(y * e, fma(0.375, e, 0.5), y);
}

// 1/x: the hardware estimate y (measured within 2^-19.9) and the geometric
// series in e = 1 - x y to e^2
__device__ __forceinline__ double wall_rcp(double x)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}

// One source's contribution (not the target itself).  s: the source's x y z,
// and its force and torque times 1/(8 pi).  With I = 1/|(dx, dy, zs)|,
// h = z_j / zs and q = (zs I)^2; the image's constants carry 4/3 (its prefactor
// is 1/(6 pi)).  The reference's terms are those of pair_ss_wall.
__device__ __forceinline__ void wall_pair(double xi, double yi, double zi, const double *s, double *v, double *w)
{
    const double fx = s[3], fy = s[4], fz = s[5], tx = s[6], ty = s[7], tz = s[8];
    const double dx = xi - s[0], dy = yi - s[1], dz = zi - s[2], zs = zi + s[2];
    const double rho = fma(dy, dy, dx * dx);
    const double i1 = wall_rsqrt(fma(dz, dz, rho)), I = wall_rsqrt(fma(zs, zs, rho));
    const double h = s[2] * wall_rcp(zs);
    // free space: v = At F + Bc (d.F) d + i3 T x d, w = -i3/2 T + 3/2 i5 (d.T) d + i3 F x d
    const double i2 = i1 * i1, i3 = i2 * i1, i5 = i3 * i2;
    const double At = fma(2.0 / 3.0, i3, i1), Bc = fma(-2.0, i5, i3);
    const double pF = fma(dy, fy, dx * fx), pT = fma(dy, ty, dx * tx);
    const double Bt = Bc * fma(dz, fz, pF), Br = 1.5 * i5 * fma(dz, tz, pT);
    // image scalars
    const double gz = zs * I, q = gz * gz, I2 = I * I, I3 = I2 * I, I4 = I2 * I2, I5 = I4 * I;
    const double gf = I * fma(zs, fz, pF), gt = I * fma(zs, tz, pT);
    const double hq = h * q, t1 = fma(-h, hq, hq) * I;  // h (1 - h) q I
    const double hm = -2.0 * h, hI = hm * I;            // -2 h, -2 h I
    const double A0 = fma(I3, fma(2.0, q, -2.0 / 3.0), fma(I5, fma(-10.0 / 3.0, q, 2.0 / 3.0), fma(-2.0, t1, -I)));
    const double Z1 = fma(I3, fma(-10.0, q, 2.0), fma(I5, fma(70.0 / 3.0, q, -10.0 / 3.0), fma(6.0, t1, -I)));
    const double Z2 = fma(I3, fma(20.0, q, -4.0),
                          fma(I5, fma(-140.0 / 3.0, q, 40.0 / 3.0), hI * fma(-6.0, hq, fma(6.0, q, -1.0))));
    const double Z3 = fma(-20.0 / 3.0, I5, -hI);
    const double Z4 = -fma(fma(hm, hI, 4.0 * I3), q, I5 * fma(-20.0, q, 8.0 / 3.0));
    // force along the wall-normal and radial directions of the image
    const double S1 = fma(Z1, gf, Z2 * (gz * fz));
    // couplings, of a source at height fraction h (w from F) and 1 - h (v from T)
    const double hk = h * I2, hk1 = I2 - hk, q12 = 12.0 * q, k4 = I4 * fma(-20.0, q, 2.0), k10 = 10.0 * I4;
    const double P1 = fma(q12, hk, k4), P1c = fma(q12, hk1, k4);
    const double P2 = fma(6.0, hk, -k10), P2c = fma(6.0, hk1, -k10);
    const double b = fma(2.0, I4, I2);
    const double u = gz * fma(-2.0, hk, b), uc = gz * fma(-2.0, hk1, b);
    const double E = fma(I2, I, -i3);
    const double M = fma(dx, ty, -(dy * tx)), N = fma(dy, fx, -(dx * fy));
    const double U1 = fma(i3, dz, -u), U2 = fma(i3, dz, uc);
    // v
    const double A = At + A0;
    const double W = fma(I, fma(gz * P2c, M * I, S1), Bt);
    const double e1 = tz * E;
    v[0] = fma(A, fx, v[0]); v[0] = fma(W, dx, v[0]); v[0] = fma(U2, ty, v[0]); v[0] = fma(e1, dy, v[0]);
    v[1] = fma(A, fy, v[1]); v[1] = fma(W, dy, v[1]); v[1] = fma(-U2, tx, v[1]); v[1] = fma(-e1, dx, v[1]);
    v[2] = fma(A + Z4, fz, v[2]); v[2] = fma(Bt, dz, v[2]); v[2] = fma(gz, fma(Z3, gf, S1), v[2]);
    v[2] = fma(M, fma(I, fma(-q, P2c, P1c), E), v[2]);
    // w
    const double sF = fma(fz, P1, -(gz * gf) * P2);
    const double c = fma(-3.0 * I5, M, fma(I, sF, fz * E));
    const double Aw = fma(I3, fma(-3.0, q, 0.5), -0.5 * i3);
    const double a1 = -1.5 * I3 * gt;
    const double Ww = fma(I, a1, Br);
    w[0] = fma(Aw, tx, w[0]); w[0] = fma(Ww, dx, w[0]); w[0] = fma(U1, fy, w[0]); w[0] = fma(c, dy, w[0]);
    w[1] = fma(Aw, ty, w[1]); w[1] = fma(Ww, dy, w[1]); w[1] = fma(-U1, fx, w[1]); w[1] = fma(-c, dx, w[1]);
    w[2] = fma(Aw, tz, w[2]); w[2] = fma(Br, dz, w[2]); w[2] = fma(-a1, gz, w[2]); w[2] = fma(-E, N, w[2]);
}

// A segment on itself (cuda_functions.cu:78-107); the loads carry 1/(8 pi).
__device__ __forceinline__ void wall_self(double z, const double *s, double *v, double *w)
{
    const double h1 = 1.0 / z, h3 = h1 * h1 * h1, h4 = h3 * h1, h5 = h4 * h1, k = 4.0 / 3.0;
    const double p = k - (9.0 * h1 - 2.0 * h3 + h5) * (k / 16.0), q = k - (9.0 * h1 - 4.0 * h3 + h5) * (k / 8.0);
    const double c = (k * 3.0 / 32.0) * h4;
    const double pr = 1.0 - (k * 15.0 / 64.0) * h3, qr = 1.0 - (k * 3.0 / 32.0) * h3;
    v[0] += p * s[3] + c * s[7];
    v[1] += p * s[4] - c * s[6];
    v[2] += q * s[5];
    w[0] += pr * s[6] - c * s[4];
    w[1] += pr * s[7] + c * s[3];
    w[2] += qr * s[8];
}

__global__ void __launch_bounds__(kWallTpb) rpy_wall_kernel(const WallSum a, int chunk)
{
    __shared__ __align__(16) double src[kWallTile][10];
    __shared__ double red[kWallWarps][6][33];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int j_begin = blockIdx.y * chunk, j_end = min(j_begin + chunk, a.n_src);
    const int group0 = blockIdx.x * 32, ti = a.tgt_start + min(group0 + lane, a.n_tgt - 1);
    const double xi = a.x[3 * (size_t)ti], yi = a.x[3 * (size_t)ti + 1], zi = a.x[3 * (size_t)ti + 2];
    double v[3] = {0.0, 0.0, 0.0}, w[3] = {0.0, 0.0, 0.0};
    for (int j0 = j_begin; j0 < j_end; j0 += kWallTile) {
        const int jn = min(kWallTile, j_end - j0);
        __syncthreads();
        for (int e = tid; e < 3 * jn; e += kWallTpb) src[e / 3][e % 3] = a.x[3 * (size_t)j0 + e];
        for (int e = tid; e < 6 * jn; e += kWallTpb) src[e / 6][3 + e % 6] = a.f[6 * (size_t)j0 + e] * (1.0 / (8.0 * kPi));
        __syncthreads();
        const int per = (jn + kWallWarps - 1) / kWallWarps, b = min(warp * per, jn), e = min(b + per, jn);
#pragma unroll 1
        for (int j = b; j < e; ++j) {
            if (j0 + j == ti)
                wall_self(zi, src[j], v, w);
            else
                wall_pair(xi, yi, zi, src[j], v, w);
        }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        red[warp][c][lane] = v[c];
        red[warp][3 + c][lane] = w[c];
    }
    __syncthreads();
    const int nt = min(32, a.n_tgt - group0);
    const size_t base = (size_t)group0 * 6, count = (size_t)a.n_tgt * 6;
    for (int o = tid; o < nt * 6; o += kWallTpb) {
        const int i = o / 6, c = o - 6 * i;
        const double t = (red[0][c][i] + red[1][c][i]) + (red[2][c][i] + red[3][c][i]);
        if (a.partial != nullptr)
            a.partial[blockIdx.y * count + base + o] = t;
        else
            a.out[base + o] = t;
    }
}

// Sources per split: the smallest power of two from 4 (one source per warp)
// that leaves no more than 24 CTAs per SM, whose set-up then costs little.
static int wall_chunk(int n_tgt, int n_src, int sm_count)
{
    const long long groups = (n_tgt + 31) / 32;
    long long chunk = 4;
    while (groups * ((n_src + chunk - 1) / chunk) > 24ll * sm_count && chunk < n_src) chunk *= 2;
    while ((n_src + chunk - 1) / chunk > 65535) chunk *= 2;
    return (int)chunk;
}

int wall_splits(int n_tgt, int n_src, int sm_count)
{
    if (n_tgt <= 0 || n_src <= 0) return 1;
    const int chunk = wall_chunk(n_tgt, n_src, sm_count);
    return (n_src + chunk - 1) / chunk;
}

gmi_status launch_wall_fp64(cudaStream_t stream, int sm_count, const WallSum &a, int *launched)
{
    const int chunk = wall_chunk(a.n_tgt, a.n_src, sm_count), splits = (a.n_src + chunk - 1) / chunk;
    rpy_wall_kernel<<<dim3((a.n_tgt + 31) / 32, splits), kWallTpb, 0, stream>>>(a, chunk);
    GMI_CUDA_TRY(cudaGetLastError());
    *launched = 1;
    if (a.partial != nullptr) {
        const int count = a.n_tgt * 6;
        GMI_CUDA_TRY(launch_chained(true, reduce_splits_tree, dim3((count + 63) / 64), dim3(64), stream, a.partial, splits,
                                    count, a.out, 0));
        *launched = 2;
    }
    return GMI_OK;
}

}  // namespace gmi
