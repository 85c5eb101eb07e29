// gmi_fx_kernels.cu -- the FP64-grade free-space pair sums (precision
// GMI_FP64) in 64-bit fixed point.
//
// Two kernels per sum, or one for small sums.  The pack kernel turns the
// sources into integer records (gmi_pairs_fx.cuh), one CTA per block of 512
// with the block's exponent found by a block maximum.  In the pair kernel a CTA
// owns 32 targets, one per lane, and a contiguous slice ("split") of the
// sources, staged in tiles of 128 into shared memory by bulk copies; its four
// warps take a quarter of each tile each, fold their integer sums into FP64 once
// per block and meet in shared memory at the end.  32 targets per CTA rather than
// 128 let a few hundred targets reach every SM.  With several splits
// reduce_splits_tree adds the partial sums.
//
// A block whose loads or positions the formats do not hold (not finite, a load
// beyond 2^+-900, a particle further than about 400 radii from the first
// source) is marked by the pack kernel, and its pairs, and all pairs of a
// warp with such a target, are summed in FP64 from the original arrays.
//
// What bounds it: instruction issue, M_ss about 470 instructions a pair and warp
// (61 wide integer multiplies, 140 FP32, 200 integer) at 1.5 cycles each; the
// FP64 kernel executed 65 FP64 instructions at 76 cycles each.  Integer limbs
// alone (530 instructions, 146 of them wide multiplies) took 1.8 cycles each.
// FP64 kernel -> integer limbs -> limb and FP32 (this one):
//   12,800 segments                  20.4 -> 3.90 -> 2.86 ms  (5.0 TFLOP/s at 87 flop a pair)
//   4096 blobs                       1223 -> 229 -> 178 us
//   12,800 segments, 4096 blobs,
//   both ways                        9.72 -> 1.80 -> 1.38 ms
// Nothing outside the pair loop runs in FP64 (76 cycles an instruction, 95 a
// conversion): positions and loads become integers, and sums FP64 numbers, by
// integer instructions.  With FP64 there, 642 segments took 28.6 us (now 20.5),
// 962 41.0 (34.8), 1669 blobs 55.3 (45.1), a solve of 962 particles 4.25 ms (3.80).
// A sum of wide sources only (gmi_pairs_fx.cuh), such as torques without forces,
// takes 22 % longer in M_ss and 9 % in M_bs and M_sb.
// Error against extended precision (2-norm, mean of four draws) as a part of the FP64
// kernels': 60 to 1500 segments 0.56 to 0.99, torques alone 0.47 to 0.92; 50 to 1200
// blobs 0.59 to 0.86; segments on blobs and back 0.64 to 0.89 (radii 0.75 to 1.3).
#include <algorithm>

#include "gmi_fx_kernels.hpp"
#include "gmi_pair_kernels.hpp"
#include "gmi_pairs.cuh"
#include "gmi_pairs_fx.cuh"

namespace gmi {

static_assert((int)kFxSS == (int)kSS && (int)kFxBB == (int)kBB && (int)kFxSB == (int)kSB && (int)kFxBS == (int)kBS,
              "FxKind follows PairKind");

constexpr int kFxBlock = 512;  // sources per block: one exponent, one fold
constexpr int kFxTpb = 128;    // four warps
constexpr int kFxWarps = kFxTpb / 32;
constexpr int kFxStages = 2;
constexpr int kFxInlinePerSm = 4;  // CTAs per SM up to which a CTA packs its own sources
constexpr int kFxBadTile = -(1 << 15);  // in place of a block's exponent: sum it in FP64
static_assert(kFxBlock == kFxWarps * kFxFold && kFxBlock % kFxTile == 0, "a warp's quarter of a block is one fold");
static_assert(kFxTile == 32 * kFxWarps, "fx_place: four warps hold a tile's sources");

template <int KIND> struct FxTraits {
    static constexpr bool torque = KIND == kFxSS || KIND == kFxBS;
    static constexpr int nout = (KIND == kFxSS || KIND == kFxSB) ? 6 : 3;
    static constexpr int nf = torque ? 6 : 3;
    // 16-byte quarters per record: X0 X1 | X2 F0.h F0.hf | F0.lf F1 | F2 meta | T0 T1 | T2 T's gap, pad,
    // meta: the block's exponent << 16 | the tile's records that are not wide << 8 | F's gap
    static constexpr int quads = torque ? 6 : 4;
};

struct FxLaunch {
    const double *xt, *xs, *fs;
    const int4 *rec;
    int tgt_start, n_tgt, n_src, chunk;
    double *out, *partial;
    int accumulate;
    unsigned *err;
    const int *skip;
    unsigned long long wait_ns;
    FxConsts K;
    EqualK<double> eq;
    UnequalK<double> uq;
};

// One source on its way into a record: its position, its loads and their
// exponent (torques over U), that of its force and of its torque.
template <int KIND> struct FxPacking {
    long long X[3];
    double F[FxTraits<KIND>::nf];
    int e, f, t;
};
constexpr int kFxMark = 0x7fffffff;  // as an exponent: the formats do not hold this source

template <int KIND>
__device__ __forceinline__ FxPacking<KIND> fx_read_source(const double *__restrict__ x, const double *__restrict__ f,
                                                          int i, const FxConsts &K)
{
    using Tr = FxTraits<KIND>;
    FxPacking<KIND> p;
    bool ok = true;
#pragma unroll
    for (int c = 0; c < 3; ++c) ok = fx_position(x[3 * (size_t)i + c], K, fx_origin(x[c], K), &p.X[c]) && ok;
    p.f = p.t = kFxNoLoad;
#pragma unroll
    for (int c = 0; c < Tr::nf; ++c) {
        p.F[c] = f[Tr::nf * (size_t)i + c];
        if (c < 3)
            p.f = max(p.f, fx_exponent(p.F[c], 0));
        else
            p.t = max(p.t, fx_exponent(p.F[c], K.unit_exp));
    }
    p.e = max(p.f, p.t);
    if (!ok || !fx_exponent_held(p.e)) p.e = kFxMark;
    return p;
}

// The largest exponent of a CTA of NW warps, one source per thread.
template <int NW> __device__ __forceinline__ int fx_block_max(int e, int *wmax)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) e = max(e, __shfl_xor_sync(0xffffffffu, e, o));
    if ((threadIdx.x & 31) == 0) wmax[threadIdx.x >> 5] = e;
    __syncthreads();
    e = wmax[0];
#pragma unroll
    for (int w = 1; w < NW; ++w) e = max(e, wmax[w]);
    return e;
}

// Where a CTA's sources go in their tiles, the wide ones last, so that each kind
// has a loop of its own: a choice in the one loop cost M_ss 4 % of its time whether
// or not it met a wide source.  even: records of the tile that are not wide.
struct FxPlace {
    int at, even;
};
template <int KIND, int NW> __device__ __forceinline__ FxPlace fx_place(bool present, bool wide, int *counts)
{
    const int tid = threadIdx.x, warp = tid >> 5, first = warp & ~(kFxWarps - 1);
    if (KIND == kFxBB) return FxPlace{tid, kFxTile};
    const unsigned mine = __ballot_sync(0xffffffffu, present && !wide);
    if ((tid & 31) == 0) counts[warp] = __popc(mine);
    __syncthreads();
    int before = __popc(mine & ((1u << (tid & 31)) - 1u)), even = 0;
#pragma unroll
    for (int w = 0; w < kFxWarps; ++w) {
        const int n = counts[first + w];
        before += first + w < warp ? n : 0;
        even += n;
    }
    const int start = 32 * first;
    return FxPlace{wide ? even + tid - before : start + before, even};
}

// The record of a source in a block whose largest exponent is E.
template <int KIND>
__device__ __forceinline__ void fx_write_record(const FxPacking<KIND> &p, int E, const FxHeld &h, int even,
                                                const FxConsts &K, int4 *r)
{
    using Tr = FxTraits<KIND>;
    const bool bad = E == kFxMark;
    const int tile = bad ? kFxBadTile : E;
    const int meta = (int)((unsigned)tile << 16) | even << 8 | h.gap;
    const auto lo = [](long long v) { return (int)(unsigned)v; };
    const auto hi = [](long long v) { return (int)(v >> 32); };
    fxop F[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        long long v;
        fx_fixed(p.F[c], 62 - (tile - h.gap), &v);
        F[c] = bad ? fxop{0, 0.0f, 0.0f} : fx_split(v);
    }
    r[0] = make_int4(lo(p.X[0]), hi(p.X[0]), lo(p.X[1]), hi(p.X[1]));
    r[1] = make_int4(lo(p.X[2]), hi(p.X[2]), F[0].h, __float_as_int(F[0].hf));
    r[2] = make_int4(__float_as_int(F[0].lf), F[1].h, __float_as_int(F[1].hf), __float_as_int(F[1].lf));
    r[3] = make_int4(F[2].h, __float_as_int(F[2].hf), __float_as_int(F[2].lf), meta);
    if constexpr (Tr::torque) {
        long long T[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            fx_fixed(p.F[3 + c], 62 - (tile - h.tgap) - K.unit_exp, &T[c]);
            if (bad) T[c] = 0;
        }
        r[4] = make_int4(lo(T[0]), hi(T[0]), lo(T[1]), hi(T[1]));
        r[5] = make_int4(lo(T[2]), hi(T[2]), h.tgap, 0);
    }
}

// A CTA's records, NW tiles' quarters, the thread's source p into its tile of
// `rec` (records of the CTA's first source on).
template <int KIND, int NW>
__device__ __forceinline__ void fx_write_records(const FxPacking<KIND> &p, bool present, const FxConsts &K, int *ints,
                                                 int4 *rec)
{
    int E = fx_block_max<NW>(p.e, ints);
    if (E == kFxNoLoad) E = 0;
    FxHeld h{0, 0, false};
    if (E != kFxMark) h = fx_held<KIND>(p.f, p.t, E);
    const FxPlace to = fx_place<KIND, NW>(present, h.wide, ints + NW);
    if (present) fx_write_record<KIND>(p, E, h, to.even, K, rec + (size_t)to.at * FxTraits<KIND>::quads);
}

template <int KIND>
__global__ void __launch_bounds__(kFxBlock) fx_pack_kernel(const double *__restrict__ x, const double *__restrict__ f,
                                                          int n, FxConsts K, int4 *__restrict__ rec, const int *skip)
{
    __shared__ int ints[2 * kFxBlock / 32];
    pdl_wait();
    if (skip != nullptr && *skip != 0) return;
    const int i = blockIdx.x * kFxBlock + threadIdx.x;
    FxPacking<KIND> p;
    p.e = p.f = p.t = kFxNoLoad;
    if (i < n) p = fx_read_source<KIND>(x, f, i, K);
    fx_write_records<KIND, kFxBlock / 32>(p, i < n, K, ints,
                                          rec + (size_t)blockIdx.x * kFxBlock * FxTraits<KIND>::quads);
}

struct FxSum {
    double v[6];
};

// M_bb's near field, out of line as ss_near_coeffs: A, and B times dF
static __device__ __noinline__ double2 fx_bb_near_fp64(double w, double f6pma, double d)
{
    return make_double2((1.0 - 3.0 * w) * f6pma, w * f6pma * d);
}

// A pair in FP64, far pairs in as few FP64 instructions as it takes: one factor
// 1/(8 pi mu) on 1/r scales all coefficients, C d serves both cross products, and the
// root is the hardware's estimate with one third-order step (gmi_wall_kernel.cu; the
// square is held between 1e-300 and the largest number by an integer instruction, for
// the pair at r = 0).  54 a pair in M_ss and 27 in M_bb, where pair_ss and pair_bb
// execute 65 and 33.  A near pair only has other coefficients: a warp meets its own
// 32 targets one lane at a time.
template <int KIND>
__device__ __forceinline__ void fx_pair_fp64(double dx, double dy, double dz, const double *F, const FxLaunch &a,
                                             double f8, double q, unsigned long long near, double *v)
{
    const double r2 = fma(dx, dx, fma(dy, dy, dz * dz));
    const double x = __hiloint2double(max(min(__double2hiint(r2), 0x7fefffff), 0x01a56e1f), __double2loint(r2));
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double h = fma(-x * y, y, 1.0), ir = fma(y * h, fma(0.375, h, 0.5), y);
    const double dF = fma(dx, F[0], fma(dy, F[1], dz * F[2]));
    double dT = 0.0, A, B, C, Ar = 0.0, Br = 0.0;
    if constexpr (KIND == kFxSS) dT = fma(dx, F[3], fma(dy, F[4], dz * F[5]));
    if ((unsigned long long)__double_as_longlong(r2) > near) {
        const double ir2 = ir * ir, c1 = f8 * ir, c5 = c1 * ir2 * ir2;
        C = c1 * ir2;
        A = fma(q, C, c1);
        B = fma(-3.0 * q, c5, C) * dF;
        if constexpr (KIND == kFxSS) {
            Ar = -0.5 * C;
            Br = 1.5 * c5 * dT;
        }
    } else if constexpr (KIND == kFxSS) {
        ss_near_coeffs<double>(r2, ir, dF, dT, a.eq, A, B, Ar, Br, C);
    } else if constexpr (KIND == kFxBB) {
        const double2 n = fx_bb_near_fp64(r2 * ir * a.eq.q32, a.eq.f6pma, ir * ir * dF);
        A = n.x;
        B = n.y;
    } else {
        unequal_coeffs<double>(r2, ir, dF, a.uq, A, B, C);
    }
    v[0] = fma(B, dx, fma(A, F[0], v[0]));
    v[1] = fma(B, dy, fma(A, F[1], v[1]));
    v[2] = fma(B, dz, fma(A, F[2], v[2]));
    if constexpr (KIND == kFxBB) return;
    const double cx = C * dx, cy = C * dy, cz = C * dz;
    if constexpr (FxTraits<KIND>::torque) {
        v[0] = fma(F[4], cz, fma(-F[5], cy, v[0]));
        v[1] = fma(F[5], cx, fma(-F[3], cz, v[1]));
        v[2] = fma(F[3], cy, fma(-F[4], cx, v[2]));
    }
    if constexpr (FxTraits<KIND>::nout == 6) {
        v[3] = fma(F[1], cz, fma(-F[2], cy, v[3]));
        v[4] = fma(F[2], cx, fma(-F[0], cz, v[4]));
        v[5] = fma(F[0], cy, fma(-F[1], cx, v[5]));
    }
    if constexpr (KIND == kFxSS) {
        v[3] = fma(Br, dx, fma(Ar, F[3], v[3]));
        v[4] = fma(Br, dy, fma(Ar, F[4], v[4]));
        v[5] = fma(Br, dz, fma(Ar, F[5], v[5]));
    }
}

// The sources [j0, j1) on one target in FP64, for the blocks and targets that
// the fixed-point formats do not hold.  M_bb four at a time, for the loads in
// flight (the others gain nothing and lose 0.6 % of the sums that do fit).
// What bounds it is the FP64 pipe, and that the splits suit the fixed-point loop: at
// 1100 particles 315 CTAs load some SMs with three of them, where two are the mean.
// With pair_ss and pair_bb here sets spread over 2400 radii took up to 1.28 of the
// time of the tiled and warp FP64 kernels (now 0.5 to 0.98, but 1.17 for M_ss of 1150);
// us, those kernels -> pair_* -> this:
//   M_ss 300 60 -> 38 -> 35, 1100 180 -> 232 -> 195, 4000 2340 -> 1976 -> 1602
//   M_bb 300 35 -> 23 -> 21, 1100 103 -> 131 -> 101, 4000 1222 -> 1236 -> 858
//   M_bs 300 47 -> 25 -> 23, 1100 133 -> 146 -> 123, 4000 1571 -> 1316 -> 1104
template <int KIND>
static __device__ __noinline__ FxSum fx_sum_fp64(const FxLaunch &a, int ti, int j0, int j1)
{
    FxSum s{};
    const double xi = a.xt[3 * (size_t)ti], yi = a.xt[3 * (size_t)ti + 1], zi = a.xt[3 * (size_t)ti + 2];
    constexpr bool kOneSet = KIND == kFxSS || KIND == kFxBB;
    const double f8 = kOneSet ? a.eq.f8pm : a.uq.f8pm, q = kOneSet ? a.eq.two_a2 * (1.0 / 3.0) : a.uq.far_c;
    const unsigned long long near = (unsigned long long)__double_as_longlong(kOneSet ? a.eq.four_a2 : a.uq.sum2);
    constexpr int kAtOnce = KIND == kFxBB ? 4 : 1;
#pragma unroll kAtOnce
    for (int j = j0; j < j1; ++j) {
        double F[6] = {0, 0, 0, 0, 0, 0};
        for (int c = 0; c < FxTraits<KIND>::nf; ++c) F[c] = a.fs[FxTraits<KIND>::nf * (size_t)j + c];
        fx_pair_fp64<KIND>(xi - a.xs[3 * (size_t)j], yi - a.xs[3 * (size_t)j + 1], zi - a.xs[3 * (size_t)j + 2], F, a, f8,
                           q, near, s.v);
    }
    return s;
}

__device__ __forceinline__ long long fx_word(int lo, int hi)
{
    return (long long)(((unsigned long long)(unsigned)hi << 32) | (unsigned)lo);
}

template <int KIND> __device__ __forceinline__ FxSource fx_load_source(const int4 *q)
{
    const int4 a = q[0], b = q[1], c = q[2], d = q[3];
    FxSource s;
    s.X[0] = fx_word(a.x, a.y);
    s.X[1] = fx_word(a.z, a.w);
    s.X[2] = fx_word(b.x, b.y);
    s.F[0] = fxop{b.z, __int_as_float(b.w), __int_as_float(c.x)};
    s.F[1] = fxop{c.y, __int_as_float(c.z), __int_as_float(c.w)};
    s.F[2] = fxop{d.x, __int_as_float(d.y), __int_as_float(d.z)};
    s.gap = d.w & 255;
    s.tgap = 0;
    if constexpr (FxTraits<KIND>::torque) {
        const int4 e = q[4], f = q[5];
        s.T[0] = fx_word(e.x, e.y);
        s.T[1] = fx_word(e.z, e.w);
        s.T[2] = fx_word(f.x, f.y);
        s.tgap = f.z;
    }
    return s;
}

// bulk copy of whole records (a multiple of 16 bytes) into shared memory
__device__ __forceinline__ void bulk_load(void *smem_dst, const void *src, unsigned bytes, uint64_t *bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(smem_dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

// CTAs per SM that the registers are held to.  M_ss: 3 2.80 ms (12,800
// segments), 4 2.85; M_bb: 6 185 us (4096 blobs), 5 189, 7 190, 4 194; both
// ways between the two: 4 1.37 ms, 3 1.42, 5 1.40.
template <int KIND> constexpr int kFxCtas = KIND == kFxSS ? 3 : KIND == kFxBB ? 6 : 4;

// kInline: no pack kernel ran; the split is at most one tile, whose records the
// CTA makes itself.
template <int KIND, bool kInline>
__global__ void __launch_bounds__(kFxTpb, kFxCtas<KIND>) rpy_fx_kernel(const __grid_constant__ FxLaunch a)
{
    using Tr = FxTraits<KIND>;
    constexpr int NOUT = Tr::nout;
    __shared__ __align__(128) int4 ring[kFxStages][kFxTile * Tr::quads];
    __shared__ long long red[2][kFxWarps][NOUT][33];
    __shared__ uint64_t bars[kFxStages];
    __shared__ int ints[2 * kFxWarps];

    pdl_wait();
    if (a.skip != nullptr && *a.skip != 0) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int j_begin = blockIdx.y * a.chunk, j_end = min(j_begin + a.chunk, a.n_src);
    const int ntiles = (j_end - j_begin + kFxTile - 1) / kFxTile;
    if (!kInline) {
        if (tid == 0) {
#pragma unroll
            for (int s = 0; s < kFxStages; ++s) mbar_init(&bars[s], 1);
            fence_mbar_init();
        }
        __syncthreads();
    }
    int issued = 0;  // tiles requested so far (meaningful on thread 0)
    const auto request = [&](int t) {
        const int j0 = j_begin + t * kFxTile;
        const unsigned bytes = (unsigned)min(kFxTile, j_end - j0) * (Tr::quads * 16u);
        mbar_arrive_expect_tx(&bars[t % kFxStages], bytes);
        bulk_load(ring[t % kFxStages], a.rec + (size_t)j0 * Tr::quads, bytes, &bars[t % kFxStages]);
    };
    if (!kInline && tid == 0)
        for (; issued < kFxStages && issued < ntiles; ++issued) request(issued);
    if (kInline) {
        FxPacking<KIND> p;
        p.e = p.f = p.t = kFxNoLoad;
        const int i = j_begin + tid;
        if (i < j_end) p = fx_read_source<KIND>(a.xs, a.fs, i, a.K);
        fx_write_records<KIND, kFxWarps>(p, i < j_end, a.K, ints, ring[0]);
        __syncthreads();
    }

    const int group0 = blockIdx.x * 32;
    const int ti = a.tgt_start + min(group0 + lane, a.n_tgt - 1);
    long long X[3];
    bool ok = true;
#pragma unroll
    for (int c = 0; c < 3; ++c)
        ok = fx_position(a.xt[3 * (size_t)ti + c], a.K, fx_origin(a.xs[c], a.K), &X[c]) && ok;
    const bool warp_ok = __all_sync(0xffffffffu, ok);
    double tot[NOUT];
#pragma unroll
    for (int c = 0; c < NOUT; ++c) tot[c] = 0.0;

    bool timed_out = false;
    FxAcc<NOUT> acc;
    fx_clear(acc);
    int E = 0;             // of the block in acc
    bool earlier = false;  // tot holds something (the same in every thread)
    int t = 0;
    for (; t < ntiles; ++t) {
        const int s = t % kFxStages;
        if (!kInline) {
            const bool arrived = mbar_wait_bounded(&bars[s], (t / kFxStages) & 1, a.wait_ns);
            if (__syncthreads_or(!arrived)) {
                timed_out = true;
                break;
            }
            // every thread has finished tile t - 1: its stage can be refilled
            if (tid == 0 && t >= 1 && issued < ntiles) request(issued++);
        }
        const int j0 = j_begin + t * kFxTile, jn = min(kFxTile, j_end - j0);
        const int per = (jn + kFxWarps - 1) / kFxWarps, b = min(warp * per, jn), e = min(b + per, jn);
        const int4 *tile = ring[s];
        const int Et = tile[3].w >> 16;
        if (Et == kFxBadTile || !warp_ok) {  // the whole block
            const FxSum r = fx_sum_fp64<KIND>(a, ti, j0 + b, j0 + e);
#pragma unroll
            for (int c = 0; c < NOUT; ++c) tot[c] += r.v[c];
            earlier = true;
            continue;
        }
        E = Et;
        // the wide sources are the tile's last
        const int mid = KIND == kFxBB ? e : min(e, max(b, tile[3].w >> 8 & 255));
        unsigned close = 0;  // of the warp's sources, those close to the lane's target
        for (int j = b; j < mid;) {
            const int stop = min(j + kFxSettle[KIND], mid);
#pragma unroll 1
            for (; j < stop; ++j)
                fx_pair<KIND, false>(X, fx_load_source<KIND>(tile + j * Tr::quads), a.K, acc, close, 1u << (j - b));
            fx_settle(acc);
        }
        if (KIND != kFxBB) {
#pragma unroll 1
            for (int j = mid; j < e; ++j) {
                fx_pair<KIND, true>(X, fx_load_source<KIND>(tile + j * Tr::quads), a.K, acc, close, 1u << (j - b));
                fx_settle(acc);
            }
        }
        if constexpr (KIND == kFxSS) {
#pragma unroll 1
            for (; close != 0; close &= close - 1) {
                const int j = b + __ffs(close) - 1;
                const FxSource src = fx_load_source<KIND>(tile + j * Tr::quads);
                if (j < mid)
                    fx_close_cross<false>(X, src, a.K, acc);
                else
                    fx_close_cross<true>(X, src, a.K, acc);
                fx_settle(acc);
            }
        }
        if (t + 1 < ntiles && (j0 + kFxTile) % kFxBlock == 0) {  // the block's last tile
#pragma unroll
            for (int c = 0; c < NOUT; ++c)
                tot[c] += fx_value(fx_total(acc, c), E, c < 3 ? a.K.vscale : a.K.wscale, c < 3 ? a.K.vfix : a.K.wfix);
            fx_clear(acc);
            earlier = true;
        }
    }

    if (timed_out) {
        if (tid == 0) {
            atomicOr(a.err, kDevErrWaitTimeout);
            // let the copies still in flight land (bounded) before the CTA exits
            for (int u = t; u < issued; ++u) (void)mbar_wait_bounded(&bars[u % kFxStages], (u / kFxStages) & 1);
        }
        return;
    }

    // the warps' sums of the last block meet as integers, so they are rounded
    // once; earlier blocks' (of splits beyond one block) in FP64
#pragma unroll
    for (int c = 0; c < NOUT; ++c) {
        const FxTotal v = fx_total(acc, c);
        red[0][warp][c][lane] = v.a;
        red[1][warp][c][lane] = v.b;
    }
    __syncthreads();
    const int nt = min(32, a.n_tgt - group0);
    const size_t base = (size_t)group0 * NOUT, count = (size_t)a.n_tgt * NOUT;
    constexpr int kPer = (32 * NOUT + kFxTpb - 1) / kFxTpb;
    double sum[kPer];
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        const int o = tid + k * kFxTpb, i = o / NOUT, c = o - i * NOUT;
        if (o >= nt * NOUT) continue;
        FxTotal v{0, 0};
#pragma unroll
        for (int w = 0; w < kFxWarps; ++w) {
            v.a += red[0][w][c][i];
            v.b += red[1][w][c][i];
        }
        sum[k] = fx_value(v, E, c < 3 ? a.K.vscale : a.K.wscale, c < 3 ? a.K.vfix : a.K.wfix);
    }
    if (earlier) {
        __syncthreads();
#pragma unroll
        for (int c = 0; c < NOUT; ++c) red[0][warp][c][lane] = __double_as_longlong(tot[c]);
        __syncthreads();
    }
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        const int o = tid + k * kFxTpb, i = o / NOUT, c = o - i * NOUT;
        if (o >= nt * NOUT) continue;
        double v = sum[k];
        if (earlier) {
            const auto r = [&](int w) { return __longlong_as_double(red[0][w][c][i]); };
            v += (r(0) + r(1)) + (r(2) + r(3));
        }
        if (a.partial != nullptr)
            a.partial[blockIdx.y * count + base + o] = v;
        else
            a.out[base + o] = a.accumulate ? a.out[base + o] + v : v;
    }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
static int quads_of(int kind) { return (kind == kSS || kind == kBS) ? 6 : 4; }
static int nout_of(int kind) { return (kind == kBB || kind == kBS) ? 3 : 6; }

size_t fx_record_bytes(int kind) { return (size_t)quads_of(kind) * 16; }

bool fx_supported(int kind, double as, double ab, double mu)
{
    FxConsts K;
    return kind != kSSWall && fx_consts(kind, as, ab, mu, &K);
}

using FxPairFn = void (*)(FxLaunch);
using FxPackFn = void (*)(const double *, const double *, int, FxConsts, int4 *, const int *);

template <bool kInline> static FxPairFn pair_fn(int kind)
{
    return kind == kSS ? rpy_fx_kernel<kFxSS, kInline> : kind == kBB ? rpy_fx_kernel<kFxBB, kInline>
         : kind == kSB ? rpy_fx_kernel<kFxSB, kInline> : rpy_fx_kernel<kFxBS, kInline>;
}
static FxPackFn pack_fn(int kind)
{
    return kind == kSS ? fx_pack_kernel<kFxSS> : kind == kBB ? fx_pack_kernel<kFxBB>
         : kind == kSB ? fx_pack_kernel<kFxSB> : fx_pack_kernel<kFxBS>;
}

int fx_splits(int n_tgt, int n_src, int sm_count)
{
    if (n_tgt <= 0 || n_src <= 0) return 1;
    const int chunk = fx_chunk((n_tgt + 31) / 32, n_src, sm_count, 1 << 20);
    return (n_src + chunk - 1) / chunk;
}

gmi_status launch_pair_fx(const FxPairSum &s, int *launched)
{
    *launched = 0;
    if (s.splits_out) *s.splits_out = 1;
    if (s.n_tgt <= 0) return GMI_OK;
    const int nout = nout_of(s.kind);
    if (s.n_src <= 0) {
        if (!s.accumulate)
            GMI_CUDA_TRY(cudaMemsetAsync(s.out, 0, (size_t)s.n_tgt * nout * sizeof(double), s.stream));
        return GMI_OK;
    }
    FxLaunch a{};
    if (!fx_consts(s.kind, s.as, s.ab, s.mu, &a.K)) {
        set_last_error_msg("launch_pair_fx: radii outside the fixed-point formats");
        return GMI_ERR_ARG;
    }
    PairConsts c;
    fill_consts(c, s.as, s.as, s.ab, s.mu);
    a.eq = EqualK<double>{c.eq[0], c.eq[1], c.eq[2], c.eq[3], c.eq[4], c.eq[5], c.eq[6], c.eq[7], c.eq[8]};
    a.uq = UnequalK<double>{c.uq[0], c.uq[1], c.uq[2], c.uq[3], c.uq[4],  c.uq[5], c.uq[6],
                            c.uq[7], c.uq[8], c.uq[9], c.uq[10], c.uq[11], c.uq[12]};
    const int groups = (s.n_tgt + 31) / 32;
    const size_t per_split = (size_t)s.n_tgt * nout * sizeof(double);
    int most = (int)std::min<size_t>(s.partial_bytes / per_split, 1 << 20);
    if (s.max_splits > 0) most = std::min(most, s.max_splits);
    a.chunk = fx_chunk(groups, s.n_src, s.sm_count, std::max(1, most));
    const int splits = (s.n_src + a.chunk - 1) / a.chunk;
    a.xt = s.xt;
    a.xs = s.xs;
    a.fs = s.fs;
    a.rec = static_cast<const int4 *>(s.rec);
    a.tgt_start = s.tgt_start;
    a.n_tgt = s.n_tgt;
    a.n_src = s.n_src;
    a.out = s.out;
    a.partial = splits > 1 || s.staged ? s.partial : nullptr;
    a.accumulate = s.accumulate;
    a.err = s.err;
    a.skip = s.skip;
    a.wait_ns = s.wait_ns;
    // a CTA packs its own sources where the packing kernel and its boundary
    // (5 us) cost more than packing each tile once per target group
    // (slices of less than a tile always: their records do not cross the slice)
    const bool packs_itself =
        a.chunk < kFxTile || (a.chunk == kFxTile && (long long)groups * splits <= kFxInlinePerSm * s.sm_count);
    *launched = packs_itself ? 1 : 2;
    if (!packs_itself)
        GMI_CUDA_TRY(launch_chained(s.pdl != 0, pack_fn(s.kind), dim3((s.n_src + kFxBlock - 1) / kFxBlock), dim3(kFxBlock),
                                    s.stream, a.xs, a.fs, s.n_src, a.K, static_cast<int4 *>(s.rec), a.skip));
    GMI_CUDA_TRY(launch_chained(s.pdl != 0 || !packs_itself, packs_itself ? pair_fn<true>(s.kind) : pair_fn<false>(s.kind),
                                dim3(groups, splits), dim3(kFxTpb), s.stream, a));
    if (s.splits_out) {
        *s.splits_out = splits;
    } else if (a.partial != nullptr) {
        // a kernel of its own: the last CTA of a target group adding the
        // group's partials took 2 us longer (320 segments: 18.5, 16.4 us)
        const int count = s.n_tgt * nout;
        GMI_CUDA_TRY(launch_chained(true, reduce_splits_tree, dim3((count + 63) / 64), dim3(64), s.stream, a.partial,
                                    splits, count, s.out, s.accumulate));
        ++*launched;
    }
    return GMI_OK;
}

}  // namespace gmi
