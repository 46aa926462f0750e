// tb_fixed.cuh -- 64-bit fixed-point arithmetic of the FP64 form's recurrence.
//
// GB300 issues two FP64 multiply-adds per clock and SM, but 25 of the integer
// mad.wide.s32 (32 x 32 + 64 bits; measured with changing operands).  The
// entries of X and of T_k(X) are bounded by one when X is scaled by its own
// Gershgorin interval (every row of |X| then sums to at most one and
// |T_k(X) e_j| <= 1), so both are held as integers of 2^-60, split into two
// balanced limbs v = hi 2^30 + lo, lo in [-2^29, 2^29): a product takes three
// mad.wide (hi hi, hi lo, lo hi; lo lo is below a quarter of the last place),
// 8.5 products a clock where FP64 has 1.7 (measured).
//
// Head room of the 64-bit accumulators for one output entry: sum |x_hi t_hi|
// <= 2^60 (row of X times column of T); sum |x_hi t_lo| <= 2^30 2^29 (rows of
// |X| sum to one); sum |x_lo t_hi| <= 2^29 sqrt(d) 2^30 over d entries of a
// row, flushed every kFxFlush blocks (d = 128: 2^62.5).
#pragma once

#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "tb_internal.h"

namespace tb {

constexpr int kFxBits = 60, kFxLimb = 30;
constexpr int64_t kFxOne = 1ll << kFxBits;
constexpr double kFxScale = 1152921504606846976.0;  // 2^60
constexpr int kFxFlush = 32;                        // blocks between flushes of the middle sums

__device__ __forceinline__ int64_t fx_mad(int32_t a, int32_t b, int64_t c)
{
    int64_t r;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
    return r;
}

__device__ __forceinline__ void fx_split(int64_t v, int32_t &hi, int32_t &lo)
{
    const int64_t t = v + (1ll << (kFxLimb - 1));
    hi = (int32_t)(t >> kFxLimb);
    lo = (int32_t)((uint32_t)t & ((1u << kFxLimb) - 1u)) - (1 << (kFxLimb - 1));
}

__device__ __forceinline__ int64_t fx_join(int32_t hi, int32_t lo) { return fx_mad(hi, 1 << kFxLimb, lo); }

// (v + s - b)/a for a diagonal entry, v/a else, to the nearest 2^-60: the
// quotient's remainder (by a multiplication with 1/a: any quotient near it
// will do) and the rounding errors of the two sums are carried along.  A NaN
// or an entry beyond `most` (one, never passed within Gershgorin's bounds; 1.9
// on a refined interval) is left out and poisons the evaluation: its moments
// are then written as NaN, as FP64 arithmetic would give them, and the
// stochastic passes are made again in FP64.
__device__ __forceinline__ int64_t fx_scaled(double v, double s0, bool diag, DevState *st, double most = 1.0 + 1e-9)
{
    const double a = st->a, inv = 1.0 / a;
    double err = 0.0;
    if (diag) {
        const double b = st->b, s = v + s0, bs = s - v;
        err = (v - (s - bs)) + (s0 - bs);
        const double d = s - b, bd = d - s;
        err += (s - (d - bd)) - (b + bd);
        v = d;
    }
    const double q = v * inv, rem = fma(-q, a, v) + err;
    if (!(fabs(q) <= most)) {
        st->poison = 1;
        return 0;
    }
    const double s = q * kFxScale;  // exact
    const int64_t w = (int64_t)s;   // |s| >= 2^53 is whole already
    return w + (int64_t)rint((s - (double)w) + rem * inv * kFxScale);
}

// One entry's product sums: hh in units of 2^-60, mid in 2^-90.
struct FxAcc {
    int64_t hh, mid;
};

__device__ __forceinline__ void fx_mul_add(FxAcc &s, int32_t xh, int32_t xl, int32_t th, int32_t tl)
{
    s.hh = fx_mad(xh, th, s.hh);
    s.mid = fx_mad(xh, tl, s.mid);
    s.mid = fx_mad(xl, th, s.mid);
}

__device__ __forceinline__ void fx_flush(FxAcc &s)
{
    s.hh += s.mid >> kFxLimb;
    s.mid &= (1ll << kFxLimb) - 1;
}

// sum, and 2 sum, rounded to the last place
__device__ __forceinline__ int64_t fx_sum(const FxAcc &s) { return s.hh + ((s.mid + (1ll << (kFxLimb - 1))) >> kFxLimb); }
__device__ __forceinline__ int64_t fx_twice(const FxAcc &s)
{
    return 2 * s.hh + ((s.mid + (1ll << (kFxLimb - 2))) >> (kFxLimb - 1));
}

// <T_k, T_k> and <T_k, T_{k+1}> of a lane's entries: the lo lo part of the
// square has a sign, so it is kept (2^-120); that of the cross product has none.
struct FxDots {
    int64_t ehh = 0, emid = 0, elo = 0, ohh = 0, omid = 0;
    __device__ __forceinline__ void add(int32_t th, int32_t tl, int32_t nh, int32_t nl)
    {
        ehh = fx_mad(th, th, ehh);
        emid = fx_mad(th, tl, emid);
        elo = fx_mad(tl, tl, elo);
        ohh = fx_mad(th, nh, ohh);
        omid = fx_mad(th, nl, omid);
        omid = fx_mad(tl, nh, omid);
    }
    __device__ __forceinline__ int64_t even() const
    {
        return ehh + ((2 * emid + (elo >> kFxLimb) + (1ll << (kFxLimb - 1))) >> kFxLimb);
    }
    __device__ __forceinline__ int64_t odd() const { return ohh + ((omid + (1ll << (kFxLimb - 1))) >> kFxLimb); }
};

}  // namespace tb
