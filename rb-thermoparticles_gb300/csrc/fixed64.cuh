// fixed64.cuh — FP64 sums and sums of products of one node carried by the integer units.
//
// GB300 executes an FP64 instruction of a warp in 64 cycles of a scheduler (measured: DFMA 64, DADD
// 76, int64 <-> double conversions 64) and a 32-bit integer instruction in 2, so a 64-bit integer
// addition costs a sixteenth of an FP64 one.  A set of doubles that is only added up is therefore
// written on a common grid as 64-bit integers, added exactly, and the result rounded once to
// FP64.  The grid is 2^5 finer than the last place of the set's largest member (FX_GUARD), so a
// member is rounded by at most 2^-57 of the largest one: less than the roundings of a chain of FP64
// additions, which each cost up to 2^-53 of the partial sum.  That is a bound on the sum, not on
// its members: one more than 2^5 below the largest keeps fewer than 53 bits.  A population that is
// collided on the grid of much larger coefficients (those of the force in a fluid at rest) is
// therefore less exact by itself than in FP64, though not against the largest of its node (mean over
// the 27 of f with u and rho of 1e-9, force 1e-5: 1e-14 of itself against 5e-16, 4.6e-17 of the largest
// against 4.3e-17; with u 0.03, rho 1e-3, force 1e-6: 1.1e-15 against 1.3e-15, 5.1e-17 against 7.3e-17).
// No rounding favours a side, because one that does adds up in a box of fixed mass, step after step.  On
// the grid a member is rounded to odd (von Neumann's rounding: cut off, and the last place set if
// anything but zeros was cut), which costs three instructions where rounding to nearest costs nine and
// errs by up to one unit to either side alike; the result is rounded to nearest with ties to even,
// which are frequent, since many members are only a few places below the largest.  Closed 16x12x8
// cavities at Ra 2e4 and 1e5, mass after 20,000 steps: 1.2e-15 and 4e-15 (9e-15 and -4e-15 with FP64
// formulas; -2.4e-12 and -3.1e-12 with members cut off, 3e-13 and -3e-13 with ties away from zero).  At
// 320x320x160 the step took 4.00 ms with members cut off, 4.45 with them rounded to odd, 4.76 to nearest.
// Conversions work on sign and magnitude, so the arithmetic is exactly odd: negated inputs give
// negated results, and zeros stay zeros.  Room: 53 + FX_GUARD bits of a member leave a factor of 31 for
// the sum.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

namespace rbtp {

constexpr int FX_GUARD = 5;
// The grid never gets finer than that of 2^-895, so that zeros and subnormals become 0 (their
// leading bit is implied only in normal numbers).  From 2^16 on (and for infinities and NaN) callers
// take the plain FP64 path: no flow has such values, and the sums that a huge one takes no part in
// would lose the digits that it shifts off the grid.
constexpr uint32_t FX_TOP_MIN = 128u << 20, FX_TOP_MAX = (1023u + 16u) << 20;

__host__ __device__ __forceinline__ uint32_t fx_hi(double d)
{
#ifdef __CUDA_ARCH__
    return (uint32_t)__double2hiint(d);
#else
    uint64_t u;
    memcpy(&u, &d, 8);
    return (uint32_t)(u >> 32);
#endif
}
__host__ __device__ __forceinline__ uint32_t fx_lo(double d)
{
#ifdef __CUDA_ARCH__
    return (uint32_t)__double2loint(d);
#else
    uint64_t u;
    memcpy(&u, &d, 8);
    return (uint32_t)u;
#endif
}
__host__ __device__ __forceinline__ double fx_double(uint32_t hi, uint32_t lo)
{
#ifdef __CUDA_ARCH__
    return __hiloint2double((int)hi, (int)lo);
#else
    const uint64_t u = ((uint64_t)hi << 32) | lo;
    double d;
    memcpy(&d, &u, 8);
    return d;
#endif
}
// shifts that give 0 from 64 places on (the device instruction clamps)
__host__ __device__ __forceinline__ uint64_t fx_shr(uint64_t v, uint32_t s)
{
#ifdef __CUDA_ARCH__
    uint64_t r;
    asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(s));
    return r;
#else
    return s > 63 ? 0 : v >> s;
#endif
}
__host__ __device__ __forceinline__ uint64_t fx_shl(uint64_t v, uint32_t s)
{
#ifdef __CUDA_ARCH__
    uint64_t r;
    asm("shl.b64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(s));
    return r;
#else
    return s > 63 ? 0 : v << s;
#endif
}

// Sign-free high word: its bits 20-30 are the biased exponent, and it orders doubles by magnitude.
__host__ __device__ __forceinline__ uint32_t fx_mag(double d) { return fx_hi(d) & 0x7fffffffu; }
// top becomes the largest of top and the fx_mag of d and e.  Read as floats, magnitudes order the same
// way, up to the floats' infinity; beyond that any value means "too large" (one instruction for two).
__host__ __device__ __forceinline__ void fx_cover(uint32_t &top, double d, double e)
{
#ifdef __CUDA_ARCH__
    float r;
    asm("max.NaN.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(__uint_as_float(top)), "f"(__uint_as_float(fx_hi(d))),
        "f"(__uint_as_float(fx_hi(e))));
    top = __float_as_uint(r);
#else
    const uint32_t a = fx_mag(d), c = fx_mag(e), m = a > c ? a : c;
    top = m > top ? m : top;
#endif
}
// Grid of a set from the largest fx_mag of its members (at least FX_TOP_MIN).
__host__ __device__ __forceinline__ uint32_t fx_grid(uint32_t top) { return top | 0xfffffu; }

// v with the sign of the word s (a predicated negation on the device)
__host__ __device__ __forceinline__ int64_t fx_signed(uint64_t v, uint32_t s)
{
#ifdef __CUDA_ARCH__
    int64_t r = (int64_t)v;
    asm("{\n\t.reg .pred p;\n\tsetp.lt.s32 p, %1, 0;\n\t@p neg.s64 %0, %0;\n\t}" : "+l"(r) : "r"(s));
    return r;
#else
    return (int32_t)s < 0 ? -(int64_t)v : (int64_t)v;
#endif
}
// 127 + the place of the leading bit of m (< 2^63), or 0 for m = 0: the exponent of m as a float,
// rounded towards zero
__host__ __device__ __forceinline__ uint32_t fx_leading(uint64_t m)
{
#ifdef __CUDA_ARCH__
    const float h = __uint2float_rz((uint32_t)(m >> 32)), l = __uint2float_rz((uint32_t)m);
    return __float_as_uint(__fmaf_rz(h, 4294967296.0f, l)) >> 23;
#else
    return m ? 127u + (63u - (uint32_t)__builtin_clzll(m)) : 0u;
#endif
}

// v with its last place set where x, what was cut off it, is not zero; a v of zero stays (its low word
// stands for v, which only misses the multiples of 2^32).  The minimum is written out because the
// compiler makes a comparison and a selection of it (320x320x160: 4.59 against 4.45 ms per step).
__host__ __device__ __forceinline__ uint64_t fx_odd(uint64_t v, uint32_t x)
{
    uint32_t s;
#ifdef __CUDA_ARCH__
    asm("{\n\tmin.u32 %0, %1, %2;\n\tmin.u32 %0, %0, 1;\n\t}" : "=r"(s) : "r"(x), "r"((uint32_t)v));
#else
    s = x != 0u && (uint32_t)v != 0u;
#endif
    return v | s;
}
// the bits of hi that a right shift of it by s places cuts off, at the top of a word (beyond 32 all of hi)
__host__ __device__ __forceinline__ uint32_t fx_cut(uint32_t hi, uint32_t s)
{
#ifdef __CUDA_ARCH__
    return __funnelshift_rc(0u, hi, s);
#else
    return s == 0u ? 0u : (s > 31u ? hi : hi << (32u - s));
#endif
}

// |d| / unit rounded to odd (d on the grid, see above), with d's sign; unit = 2^(E - 1075 - FX_GUARD),
// E = grid >> 20.  What was cut off is looked for in the low word of the significand.
__host__ __device__ __forceinline__ int64_t fx_from(double d, uint32_t grid)
{
    const uint32_t hi = fx_hi(d), lo = fx_lo(d);
    const uint32_t down = (grid - (hi & 0x7fffffffu)) >> 20;   // E - exponent of d: the low 20 bits never borrow
    const uint32_t mh = ((hi << FX_GUARD | lo >> (32 - FX_GUARD)) & ((1u << (20 + FX_GUARD)) - 1u)) |
                        (1u << (20 + FX_GUARD));
    const uint32_t ml = lo << FX_GUARD;
    return fx_signed(fx_odd(fx_shr((uint64_t)mh << 32 | ml, down), fx_cut(ml, down)), hi);
}

// v units of a grid (E = grid >> 20), times 2^up, rounded to the nearest double, ties to even.
__host__ __device__ __forceinline__ double fx_to(int64_t v, uint32_t grid, int up = 0)
{
    const uint32_t sign = (uint32_t)((uint64_t)v >> 32);
    const uint64_t m = (uint64_t)fx_signed((uint64_t)v, sign);
    const uint32_t e = fx_leading(m);
    // leading bit to bit 62, 10 places rounded off; bit 20 of the high word then adds one to the exponent
    // (two when the rounding carried over)
    const uint64_t n = fx_shl(m, 189u - e), q = (n + 0x1ffu + ((uint32_t)n >> 10 & 1u)) >> 10;
    const uint32_t base = (grid & 0xfff00000u) + ((uint32_t)(up - 180 - FX_GUARD) << 20);
    const uint32_t hi = (uint32_t)(q >> 32) + (e << 20) + base;
    return fx_double(e == 0u ? 0u : (hi | (sign & 0x80000000u)), (uint32_t)q);
}

// A factor |k| < 1 of products formed on a grid: its significand, leading bit at bit 63, and its
// high word for sign and exponent.
struct FxFactor {
    uint32_t mh, ml, hi;
};
__host__ __device__ __forceinline__ FxFactor fx_factor(double k)
{
    const uint32_t hi = fx_hi(k), lo = fx_lo(k);
    return {hi << 11 | lo >> 21 | 0x80000000u, lo << 11, hi};
}
__host__ __device__ __forceinline__ uint32_t fx_mulhi(uint32_t a, uint32_t b)
{
#ifdef __CUDA_ARCH__
    return __umulhi(a, b);
#else
    return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}
// Places between the product of the factor with a double of exponent 0 and the grid times 2^up, as
// an exponent field with its low 20 bits set.
__host__ __device__ __forceinline__ uint32_t fx_places(FxFactor k, uint32_t grid, int up)
{
    return grid - (k.hi & 0x7ff00000u) + ((uint32_t)(up + 1023 + FX_GUARD) << 20);
}
// |k d| / unit rounded to odd, with the product's sign: the upper 64 of the 128 bits of the significands'
// product (less at most 3 units of its last place), moved to the grid.  Some of the 106 bits are
// always taken to be cut off.  The grid must leave at least 2 places, so that the result stays below 2^62.
__host__ __device__ __forceinline__ int64_t fx_times(FxFactor k, double d, uint32_t places)
{
    const uint32_t hi = fx_hi(d), lo = fx_lo(d);
    const uint32_t mh = hi << 11 | lo >> 21 | 0x80000000u, ml = lo << 11;
    const uint64_t p = (uint64_t)mh * k.mh + fx_mulhi(mh, k.ml) + fx_mulhi(ml, k.mh);
    return fx_signed(fx_odd(fx_shr(p, (places - (hi & 0x7fffffffu)) >> 20), 1u), hi ^ k.hi);
}

}  // namespace rbtp
