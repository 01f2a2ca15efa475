/*
 * pt_convert.cuh -- FP64 <-> FP32 conversions on the integer pipe.
 *
 * GB300 runs 2 FP64 operations per cycle per SM, and the hardware
 * conversions between double and float go through that FP64 pipe.  The
 * mixed-precision evaluation converts six to twelve values per force
 * evaluation, so these bit-level versions (shifts, masks and adds on the
 * 64-lane integer pipe) keep the FP64 pipe for the arithmetic that must stay
 * FP64.  IEEE-754 binary64 and binary32 formats, round-to-nearest-even.
 *
 * Range: results below the smallest normal float flush to a signed zero and
 * above the largest float round to infinity; NaN stays NaN.  Mixed precision
 * converts momenta, in-cell offsets, position increments and forces, whose
 * magnitudes sit far inside that range.
 */
#ifndef PT_CONVERT_CUH
#define PT_CONVERT_CUH

#include <stdint.h>

/* double -> float outside the float normal range: zero, infinity, NaN. */
__device__ __noinline__ inline float pt_d2f_special(uint32_t hi, uint32_t lo)
{
    const uint32_t sign = hi & 0x80000000u, e = (hi >> 20) & 0x7ffu;
    if (e == 0x7ffu && ((hi & 0xfffffu) | lo)) return __uint_as_float(sign | 0x7fc00000u);
    return __uint_as_float(e < 897u ? sign : sign | 0x7f800000u);
}

/* double -> float, round to nearest even: in the float normal range the
 * exponent is rebiased by dropping its two top bits and flipping the next
 * (biased 897..1150 -> 1..254), and the 29 dropped bits decide the rounding
 * (whose carry may bump the exponent). */
__device__ __forceinline__ float pt_d2f(double x)
{
    const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
    if ((hi & 0x7fffffffu) - 0x38100000u >= 0x47f00000u - 0x38100000u) return pt_d2f_special(hi, lo);
    const uint32_t f = ((__funnelshift_l(lo, hi, 3) & 0x7fffffffu) ^ 0x40000000u) | (hi & 0x80000000u);
    return __uint_as_float(f + ((lo & 0x1fffffffu) + (f & 1u) > 0x10000000u ? 1u : 0u));
}

/* float -> double, exact (float subnormals flush to zero). */
__device__ __forceinline__ double pt_f2d(float f)
{
    const uint32_t b = __float_as_uint(f), a = b & 0x7fffffffu;
    uint32_t hi = (a >> 3) + 0x38000000u, lo = b << 29;
    if (a >= 0x7f800000u) hi += 0x38000000u;               /* inf, NaN */
    if (a < 0x00800000u) hi = lo = 0u;
    return __hiloint2double((int)(hi | (b & 0x80000000u)), (int)lo);
}

#endif /* PT_CONVERT_CUH */
