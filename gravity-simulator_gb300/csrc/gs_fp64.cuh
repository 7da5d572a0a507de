// gs_fp64.cuh -- FP64 helpers that stay off the FP64 pipe where they can.
//
// On this GPU an FP64 instruction (comparisons included) holds its SM
// sub-partition's pipe for 64 cycles whatever its lanes do, so tests on FP64
// values are made on their bits, and quotients by divisors known in advance are
// four instructions instead of a division's nine.
#pragma once

#include <cuda_runtime.h>

namespace gs {

// |x| as an integer that orders like it (NaN last).
__device__ __forceinline__ long long abs_bits(double x)
{
    return __double_as_longlong(x) & 0x7fffffffffffffffll;
}

__device__ __forceinline__ bool finite_bits(double x)
{
    return abs_bits(x) < 0x7ff0000000000000ll;
}

__device__ __forceinline__ bool is_zero(double x) { return abs_bits(x) == 0; }

// Exponent of |x| between those of 2^-e and 2^e.
__device__ __forceinline__ bool exponent_within(double x, int e)
{
    const int ex = (__double2hiint(x) >> 20) & 0x7ff;
    return ex >= 1023 - e && ex < 1023 + e;
}

// RN(x / d) from the double-word reciprocal of d, zh = RN(1/d) and
// zl = RN(1/d - zh): q = RN(x zh + RN(x zl)) is within an ulp of x / d (Brisebarre,
// Muller and Raina, IEEE Trans. Computers 53(8), 2004), and the exact remainder
// x - q d corrects it (Markstein, IBM J. Res. Dev. 34(1), 1990).  ok: d and its
// reciprocal are far from the subnormal range; operands near it take the division.
__device__ __forceinline__ double div_known(double x, double d, double zh, double zl, bool ok)
{
    if (!ok || !exponent_within(x, 900)) return __ddiv_rn(x, d);
    const double q = __fma_rn(x, zh, __dmul_rn(x, zl));
    const double r = __fma_rn(-q, d, x);
    return __fma_rn(r, zh, q);
}

__device__ __forceinline__ void reciprocal2(double d, double &zh, double &zl)
{
    zh = __ddiv_rn(1.0, d);
    zl = __ddiv_rn(__fma_rn(-zh, d, 1.0), d);
}

}  // namespace gs
