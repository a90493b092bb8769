// Sums of doubles on the integer pipes.
//
// GB300 adds doubles at 2 lanes per cycle and SM and integers at 64. A stencil residual
// b + diag*x - sum(x_nb) is a sum: within a tile whose values share one exponent E, each
// double is shifted into a 64-bit integer (units of 2^(E-1081): 59 bits below the largest
// value), the sum is exact, and one conversion rounds it to double. Values within a factor
// 64 of the tile's largest convert without loss (53 + 6 bits), smaller ones to 2^-59 of it,
// where the double sum rounds every partial sum to 2^-53 of itself. A tile in which some
// thread's own values are all more than 64 times smaller than the largest, or not finite,
// is summed in doubles instead,
// as one whose sums could leave the range of the doubles.
#pragma once
#include "nyles_common.cuh"

namespace nyles {

constexpr int FX_RANGE = 6;          // exponents below the tile's largest that stay exact
constexpr int FX_EMIN = 128;         // biased exponents below this: sum in doubles
constexpr int FX_EMAX = 0x7f6;       // and above this: a sum of eight residuals reaches 2^7 times the largest value

// |x|'s upper word: ordered as |x|, its exponent in bits 20..30
__device__ __forceinline__ unsigned int fx_mag(double x) { return (unsigned int)__double2hiint(x) & 0x7fffffffu; }

// x in units of 2^(E-1081) (truncated below), |x| < 2^(E-1022): at most 59 bits. What the
// truncation takes from the x of a residual it takes from the centre's and the neighbours'
// terms alike.
__device__ __forceinline__ long long fx_from(double x, int E) {
    const unsigned int hi = (unsigned int)__double2hiint(x), lo = (unsigned int)__double2loint(x);
    const unsigned int e = (hi >> 20) & 0x7ffu;
    const unsigned int mh = __funnelshift_l(lo, hi, 11) | 0x80000000u;
    unsigned long long m = ((unsigned long long)mh << 32) | (lo << 11);
    asm("shr.b64 %0, %0, %1;" : "+l"(m) : "r"((unsigned int)E + 5u - e));   // amounts above 63 give 0 (x = 0)
    return (int)hi < 0 ? -(long long)m : (long long)m;
}

// x in the same units, to the nearest: for the right-hand side, whose truncation would leave
// the residual a mean, which the coarse levels amplify (the constant of a 256^3 pressure was
// 2e-12 off with it and is 6e-14 off without, 1.3e-13 with double sums)
__device__ __forceinline__ long long fx_round(double x, int E) {
    const unsigned int hi = (unsigned int)__double2hiint(x), lo = (unsigned int)__double2loint(x);
    const unsigned int e = (hi >> 20) & 0x7ffu;
    const unsigned int mh = __funnelshift_l(lo, hi, 11) | 0x80000000u;
    unsigned long long m = ((unsigned long long)mh << 32) | (lo << 11);
    asm("shr.b64 %0, %0, %1;" : "+l"(m) : "r"((unsigned int)E + 4u - e));
    m = (m >> 1) + (m & 1ull);
    return (int)hi < 0 ? -(long long)m : (long long)m;
}

// f * d for a small d >= 0, modulo 2^64
__device__ __forceinline__ long long fx_mul(long long f, unsigned int d) {
    const unsigned long long lo = (unsigned long long)(unsigned int)f * d;
    return (long long)(lo + ((unsigned long long)((unsigned int)((unsigned long long)f >> 32) * d) << 32));
}

// r * 2^(E-1081) to the nearest double (half away from zero)
__device__ __forceinline__ double fx_to_double(long long r, int E) {
    unsigned long long m = r < 0 ? 0ull - (unsigned long long)r : (unsigned long long)r;
    const int lz = __clzll((long long)m);
    m <<= lz & 63;
    // 53 bits with the leading one, which adds 1 to the exponent field, as a carry of the
    // rounding may
    unsigned long long b = (m >> 11) + ((m >> 10) & 1ull);
    b += (unsigned long long)(unsigned int)(E + 4 - lz) << 52;
    if (lz == 64) b = 0;
    b |= (unsigned long long)r & 0x8000000000000000ull;
    return __longlong_as_double((long long)b);
}

}  // namespace nyles
