// Sums of doubles on the integer pipes.
//
// GB300 adds doubles at 2 lanes per cycle and SM and integers at 64. A stencil residual
// b + diag*x - sum(x_nb) is a sum: within a tile whose largest value has the exponent E, each
// double is shifted into a 64-bit integer (units of 2^(E-1081): 59 bits below the largest
// value), the sum is exact, and one conversion rounds it to double. Values within a factor
// 64 of the tile's largest convert without loss (53 + 6 bits), smaller ones to 2^-59 of it.
// A sum whose own largest operand lies within that factor therefore loses at most 6.5 units of 2^-52 of
// that operand (six neighbours or six times the centre cut off, b rounded), where the roundings
// of the double sum's partial sums reach 20. Random operands at the very limit: 3.1 units of 2^-53 rms, 2.9 in
// doubles (a half-sweep's sum without the centre 1.3 and 1.5; neighbours within 5% of each other, as of
// smooth fields, 0.8 and 4.8); at twice the limit 7.2. A sum whose operands are all smaller is formed in doubles. Tiles with
// values beyond FX_EMIN..FX_EMAX, which includes infinities and NaN, are summed in doubles as a whole.
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
// terms alike: rounded instead (fx_round), three cases in three seeds each were as far from 64 bits
// (256^3 Rayleigh-Taylor 1.3e-13, 1.6e-13 and 1.8e-13 both ways) and 1.2 to 1.6% slower.
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

// |f|'s upper word, less 1 in it for some negative f. The or of a sum's operands' is below FX_FOLD_MIN where
// all of them lie below 2^(E-1023-FX_RANGE).
__device__ __forceinline__ unsigned int fx_fold(long long f) {
    const int hi = (int)((unsigned long long)f >> 32);
    return (unsigned int)(hi ^ (hi >> 31));
}
constexpr unsigned int FX_FOLD_MIN = 1u << (59 - 1 - FX_RANGE - 32);

// +-m * 2^(E-1081) to the nearest double (half away from zero)
__device__ __forceinline__ double fx_pack(bool neg, unsigned long long m, int E) {
    const int lz = __clzll((long long)m);
    m <<= lz & 63;
    // 53 bits with the leading one, which adds 1 to the exponent field, as a carry of the
    // rounding may
    unsigned long long b = (m >> 11) + ((m >> 10) & 1ull);
    b += (unsigned long long)(unsigned int)(E + 4 - lz) << 52;
    if (lz == 64) b = 0;
    b |= (unsigned long long)neg << 63;
    return __longlong_as_double((long long)b);
}
__device__ __forceinline__ double fx_to_double(long long r, int E) {
    return fx_pack(r < 0, r < 0 ? 0ull - (unsigned long long)r : (unsigned long long)r, E);
}

// A sum of up to eight integers of 63 bits: `lo` modulo 2^64, `hi` the sum of their parts above 2^35
struct FxWide {
    unsigned long long lo;
    int hi;
    __device__ __forceinline__ void set(long long r) { lo = (unsigned long long)r; hi = fx_high(r); }
    __device__ __forceinline__ void add(long long r) { lo += (unsigned long long)r; hi += fx_high(r); }
    __device__ static __forceinline__ int fx_high(long long r) { return (int)((unsigned long long)r >> 32) >> 3; }
    // to the nearest double, as fx_to_double
    __device__ __forceinline__ double value(int E) const {
        // the parts below 2^35 that `hi` leaves out add up to less than 8 of its units
        long long c = (((long long)hi + 7) - (long long)(lo >> 35)) >> 29;   // the sum is c 2^64 + lo
        unsigned long long m = lo;
        const bool neg = c < 0;
        if (neg) {
            c = -c - (m != 0);
            m = 0ull - m;
        }
        if (c) {
            const int s = 64 - __clzll(c);
            m = (m >> s) | ((unsigned long long)c << (64 - s));
            E += s;
        }
        return fx_pack(neg, m, E);
    }
};

}  // namespace nyles
