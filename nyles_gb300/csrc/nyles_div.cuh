// Quotient of doubles by functional iteration (M. J. Flynn, "On Division by Functional Iteration", IEEE
// Transactions on Computers C-19, 1970): with y near 1/x and e = 1 - x y,
//     a / x = a y / (1 - e) = a y (1 + e + e^2 + ...),
// here up to e^2, in Horner's form on a y. The first term left out is e^3: below 2^-59 of the quotient for
// |e| <= 2^-20 + 2^-22, which the hardware's approximate reciprocal keeps (measured over mantissas and
// exponents by tests/test_gpu_div.py, with the quotients beside CUDA's own division: within 2 units in the
// last place). Two roundings count, of a y and of the last step: 2^-52 relative.
// For 2^-1022 <= x < 2^1022, where y is a normal number, and |a y| within the doubles.
// 4 FP64 instructions where a 256^3 right-hand side by lines takes 12.77 ms, 13.30 with __drcp_rn and a
// multiplication, 13.79 with the division.
#pragma once

namespace nyles {

__device__ __forceinline__ double div_seed(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    return y;
}
__device__ __forceinline__ double div_series(double a, double x) {
    const double y = div_seed(x), e = fma(-x, y, 1.0), q = a * y;
    return fma(e, fma(e, q, q), q);
}

}  // namespace nyles
