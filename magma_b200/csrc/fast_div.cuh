// fast_div.cuh -- repeated IEEE division by one FP64 number (a diagonal entry of a triangular
// factor): the same quotients as the division, from a reciprocal formed once.
#pragma once

namespace mb200 {

// A diagonal entry prepared for div_fast: d, the rounded reciprocal and its error term.
struct Divisor {
    double d, hi, lo;
};
__device__ __forceinline__ Divisor make_divisor(double d) {
    const double r = 1.0 / d;
    return {d, r, __fma_rn(-d, r, 1.0) * r};
}
// Operands for which div_fast's products neither overflow nor lose bits: a zero or in
// 2^-700 .. 2^700, d in 2^-250 .. 2^250.
__device__ __forceinline__ bool div_fast_num(double a) {
    const unsigned h = (unsigned)__double2hiint(a) & 0x7fffffffu;
    return h - (323u << 20) < (1400u << 20) || (h | (unsigned)__double2loint(a)) == 0;
}
__device__ __forceinline__ bool div_fast_den(double d) {
    return ((unsigned)__double2hiint(d) & 0x7fffffffu) - (773u << 20) < (500u << 20);
}
// a / d, correctly rounded (Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", 1990: for q within one ulp of a / d, the exact residual r = a - d q
// and rd the rounded reciprocal, q + r rd rounds to the quotient). a (hi + lo) rounds to within
// one ulp. Four operations on the chain of a substitution step; a division is about 130 cycles.
// A zero a keeps its sign through a * hi.
__device__ __forceinline__ double div_fast(double a, const Divisor& v) {
    const double q = __fma_rn(a, v.hi, a * v.lo);
    const double x = __fma_rn(__fma_rn(-v.d, q, a), v.hi, q);
    return (((unsigned)__double2hiint(a) & 0x7fffffffu) | (unsigned)__double2loint(a)) == 0 ? a * v.hi : x;
}
// The division itself, for the operands div_fast does not take; kept out of the unrolled steps.
static __device__ __noinline__ double div_slow(double a, double d) { return a / d; }

}  // namespace mb200
