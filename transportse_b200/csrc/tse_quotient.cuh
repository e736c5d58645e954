// Quotients that share a divisor, correctly rounded.
//
// FP64 divisions bound the two flux kernels, 26 a cell in compute_q and 25 in
// flow_error by the formulas: an operator's branch for special operands keeps
// one from overlapping the next, and each does its own reciprocal.  Here a
// reciprocal is formed once a divisor (CUDA's rounded one), and a quotient by it
// takes two fused corrections (Markstein 1990, "Computation of elementary
// functions on the IBM RISC System/6000"): a y is within a few units of a / b,
// the first correction makes it one of the two neighbours of a / b, and from
// such a q and y = RN(1 / b), q + (a - b q) y is RN(a / b).  The results are the
// divided quotients' bits as long as no operand is near an end of the exponent
// range; callers divide where one is.
//
// us at 255 x 256 x 127 (B200), fluxes and flow error: 286 and 221; with a
// reciprocal refined by hand 308 and 211, with the operator's divisions 340 and
// 305.
#pragma once

namespace tse {

struct Divisor {
    double b, y;
};
__device__ __forceinline__ Divisor divisor(double b) { return {b, __drcp_rn(b)}; }
__device__ __forceinline__ double quotient(double a, const Divisor& d) {
    double q = a * d.y;
    q = __fma_rn(__fma_rn(-d.b, q, a), d.y, q);
    return __fma_rn(__fma_rn(-d.b, q, a), d.y, q);
}
// a may be zero: keeps its sign
__device__ __forceinline__ double quotient_0(double a, const Divisor& d) {
    return a == 0.0 ? a * d.y : quotient(a, d);
}
__device__ __forceinline__ Divisor half(const Divisor& s) { return {0.5 * s.b, 2.0 * s.y}; }
// positive, within 2^-80 .. 2^80: what the formulas derive from such inputs
// stays within 2^-900 .. 2^900
__device__ __forceinline__ bool plain_positive(double v) {
    return (unsigned)__double2hiint(v) - (943u << 20) <= (160u << 20);
}
// 0 or of magnitude 2^-300 .. 2^300
__device__ __forceinline__ bool plain_signed(double v) {
    return v == 0.0 || ((unsigned)__double2hiint(v) & 0x7fffffffu) - (723u << 20) <= (600u << 20);
}

}  // namespace tse
