// ucb_exact.cuh — the exact form's division by six (NVRTC header, before the step body).
//
// The codegen RK4 template ends every component with "h * (...) / 6". Written out in full,
// the three divisions of a step are about 300 of its 480 cycles at one warp a scheduler: a
// reciprocal seed, a chain of corrections and a branch to the rare cases each. Two FMAs after
// one product give the same bits when the divisor is a constant (Brisebarre, Muller & Raina,
// "Accelerating correctly rounded floating-point division when the divisor is known in
// advance", IEEE Trans. Computers 53, 2004): with r = RN(1/6), q = RN(x r) is within one ulp
// of x / 6, the remainder x - 6 q is exact, and q + r (x - 6 q) differs from x / 6 by less
// than 2^-50 ulp before it is rounded — while x / 6 is a multiple of ulp / 6 and odd
// multiples of half an ulp are not, so it lies at least ulp / 6 from any rounding boundary.
// (The remainder is taken with the other sign, so that -0 / 6 stays -0.)
// The remainder has to be a normal number: `range` gathers the largest distance of an
// argument from the smallest exponent allowed (zero counts as in range), and steps with a
// nonzero argument below 2^-959 (2^-63 in FP32), an infinity or a NaN among them are taken
// again with the division, and the trajectory's later steps too (Stepper and meet of
// ucb_device.cuh: what that costs) — one branch for a block of steps, where a branch a component
// cost as much as the division.
// B200, cycles of a Lorenz step at one warp a scheduler: 492 -> 214 (FP64), 437 -> 292 (FP32);
// FP64 maps, whole calls: Rossler 300^2 19.9 -> 14.8 ms, curve of 200 values 12.7 -> 5.4 ms,
// hyper-chaotic Rossler spectrum 200^2 18.3 -> 13.5 ms.
#pragma once

#ifdef UCB_NUMB_F32
constexpr unsigned int kSixthRange = 0x5F7FFFFFu;  // exponent field 64 .. 254
__device__ __forceinline__ float ucb_sixth(float x, unsigned int& range) {
    const unsigned int b = (unsigned int)__float_as_int(x) & 0x7FFFFFFFu;
    const unsigned int e = b ? b - 0x20000000u : 0u;
    range = e > range ? e : range;
    const float r = 1.0f / 6.0f;
    const float q = __fmul_rn(x, r);
    return __fmaf_rn(__fmaf_rn(6.0f, q, -x), -r, q);
}
#else
constexpr unsigned int kSixthRange = 0x7BEFFFFFu;  // exponent field 64 .. 2046
__device__ __forceinline__ double ucb_sixth(double x, unsigned int& range) {
    const unsigned int hi = (unsigned int)__double2hiint(x) & 0x7FFFFFFFu;
    const unsigned int e = (hi | (unsigned int)__double2loint(x)) ? hi - 0x04000000u : 0u;
    range = e > range ? e : range;
    const double r = 1.0 / 6.0;
    const double q = __dmul_rn(x, r);
    return __fma_rn(__fma_rn(6.0, q, -x), -r, q);
}
#endif
