// FP64 quotients that overlap. The compiler's division is a call-like sequence with a branch: independent
// divisions of a thread run one after another, 113 cycles each on a B200 with one warp per scheduler
// (eight independent ones: 113 cycles each as well). Here a group of quotients is formed by straight-line
// FMAs, so their chains overlap, and one branch covers the group: where an operand's exponent is extreme
// (or an operand is zero, infinite or NaN where that matters) the caller takes the plain divisions.
//
// Method (P. W. Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor", IBM J.
// Res. Dev. 34, 1990): a reciprocal r of b within one ulp, refined by y + y (1 - b y) with the bracket
// exact in one FMA, is 1 / b rounded, unless b's mantissa is all ones; and with that r and q = a r, the remainder
// a - b q is exact in one FMA and q + (a - b q) r rounds to a / b. The first r here is the hardware's approximation
// y0 (rcp.approx.ftz.f64) with two terms of the series about it, y0 (1 + e + e^2), e = 1 - b y0, rounded up: for the
// mantissa of all ones that is the neighbour above 1 / b, from which the refinement rounds rightly too (from the one
// below it meets a tie). Without the refinement r is a last place off for one divisor in some 3500, and 2^k
// divided by that mantissa was wrong in its last place.
//
// So the results equal IEEE division for the operands that quot_ok accepts: positive divisors (the rounding up, and
// the sign of a zero dividend's quotient, are for those). tests/test_quot.py compares random operands with the
// device's division; tests/test_quot_directed.py, with the host's, operands next to the midpoints of two
// neighbours, divisors just below a power of two, and zeros.
//
// Measured per quotient (B200, groups of 8 per thread, cycles of a warp): 32 at 1 warp per scheduler, 52 at
// 2, 88 at 4, 168 at 8, against 113, 113, 122 and 185 for the compiler's. The reaction and turbulence
// closure 148 -> 128 us on the 41x181x361 shell, a whole dry iteration there 1604 -> 1510 us with quot1 in
// the stage kernel's heating and buoyancy terms. A group keeps its operands and reciprocals live, so a
// kernel at its register limit takes quot1: the stage kernel with its quotients in one group spilt 224
// bytes and took 263 us instead of 200.
#pragma once

namespace atjup {

__device__ __forceinline__ double rcp_of(double b) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    const double e = __fma_rn(-b, y, 1.0);
    y = __fma_ru(y, __fma_rn(e, e, e), y);
    return __fma_rn(y, __fma_rn(-b, y, 1.0), y);
}

// a / b given r = rcp_of(b)
__device__ __forceinline__ double quot(double a, double b, double r) {
    const double q = a * r;
    return __fma_rn(-__fma_rn(b, q, -a), r, q);
}

// operands whose quotient the method rounds correctly: b positive, its exponent and a's within 2^+-400, or a = 0
__device__ __forceinline__ bool quot_ok(double a, double b) {
    const unsigned ea = ((unsigned)__double2hiint(a) >> 20) & 0x7ffu;
    const unsigned eb = (unsigned)__double2hiint(b) >> 20;            // with the sign: negative ones are out of range
    return (ea - 623u <= 800u || a == 0.0) && eb - 623u <= 800u;
}

// a / b on its own: a chain of eight FMAs and the approximation
__device__ __forceinline__ double quot1(double a, double b) {
    return quot_ok(a, b) ? quot(a, b, rcp_of(b)) : a / b;
}

// o[q] = a[q] / b[q], the whole group at once
template <int N>
__device__ __forceinline__ void quots(const double (&a)[N], const double (&b)[N], double (&o)[N]) {
    bool ok = true;
#pragma unroll
    for (int q = 0; q < N; q++) ok = ok && quot_ok(a[q], b[q]);
    if (ok) {
#pragma unroll
        for (int q = 0; q < N; q++) o[q] = quot(a[q], b[q], rcp_of(b[q]));
    } else {
#pragma unroll
        for (int q = 0; q < N; q++) o[q] = a[q] / b[q];
    }
}
// o[q] = a[q] / b with r = rcp_of(b) (or the host's 1.0 / b, the same bits): a divisor used many times
template <int N>
__device__ __forceinline__ void quots_by(const double (&a)[N], double b, double r, double (&o)[N]) {
    bool ok = true;
#pragma unroll
    for (int q = 0; q < N; q++) ok = ok && quot_ok(a[q], b);
    if (ok) {
#pragma unroll
        for (int q = 0; q < N; q++) o[q] = quot(a[q], b, r);
    } else {
#pragma unroll
        for (int q = 0; q < N; q++) o[q] = a[q] / b;
    }
}
// o[q] = a[q] / b[q] with r[q] = rcp_of(b[q])
template <int N>
__device__ __forceinline__ void quots(const double (&a)[N], const double (&b)[N], const double (&r)[N], double (&o)[N]) {
    bool ok = true;
#pragma unroll
    for (int q = 0; q < N; q++) ok = ok && quot_ok(a[q], b[q]);
    if (ok) {
#pragma unroll
        for (int q = 0; q < N; q++) o[q] = quot(a[q], b[q], r[q]);
    } else {
#pragma unroll
        for (int q = 0; q < N; q++) o[q] = a[q] / b[q];
    }
}
__device__ __forceinline__ double quot1_by(double a, double b, double r) {
    return quot_ok(a, b) ? quot(a, b, r) : a / b;
}
// FP32 divisions overlap as they are
template <int N>
__device__ __forceinline__ void quots(const float (&a)[N], const float (&b)[N], float (&o)[N]) {
#pragma unroll
    for (int q = 0; q < N; q++) o[q] = a[q] / b[q];
}

}  // namespace atjup
