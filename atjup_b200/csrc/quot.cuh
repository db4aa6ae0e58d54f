// FP64 quotients that overlap. The compiler's division is a call-like sequence with a branch: independent
// divisions of a thread run one after another, 113 cycles each on a B200 with one warp per scheduler
// (eight independent ones: 113 cycles each as well). Here a group of quotients is formed by straight-line
// FMAs, so their chains overlap, and one branch covers the group: where an operand's exponent is extreme
// (or an operand is zero, infinite or NaN where that matters) the caller takes the plain divisions.
//
// Method: Newton's iteration for the reciprocal from the hardware's approximation (rcp.approx.ftz.f64),
// the first step cubic, then Markstein's quotient correction (P. W. Markstein, "Computation of elementary
// functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990): with r the correctly
// rounded reciprocal of b and q = a r, the remainder a - b q is exact in one FMA and q + (a - b q) r
// rounds to a / b. The results equal IEEE division for operands that quot_ok accepts (tests/test_quot.py
// compares them on the GPU).
//
// Measured per quotient (B200, groups of 8 per thread, cycles of a warp): 39 at 1 warp per scheduler, 55 at
// 2, 79 at 4, 150 at 8, against 113, 113, 122 and 185 for the compiler's. The reaction and turbulence
// closure 148 -> 128 us on the 41x181x361 shell, a whole dry iteration there 1604 -> 1510 us with quot1 in
// the stage kernel's heating and buoyancy terms. A group keeps its operands and reciprocals live, so a
// kernel at its register limit takes quot1: the stage kernel with its quotients in one group spilt 224
// bytes and took 263 us instead of 200.
#pragma once

namespace atjup {

__device__ __forceinline__ double rcp_of(double b) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    double e = __fma_rn(-b, y, 1.0);
    return __fma_rn(y, __fma_rn(e, e, e), y);
}

// a / b given r = rcp_of(b)
__device__ __forceinline__ double quot(double a, double b, double r) {
    const double q = a * r;
    return __fma_rn(__fma_rn(-b, q, a), r, q);
}

// operands whose quotient the method rounds correctly: b's and a's exponents within 2^+-400, or a = 0
__device__ __forceinline__ bool quot_ok(double a, double b) {
    const unsigned ea = ((unsigned)__double2hiint(a) >> 20) & 0x7ffu;
    const unsigned eb = ((unsigned)__double2hiint(b) >> 20) & 0x7ffu;
    return (ea - 623u <= 800u || a == 0.0) && eb - 623u <= 800u;
}

// a / b on its own: a chain of six FMAs and the approximation
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
