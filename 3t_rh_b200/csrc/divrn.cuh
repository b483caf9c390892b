// Correctly rounded FP64 division a / b by a reciprocal shared between
// several divisions with the same divisor, for the no-contraction build:
// every quotient equals the IEEE quotient bit for bit, at 5 (or, for the
// constants 3 and 6, 3) FP64 operations once the reciprocal is known.
//
// Method: Markstein's correction step (P. Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", IBM J. Res.
// Dev. 34(1), 1990; also Cornea, Harrison, Tang, "Scientific Computing on
// Itanium-based Systems", 2002). Let y = RN(1/b) and q a faithful
// approximation of z = a/b (one of the two doubles around z). Then
// r = a - b q is a double (computed exactly by one FMA) and
// RN(q + r y) = RN(z). Proof, b = B 2^(eb-52) with B in [2^52, 2^53), z in
// [2^E, 2^(E+1)): every midpoint mu between doubles near z is
// M 2^(E-53), M odd, so a - b mu = N 2^(eb+E-105) with N a nonzero integer
// (a quotient of two doubles is never a midpoint); r = R 2^(eb+E-104) with
// |R| < B; b y - 1 = K 2^-105 with |K| <= B/2 (y is within half an ulp of
// 1/b). Then b (q + r y - mu) = (a - b mu) + r (b y - 1)
//                             = 2^(eb+E-105) (N + R K 2^-104),
// and |R K 2^-104| < B^2 2^-105 < 1 <= |N|: q + r y lies on the same side of
// every midpoint as z (and is none), so both round to the same double.
//
// A faithful q: q0 = RN(a y) is within 1.5 ulp of z (|a y - z| < z 2^-53);
// q1 = RN(q0 + RN(a - b q0) y) is within (1/2 + 2^-51) ulp, hence faithful;
// q2 = RN(q1 + (a - b q1) y) = RN(z). For b = 3 or 6, RN(1/b) = (1 - 2^-54)/b
// exactly, so a y lies within half an ulp below z and RN(a y) is already
// faithful: one correction suffices.
//
// The argument needs no overflow, underflow or special value anywhere: the
// fast sequence is taken only when both exponents are within [-450, 450]
// (then z lies in [2^-901, 2^901], y in [2^-451, 2^450] and a nonzero r
// above 2^-557: all normal numbers); a zero numerator over such a divisor
// is the signed zero a y; anything else (subnormal, huge, infinite, NaN, a
// divisor out of range) takes the IEEE division. tests/test_gpu_math.py compares
// every routine here with the IEEE quotient bit for bit on random,
// near-midpoint and special operands (rh3t_div_check).
#pragma once

namespace rh3t {

__device__ __forceinline__ bool div_in_range(double x) {
    const unsigned e = (unsigned)__double2hiint(x) & 0x7ff00000u;
    return e - 0x23d00000u <= 0x38400000u; // biased exponent in [1023 - 450, 1023 + 450]
}

// the IEEE quotient, out of line: the rare operands outside the fast range
// take it, and one copy of its code serves every call site (the callers'
// code stays small enough for the instruction cache)
static __device__ __noinline__ double div_ieee(double a, double b) { return __ddiv_rn(a, b); }

// operands outside the fast range (b_ok: b is in it, y = RN(1/b)): a zero
// numerator over such a divisor, common where a flow is uniform, gives the
// signed zero a y (y is finite, nonzero and of b's sign, so the sign is a's
// XOR b's, as in IEEE division); anything else takes the IEEE quotient. The
// zero test is inline: zero numerators are too frequent for a call (batch
// of half-cylinder instances: with zeros through the IEEE division the flux
// kernels ran 9% and the RHS 26% slower, with the test out of line 2% and 6%)
__device__ __forceinline__ double div_edge(double a, double b, double y, bool b_ok) {
    return (b_ok && a == 0.0) ? __dmul_rn(a, y) : div_ieee(a, b);
}

struct Recip {
    double b, y;
    bool ok;
};

__device__ __forceinline__ Recip recip(double b) {
    Recip d;
    d.b = b;
    d.y = __ddiv_rn(1.0, b);
    d.ok = div_in_range(b);
    return d;
}

// a / d.b, correctly rounded
__device__ __forceinline__ double div_rn(double a, const Recip& d) {
    if (!(d.ok && div_in_range(a))) return div_edge(a, d.b, d.y, d.ok);
    double q = __dmul_rn(a, d.y);
    double r = __fma_rn(-d.b, q, a);
    q = __fma_rn(r, d.y, q);
    r = __fma_rn(-d.b, q, a);
    return __fma_rn(r, d.y, q);
}

// a / 3.0 and a / 6.0, correctly rounded
__device__ __forceinline__ double div3_rn(double a) {
    const double y = 0x1.5555555555555p-2; // RN(1/3)
    if (!div_in_range(a)) return div_edge(a, 3.0, y, true);
    const double q = __dmul_rn(a, y);
    const double r = __fma_rn(-3.0, q, a);
    return __fma_rn(r, y, q);
}
__device__ __forceinline__ double div6_rn(double a) {
    const double y = 0x1.5555555555555p-3; // RN(1/6)
    if (!div_in_range(a)) return div_edge(a, 6.0, y, true);
    const double q = __dmul_rn(a, y);
    const double r = __fma_rn(-6.0, q, a);
    return __fma_rn(r, y, q);
}

// ---------------------------------------------------------------- branch-free form
// The same quotients without a branch each: the caller tests the operands of
// a whole group of divisions once (den_near for the divisors, num_near or a
// bound of its own for the numerators) and takes the routines above, or IEEE
// divisions, for the group that fails. A branch per quotient made each
// division a basic block of its own, a chain of five dependent FP64 operations
// with nothing to overlap it; in this form the scheduler interleaves the
// chains of a group.
//
// recip_near(b): the PTX approximation rcp.approx.ftz.f64 (it reads the upper
// 32 bits of b; |1 - b y| <= 2^-19.9, measured over all 2^20 leading fractions
// and both extremes of the lower word) and two Newton steps y <- y + y (1 - b y),
// each by two FMAs: the error before the last rounding is 2^-79, so y lies
// within (1/2 + 2^-26) ulp of 1/b. The argument above then holds with
// |K| <= (1 + 2^-25) B / 2, and with |R| <= (1/2 + 2^-51) B (q1 is that close
// to z): |R K 2^-104| < B^2 2^-106 (1 + 2^-24) < 1 for every B below
// 2^53 (1 - 2^-20). den_near refuses the divisors above that (leading 20
// fraction bits all ones).
//
// With yl = (1 - b y) y, the reciprocal y + yl holds 1/b to 2^-100, and
// q = RN(a y + a yl) is within (1/2 + 2^-50) ulp of z: faithful in two operations,
// so the one correction that follows rounds correctly (the argument above
// with this q for q1): four operations a quotient instead of five. The
// quotient's sign is the numerator's (b > 0), set explicitly because a zero
// numerator would lose it; den_near refuses b <= 0.
struct RecipN {
    double b, y, yl;
};
__device__ __forceinline__ RecipN recip_near(double b) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    double e = __fma_rn(-b, y, 1.0);
    y = __fma_rn(y, e, y);
    e = __fma_rn(-b, y, 1.0);
    y = __fma_rn(y, e, y);
    e = __fma_rn(-b, y, 1.0);
    return {b, y, __dmul_rn(e, y)};
}

// b > 0, exponent in [-450, 450], leading 20 fraction bits not all ones
__device__ __forceinline__ bool den_near(double b) {
    const unsigned h = (unsigned)__double2hiint(b);
    return h - 0x23d00000u <= 0x384fffffu && (h & 0xfffffu) != 0xfffffu;
}

// div_near(a, recip_near(b)) rounds correctly beyond the operands that den_near and
// num_near admit: for b as den_near wants it and a zero, or with an exponent of -969 or
// more and a quotient within 2^-1000..2^1000. The residual a - b q is a multiple of
// 2^(e - 105), e the exponent of a, so it is exact; q is normal; and what a yl loses as a
// subnormal (2^-1075) is at most 2^-23 ulp of the quotient: the first quotient
// is within (1/2 + 2^-22) ulp, and the argument holds with its margin
// ((1 + 2^-22) (1 + 2^-25) (1 - 2^-19) < 1). The tests of a group bound numerators and
// divisors so that this holds for each of its quotients.

// a is zero, or its exponent is in [-450, 450]
__device__ __forceinline__ bool num_near(double a) {
    const unsigned h = (unsigned)__double2hiint(a) & 0x7fffffffu;
    return h - 0x23d00000u <= 0x384fffffu || (h | (unsigned)__double2loint(a)) == 0u;
}

// Divisors b > 0 with an exponent in [-100, 100] (leading 20 fraction bits not all
// ones) admit numerators down to 2^-880: the quotient is at least 2^-981.
__device__ __forceinline__ bool den_mid_near(double b) {
    const unsigned h = (unsigned)__double2hiint(b);
    return h - 0x39b00000u <= 0x0c8fffffu && (h & 0xfffffu) != 0xfffffu;
}
__device__ __forceinline__ bool num_small_near(double a) {
    const unsigned h = (unsigned)__double2hiint(a) & 0x7fffffffu;
    return h - 0x08f00000u <= 0x532fffffu || (h | (unsigned)__double2loint(a)) == 0u;
}

// b > 0, exponent in [-100, 450], leading 20 fraction bits not all ones: the numerators'
// lower bound is the caller's
__device__ __forceinline__ bool den_wide_near(double b) {
    const unsigned h = (unsigned)__double2hiint(b);
    return h - 0x39b00000u <= 0x226fffffu && (h & 0xfffffu) != 0xfffffu;
}

// a / d.b, correctly rounded
__device__ __forceinline__ double div_near(double a, const RecipN& d) {
    const double q = __fma_rn(a, d.y, __dmul_rn(a, d.yl));
    const double r = __fma_rn(-d.b, q, a);
    const double z = __fma_rn(r, d.y, q);
    return __hiloint2double((__double2hiint(z) & 0x7fffffff) | (__double2hiint(a) & 0x80000000), __double2loint(z));
}

// c / b, correctly rounded, for one quotient by b (c > 0): the reciprocal's
// low part would serve this quotient alone, so the correction runs twice
// instead
__device__ __forceinline__ double div_once(double c, double b) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    double e = __fma_rn(-b, y, 1.0);
    y = __fma_rn(y, e, y);
    e = __fma_rn(-b, y, 1.0);
    y = __fma_rn(y, e, y);
    double q = __dmul_rn(c, y);
    double r = __fma_rn(-b, q, c);
    q = __fma_rn(r, y, q);
    r = __fma_rn(-b, q, c);
    return __fma_rn(r, y, q);
}

// a / 3 for every finite a (the residual taken as 3 q - a and the correction
// as -y, so that a zero numerator keeps its sign): the residual is a small
// multiple of ulp(q), or of 2^-1074, so it is exact down to the subnormals, where a / 3 is
// never a tie. a / 6 likewise, except that a subnormal quotient can be a tie,
// a = (6 k + 3) 2^-1074: q is k there (a y lies just below the tie) and the residual
// three units, which y, less than 1 / 6, would leave at k. For an odd k the next
// double above y, more than 1 / 6, takes it to the even k + 1; the residuals of other
// quotients there are four units at most, and either y rounds them alike.
__device__ __forceinline__ double div3_near(double a) {
    const double y = 0x1.5555555555555p-2;
    const double q = __dmul_rn(a, y);
    return __fma_rn(__fma_rn(3.0, q, -a), -y, q);
}
__device__ __forceinline__ double div6_near(double a) {
    const double q = __dmul_rn(a, 0x1.5555555555555p-3);
    const int odd = (__double2hiint(q) & 0x7ff00000) == 0 ? __double2loint(q) & 1 : 0; // of a subnormal q
    const double y = __hiloint2double(0x3fc55555, 0x55555555 + odd);
    return __fma_rn(__fma_rn(6.0, q, -a), -y, q);
}
__device__ __forceinline__ bool finite_near(double a) { return ((unsigned)__double2hiint(a) & 0x7fffffffu) < 0x7ff00000u; }

} // namespace rh3t
