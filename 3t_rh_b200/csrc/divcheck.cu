// Diagnostic (no reference counterpart): the shared-reciprocal divisions of
// divrn.cuh against the IEEE quotient, bit for bit, on operands generated on
// the device: random ones, divisors with all-ones significands, quotients
// next to a rounding midpoint, operands at and beyond the fast path's
// exponent range, and special values; and the reciprocals of a face's
// L-row divisors that roe_div (physics.cuh) forms by scaling 1/(12 c^2). The
// branch-free routines are checked on the same operands, zeros and subnormal
// sixths among them, and on others in the widest range in which each is used.
#include <cstdint>

#include <cuda_runtime.h>

#include "physics.cuh"

namespace rh3t {

__device__ __forceinline__ uint64_t mix64(uint64_t x) { // splitmix64 finaliser
    x += 0x9e3779b97f4a7c15ull;
    x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
    x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
    return x ^ (x >> 31);
}

// a double with random sign, random 52-bit fraction and exponent e (e in [-1023, 1023])
__device__ __forceinline__ double make_double(uint64_t h, int e) {
    const uint64_t frac = h & 0x000fffffffffffffull;
    const uint64_t sign = (h >> 63) << 63;
    return __longlong_as_double((long long)(sign | ((uint64_t)(e + 1023) << 52) | frac));
}

// a value whose quotient by b lies next to a rounding midpoint: RN(b mu),
// mu = q + ulp(q) / 2 for a random q with exponent e, moved by up to 3 ulps
__device__ __forceinline__ double near_midpoint(double b, uint64_t hq, int e, int shift) {
    const double q = make_double(hq & ~(1ull << 63), e);
    const double half_ulp = __longlong_as_double((long long)((__double_as_longlong(q) & 0x7ff0000000000000ll) -
                                                             (53ll << 52)));
    const double a = __fma_rn(b, q, b * half_ulp);
    return __longlong_as_double(__double_as_longlong(a) + shift);
}

__device__ __forceinline__ bool same_bits(double x, double y) {
    if (isnan(x) && isnan(y)) return true;
    return __double_as_longlong(x) == __double_as_longlong(y);
}

constexpr int DIV_CATEGORIES = 7;

// exponent of a normal number
__device__ __forceinline__ int exponent(double a) { return ((__double2hiint(a) >> 20) & 0x7ff) - 1023; }

// a and b within what div_near admits: b > 0 with an exponent in [-450, 450] and
// leading fraction bits that are not all ones, a zero or of exponent -969 or more with
// |a / b| in [2^-1000, 2^1000]
__device__ __forceinline__ bool div_near_admits(double a, double b) {
    if (!den_near(b)) return false;
    if (a == 0.0) return true;
    const int e = exponent(a) - exponent(b);
    return isfinite(a) && exponent(a) >= -969 && e >= -999 && e <= 999;
}

// the branch-free quotient of case (a, b), or `want` where it is not used for such
// operands (a / 3 and a / 6: any finite a, subnormals among them). Every routine's
// range tests have to imply what is checked here.
__device__ __forceinline__ double near_quotient(int cat, double a, double b, double want) {
    if (cat == 4 || cat == 5) {
        if (!isfinite(a)) return want;
        if (a != 0.0) {
            // the same operand scaled into the subnormal range and its edge, and a
            // quotient by 6 that is a tie there
            const unsigned w = (unsigned)__double2loint(a);
            const int sh = (int)(w % 120u) - 1070;
            const unsigned long long odd = 6ull * ((unsigned long long)__double_as_longlong(a) >> (14 + w % 49u)) + 3ull;
            const double t = scalbn(a, sh - ilogb(a)), u = (double)odd * 0x1p-1074; // (below 2^53 units: exact)
            if (cat == 4 && !same_bits(div3_near(t), __ddiv_rn(t, 3.0))) return div3_near(t);
            if (cat == 5 && !same_bits(div6_near(t), __ddiv_rn(t, 6.0))) return div6_near(t);
            if (cat == 5 && !same_bits(div6_near(u), __ddiv_rn(u, 6.0))) return div6_near(u);
            if (cat == 5 && !same_bits(div6_near(-u), __ddiv_rn(-u, 6.0))) return div6_near(-u);
        }
        return cat == 4 ? div3_near(a) : div6_near(a);
    }
    const bool groups = (den_near(b) && num_near(a)) || (den_mid_near(b) && num_small_near(a));
    if (!div_near_admits(a, b)) return groups ? NAN : want; // (a group's tests admit too much)
    const double q = div_near(a, recip_near(b));
    if (!same_bits(q, want)) return q;
    return a > 0.0 && den_near(b) && num_near(a) ? div_once(a, b) : q;
}

// category of case k: 0 random, 1 all-ones divisors, 2 near-midpoint
// quotients, 3 range edges and special values, 4 a / 3, 5 a / 6, 6 the
// reciprocals of 6 c^2 and 3 c^2 in roe_div (c^2 > 0 with exponents over and
// beyond the fast range, all-ones significands among them)
__global__ void k_div_check(long long n, unsigned long long seed, unsigned long long* bad, double* first) {
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += stride) {
        const int cat = (int)(k % DIV_CATEGORIES);
        const uint64_t h1 = mix64(seed ^ (uint64_t)k), h2 = mix64(h1), h3 = mix64(h2);
        double a, b, got;
        if (cat == 0) {
            a = make_double(h1, (int)(h3 % 941) - 470);
            b = make_double(h2, (int)((h3 >> 16) % 941) - 470);
            if ((h3 >> 40) % 3 == 0) { // small numerators, as velocities ahead of a front
                a = make_double(h1, (int)(h3 % 540) - 980);
                b = make_double(h2 & ~(1ull << 63), (int)((h3 >> 16) % 556) - 102);
            }
        } else if (cat == 1) {
            a = make_double(h1, (int)(h3 % 401) - 200);
            const uint64_t frac = 0x000fffffffffffffull - (h2 & 0xffull) - (((h3 >> 40) & 1) ? ((h2 >> 8) & 0xffffull) : 0);
            b = __longlong_as_double((long long)(((uint64_t)((int)((h3 >> 16) % 401) - 200 + 1023) << 52) | frac));
        } else if (cat == 2) {
            b = make_double(h1, (int)(h3 % 201) - 100);
            int e = (int)((h3 >> 16) % 201) - 100;
            if ((h3 >> 50) & 1) { // quotients down to 2^-1000, numerators to 2^-969
                b = make_double(h1 & ~(1ull << 63), (int)(h3 % 901) - 450);
                e = max(-1000, -969 - exponent(b)) + (int)((h3 >> 16) % 64);
            }
            const double scale = e < -900 ? 0x1p-200 : 1.0; // (half an ulp of 2^-1000 is no normal number)
            a = scale * near_midpoint(b, h2, e < -900 ? e + 200 : e, (int)((h3 >> 40) % 7) - 3);
        } else if (cat == 3) {
            const double specials[12] = {0.0, -0.0, INFINITY, -INFINITY, NAN, 4.9e-324, 2.2250738585072014e-308,
                                         1.7976931348623157e308, 0x1p-450, 0x1p450, 0x1.fffffffffffffp-451,
                                         0x1.fffffffffffffp450};
            a = (h3 & 3) == 0 ? specials[h1 % 12] : make_double(h1, (int)(h3 % 2047) - 1023);
            b = (h3 & 12) == 0 ? specials[h2 % 12] : make_double(h2, (int)((h3 >> 16) % 2047) - 1023);
            // next to the fast path's exponent range [-450, 450], on both sides
            if ((h3 >> 20) % 5 == 0) a = make_double(h1, ((h3 >> 44) & 1 ? 1 : -1) * ((int)((h3 >> 24) % 7) + 447));
            if ((h3 >> 28) % 5 == 0) b = make_double(h2, ((h3 >> 45) & 1 ? 1 : -1) * ((int)((h3 >> 32) % 7) + 447));
        } else if (cat == 6) {
            uint64_t hc = h1 & ~(1ull << 63);
            if ((h3 & 7) == 0) hc |= 0x000fffffffffffffull;
            const double cs2 = make_double(hc, (int)(h3 % 921) - 460);
            Roe q{};
            q.cs2 = cs2;
            q.den = 12.0 * cs2;
            q.b = 1.0;
            DevParams P{};
            P.gamma_e = 5.0 / 3.0;
            P.gamma_i = 5.0 / 3.0;
            P.gamma_r = 4.0 / 3.0;
            const RoeDiv rd = roe_div(q, P);
            const double w6 = __ddiv_rn(1.0, 6.0 * cs2), w3 = __ddiv_rn(1.0, 3.0 * cs2);
            a = cs2;
            b = 6.0 * cs2;
            if (!same_bits(rd.c6.y, w6) || !same_bits(rd.c3.y, w3) || rd.c6.b != 6.0 * cs2 || rd.c3.b != 3.0 * cs2) {
                atomicAdd(&bad[cat], 1ull);
                if (atomicAdd(&bad[DIV_CATEGORIES], 1ull) == 0) {
                    first[0] = a;
                    first[1] = b;
                    first[2] = same_bits(rd.c6.y, w6) ? rd.c3.y : rd.c6.y;
                }
            }
            continue;
        } else {
            b = cat == 4 ? 3.0 : 6.0;
            if ((h3 & 1) == 0) a = make_double(h1, (int)(h3 % 1001) - 500);
            else a = near_midpoint(b, h2, (int)((h3 >> 16) % 201) - 100, (int)((h3 >> 40) % 7) - 3);
            if ((h3 >> 50) % 64 == 0) a = (h3 >> 56) & 1 ? -0.0 : 0.0;
        }
        double want = __ddiv_rn(a, b);
        if (cat == 4) got = div3_rn(a);
        else if (cat == 5) got = div6_rn(a);
        else got = div_rn(a, recip(b));
        if (same_bits(got, want)) got = near_quotient(cat, a, b, want);
        if (cat == 0 && same_bits(got, want)) { // and a WENO5's alpha, over the range of its divisors
            const double c = h3 % 3 == 0 ? 0.1 : (h3 % 3 == 1 ? 0.6 : 0.3);
            const double s = make_double(h2 & ~(1ull << 63), (int)((h3 >> 30) % 1412) - 960);
            if (((unsigned)__double2hiint(s) & 0xfffffu) != 0xfffffu) {
                a = c;
                b = s;
                got = div_once(c, s);
                want = __ddiv_rn(c, s);
            }
        }
        if (!same_bits(got, want)) {
            atomicAdd(&bad[cat], 1ull);
            if (atomicAdd(&bad[DIV_CATEGORIES], 1ull) == 0) {
                first[0] = a;
                first[1] = b;
                first[2] = got;
            }
        }
    }
}

} // namespace rh3t

// counts[0..6]: mismatches per category (0 random, 1 all-ones divisors, 2
// near-midpoint quotients, 3 range edges and special values, 4 a / 3,
// 5 a / 6, 6 roe_div's reciprocals of 6 c^2 and 3 c^2); first[3]: a, b and
// the routine's quotient of one mismatch (category 6: c^2, 6 c^2 and the
// reciprocal)
extern "C" int rh3t_div_check(int32_t device, int64_t n, uint64_t seed, int64_t* counts, double* first) {
    if (!counts || !first || n < 0) return 7; // RH3T_ERR_INVALID_ARGUMENT
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev) return 10; // RH3T_ERR_NO_DEVICE
    if (cudaSetDevice(device) != cudaSuccess) return 8;
    unsigned long long* d_bad = nullptr;
    double* d_first = nullptr;
    if (cudaMalloc(&d_bad, (rh3t::DIV_CATEGORIES + 1) * sizeof(unsigned long long)) != cudaSuccess) return 8;
    if (cudaMalloc(&d_first, 3 * sizeof(double)) != cudaSuccess) {
        cudaFree(d_bad);
        return 8;
    }
    cudaError_t e = cudaMemset(d_bad, 0, (rh3t::DIV_CATEGORIES + 1) * sizeof(unsigned long long));
    if (e == cudaSuccess) e = cudaMemset(d_first, 0, 3 * sizeof(double));
    if (e == cudaSuccess && n > 0) {
        rh3t::k_div_check<<<148 * 16, 256>>>((long long)n, (unsigned long long)seed, d_bad, d_first);
        e = cudaGetLastError();
    }
    unsigned long long h[rh3t::DIV_CATEGORIES + 1] = {0};
    if (e == cudaSuccess) e = cudaMemcpy(h, d_bad, sizeof(h), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(first, d_first, 3 * sizeof(double), cudaMemcpyDeviceToHost);
    cudaFree(d_bad);
    cudaFree(d_first);
    if (e != cudaSuccess) return 8; // RH3T_ERR_CUDA
    for (int k = 0; k < rh3t::DIV_CATEGORIES; ++k) counts[k] = (int64_t)h[k];
    return 0;
}
