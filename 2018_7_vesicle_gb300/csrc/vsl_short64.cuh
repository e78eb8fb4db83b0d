// vsl_short64.cuh -- short FP64 quotients for the plain form's kernels.
//
// The FP64 pipe bounds those kernels (two lanes per SM and clock on GB300), and a general
// division is about ten of its instructions.  A quotient whose divisor's reciprocal is known
// takes three: multiply, remainder, correction (Markstein, IBM J. Res. Dev. 34, 1990), and is
// the correctly rounded one.  A reciprocal takes three more, from the documented PTX
// approximation rcp.approx.ftz.f64 (20 bits) and one third-order Newton step (its error is that
// of the approximation cubed), and serves every quotient by the same divisor.  Neither handles
// overflow or underflow: the callers check their operands' range and keep the general code for
// the rest.  (tests/test_quotient_host.py replays both on the CPU.)
#pragma once

#include <cmath>
#include <cuda_runtime.h>

namespace vsl {
namespace {

// a / d for the divisor d whose reciprocal r is 1 / d to within an ulp
__device__ __forceinline__ double quotient(double a, double d, double r)
{
    const double q = __dmul_rn(a, r);
    const double z = __fma_rn(__fma_rn(-d, q, a), r, q);
    // the first product's sign: the correction would turn a quotient of -0 into +0
    return __hiloint2double((__double2hiint(z) & 0x7fffffff) | (__double2hiint(q) & (int)0x80000000),
                            __double2loint(z));
}

// 1 / d to within an ulp for a normal d whose reciprocal is normal
__device__ __forceinline__ double reciprocal(double d)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
    const double e = __fma_rn(-d, y, 1.0);  // at most about 2^-19
    return __fma_rn(y, __fma_rn(e, e, e), y);
}

// magnitude bits of the high word
__device__ __forceinline__ int mag_hi(double x) { return __double2hiint(x) & 0x7fffffff; }
// zero, or of magnitude 2^lo .. 2^hi
__device__ __forceinline__ bool within64(double x, int lo, int hi)
{
    const unsigned m = (unsigned)mag_hi(x);
    return m - (unsigned)((1023 + lo) << 20) < (unsigned)((hi - lo) << 20) || (m | (unsigned)__double2loint(x)) == 0u;
}

// a double whose quotients are the short ones; the compiler shares the reciprocals of equal
// divisors
struct Short64 {
    double v;
    __device__ __forceinline__ Short64() {}
    __device__ __forceinline__ Short64(double x) : v(x) {}
    __device__ __forceinline__ Short64(int x) : v((double)x) {}
    friend __device__ __forceinline__ Short64 operator+(Short64 a, Short64 b) { return __dadd_rn(a.v, b.v); }
    friend __device__ __forceinline__ Short64 operator-(Short64 a, Short64 b) { return __dadd_rn(a.v, -b.v); }
    friend __device__ __forceinline__ Short64 operator-(Short64 a) { return -a.v; }
    friend __device__ __forceinline__ Short64 operator*(Short64 a, Short64 b) { return __dmul_rn(a.v, b.v); }
    friend __device__ __forceinline__ Short64 operator/(Short64 a, Short64 b) { return quotient(a.v, b.v, reciprocal(b.v)); }
};
__device__ __forceinline__ double raw64(double x) { return x; }
__device__ __forceinline__ double raw64(Short64 x) { return x.v; }

// a divisor known on the host, with its correctly rounded reciprocal
struct Divisor64 {
    double d, r;
};
inline Divisor64 divisor64(double d) { return Divisor64{d, 1.0 / d}; }
__device__ __forceinline__ double operator/(double a, const Divisor64 &c) { return a / c.d; }
__device__ __forceinline__ Short64 operator/(Short64 a, const Divisor64 &c) { return quotient(a.v, c.d, c.r); }

// are the spacings within the range that the short quotients' callers assume
inline bool ordinary_spacing(double h) { return h > std::ldexp(1.0, -60) && h < std::ldexp(1.0, 60); }

}  // namespace
}  // namespace vsl
