// vsl_short64.cuh -- short FP64 quotients for the plain form's kernels.
//
// The FP64 pipe bounds those kernels (two lanes per SM and clock on GB300), and a general
// division is about ten of its instructions.  A quotient whose divisor's reciprocal is known
// takes three: multiply, remainder, correction.  With the correctly rounded reciprocal it is the
// correctly rounded quotient (Markstein, IBM J. Res. Dev. 34, 1990; Brisebarre, Muller and Raina,
// IEEE Trans. Comput. 53, 2004).  A reciprocal takes three more and serves every quotient by the
// same divisor.  Neither handles overflow or underflow (nor an intermediate that underflows): the
// callers check their operands' range and keep the general code for the rest.
// (tests/test_quotient_exact_host.py runs this file on the CPU.)
#pragma once

#include <cmath>
#include <cuda_runtime.h>

#include "vsl_device.cuh"

namespace vsl {
namespace {

// a / d for the divisor d whose reciprocal is r
__device__ __forceinline__ double quotient(double a, double d, double r)
{
    const double q = __dmul_rn(a, r);
    const double z = __fma_rn(__fma_rn(-d, q, a), r, q);
    // the first product's sign: the correction would turn a quotient of -0 into +0
    return __hiloint2double((__double2hiint(z) & 0x7fffffff) | (__double2hiint(q) & (int)0x80000000),
                            __double2loint(z));
}

// 1 / d for a normal d whose reciprocal is normal, as the quotients above need it: with a
// reciprocal y off the exact one by (1/2 + e) ulp a quotient can round wrongly only if the
// divisor's significand (in 1 .. 2) is at least 2 - 4 e.  The hardware's FP32 reciprocal of the
// significand is within 2^-22.4 and one third-order Newton step cubes that, so e is 2^-15; divisors
// next to two (the upper 2^-12) take one more step, which rounds correctly (Markstein) but for the
// significand of ones alone, whose reciprocal is the odd one next to a power of two.  The seed is
// integer work and free beside the FP64 pipe (against a seed of 20 bits and no guard: steps of 128^3
// and up 0.5 .. 1.2 % faster, 64^3 reinitializations, which wait on the chain, 1.4 % slower).
__device__ __forceinline__ double reciprocal(double d)
{
    const int hi = __double2hiint(d), lo = __double2loint(d);
    const int s = __float_as_int(rcp_ftz(__int_as_float(0x3f800000 | ((hi << 3 | (int)((unsigned)lo >> 29)) & 0x7fffff))));
    double y = __hiloint2double(((s >> 3) + ((896 + 1023) << 20) - (hi & 0x7ff00000)) | (hi & (int)0x80000000), s << 29);
    const double e = __fma_rn(-d, y, 1.0);
    y = __fma_rn(y, __fma_rn(e, e, e), y);
    if (__builtin_expect((hi & 0xfff00) == 0xfff00, 0)) {
        y = __fma_rn(y, __fma_rn(-d, y, 1.0), y);
        if ((hi & 0xfffff) == 0xfffff && lo == -1) y = __hiloint2double(__double2hiint(y), __double2loint(y) | 1);
    }
    return y;
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
