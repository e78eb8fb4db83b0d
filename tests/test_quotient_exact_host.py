"""csrc/vsl_short64.cuh itself on the CPU (its text compiled by the host compiler, the intrinsics
replaced): the short FP64 quotients are the correctly rounded ones, the sign of a zero included,
for a hardware FP32 reciprocal anywhere within its documented ulp.  Divisors whose significand lies
next to two or to one against numerators next to powers of two, the numerators that put a quotient
next to the midpoint of two neighbours, and random ones.  Bit patterns are compared."""
import ctypes
import os
import re
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "2018_7_vesicle_gb300", "csrc")

SHIM = r"""
#include <cmath>
#include <cstdint>
#include <cstring>
#include <limits>
#define __device__
#define __forceinline__ inline
template <class A, class B> static A cast(B b) { A a; std::memcpy(&a, &b, sizeof a); return a; }
static int seed_ulp = 0;  // what the hardware reciprocal is off by
static float rcp_ftz(float x)
{
    const float y = 1.f / x;
    return seed_ulp == 0 ? y : std::nextafterf(y, seed_ulp < 0 ? 0.f : INFINITY);
}
static double __dmul_rn(double a, double b) { volatile double r = a * b; return r; }
static double __dadd_rn(double a, double b) { volatile double r = a + b; return r; }
static double __fma_rn(double a, double b, double c) { return std::fma(a, b, c); }
static int __double2hiint(double x) { return (int)(cast<uint64_t>(x) >> 32); }
static int __double2loint(double x) { return (int)(uint32_t)cast<uint64_t>(x); }
static double __hiloint2double(int h, int l) { return cast<double>((uint64_t)(uint32_t)h << 32 | (uint32_t)l); }
static float __int_as_float(int i) { return cast<float>(i); }
static int __float_as_int(float f) { return cast<int>(f); }
"""

CHECK = r"""
using namespace vsl;
static uint64_t s = 88172645463325252ULL;
static uint64_t rnd() { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s * 2685821657736338717ULL; }
static double sig(uint64_t m, int e) { return std::ldexp((double)((m & ((1ULL << 52) - 1)) | (1ULL << 52)), e - 52); }
static bool wrong(double a, double d)
{
    volatile double want = a / d;
    const double got = quotient(a, d, reciprocal(d)), known = quotient(a, d, 1.0 / d);
    const double typed = (Short64(a) / Short64(d)).v;
    return cast<uint64_t>(got) != cast<uint64_t>((double)want) || cast<uint64_t>(known) != cast<uint64_t>((double)want) ||
           cast<uint64_t>(typed) != cast<uint64_t>((double)want);
}
extern "C" long edges(int ulp)
{
    seed_ulp = ulp;
    long bad = 0;
    const uint64_t one = 1ULL << 52;
    for (long m = 0; m <= 4096; ++m)
        for (int side = 0; side < 3; ++side) {
            // next to two, next to one, and the divisors next to two whose reciprocals lie near midpoints
            const uint64_t w = side == 0 ? one - 1 - m : (side == 1 ? m : one - 1 - 2 * (rnd() >> 40));
            const double d = sig(w, (int)(m % 7) - 3), n = m % 2 ? -1.0 : 1.0;
            for (int t = 0; t <= 8; ++t) {
                bad += wrong(n * sig(t, 0), d) + wrong(n * sig(one - 1 - t, 5), d) + wrong(n * sig(t, 0), -d);
            }
            bad += wrong(0.0, d) + wrong(-0.0, d) + wrong(0.0, -d) + wrong(-0.0, -d);
            bad += wrong(0.1, d) + wrong(0.6, d) + wrong(0.3, d);
        }
    return bad;
}
// For an odd significand D there is one odd M modulo 2^k with D M = +-1, and the numerator
// A = (D M -+ 1) / 2^k is as near the midpoint M / 2 as any: all of them.
extern "C" long midpoints(long n, int ulp)
{
    seed_ulp = ulp;
    long bad = 0;
    for (long q = 0; q < n; ++q) {
        const uint64_t one = 1ULL << 52;
        const uint64_t D = (q % 2 ? (2 * one - 1 - 2 * (rnd() >> (12 + rnd() % 48))) : (rnd() >> 12 | one)) | 1;
        uint64_t inv = D;
        for (int it = 0; it < 6; ++it) inv *= 2 - D * inv;
        for (int k = 53; k <= 54; ++k)
            for (int sign = -1; sign <= 1; sign += 2) {
                uint64_t M = (sign > 0 ? inv : 0 - inv) & ((1ULL << k) - 1);
                for (int more = 0; more < 2; ++more, M += 1ULL << k) {
                    if (M < 2 * one || M >= 4 * one) continue;
                    const unsigned __int128 A = ((unsigned __int128)D * M - (unsigned __int128)(__int128)sign) >> k;
                    if (A < one || A >= 2 * one) continue;
                    bad += wrong((double)(uint64_t)A, (double)D);
                }
            }
    }
    return bad;
}
extern "C" long random_pairs(long n, int ulp)
{
    seed_ulp = ulp;
    long bad = 0;
    for (long k = 0; k < n; ++k) {
        const double d = sig(rnd(), (int)(rnd() % 40) - 20);
        double a = sig(rnd(), (int)(rnd() % 40) - 20);
        if (k % 4 == 0) a = std::fma(sig(rnd(), 0), d, 0.5 * std::ldexp(d, -52));
        bad += wrong(k % 3 ? a : -a, d);
    }
    return bad;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    with open(os.path.join(CSRC, "vsl_short64.cuh")) as f:
        text = re.sub(r"^#(include|pragma).*$", "", f.read(), flags=re.M)
    d = tmp_path_factory.mktemp("quotient")
    (d / "q.cpp").write_text(SHIM + text + CHECK)
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-o", str(d / "q.so"),
                    str(d / "q.cpp")], check=True)
    so = ctypes.CDLL(str(d / "q.so"))
    so.edges.restype, so.edges.argtypes = ctypes.c_long, [ctypes.c_int]
    for f in (so.midpoints, so.random_pairs):
        f.restype, f.argtypes = ctypes.c_long, [ctypes.c_long, ctypes.c_int]
    return so


@pytest.mark.parametrize("seed_ulp", [-1, 0, 1])
def test_short_quotients_are_correctly_rounded(lib, seed_ulp):
    assert lib.edges(seed_ulp) == 0
    assert lib.midpoints(400_000, seed_ulp) == 0
    assert lib.random_pairs(500_000, seed_ulp) == 0


# The FP32 quotient of the adjoint's uniform stencils (Short32 of csrc/vsl_adjoint.cu): the hardware
# reciprocal is either neighbour of the exact one, and the correctly rounded one for the significand
# of ones (tests/test_gpu_quotient32.py).
SHIM32 = r"""
static float __fmul_rn(float a, float b) { volatile float r = a * b; return r; }
static float __fmaf_rn(float a, float b, float c) { return std::fmaf(a, b, c); }
static float neighbour(float x)
{
    const double exact = 1.0 / (double)x;
    const float y = (float)exact;
    if ((~cast<uint32_t>(x) & 0x7fffff) == 0) return y;
    if (seed_ulp < 0) return (double)y > exact ? std::nextafterf(y, 0.f) : y;
    return (double)y < exact ? std::nextafterf(y, INFINITY) : y;
}
#define rcp_ftz neighbour
"""
CHECK32 = r"""
static uint32_t s32 = 2463534242u;
static uint32_t rnd32() { s32 ^= s32 << 13; s32 ^= s32 >> 17; s32 ^= s32 << 5; return s32; }
static float sig32(uint32_t m, int e) { return std::ldexp((float)((m & 0x7fffff) | 0x800000), e - 23); }
static bool wrong32(float a, float b)
{
    volatile float want = a / b;
    return (Short32(a) / Short32(b)).v != want;
}
/* every divisor's significand against powers of two and their neighbours, a weight of the scheme, a
   random numerator and those whose quotients lie nearest to the midpoint of two neighbours */
extern "C" long all_significands(int ulp)
{
    seed_ulp = ulp;
    long bad = 0;
    const uint32_t one = 1u << 23;
    for (uint32_t m = 0; m < one; ++m) {
        const float b = sig32(m, (int)(m % 41) - 20);
        bad += wrong32(1.f, b) + wrong32(-0x1.fffffep3f, b) + wrong32(0.6f, b) + wrong32(sig32(rnd32(), 0), b);
        const uint64_t D = m | one;
        if (D % 2 == 0) continue;
        uint64_t inv = D;
        for (int it = 0; it < 6; ++it) inv *= 2 - D * inv;
        for (int k = 24; k <= 25; ++k)
            for (int sign = -1; sign <= 1; sign += 2) {
                const uint64_t M = (sign > 0 ? inv : 0 - inv) & ((1ULL << k) - 1);
                const uint64_t A = (D * M - (uint64_t)(int64_t)sign) >> k;
                if (M >= 2 * one && M < 4 * one && A >= one && A < 2 * one) bad += wrong32((float)A, (float)D);
            }
    }
    return bad;
}
/* numerators down to 2^-100 over divisors of 1 .. 2 */
extern "C" long small_numerators(long n, int ulp)
{
    seed_ulp = ulp;
    long bad = 0;
    for (long q = 0; q < n; ++q) bad += wrong32(sig32(rnd32(), -(int)(rnd32() % 101)), sig32(rnd32(), 0));
    return bad;
}
"""


@pytest.fixture(scope="module")
def lib32(tmp_path_factory):
    with open(os.path.join(CSRC, "vsl_adjoint.cu")) as f:
        struct = re.search(r"^struct Short32 \{.*?^\};", f.read(), flags=re.M | re.S).group(0)
    d = tmp_path_factory.mktemp("quotient32")
    (d / "q.cpp").write_text(SHIM + SHIM32 + struct + CHECK32)
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-o", str(d / "q.so"),
                    str(d / "q.cpp")], check=True)
    so = ctypes.CDLL(str(d / "q.so"))
    so.all_significands.restype, so.all_significands.argtypes = ctypes.c_long, [ctypes.c_int]
    so.small_numerators.restype, so.small_numerators.argtypes = ctypes.c_long, [ctypes.c_long, ctypes.c_int]
    return so


@pytest.mark.parametrize("seed_ulp", [-1, 1])
def test_fp32_short_quotients_are_correctly_rounded(lib32, seed_ulp):
    assert lib32.all_significands(seed_ulp) == 0
    assert lib32.small_numerators(1_000_000, seed_ulp) == 0
