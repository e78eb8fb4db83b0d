"""The short FP64 quotients of csrc/vsl_stage64.cuh on the CPU: the reciprocal by one
third-order Newton step from an approximation of 20 bits, and Markstein's remainder
correction, against the correctly rounded quotient.  Divisors near powers of two and
numerators whose quotients lie next to midpoints included."""
import ctypes
import subprocess

import pytest

SRC = r"""
#include <math.h>
#include <stdint.h>
#include <string.h>
static uint64_t s = 88172645463325252ULL;
static uint64_t rnd(void) { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s * 2685821657736338717ULL; }
static double of(uint64_t m, int e) { return ldexp((double)((m >> 11) | (1ULL << 52)), e - 52); }
static double top20(double x) { uint64_t b; memcpy(&b, &x, 8); b &= ~0xffffffffULL; memcpy(&x, &b, 8); return x; }
static double quotient(double a, double d, double r) { double q = a * r; return fma(fma(-d, q, a), r, q); }
static double reciprocal(double d) {
    double y = top20(1.0 / top20(d)), e = fma(-d, y, 1.0);
    return fma(y, fma(e, e, e), y);
}
/* kind 0: reciprocal by Newton, 1: a correctly rounded reciprocal (the grid spacing's) */
long check(long n, int kind) {
    long bad = 0;
    for (long k = 0; k < n; ++k) {
        uint64_t m = rnd() >> 1;
        double d = of(k % 8 == 0 ? ((uint64_t)-1) >> (1 + rnd() % 3) & ~(rnd() >> 20) : m, (int)(rnd() % 40) - 20);
        double a = of(rnd() >> 1, (int)(rnd() % 40) - 20);
        if (k % 4 == 0) { /* a quotient within an ulp of a midpoint */
            double q = of(rnd() >> 1, 0);
            a = fma(q, d, 0.5 * ldexp(d, -52));
        }
        if (k % 16 == 1) a = 0.0;
        if (k % 3 == 0) a = -a;
        volatile double want = a / d;
        if (quotient(a, d, kind ? 1.0 / d : reciprocal(d)) != want) ++bad;
    }
    return bad;
}
"""


@pytest.mark.parametrize("kind", [0, 1])
def test_quotients_round_correctly(tmp_path, kind):
    (tmp_path / "q.c").write_text(SRC)
    so = tmp_path / "q.so"
    subprocess.run(["gcc", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-o", str(so), str(tmp_path / "q.c"), "-lm"],
                   check=True)
    lib = ctypes.CDLL(str(so))
    lib.check.restype, lib.check.argtypes = ctypes.c_long, [ctypes.c_long, ctypes.c_int]
    assert lib.check(4_000_000, kind) == 0


# The FP32 quotient of the adjoint's uniform stencils (csrc/vsl_adjoint.cu): a Newton step from a
# reciprocal that is off by up to an ulp, and the same remainder correction.
SRC32 = r"""
#include <math.h>
#include <stdint.h>
#include <string.h>
static uint32_t s = 2463534242u;
static uint32_t rnd(void) { s ^= s << 13; s ^= s >> 17; s ^= s << 5; return s; }
static float bits(uint32_t m, int e) { return ldexpf((float)((m & 0x7fffff) | 0x800000), e - 23); }
long check(long n) {
    long bad = 0;
    for (long k = 0; k < n; ++k) {
        float b = bits(k % 8 == 0 ? 0x7fffffu - rnd() % 4 : (k % 8 == 1 ? rnd() % 4 : rnd()), (int)(rnd() % 40) - 20);
        float a = bits(rnd(), (int)(rnd() % 40) - 20);
        if (k % 4 == 2) a = fmaf(bits(rnd(), 0), b, 0.5f * ldexpf(b, -23));
        if (k % 16 == 3) a = 0.f;
        if (k % 3 == 0) a = -a;
        float y0 = 1.f / b;
        y0 = k % 5 < 2 ? nextafterf(y0, 0.f) : (k % 5 < 4 ? nextafterf(y0, INFINITY) : y0);
        float y = fmaf(fmaf(-b, y0, 1.f), y0, y0), q = a * y;
        volatile float want = a / b;
        if (fmaf(fmaf(-b, q, a), y, q) != want) ++bad;
    }
    return bad;
}
"""


def test_fp32_quotients_round_correctly(tmp_path):
    (tmp_path / "q32.c").write_text(SRC32)
    so = tmp_path / "q32.so"
    subprocess.run(["gcc", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-o", str(so), str(tmp_path / "q32.c"),
                    "-lm"], check=True)
    lib = ctypes.CDLL(str(so))
    lib.check.restype, lib.check.argtypes = ctypes.c_long, [ctypes.c_long]
    assert lib.check(8_000_000) == 0
