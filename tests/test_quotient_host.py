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
