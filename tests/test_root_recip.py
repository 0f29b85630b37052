"""The FP64 reciprocal and square root the sweep kernel forms from the
hardware's approximations (recip, root, root_inverse in csrc/sweep_core.cuh):
one third-order Householder step from an approximation y0 and the correction
by the exact remainder.  The device sequence is round-to-nearest multiplies
and fused multiply-adds, so the same sequence in C with fma() on the host is
the same arithmetic; the approximation is stood in for by the exact value with
a relative error of up to 2^-20 and its low word cleared, coarser than the
hardware's.

After the step y is within 1.5 units in the last place (2^-60 from the series,
the rest from three roundings), so the remainder's correction is off by less
than 2^-50 of a unit before its rounding: no mismatch against the IEEE 1/x and
sqrt is expected among 5e6 operands, and none is allowed.  (A significand of
all ones is the one operand whose reciprocal lies that close to a midpoint:
recip sets the result's last bit there.)  1/sqrt, which has no
correction, stays within 2 units of the rounded quotient."""
import shutil
import subprocess

import pytest

SRC = r"""
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
static uint64_t s = 0x9E3779B97F4A7C15ull;
static uint64_t rnd(void) { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s; }
static uint64_t bits(double x) { uint64_t b; memcpy(&b, &x, 8); return b; }
static double from(uint64_t b) { double x; memcpy(&x, &b, 8); return x; }
static double coarse(double y) {
    const double e = ((double)(rnd() >> 11) / 4503599627370496.0 - 1.0) * 0x1p-20;
    return from(bits(y * (1.0 + e)) & 0xFFFFFFFF00000000ull);
}
static double near_recip(double x) {
    const double y = coarse(1.0 / x), e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}
static double recip(double x) {
    const double y = near_recip(x), r = fma(y, fma(-x, y, 1.0), y);
    const int ones = (bits(x) & 0xFFFFFFFFFFFFFull) == 0xFFFFFFFFFFFFFull;
    return from(bits(r) | (uint64_t)ones);
}
static double root_inverse(double x) {
    const double y = coarse(1.0 / sqrt(x)), e = fma(-(x * y), y, 1.0);
    return fma(y * e, fma(0.375, e, 0.5), y);
}
static double root(double x) {
    const double y = root_inverse(x), g = x * y;
    return fma(fma(-g, g, x), 0.5 * y, g);
}
static long long ulps(double a, double b) { return llabs((long long)(bits(a) - bits(b))); }
int main(int argc, char** argv) {
    long long n = atoll(argv[1]), bad = 0, far = 0;
    for (long long it = 0; it < n; ++it) {
        const uint64_t r = rnd();
        uint64_t m = rnd() & 0xFFFFFFFFFFFFFull;
        if ((it & 3) == 1) m |= 0xFFFFFFFFFFF00ull;
        if ((it & 3) == 2) m &= 0xFFFF0000000FFull;
        const double x = from(((uint64_t)(r % 1600 + 223) << 52) | m);
        if (recip(x) != 1.0 / x) ++bad;
        if (root(x) != sqrt(x)) ++bad;
        if (ulps(near_recip(x), 1.0 / x) > 2 || ulps(root_inverse(x), 1.0 / sqrt(x)) > 2) ++far;
    }
    printf("%lld %lld\n", bad, far);
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("gcc") is None, reason="gcc not found")
def test_recip_and_root_are_correctly_rounded(tmp_path):
    c = tmp_path / "rr.c"
    c.write_text(SRC)
    exe = tmp_path / "rr"
    subprocess.run(["gcc", "-O2", "-ffp-contract=off", "-o", str(exe), str(c), "-lm"], check=True)
    out = subprocess.run([str(exe), "5000000"], check=True, capture_output=True, text=True).stdout.split()
    assert out == ["0", "0"]
