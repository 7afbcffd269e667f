"""The branch-free reciprocal, division and roots of the exact Riemann solver
and the mixed kernels (``rcp_nr``, ``div_by``, ``rsqrt_nr``, ``sqrt_nr`` in
flash5_b200/csrc/exact_rs.cuh), restated in C with truncated 20-bit seeds
and compared with long double results (64-bit significands) over the
operands' whole range.

Bound: the last step adds a correction from an exact residual, so a result
is one rounding (0.5 ulp) of a value that is off by the cube of the seed's
2^-20, 2^-60 relative and 2^-7 ulp at most: below 0.51 with the 2^-11 ulp
of the reference.
"""
import os
import subprocess

import pytest

SRC = r"""
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>
static uint64_t s = 0x243F6A8885A308D3ull;
static uint64_t nx(void) { s += 0x9E3779B97F4A7C15ull; uint64_t z = s;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull; z = (z ^ (z >> 27)) * 0x94D049BB133111EBull; return z ^ (z >> 31); }
static double rnd(int lo, int hi) { uint64_t m = nx() & 0xFFFFFFFFFFFFFull; int e = lo + (int)(nx() % (uint64_t)(hi - lo));
  if (nx() % 8 == 0) m = nx() & 1 ? 0xFFFFFFFFFFFFFull - (nx() & 15) : nx() & 15;
  uint64_t b = ((uint64_t)(e + 1023) << 52) | m; double d; memcpy(&d, &b, 8); return d; }
/* a seed keeps 20 bits of the result for the operand's leading 32 bits */
static double cut(double b) { uint64_t u; memcpy(&u, &b, 8); u &= 0xFFFFFFFF00000000ull; memcpy(&b, &u, 8); return b; }
static double rcp_nr(double b) { const double y = cut(1. / cut(b)), e = fma(-b, y, 1.); return fma(y, fma(e, e, e), y); }
static double div_by(double x, double b, double y) { const double q = x * y; return fma(fma(-q, b, x), y, q); }
static double rsqrt_nr(double a) { const double y = cut(1. / sqrt(cut(a))), e = fma(-a, y * y, 1.);
  return fma(y * e, fma(e, .375, .5), y); }
static double sqrt_nr(double a) { const double y = rsqrt_nr(a), q = a * y; return fma(.5 * y, fma(-q, q, a), q); }
static double worst[4]; static long off[4];
static void take(int k, double got, long double want) {
  int e; frexpl(want, &e);
  const double u = (double)fabsl(((long double)got - want) / ldexpl(1.L, e - 53));
  if (!(u <= worst[k])) worst[k] = u;
  off[k] += got != (double)want;
}
int main(void) {
  const long N = 4000000;
  for (long i = 0; i < N; ++i) {
    const double b = i % 3 ? rnd(-40, 40) : rnd(-500, 500), x = i % 3 ? rnd(-60, 60) : rnd(-400, 400);
    take(0, rcp_nr(b), 1.L / b);
    take(1, div_by(x, b, rcp_nr(b)), (long double)x / b);
    take(2, rsqrt_nr(b), 1.L / sqrtl(b));
    take(3, sqrt_nr(b), sqrtl(b));
  }
  for (int k = 0; k < 4; ++k) printf("%d: worst %.4f ulp, not correctly rounded %.2e\n", k, worst[k], off[k] / (double)N);
  for (int k = 0; k < 4; ++k) if (!(worst[k] <= 0.51)) return 1;
  return 0;
}
"""


def test_results_are_one_rounding_off(tmp_path):
    c = tmp_path / "nr.c"
    exe = tmp_path / "nr"
    c.write_text(SRC)
    try:
        subprocess.run(["gcc", "-O2", "-ffp-contract=off", "-o", str(exe), str(c), "-lm"], check=True,
                       capture_output=True, text=True)
    except (OSError, subprocess.CalledProcessError) as e:
        pytest.skip(f"no C compiler: {e}")
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout


RANGES = r"""
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>
static int hi(double x) { uint64_t u; memcpy(&u, &x, 8); return (int)(uint32_t)(u >> 32); }
static int in_range(double x) { return (unsigned)hi(x) - 0x2D300000u < 0x25800000u; }
static int at_least(double x, int lo) { return hi(x) > lo && hi(x) < 0x52B00000; }
int main(void) {
  const double v[] = {0., -0., 5e-324, -5e-324, 1e-310, -1e-310, 1e-100, -1e-100, 0x1p-301, 0x1p-300, 1e-16, -1e-16, 1.,
                      -1., 0x1.fp299, 0x1p300, -0x1p300, 1e308, INFINITY, -INFINITY, NAN, -NAN};
  const int lo = hi(0x1p-300);
  for (unsigned k = 0; k < sizeof v / sizeof *v; ++k) {
    const int in = v[k] >= 0x1p-300 && v[k] < 0x1p300;
    if (in_range(v[k]) != in) { printf("in_range %g\n", v[k]); return 1; }
    /* at_least needs the high word above lo's: a double or so above it */
    if (at_least(v[k], lo) != (in && v[k] >= 0x1.00001p-300)) { printf("at_least %g\n", v[k]); return 1; }
    if (at_least(v[k], hi(1e-16)) != (in && v[k] > 1.01e-16)) { printf("at_least tiny %g\n", v[k]); return 1; }
  }
  return 0;
}
"""


def test_range_tests(tmp_path):
    """The tests on high words that choose between the branch-free forms and
    the general ones (``in_range``, and ``at_least`` of the mixed HLLC), with
    negative numbers, zeros of both signs, subnormals, infinities and NaN."""
    c = tmp_path / "ranges.c"
    exe = tmp_path / "ranges"
    c.write_text(RANGES)
    try:
        subprocess.run(["gcc", "-O2", "-fwrapv", "-o", str(exe), str(c), "-lm"], check=True, capture_output=True, text=True)
    except (OSError, subprocess.CalledProcessError) as e:
        pytest.skip(f"no C compiler: {e}")
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
