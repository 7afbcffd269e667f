"""The divisions of the FP64 kernels (flash5_b200/csrc/hy_core.cuh): the
branch-free one of the direction kernels (``Arith<true>``, Newton's
iteration from a 20-bit seed, restated here with a truncated seed) and the
division used by the FP64 species pass (``div_rn`` in
flash5_b200/csrc/hy_core.cuh): x / b from rb = RN(1 / b) with one FMA
correction (Markstein's theorem).  Restated here in C and compared bit for
bit with IEEE division on random operands (constants 3 and 6 of the PPM
formulas, runtime grid spacings, significands of all ones) and on the
special values that take the plain division.  The FP64 GPU parity tests
check the device function itself against the oracle's divisions."""
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
  uint64_t b = ((uint64_t)(e + 1023) << 52) | m; if (nx() & 1) b |= 1ull << 63; double d; memcpy(&d, &b, 8); return d; }
static double div_rn(double x, double b, double rb) {
  const double q0 = x * rb;
  const double a = fabs(q0), ax = fabs(x);
  if (a > 0x1p-960 && a < 0x1p1000 && ax > 0x1p-960 && ax < 0x1p1000) return fma(fma(-q0, b, x), rb, q0);
  return x / b;
}
static long bad = 0;
static void check(double x, double b) {
  double q = div_rn(x, b, 1. / b), r = x / b;
  if (memcmp(&q, &r, 8) && !(isnan(q) && isnan(r))) { if (bad < 5) printf("x=%a b=%a q=%a r=%a\n", x, b, q, r); ++bad; }
}
/* Arith<true>: the seed keeps 20 bits of the reciprocal of b's leading 32 */
static double seed(double b) { uint64_t u; memcpy(&u, &b, 8); u &= 0xFFFFFFFF00000000ull; memcpy(&b, &u, 8);
  double y = 1. / b; memcpy(&u, &y, 8); u &= 0xFFFFFFFF00000000ull; memcpy(&y, &u, 8); return y; }
/* the stated range: b and x (or x = 0) in [2^-500, 2^500), b's significand not all ones */
static int refused(double x, double b) {
  uint64_t u; memcpy(&u, &b, 8); u &= 0xFFFFFFFFFFFFFull;
  return !(fabs(b) >= 0x1p-500 && fabs(b) < 0x1p500) || u == 0xFFFFFFFFFFFFFull ||
         !(x == 0. || (fabs(x) >= 0x1p-500 && fabs(x) < 0x1p500));
}
/* the kernels' test of it (Arith<true>::check and rcp), on the words */
static int bad_bits(double x, double b) {
  uint64_t ub, ux; memcpy(&ub, &b, 8); memcpy(&ux, &x, 8);
  const uint32_t hi = (uint32_t)(ub >> 32), v = (uint32_t)(ux >> 32) & 0x7fffffffu;
  const int r = (hi & 0x7fffffffu) - 0x20B00000u >= 0x3E800000u || ((hi | 0xfff00000u) & (uint32_t)ub) == 0xffffffffu;
  return r || (v - 0x20B00000u >= 0x3E800000u && (v | (uint32_t)ux) != 0u);
}
static double div_bf(double x, double b) {
  double y = seed(b);
  const double e = fma(-b, y, 1.);
  y = fma(y, fma(e, e, e), y);
  const double r = fma(y, fma(-b, y, 1.), y), q0 = x * r;
  return fma(-fma(q0, b, -x), r, q0);
}
static void checkf(double x, double b) {
  double q = div_bf(x, b), r = x / b;
  if (refused(x, b) != bad_bits(x, b)) { if (bad < 5) printf("range test: x=%a b=%a\n", x, b); ++bad; }
  if (!bad_bits(x, b) && memcmp(&q, &r, 8)) { if (bad < 5) printf("x=%a b=%a q=%a r=%a\n", x, b, q, r); ++bad; }
}
int main(void) {
  const double cs[] = {3., 6.};
  for (int c = 0; c < 2; ++c)
    for (long i = 0; i < 4000000; ++i) check(i % 7 ? rnd(-60, 60) : rnd(-1021, 1023), cs[c]);
  for (long i = 0; i < 8000000; ++i) {
    double b = rnd(-40, 40);
    if (i % 5 == 0) { uint64_t bb; memcpy(&bb, &b, 8); bb |= 0xFFFFFFFFFFFF0ull; memcpy(&b, &bb, 8); }
    check(rnd(-60, 60), b);
  }
  const double sp[] = {0., -0., 1e-310, -1e-310, 5e-324, 1e308, -1e308, INFINITY, -INFINITY, NAN};
  for (int i = 0; i < 10; ++i) { check(sp[i], 3.); check(sp[i], 6.); check(sp[i], 1e-3); check(sp[i], 7.5e9); }
  long b0 = bad;
  for (long i = 0; i < 12000000; ++i) {
    const double x = i % 3 ? rnd(-60, 60) : rnd(-499, 499);
    double b = fabs(i % 5 ? rnd(-40, 40) : rnd(-499, 499));
    if (i % 7 == 0) { uint64_t bb; memcpy(&bb, &b, 8); bb |= 0xFFFFFFFFFFFF0ull; memcpy(&b, &bb, 8); }
    checkf(x, b);
  }
  for (long i = 0; i < 3000000; ++i) { checkf(rnd(-60, 60), 3.); checkf(rnd(-60, 60), 6.); checkf(rnd(-60, 60), 12.); }
  const double z[] = {0., -0.};
  for (int i = 0; i < 2; ++i) { checkf(z[i], 3.); checkf(z[i], 0.7); }
  const double out[] = {5e-324, -1e-315, 0x1p-1043, 1e-310, 1e200, INFINITY, NAN, -1e-160, 0x1.fp-501, 0x1p500};
  for (int i = 0; i < 10; ++i) if (!refused(out[i], 1.5) || !bad_bits(out[i], 1.5)) { printf("not refused %g\n", out[i]); ++bad; }
  for (long i = 0; i < 1000000; ++i) {           /* subnormal numerators */
    uint64_t u = (nx() & 0xFFFFFFFFFFFFFull) >> (nx() % 52); double x; memcpy(&x, &u, 8);
    checkf(nx() & 1 ? x : -x, i % 4 ? fabs(rnd(-40, 40)) : (i % 3 ? 6. : 12.));
  }
  { uint64_t ones = 0x3FFFFFFFFFFFFFFFull; double b; memcpy(&b, &ones, 8); if (!bad_bits(1., b)) ++bad; }
  if (!bad_bits(1., 0.) || !bad_bits(1., 1e300) || !bad_bits(1., 0x1p500) || !bad_bits(1., 0x1.fp-501)) ++bad;
  printf("branch-free: mismatches %ld\n", bad - b0);
  printf("mismatches %ld\n", bad);
  return bad != 0;
}
"""


def test_div_rn_equals_division(tmp_path):
    c = tmp_path / "div_rn.c"
    exe = tmp_path / "div_rn"
    c.write_text(SRC)
    try:
        subprocess.run(["gcc", "-O2", "-ffp-contract=off", "-o", str(exe), str(c), "-lm"], check=True,
                       capture_output=True, text=True)
    except (OSError, subprocess.CalledProcessError) as e:
        pytest.skip(f"no C compiler: {e}")
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
