"""CPU: the 64-bit fixed-point arithmetic of the DCT kernels (pypde_gb300/csrc/pgx_fixed.cuh).

The header compiles for the host with the device's integer operations; a small g++ harness compares
products, conversions and the cosine tables with 128-bit and long double arithmetic.  Bounds: a
product drops the low x low word product (|.| <= 2^31 2^31 / 2^62 = 1 unit), rounds its cross terms
to half a unit and shifts once more (half a unit): 2 units; a complex product has two of each: 3.
"""
import os
import shutil
import subprocess
import tempfile

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "pypde_gb300", "csrc")

HARNESS = r"""
#include <stdio.h>
#include <math.h>
#include <stdint.h>
#include "pgx_fixed.cuh"
typedef __int128 i128;
static uint64_t state = 0x9E3779B97F4A7C15ULL;
static uint64_t next64(void) {  /* splitmix64 */
  uint64_t z = (state += 0x9E3779B97F4A7C15ULL);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
  return z ^ (z >> 31);
}
static int64_t below(int bits) { return (int64_t)(next64() >> (64 - bits)) * ((next64() & 1) ? 1 : -1); }
static double off(i128 exact62, int64_t got) {  /* got - exact / 2^62, in units */
  const i128 d = ((i128)got << 62) - exact62;
  return (double)d / 4611686018427387904.0;
}
int main(void) {
  double mul = 0, cmul = 0, sum = 0;
  long n = 0, bad = 0;
  for (long i = 0; i < 400000; ++i) {
    const int64_t x = below(3 + (int)(next64() % 58)), y = below(60);
    int64_t w = below(62);
    if (i % 100 == 0) w = (int64_t)1 << 62;
    if (i % 100 == 1) w = -((int64_t)1 << 62);
    const double d = off((i128)x * w, fx_mul(x, fx_coef(w)));
    if (fabs(d) > mul) mul = fabs(d);
    sum += d;
    ++n;
    const int N = 2 * (1 + (int)(next64() % 1050)), k = (int)(next64() % (2 * N));
    int64_t c, s;
    fx_cos_sin(k, 2 * N, &c, &s);
    const fx2 v = {x, y}, r = fx_cmul(v, fx_twiddle(k, N));
    const double e = fmax(fabs(off((i128)x * c + (i128)y * s, r.x)), fabs(off((i128)y * c - (i128)x * s, r.y)));
    if (e > cmul) cmul = e;
    const long double a = 2 * 3.14159265358979323846264338327950288L * k / (2 * N);
    if (fabsl(c - cosl(a) * 0x1p62L) > 4 || fabsl(s - sinl(a) * 0x1p62L) > 4) ++bad;
  }
  printf("mul %g mean %g cmul %g tables %ld\n", mul, sum / n, cmul, bad);
  for (int N = 2; N < 2104; N += 2) {
    const fx_tw w = fx_inverse(N);
    const int64_t c = (int64_t)w.rh * 4294967296LL + w.rl;
    if (fabsl((long double)c - ldexpl(1.0L / N, 62 + w.ih)) > 0.51L || c > ((int64_t)1 << 62)) ++bad;
  }
  /* doubles in: rounded to nearest; and back: exact where the value has 53 bits, else to nearest */
  long in = 0, out = 0;
  for (long i = 0; i < 600000; ++i) {
    const double x = fx_double(next64());
    if (!(fabs(x) <= 1e290)) continue;  /* a unit is up to 2^60 larger than x: it stays finite */
    int e;
    frexp(x, &e);
    int q = e + (int)(next64() % 60);
    if (q < FX_KX_MIN - FX_KX0) q = FX_KX_MIN - FX_KX0;
    const int kx = FX_KX0 + q, neg = (int)(next64() & 1);
    const int64_t v = fx_from_double(x, kx, neg, 0);
    const long double exact = ldexpl(neg ? -(long double)x : (long double)x, FX_P0 - kx);
    if (fabsl((long double)v - exact) > 0.5L) ++in;
    const double back = fx_to_double(v, kx - FX_P0);
    const long double want = ldexpl((long double)v, kx - FX_P0);
    const double up = nextafter(back, INFINITY), dn = nextafter(back, -INFINITY);
    if (fabsl(back - want) > fabsl(up - want) || fabsl(back - want) > fabsl(dn - want)) ++out;
  }
  if (fx_to_double((int64_t)1 << 60, 970) != INFINITY || fx_to_double(-((int64_t)1 << 60), 963) != -ldexp(1.0, 1023) ||
      fx_to_double(3, -1074) != 3 * 4.9406564584124654e-324 || fx_to_double(1, -1090) != 0.0 || fx_to_double(0, 5) != 0.0)
    ++out;
  printf("in %ld out %ld inverse %ld\n", in, out, bad);
  return mul > 2 || cmul > 3 || fabs(sum / n) > 0.01 || bad || in || out;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_fixed_point_products_tables_and_conversions():
    with tempfile.TemporaryDirectory() as d:
        src, exe = os.path.join(d, "h.cpp"), os.path.join(d, "h")
        with open(src, "w") as f:
            f.write(HARNESS)
        subprocess.run(["g++", "-O2", "-I", CSRC, src, "-o", exe], check=True)
        r = subprocess.run([exe], capture_output=True, text=True)
        assert r.returncode == 0, r.stdout
