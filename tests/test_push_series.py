"""The FP64 push's integer and series forms of 1 / sqrt(a) and e^{ie}, taken from the kernel's
source and compiled for the host: bit for bit against sqrt and division, and against long double
sines and cosines.

Bounds of e^{ie} as their comments derive them: below 1/16 the two series are exact to 2^-58 and
rounded to the 2^-53 spacing of doubles under 1 (2^-54), the sine's product rounds once more
(2^-53 of it); below 1/4 a Horner chain in doubles, its last two operations within an ulp of 1."""
import os
import re
import subprocess

import pytest

from conftest import PKG

HEAD = r"""
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>
#include <algorithm>
#define __device__
#define __forceinline__ inline
using std::fma; using std::sqrt;
struct C2 { double x, y; };
static inline double __longlong_as_double(long long b) { double d; memcpy(&d, &b, 8); return d; }
static inline long long __double_as_longlong(double d) { long long b; memcpy(&b, &d, 8); return b; }
static inline int __double2hiint(double d) { return (int)(__double_as_longlong(d) >> 32); }
static inline int __clz(int v) { return __builtin_clz((unsigned)v); }
static inline unsigned __umulhi(unsigned a, unsigned b) { return (unsigned)(((unsigned long long)a * b) >> 32); }
static inline unsigned long long __umul64hi(unsigned long long a, unsigned long long b) {
  return (unsigned long long)(((unsigned __int128)a * b) >> 64);
}
"""

MAIN = r"""
static long long bad = 0;
static void one(double a) {
  double ib, om;
  recip_sqrt_1m(a, ib, om);
  const double r = 1. / sqrt(a);
  if (ib != r || om != 1. - r || recip_sqrt_near1(a) != r) bad++;
}
int main() {
  const long long kOne = 0x3FF0000000000000LL, edge = 1LL << 31;
  std::mt19937_64 g(1);
  for (long long m = 1; m <= 1 << 18; m++) one(__longlong_as_double(kOne - m));
  for (long long m = edge - (1 << 18); m <= edge + (1 << 18); m++) one(__longlong_as_double(kOne - m));
  for (int i = 0; i < 3000000; i++) one(__longlong_as_double(kOne - 1 - (long long)(g() % (edge - 1))));
  for (int i = 0; i < 1000000; i++) one(__longlong_as_double(kOne - 1 - (long long)(g() >> (20 + g() % 30))));
  for (int i = 0; i < 300000; i++) one(__longlong_as_double(kOne + (long long)(g() >> (24 + g() % 30))));
  for (double a : {1., 0.5, 0.25, 2., 1e-300, 3.}) one(a);
  printf("%lld\n", bad);
  double c1 = 0, s1 = 0, c2 = 0, s2 = 0;
  for (int i = 0; i < 3000000; i++) {
    const double u = (double)(g() >> 11) * 0x1p-53;
    double e = std::ldexp(0.5 + 0.5 * u, -3 - (int)(g() % (i % 3 ? 4 : 70)));
    if (i % 1000 == 0) e = 0x1p-4 * (1 - 0x1p-53);
    if (g() & 1) e = -e;
    const C2 t = e < 0x1p-4 && e > -0x1p-4 ? expi_tiny(e) : C2{(double)cosl(e), (double)sinl(e)};
    c1 = std::max(c1, (double)fabsl((long double)t.x - cosl(e)));
    s1 = std::max(s1, (double)fabsl(((long double)t.y - sinl(e)) / sinl(e)));
    const double w = e * 2 * 0.999;
    const C2 v = expi_small(w);
    c2 = std::max(c2, (double)fabsl((long double)v.x - cosl(w)));
    s2 = std::max(s2, (double)fabsl(((long double)v.y - sinl(w)) / sinl(w)));
  }
  const C2 z = expi_tiny(0.);
  if (z.x != 1 || z.y != 0) c1 = 1;
  printf("%.17g %.17g %.17g %.17g\n", c1, s1, c2, s2);
}
"""


@pytest.fixture(scope="module")
def results(tmp_path_factory):
    text = open(os.path.join(PKG, "csrc", "kernels_plain.cu")).read()
    parts = []
    for name in ("below_pow2", "recip_sqrt_near1", "recip_sqrt_1m", "expi_small", "expi_tiny"):
        m = re.search(r"__device__ __forceinline__ \w+ %s\(.*?\n}\n" % name, text, re.S)
        assert m, name
        parts.append(m.group(0))
    d = tmp_path_factory.mktemp("series")
    src = str(d / "series.cpp")
    with open(src, "w") as f:
        f.write(HEAD + "".join(parts) + MAIN)
    exe = str(d / "series")
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-o", exe, src])
    return subprocess.check_output([exe], text=True).split()


def test_reciprocal_square_root_is_the_rounded_quotient_of_the_rounded_root(results):
    assert results[0] == "0"


def test_small_rotations_keep_their_bounds(results):
    c1, s1, c2, s2 = (float(v) for v in results[1:])
    assert c1 <= 2.0 ** -54 + 2.0 ** -57
    assert s1 <= 2.0 ** -53 + 2.0 ** -54 + 2.0 ** -57
    assert c2 <= 2.0 ** -53 and s2 <= 2.0 ** -52
