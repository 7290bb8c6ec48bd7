"""The quotients and inverse square roots of the decode kernels (csrc/decode_math.h), compiled for the host.  The hardware's
approximations are replaced by every value that their documented bound of two ulps allows (rsqrtf and __fdividef, CUDA's
programming guide)."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "autoresearch-go-ane_b200", "csrc")

MAIN = r"""
#include <math.h>
#include <stdio.h>
#include <string.h>
#include "decode_math.h"
using namespace ane;
static float next(float x, int ulps) { uint32_t u; memcpy(&u, &x, 4); u += ulps; memcpy(&x, &u, 4); return x; }
static uint64_t state = 1;
static double uniform() { state = state * 6364136223846793005ull + 1442695040888963407ull; return (double)(state >> 11) / 9007199254740992.0; }
int quotients() {
  for (int d = 1; d < 65536; ++d) {
    const unsigned magic = quotient_magic(d);
    if (d <= 512)
      for (int n = 0; n < 65536; ++n) { if (quotient(n, d, magic) != n / d) return printf("%d / %d\n", n, d); }
    else
      for (int n = 0; n < 65536 + d; n += d)  // where the quotient changes
        for (int m = n - 1; m <= n; ++m) if (m >= 0 && m < 65536 && quotient(m, d, magic) != m / d) return printf("%d / %d\n", m, d);
  }
  return 0;
}
// error in ulps of the result
static double off(float got, long double want) {
  int exp;
  frexpl(want, &exp);
  return (double)(fabsl(got - want) / ldexpl(1.0L, exp - 24));
}
int inverses() {  // sums of probabilities: 1 to the number of positions, mantissas of ones among them; outputs of either sign
  int other = 0;
  for (int i = 0; i < 400000; ++i) {
    const float x = i & 7 ? (float)exp2(uniform() * (i & 1 ? 12 : 1)) : next((float)exp2(1 + i / 8 % 12), -1 - i % 3);
    const float o = (float)((uniform() - 0.5) * exp2(uniform() * 40 - 20)), y = (float)(1.0 / (double)x);
    for (int e = -2; e <= 2; ++e) {
      const float got = divide(o, x, newton_inverse(x, next(y, e)));
      other += got != o / x;
      if (off(got, (long double)o / x) > 0.5 + 0x1p-18) return printf("%a / %a = %a, not %a\n", o, x, got, o / x);
    }
  }
  if (divide(-INFINITY, 3.f, 1 / 3.f) != -INFINITY || !isnan(divide(NAN, 3.f, 1 / 3.f))) return printf("inf or NaN\n");
  return other > 20 && printf("%d quotients differ from IEEE division\n", other);
}
int inverse_square_roots() {  // mean squares from eps to the largest
  for (int i = 0; i < 400000; ++i) {
    const float x = (float)(1e-5f + exp2(uniform() * (i & 1 ? 60 : 167) - 40));
    const long double want = 1.0L / sqrtl((long double)x);
    for (int e = -2; e <= 2; ++e) {
      const float got = newton_inverse_sqrt(x, next((float)want, e));
      if (off(got, want) > 1.01) return printf("1 / sqrt(%a) = %a\n", x, got);
    }
  }
  if (newton_inverse_sqrt(INFINITY, 0.f) != 0.f || !isnan(newton_inverse_sqrt(NAN, NAN))) return printf("inf or NaN\n");
  return 0;
}
int main(int, char** argv) { return argv[1][0] == 'q' ? quotients() : argv[1][0] == 'i' ? inverses() : inverse_square_roots(); }
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    folder = tmp_path_factory.mktemp("decode_math")
    (folder / "main.cpp").write_text(MAIN)
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", CSRC, "main.cpp", "-o", "main"], cwd=folder, check=True, timeout=120)
    return folder / "main"


@pytest.mark.parametrize("what", ["quotients", "inverses", "square roots"])
def test_every_approximation_within_two_ulps_is_made_exact(program, what):
    """Whole quotients exactly; o / x within half an ulp and 2^-18 of one, where IEEE division's 2e6 results differ in at most a few
    (2^-46 from the middle between two numbers: 2^-21 of them); 1 / sqrt(x) within 1.01 ulp (half of the
    rounding of x * approx, its own, and what is of second order), where 1.f / sqrtf(x) is off by up to 1.49."""
    r = subprocess.run([program, what], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
