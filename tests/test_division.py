"""dv_div.h: division by a kept divisor gives the rounded quotient.

The header is plain C++ on the host, so it is compiled and compared here with
the machine's own division: equal bits for every x, the ones outside its range
(zeros, infinities, NaN, subnormals) among them."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <stdint.h>
#include <stdio.h>
#include <string.h>
#include "dv_div.h"
template <class R, class U> int run(const R* ds, int nd, int most_exp) {
  uint64_t s = 88172645463325252ull;
  long bad = 0;
  for (int i = 0; i < nd; ++i) {
    const R d = ds[i], y = dv::div_reciprocal(d);
    for (int k = 0; k < 400000; ++k) {
      s ^= s << 13; s ^= s >> 7; s ^= s << 17;
      U bits = (U)s;
      R x;
      memcpy(&x, &bits, sizeof(x));
      if (k % 3 == 0) x = (R)((double)(s >> 11) * 0x1p-53) * d;  // quotients near 1
      if (k % 3 == 1) x = d * (R)(1 + (int)(s & 1023));            // exact quotients
      if (k % 97 == 0) x = R(0);
      if (k % 97 == 1) x = -R(0);
      const R a = dv::div_by(x, d, y), b = x / d;
      if (memcmp(&a, &b, sizeof(a)) && !(a != a && b != b)) ++bad;
    }
  }
  return bad != 0;
}
int main() {
  const double dd[] = {1.0, 1.0000000000000002, 1.01, 1.0625, 1.09, 1.25, 1.36, 2.0, 101.0,
                       1.9999999999999998, 1e59, 1e61, 0.5};
  const float df[] = {1.0f, 1.0000001f, 1.01f, 1.0625f, 1.09f, 1.25f, 1.36f, 2.0f, 101.0f,
                      1.9999999f, 9e5f, 2e6f, 0.5f};
  const int a = run<double, uint64_t>(dd, 13, 0), b = run<float, uint32_t>(df, 13, 0);
  printf("%d %d\n", a, b);
  return a || b;
}
"""


@pytest.mark.parametrize("flags", [["-mfma"], []])
def test_div_by_equals_division(tmp_path, flags):
    src = tmp_path / "t.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "t"
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", *flags, "-I",
                           os.path.join(ROOT, "dvide_b200", "csrc"), str(src), "-o", str(exe)])
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
