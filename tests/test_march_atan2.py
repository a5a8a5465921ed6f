"""The march's arctangent (march_atan2, csrc/gi_math.h) has the bits of atan2f_ for all
arguments: every pair of special values (zeros of both signs, subnormals, infinities,
NaNs, one NaN beside a number among them), and random ones over the exponent range."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent

PROGRAM = r"""
#include "gi_math.h"
#include <cstdio>
#include <random>
int bad = 0;
void check(float y, float x) {
  const float a = gi::atan2f_(y, x), b = gi::march_atan2(y, x);
  if (a != a && b != b) return;
  if (gi::f2u(a) != gi::f2u(b) && bad++ < 20) printf("(%g, %g): atan2f_ %g march_atan2 %g\n", y, x, a, b);
}
int main() {
  const float v[] = {0.0f, 1e-45f, 1e-40f, 1.17549435e-38f, 1e-20f, 0.26794919f, 0.5f, 1.0f, 1.7320508f, 3e38f,
                     gi::kInf, gi::u2f(0x7fc00000u)};
  for (float y : v)
    for (float x : v)
      for (int s = 0; s < 4; s++) check(s & 1 ? -y : y, s & 2 ? -x : x);
  std::mt19937 g(7);
  for (int k = 0; k < 4000000; k++) {
    const unsigned a = g();
    const unsigned near = (a & 0x80ffffffu) ^ (g() & 0x81ffffffu);  // an exponent next to it
    check(gi::u2f(a), gi::u2f(k & 1 ? g() : (a & 0x7f000000u) | near));
  }
  return bad != 0;
}
"""


def test_march_atan2_has_the_bits_of_atan2(tmp_path):
    (tmp_path / "atan2.cpp").write_text(PROGRAM)
    exe = tmp_path / "atan2"
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", f"-I{ROOT / 'legitengine_gb300' / 'csrc'}",
                    str(tmp_path / "atan2.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
