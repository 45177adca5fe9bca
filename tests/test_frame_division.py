"""The camera rays' division by the frame's size (camera_direction, core/yc_shade.cuh) is done
with a reciprocal and one step along the remainder; its quotients are the division's, bit for
bit, for every frame size and the fractional pixel positions that float can hold."""
import subprocess

SRC = r"""
#include <cmath>
#include <cstdint>
#include <cstdio>
static double divided(double a, double b, double r) {
  const double q = a * r;
  return std::fma(std::fma(-q, b, a), r, q);
}
int main() {
  uint64_t x = 88172645463325252ull;
  auto next = [&] { x ^= x << 13; x ^= x >> 7; x ^= x << 17; return (uint32_t)(x >> 16); };
  for (int b = 1; b <= 65536; ++b) {
    const double r = 1.0 / (double)b;
    for (int k = 0; k < 60; ++k) {
      float f = (float)(next() % (uint32_t)b);
      f = k == 0 ? 0.0f : k < 3 ? (float)b : f + (float)next() * 2.3283064e-10f;
      if (k % 3 == 2) f = (float)next() * 2.3283064e-10f;   // the first column and row: small quotients
      const double a = 2.0 * (double)f;
      if (divided(a, (double)b, r) != a / (double)b) { std::printf("%d %.9g\n", b, f); return 1; }
    }
  }
  const double m = 4294967295.0;
  for (int k = 0; k < 4000000; ++k) {
    const double a = (double)(k < 100 ? 4294967295u - (uint32_t)k : next());
    if (divided(a, m, 1.0 / m) != a / m) { std::printf("seed %.17g\n", a); return 1; }
  }
  return 0;
}
"""


def test_quotients_are_the_divisions(tmp_path):
    (tmp_path / "d.cpp").write_text(SRC)
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-o", str(tmp_path / "d"), str(tmp_path / "d.cpp")], check=True)
    out = subprocess.run([str(tmp_path / "d")], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
