"""The double-precision quotients of the camera rays (ym::divided with the reciprocals of
yc::frame_size) and of the first light sample (ym::u01_inclusive) are the division's, bit for bit:
the shipped functions against `/`, at every frame side up to 8,192 and at sides drawn up to 2^28,
at fractional pixel positions, at numerators whose quotients lie nearest to a midpoint of two
doubles, and at seeds of all sizes."""
import os
import subprocess

from yune_gb300 import build

SRC = r"""
#include <cstdio>
#include <cstdint>
#include "ym_math.h"
#include "core/yc_internal.h"

static uint64_t x = 88172645463325252ull;
static uint32_t next() { x ^= x << 13; x ^= x >> 7; x ^= x << 17; return (uint32_t)(x >> 16); }

static bool same(const yc::PassParams& pp, float f) {
  const double a = 2.0 * (double)f;
  return ym::divided(a, pp.w, pp.inv_w) == a / (double)pp.width && ym::divided(a, pp.h, pp.inv_h) == a / (double)pp.height;
}

static bool side(int n) {
  yc::PassParams pp{};
  yc::frame_size(pp, n, n % 977 + 1);
  for (int k = 0; k < 24; ++k) {
    float f = (float)(next() % (uint32_t)n) + (float)next() * 2.3283064e-10f;
    if (k == 0) f = 0.0f;
    if (k == 1) f = (float)n;
    if (k > 1 && k % 3 == 0) f = (float)next() * 2.3283064e-10f;   // the first column: small quotients
    if (!same(pp, f)) { std::printf("%d %.9g\n", n, f); return false; }
    // the 24-bit numerators next to n times a midpoint
    const double q = 2.0 * (double)f / n, mid = q + 0.5 * (std::nextafter(q, 2.0) - q);
    float near = (float)(mid * n * 0.5);
    for (int s = 0; s < 3; ++s, near = std::nextafterf(near, 1e9f))
      if (near > 0.0f && !same(pp, near)) { std::printf("%d %.9g\n", n, near); return false; }
  }
  return true;
}

int main() {
  for (int n = 1; n <= 8192; ++n) if (!side(n)) return 1;
  for (int k = 0; k < 40000; ++k) if (!side(1 + (int)(next() % (1u << (14 + k % 15))))) return 1;
  for (int k = 0; k < 3; ++k) if (!side((1 << 28) - k)) return 1;
  for (uint32_t k = 0; k < 4000000; ++k) {
    const uint32_t seed = k < 1000 ? k : k < 2000 ? 0u - k : next() >> (k % 32);
    if (ym::u01_inclusive(seed) != (float)((double)seed / 4294967295.0)) { std::printf("seed %u\n", seed); return 1; }
    if (ym::divided((double)seed, 4294967295.0, 1.0 / 4294967295.0) != (double)seed / 4294967295.0) return 1;
  }
  return 0;
}
"""


def test_shipped_quotients_are_the_divisions(tmp_path):
    (tmp_path / "d.cpp").write_text(SRC)
    cuda = os.path.join(os.path.dirname(os.path.dirname(build.NVCC)), "include")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I" + build.CSRC,
                    "-I" + os.path.join(build.ROOT, "include"), "-I" + cuda, "-include", "cmath", "-o",
                    str(tmp_path / "d"), str(tmp_path / "d.cpp")], check=True)
    out = subprocess.run([str(tmp_path / "d")], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
