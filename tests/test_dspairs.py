"""The packed double-single arithmetic that the FP64-accurate operator runs (splits, sums, the compensated
dot product of a row of SU(3)), on the CPU against 64-bit mantissas, at the bounds its header derives."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROG = r"""
#include "dspairs.cuh"
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
using namespace gbdw;
static long double ex(float h, float l) { return (long double)h + (long double)l; }
static bool same(float a, float b) { return std::memcmp(&a, &b, 4) == 0; }
int main() {
  std::mt19937_64 rng(54321);
  std::uniform_real_distribution<double> u(-1.0, 1.0);
  std::uniform_int_distribution<int> wide(-40, 40), near(-6, 6);
  auto rnd = [&](auto& d) { const double v = u(rng); return std::ldexp(std::copysign(1.0 + std::fabs(v), v), d(rng)); };
  double split = 0, add = 0, dot = 0;
  int differ = 0;
  for (int i = 0; i < 200000; ++i) {
    const double2 a = {rnd(wide), rnd(wide)}, b = {rnd(wide), rnd(wide)};
    const ds2 x = split2(a), y = split2(b), z = x + y;
    const dsf r = ds_split(a.x), m = ds_split(a.y);
    differ += !(same(r.h, x.h.x) && same(r.l, x.l.x) && same(m.h, x.h.y) && same(m.l, x.l.y));
    split = std::fmax(split, (double)(std::fabs(ex(x.h.x, x.l.x) - (long double)a.x) / std::fabs(a.x)));
    const long double p = ex(x.h.y, x.l.y), q = ex(y.h.y, y.l.y);
    add = std::fmax(add, (double)(std::fabs(ex(z.h.y, z.l.y) - (p + q)) / (std::fabs(p) + std::fabs(q))));
    float2 s = {0, 0}, e = {0, 0};
    long double want[2] = {0, 0}, mag[2] = {0, 0};
    for (int k = 0; k < 6; ++k) {  // the second component's sign as the imaginary part's product has it
      const dsf c = ds_split(rnd(near));
      const ds2 v = split2({rnd(near), rnd(near)});
      dot2({c.h, -c.h}, {c.l, -c.l}, v, s, e);
      const long double t[2] = {ex(c.h, c.l) * ex(v.h.x, v.l.x), -ex(c.h, c.l) * ex(v.h.y, v.l.y)};
      for (int j = 0; j < 2; ++j) want[j] += t[j], mag[j] += std::fabs(t[j]);
    }
    const ds2 w = join2(s, e);
    dot = std::fmax(dot, (double)(std::fabs(ex(w.h.x, w.l.x) - want[0]) / mag[0]));
    dot = std::fmax(dot, (double)(std::fabs(ex(w.h.y, w.l.y) - want[1]) / mag[1]));
  }
  float h, l;
  int special = 0;
  split1(0.0, h, l), special += h == 0 && l == 0 && !std::signbit(h);
  split1(-0.0, h, l), special += h == 0 && l == 0 && std::signbit(h);
  split1(1e-40, h, l), special += h == 0 && l == 0;
  split1(-1e300, h, l), special += std::isinf(h) && h < 0 && l == 0;
  split1(0x1.23456789abcdep-80, h, l), special += std::fabs((double)h + l - 0x1.23456789abcdep-80) <= 0x1p-23 * 0x1.2p-80;
  std::printf("%.3e %.3e %.3e %d %d\n", split, add, dot, differ, special);
}
"""


def test_packed_pairs_keep_their_bounds(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("g++ not available")
    src, exe = tmp_path / "t.cc", tmp_path / "t"
    src.write_text(PROG)
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(ROOT, "gridbench_gb300", "csrc"),
                    str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()
    split, add, dot = map(float, out[:3])
    assert split <= 2.0 ** -47
    assert add <= 2.0 ** -46
    assert dot <= 2.0 ** -40
    assert out[3:] == ["0", "5"]  # bits unlike ds_split's; special values as they should be
