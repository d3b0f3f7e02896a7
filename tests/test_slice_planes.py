"""Where a vertex lies among the slice planes (csrc/vf_slices.h, compiled by the host
compiler with its undefined-behaviour checks): equal to a binary search for coordinates
inside and far outside the caller's box, infinities and NaN, within a few looks at the
planes.  k_tetra and k_odd_edges use the function as it is."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include <algorithm>
#include <cstdio>
#include <limits>
#include <vector>
#include "vf_slices.h"
struct Planes {
  const std::vector<float>& a;
  mutable int looks = 0;
  float operator[](uint32_t i) const { ++looks; return a[i]; }
};
int main() {
  const float inf = std::numeric_limits<float>::infinity(), nan = std::numeric_limits<float>::quiet_NaN();
  uint32_t s = 7;
  auto rnd = [&] { s ^= s << 13; s ^= s >> 17; s ^= s << 5; return (float)s / 4294967296.0f; };
  for (uint32_t n : {2u, 3u, 64u, 333u, 1000u, 4096u}) {
    std::vector<float> a(n);
    float y = -1.0f;
    for (uint32_t i = 0; i < n; ++i) { a[i] = y; y += 2.0f / (float)n; }
    std::vector<float> v = {inf, -inf, nan, 3.4e38f, -3.4e38f, 1e10f, -1e10f, 2.2e9f, 1.0f, -1.0f, 0.0f, 4e6f};
    v.insert(v.end(), a.begin(), a.end());
    for (int k = 0; k < 5000; ++k) v.push_back(3.0f * rnd() - 1.5f);
    for (float x : v) {
      const uint32_t want = x != x ? n : (uint32_t)(std::upper_bound(a.begin(), a.end(), x) - a.begin());
      Planes p{a};
      const uint32_t got = slice_above(p, n, x);
      if (got != want || p.looks > 8) { printf("n %u v %g: %u, not %u, %d looks\n", n, x, got, want, p.looks); return 1; }
    }
  }
  return 0;
}
"""


def test_slice_above(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ not found")
    src, exe = tmp_path / "slices.cpp", tmp_path / "slices"
    src.write_text(SOURCE)
    inc = os.path.join(ROOT, "voxelfragmentml_gb300", "csrc")
    r = subprocess.run([gxx, "-std=c++17", "-O1", "-Wall", "-Werror", "-fsanitize=undefined,float-cast-overflow",
                        "-fno-sanitize-recover=all", "-I", inc, str(src), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, (r.stdout, r.stderr)
