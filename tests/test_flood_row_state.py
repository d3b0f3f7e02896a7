"""The state planes of the flood's rows (csrc/vf_wave_state.h, compiled by the host
compiler): a reader of a wave may see each of a row's two words as it was before or
after the owner's claim of that wave.  Any such mix must show the same front as the
row before the claim, and nothing unclaimed or claimed that was not so before or
after it.  The flood kernel uses these functions as they are."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include <cstdio>
#include "vf_wave_state.h"
int main() {
  uint32_t s = 12345u;
  auto rnd = [&] { s ^= s << 13; s ^= s >> 17; s ^= s << 5; return s; };
  for (int trial = 0; trial < 200000; ++trial) {
    const uint32_t t = trial & 1;
    // any row before wave t: EMPTY, unclaimed, claimed by either parity
    const uint32_t occupied = rnd(), claimed = rnd() & rnd() & occupied, front = rnd() & claimed;
    uint32_t a = wave_empty_a(occupied), b = wave_empty_b(occupied);
    if (wave_claimed(a, b) || wave_front(a, b, t) || wave_unclaimed(a, b) != occupied) return 1;
    wave_claim(a, b, claimed & ~front, t);  // E((t + 1) & 1)
    wave_claim(a, b, front, t + 1);         // E(t & 1)
    if (wave_claimed(a, b) != claimed || wave_front(a, b, t) != front) return 2;
    const uint32_t open = wave_unclaimed(a, b), n = open & rnd();
    if (open != (occupied & ~claimed)) return 3;
    uint32_t na = a, nb = b;
    wave_claim(na, nb, n, t);
    if (wave_front(na, nb, t + 1) != (n | (claimed & ~front)) || wave_claimed(na, nb) != (claimed | n)) return 4;
    for (int mix = 0; mix < 4; ++mix) {
      const uint32_t ra = mix & 1 ? na : a, rb = mix & 2 ? nb : b;
      if (wave_front(ra, rb, t) != front) { printf("wave %u, mix %d\n", t, mix); return 5; }
      const uint32_t o = wave_unclaimed(ra, rb), c = wave_claimed(ra, rb);
      if ((o & ~open) || (~o & open & ~n) || (c & ~(claimed | n)) || (~c & claimed)) return 6;
    }
  }
  return 0;
}
"""


def test_no_mix_of_old_and_new_words_shows_a_claim_early(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ not found")
    src, exe = tmp_path / "state.cpp", tmp_path / "state"
    src.write_text(SOURCE)
    inc = os.path.join(ROOT, "voxelfragmentml_gb300", "csrc")
    r = subprocess.run([gxx, "-std=c++17", "-O2", "-Wall", "-Werror", "-I", inc, str(src), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, (r.returncode, r.stdout)
