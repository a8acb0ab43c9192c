"""The half-length Coulomb plans (csrc/coul_half.h) against the five passes' plans on every
grid: the allocation-free solve splits a fixed scratch array by a plan's bytes per density,
so what it accepts must not depend on the plan."""
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "v1-1_b200" / "csrc"
PROGRAM = r"""
#include <cstdio>
#include "coul_half.h"
#include "fft_lengths.h"
using namespace sincgpu;
int main() {
  for (int n = 2; n <= 128; ++n) {
    int m1 = 0, m2 = 0, P = -1;
    const int M = half_length_for(n, &m1, &m2);
    for (int i = kNumFftLens - 1; i >= 0; --i)
      if (kFftLens[i] >= 2 * n - 1) P = kFftLens[i];
    const long long five = 16LL * ((long long)n * n * P + (long long)n * P * P);
    const long long half = M > 0 ? 2LL * 16 * 2 * M * half_slots(n, m1, m2) : 0;
    std::printf("%d %d %lld %lld\n", n, M, five, half);
  }
}
"""


def test_half_length_plans_need_no_more_scratch_than_the_five_passes(tmp_path):
    src, exe = tmp_path / "p.cpp", tmp_path / "p"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", str(CSRC), str(src), "-o", str(exe)], check=True)
    rows = [tuple(map(int, l.split())) for l in subprocess.check_output([str(exe)], text=True).splitlines()]
    planned = [r for r in rows if r[1] > 0]
    assert len(planned) > 20
    for n, M, five, half in planned:
        assert n <= M and half <= five, (n, M, five, half)

