"""The generator's fixed-point forms (legionorigins_gb300/csrc/ckt_drand.cuh)
against the double arithmetic they replace, on the CPU: the affine expressions
of load_circuit (apps/circuit/circuit.cc:1121-1170) for its own constants and
others, the index draw, and the crossing threshold -- random states, edges,
and states whose value lies next to a boundary between two floats."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "legionorigins_gb300", "csrc")

SOURCE = r'''
#include <cmath>
#include <cstdio>
#include <random>
#include "ckt_drand.cuh"
using namespace ckt::drand;
int main() {
  std::mt19937_64 rng(77);
  const uint64_t M48 = (1ull << 48) - 1;
  const uint64_t edge[] = {0, 1, 2, M48, M48 - 1, 1ull << 47, (1ull << 47) - 1, 1ull << 24, 12345};
  const double sc[][2] = {{0.01, 0.1}, {0.1, 0.0}, {0.01, 0.001}, {(double)0.1f, 0.0}, {8e-7, 1e-7},
                          {0.0, 0.25}, {3.0, 1e-9}, {1e-9, 5.0}, {1.0, 1.0}, {1e15, 0.0}};
  long bad = 0, settled = 0, n = 0;
  for (const auto &p : sc) {
    const Affine a = make_affine(p[0], p[1]);
    bad += a.exponent == 0x7fffffff;
    for (int i = 0; i < 300000; i++) {
      uint64_t x = i < 9 ? edge[i] : (rng() & M48);
      if (i >= 9 && i % 4 == 0 && p[0] > 0) {
        // a state whose value lies next to the middle of two floats
        const float f = (float)(x * 0x1p-48 * p[0] + p[1]);
        const double mid = ((double)f + (double)std::nextafter(f, 1e30f)) / 2;
        const double xs = (mid - p[1]) / p[0] * 0x1p48;
        if (xs >= 0 && xs < 0x1p48 - 4) x = (uint64_t)xs + (uint64_t)(i / 4 % 3);
      }
      const float want = (float)(x * 0x1p-48 * p[0] + p[1]);
      float got;
      n++;
      if (affine_float(x, a, &got)) {
        settled++;
        bad += got != want;
      }
    }
  }
  for (const double v : {-1.0, 0.0, 1e30, 1e-30}) bad += make_affine(v, 0).exponent != 0x7fffffff;
  bad += make_affine(0.1, -0.01).exponent != 0x7fffffff;
  bad += make_affine(NAN, 0).exponent != 0x7fffffff;
  for (int i = 0; i < 1000000; i++) {
    const uint32_t m = (uint32_t)(rng() % 2147483647u) + 1;
    uint64_t x = rng() & M48;
    if (i & 1) x = (uint64_t)(((unsigned __int128)(rng() % m + 1) << 48) / m) - (i & 7) + 3;  // near k/m
    x &= M48;
    bad += trunc_mul_fast(x, m) != (uint32_t)(int)(x * 0x1p-48 * m);
  }
  for (const double pct : {-1.0, 0.0, 0.5, 33.3, 50.0, 83.25, 95.0, 99.999, 100.0, 250.0}) {
    const uint64_t thr = pct_threshold(pct), f = first_crossing(thr);
    for (int d = -3; d <= 3; d++) {
      const uint64_t x = f + d;
      if (x <= M48) bad += (x >= f) != !(100 * (x * 0x1p-48) < pct);
    }
    bad += f > 0 && !pct_below(0, thr);
    bad += f <= M48 && pct_below(M48, thr);
  }
  printf("checked %ld settled %ld bad %ld\n", n, settled, bad);
  return bad != 0 || settled < n / 2;
}
'''


@pytest.mark.skipif(shutil.which("g++") is None, reason="g++ not available")
def test_fixed_point_forms_match_double_arithmetic(tmp_path):
    src = tmp_path / "check.cc"
    src.write_text(SOURCE)
    exe = tmp_path / "check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", CSRC, "-o", str(exe),
                    str(src)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and "bad 0" in out.stdout, out.stdout + out.stderr
