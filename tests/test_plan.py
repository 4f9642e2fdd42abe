"""Sizes that kernels and their buffers agree on (csrc/ammsb_plan.h), compiled
for the host: no round of a minibatch examines more candidates than an
iteration's scratch area holds."""
import os
import subprocess

from mcmc_for_ammsb_gb300 import build

ROUNDS = r"""
#include <cstdio>
#include <initializer_list>
#include "ammsb_plan.h"
using namespace ammsb;
static long long hash_slots(long long need) { long long p = 1; while (p < need) p <<= 1; return p; }
int main() {
  long long bad = 0, checked = 0;
  for (long long m : {1, 32, 1000, 2000, 3584, 3585, 4000, 4096, 4097, 5000, 8192, 8193, 10000, 40000, 1 << 20, 1 << 24})
    for (long long nodes : {0ll, 9001ll, 4 * m + 1})  // a general edge list's nodes share the hash
      for (double accept : {1.0, 0.95, 0.5, 0.1, 0.01, 0.0}) {
        long long need_slots = 2 * m > 8192 ? 2 * m : 8192;
        if (2 * nodes > need_slots) need_slots = 2 * nodes;
        const long long hcap = hash_slots(need_slots), half = hcap / 2, room = candidate_slots(m, hcap);
        long long count = 0, seen = 0;
        for (int round = 0; round < 2000 && count < m; ++round) {
          const long long R = nonlink_round(m - count, count, half, seen, count);
          ++checked;
          if (R > room || R < m - count || edge_round(m - count, count, half) > room) {
            if (!bad++) std::printf("m %lld hash %lld: a round of %lld in %lld words\n", m, hcap, R, room);
          }
          seen += R;
          const long long got = (long long)(accept * R);
          count += got < m - count ? got : m - count;
        }
      }
  std::printf("%lld rounds checked\n", checked);
  return bad != 0;
}
"""


def test_a_round_fits_its_scratch_area(tmp_path):
    src, exe = tmp_path / "rounds.cc", str(tmp_path / "rounds")
    src.write_text(ROUNDS)
    subprocess.run([os.environ.get("CXX", "g++"), "-std=c++17", "-I", build.CSRC, str(src), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
