"""What csrc/ammsb_plan.h holds, compiled for the host: no round of a minibatch
examines more candidates than an iteration's scratch area holds, no update starts
early right behind the join of its draws, the pairs
that the samplers leave out are rows in order, and a read-out or a ring
of draws that finds no room on the device makes do with less."""
import os
import subprocess

import numpy as np

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


ORDER = r"""
#include <cstdio>
#include <initializer_list>
#include <string>
#include "ammsb_plan.h"
struct Recorder {  // F fork, J join, R and r rows (r early), T theta, X the launch that fails
  std::string* log;
  int fail;
  int put(char c) { return log->push_back((int)log->size() == fail ? 'X' : c), (int)log->size() - 1 == fail; }
  int fork() { return put('F'); }
  int rows(int, bool early) { return put(early ? 'r' : 'R'); }
  int theta(int) { return put('T'); }
  int join() { return put('J'); }
};
int main() {
  for (int count : {1, 3}) {
    std::string pair, failed;
    ammsb::launch_block_order(Recorder{&pair, -1}, count);
    ammsb::launch_block_order(Recorder{&pair, -1}, count);
    const int e = ammsb::launch_block_order(Recorder{&failed, count + 1}, count);
    std::printf("%s %s %d\n", pair.c_str(), failed.c_str(), e);
  }
}
"""


ROWS = r"""
#include <cstdio>
#include <cstdlib>
#include "ammsb_plan.h"
int main(int argc, char** argv) {  // n, then the pairs
  std::vector<int> x;
  for (int i = 2; i < argc; ++i) x.push_back(std::atoi(argv[i]));
  std::vector<int64_t> row;
  std::vector<int32_t> col;
  ammsb::symmetric_rows(std::atoi(argv[1]), [&](auto&& f) {
    for (size_t i = 0; i < x.size(); i += 2) f(x[i], x[i + 1]);
  }, &row, &col);
  for (size_t v = 0; v + 1 < row.size(); ++v, std::printf("\n"))
    for (int64_t q = row[v]; q < row[v + 1]; ++q) std::printf("%d ", (int)col[q]);
}
"""


READS = r"""
#include <cstdio>
#include <initializer_list>
#include "ammsb_plan.h"
int main() {
  for (bool room : {true, false})
    for (long long values : {1ll, 16384ll, 16385ll, 1ll << 40}) {
      int asked = 0;
      const bool on = ammsb::widen_on_device(values, [&] { return ++asked, room; });
      std::printf("%d%d ", asked, (int)on);
    }
}
"""


ROOM = r"""
#include <cstdio>
#include <initializer_list>
#include "ammsb_plan.h"
int main() {
  for (int want : {16, 8, 3, 2, 1})
    for (int room : {32, 16, 4, 3, 2, 1})  // buffer sets that fit
      std::printf("%d ", ammsb::block_with_room(want, [&](int block) { return 2 * block <= room; }));
}
"""


CALLS = r"""
#include <cstdio>
#include <initializer_list>
#include "ammsb_plan.h"
int main() {
  unsigned seed = 1;
  long long bad = 0;
  for (int D : {1, 2, 3, 8, 16})
    for (bool pairs : {true, false})
      for (bool single : {true, false})
        for (int chain = 0; chain < 200; ++chain) {
          long long drawn = D, done = 0;  // of this chain's iterations
          for (int call = 0, slot = 0, ahead = D; call < 12; ++call) {
            seed = seed * 1664525u + 1013904223u;
            const long long count = 1 + (seed >> 8) % (chain % 2 ? 3 * D + 2 : D);
            for (long long left = count; left > 0;) {
              const auto next = ammsb::next_launch(D, slot, ahead, left, call == 0 && ammsb::brief_call(D, 0, count), pairs, single);
              if (next.fork) drawn += D, ahead += D;
              bad += next.n < 1 || next.n > left || next.n > ahead + (next.whole ? next.n : 0);
              bad += next.whole ? slot % D != 0 || ahead != D || next.n != (next.both ? 2 * D : D) || (next.both && !pairs)
                                : slot % D + next.n > D || (next.n & (next.n - 1)) != 0 || (single && next.n > 1);
              if (next.whole) drawn += next.n; else ahead -= next.n;
              slot = (slot + next.n) % (2 * D);
              done += next.n, left -= next.n;
              bad += drawn - done != ahead || ahead < 1 || ahead > 2 * D || drawn % D != 0;
              // a brief call, after its own draws, makes those of blocks that it reaches;
              // another also those of the block after the one where it ends
              bad += drawn > ((done + left) / D + (call == 0 && count <= (D < 8 ? 1 : D / 4) ? 1 : 2)) * D;
            }
          }
        }
  std::printf("%lld", bad);
}
"""


def compiled_output(tmp_path, program, *args):
    src, exe = tmp_path / "program.cc", str(tmp_path / "program")
    src.write_text(program)
    subprocess.run([os.environ.get("CXX", "g++"), "-std=c++17", "-I", build.CSRC, str(src), "-o", exe], check=True)
    r = subprocess.run([exe, *map(str, args)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    return r.stdout


def test_a_round_fits_its_scratch_area(tmp_path):
    assert "rounds checked" in compiled_output(tmp_path, ROUNDS)


def test_no_update_starts_early_behind_the_join_of_its_draws(tmp_path):
    one, three = compiled_output(tmp_path, ORDER).splitlines()
    # two blocks in turn: R, not r, behind a J
    assert one == "FRTJ" "FRTJ" " FRX 1"
    assert three == "FRTrTrTJ" "FRTrTrTJ" " FRTrX 1"


def test_left_out_pairs_are_rows_in_order(tmp_path):
    rng = np.random.default_rng(0)
    for n, pairs in ((2, []), (3, [(2, 0)]), (40, [tuple(rng.choice(40, 2, replace=False)) for _ in range(300)])):
        rows = [sorted([b for a, b in pairs if a == v] + [a for a, b in pairs if b == v]) for v in range(n)]
        out = compiled_output(tmp_path, ROWS, n, *(x for p in pairs for x in p))
        assert [[int(x) for x in line.split()] for line in out.split("\n")[:n]] == rows  # repeated pairs stay


def test_a_read_without_room_for_its_staging_goes_on_on_the_host(tmp_path):
    # (asked for the buffer, widened on the device) with room, then without
    assert compiled_output(tmp_path, READS).split() == ["00", "00", "11", "11", "00", "00", "10", "10"]


def test_a_ring_without_room_takes_smaller_blocks(tmp_path):
    assert compiled_output(tmp_path, ROOM).split() == \
        "16 2 2 1 1 0  8 8 2 1 1 0  3 3 2 1 1 0  2 2 2 1 1 0  1 1 1 1 1 0".split()


def test_a_call_draws_no_block_that_it_does_not_reach(tmp_path):
    assert compiled_output(tmp_path, CALLS) == "0"
