// ammsb_plan.h -- sizes that a kernel and the buffers it writes have to agree
// on, the order of a block's launches, the rows that the samplers search, and
// choices between two ways of a call, in plain C++.
#pragma once
#include <stdint.h>

#include <vector>

#ifdef __CUDACC__
#define AMMSB_HD __host__ __device__ __forceinline__
#else
#define AMMSB_HD inline
#endif

namespace ammsb {

AMMSB_HD int64_t plan_min(int64_t a, int64_t b) { return a < b ? a : b; }
AMMSB_HD int64_t plan_max(int64_t a, int64_t b) { return a > b ? a : b; }

// Candidates that a round of a non-link minibatch examines, to find the `need`
// of m that it lacks with `count` kept: what the rounds so far (`kept` of `seen`)
// say they take (need at first), plus an eighth and 64, while the dedup hash
// stays at most half full (`half` keys) -- and never fewer than need.
AMMSB_HD int64_t nonlink_round(int64_t need, int64_t count, int64_t half, int64_t seen, int64_t kept) {
  const int64_t est = seen == 0 ? need : (kept > 0 ? (need * seen + kept - 1) / kept : half);
  const int64_t want = plan_min(est + est / 8 + 64, half);
  return plan_max(need, plan_min(half - count, want));
}

// ... and a round of a random-edge one.
constexpr int64_t kEdgeRound = 4096;
AMMSB_HD int64_t edge_round(int64_t need, int64_t count, int64_t half) {
  return plan_max(need, plan_min(half - count, kEdgeRound));
}

// Candidate words of one iteration's minibatch: the most that either round
// writes, for minibatches of m with a hash of hcap slots (a round is need <= m,
// or at most half the hash).
AMMSB_HD int64_t candidate_slots(int64_t m, int64_t hcap) { return plan_max(m, hcap / 2); }

// The launches of a block of `count` iterations, with the other block's draws
// forked alongside and joined behind: per iteration the rows (update_phi and the
// commit), then the theta step.  An update that follows a theta step inside the
// block starts early; the block's first does not, whatever is ahead of it in the
// stream, because its own draws were joined there: a programmatic launch that
// follows a joined stream takes a programmatic edge from that stream's kernel too
// (as the edges of such a capture say), which makes nothing that the kernel wrote
// visible before the wait.  Joining the draws ahead of the block's last theta step
// instead, whose wait they end before, let that update start early too: a
// 100k-node interval 5.66 to 5.54 ms, but 64 chains on streams of their own, 200
// iterations, 43.6 to 59.7 ms.
template <class Launches>
auto launch_block_order(Launches&& l, int count) {
  auto e = l.fork();
  for (int i = 0; !e && i < count; ++i) {
    e = l.rows(i, i > 0);
    if (!e) e = l.theta(i);
  }
  if (!e) e = l.join();
  return e;
}

// What a call launches next with `left` iterations to go, at ring slot `slot` of
// two blocks of D with `ahead` iterations drawn from there on: n updates -- one
// whole block with the other's draws alongside, both in turn (`both`, where
// `pairs` allows it), or a run of n (a power of two, so that few graphs are kept;
// one with `single`) inside a block, with the other block's draws forked ahead of
// it (`fork`): with a block's first launch, so that they overlap all of the call
// that is left.  A `brief` call -- one that had to make its first block's draws
// itself, and is over after a quarter of it -- leaves them to a later one unless it
// reaches the block's end: such calls that each follow a change of state or step,
// which drops the draws, make eight iterations' draws rather than sixteen (set_step
// and step(1) of the 400,000-node workload: 198 us, now 121).  Longer ones overlap
// them (64 chains on streams of their own, step(5) and step(200): 48.5 ms, 60 with
// the draws of the first call left to the second).
inline bool brief_call(int D, int ahead, int64_t n) { return ahead == 0 && n <= (D < 8 ? 1 : D / 4); }
struct NextLaunch {
  int n;
  bool whole, both, fork;
};
inline NextLaunch next_launch(int D, int slot, int ahead, int64_t left, bool brief, bool pairs, bool single) {
  const int pos = slot % D, rest = D - pos;
  if (pos == 0 && left >= D) {
    const bool both = pairs && left >= 2 * (int64_t)D;
    return {both ? 2 * D : D, true, both, false};
  }
  const int most = (int)plan_min(left, rest);
  int n = 1;
  while (!single && n < 8 && 2 * n <= most) n *= 2;
  return {n, false, false, ahead == rest && (left >= rest || (pos == 0 && !brief))};
}

// The iterations of a draws launch: `want`, or as few as alloc(block), which gives
// back what it got when it fails, finds room for (a ring of two blocks' buffer
// sets: sixteen for eight iterations, four for two, two for one).  0: none.
template <class Alloc>
int block_with_room(int want, Alloc&& alloc) {
  for (int block = want; block > 0; block = block > 2 ? 2 : block - 1)
    if (alloc(block)) return block;
  return 0;
}

// Whether BF16 rows are widened on the device for a read-out, with a staging
// buffer that stage() allocates with the first read that wants it: reads of more
// than 16,384 values, if it can be had.  2,000 values take the host's loop 22 us
// and a kernel with its copy 28, 32,000 either 28, 140,000 the host 62 and the
// kernel 35.
template <class Stage>
bool widen_on_device(int64_t values, Stage&& stage) {
  return values > 16384 && stage();
}

// Pairs of n nodes (each(f) calls f(a, b) for every one) as a symmetric CSR with
// sorted rows: their entries in any order first, whose transpose -- the same
// matrix -- has every row in order.  Sorting the rows one by one was two thirds
// of an ammsb_create where nodes have many such pairs (1M entries, 200 a row:
// 20.7 ms in all, now 5.9; 2.4M entries of 100,000 nodes: 48 ms, now 32).
template <class Each>
void symmetric_rows(int64_t n, Each&& each, std::vector<int64_t>* row, std::vector<int32_t>* col) {
  // end[v], the pointer past row v: counts, then their running sums; every entry
  // placed below its row's end leaves the rows' starts there, and the transpose,
  // placed upwards, their ends again
  row->assign((size_t)n + 1, 0);
  int64_t* end = row->data() + 1;
  each([&](int32_t a, int32_t b) { ++end[a], ++end[b]; });
  for (int64_t v = 1; v < n; ++v) end[v] += end[v - 1];
  const size_t total = (size_t)end[n - 1];
  struct Entry {
    int32_t of, with;
  };
  std::vector<Entry> any(total);
  each([&](int32_t a, int32_t b) { any[--end[a]] = {a, b}, any[--end[b]] = {b, a}; });
  col->resize(total);
  for (const Entry& e : any) (*col)[end[e.with]++] = e.of;
}

}  // namespace ammsb
