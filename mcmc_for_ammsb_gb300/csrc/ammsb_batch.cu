// ammsb_batch.cu -- many independent chains advanced together, up to sixteen
// iterations of all of them per CUDA graph launch.
//
// Each chain is an ammsb_handle of its own (its graph, held-out set, state,
// options and update_phi configuration).  The batch launches every kernel
// of the iteration once for all chains that share the kernel's compiled
// shape: a map from a block to its chain selects the chain, whose model, graph
// and buffer sets come from a device array of ChainArgs.  Chains of different row widths,
// minibatch sizes and graphs therefore run in a handful of launches per
// iteration instead of five per chain, and a block of iterations of all
// chains -- their updates and, on a second stream, one launch of all their
// next block's draws -- is captured as one graph per block of the ring.
// Every chain keeps its own step counter and Philox key, so a chain advanced
// in a batch goes through exactly the states it goes through on its own.
#include <algorithm>
#include <cstdlib>
#include <cstdio>
#include <cstring>
#include <map>
#include <string>
#include <tuple>
#include <vector>

#include "ammsb_internal.h"
#include "ammsb_phi_ring.cuh"

namespace {

// The blocks of one launch over many chains: each chain's own, in chain order.
struct BlockMap {
  std::vector<BlockOf> blocks;
  BlockOf* d = nullptr;
  void add(int chain, int n) {
    for (int i = 0; i < n; ++i) blocks.push_back(BlockOf{chain, i, n, 0});
  }
  int grid() const { return (int)blocks.size(); }
};

// One launch of the update phase: the chains sharing a kernel shape.
struct PhiGroup {
  int dtype;
  KernelCfg cfg;
  bool full;  // ring kernel: every lane's vectors inside the row
  std::vector<int> chains;
  BlockMap map, map_few;  // map_few: the ring kernel's launch for iterations of few nodes, where it has its own
  size_t smem = 0;      // ring kernel: per four-warp group
  size_t smem_few = 0;  // ring kernel: a 16-warp node
};

struct CommitGroup {
  int dtype, kq;
  int chunk;  // k_commit_star's edges per summing warp at once; 0: k_commit_beta
  BlockMap map;
  size_t smem = 0;
};

// `all`: every chain's arguments; `pdl`: as for one chain.
template <typename PiT, int L, int V, int S>
cudaError_t phi_reg_chains(const PhiGroup& g, const ChainArgs* all, int p, cudaStream_t st, bool pdl) {
  constexpr int NPB = 128 / (L * S) > 0 ? 128 / (L * S) : 1;
  return launch_k(k_update_phi_chains<PiT, L, V, S, NPB>, g.map.grid(), NPB * S * L, g.smem, st, pdl, all, g.map.d, p);
}

template <typename PiT, int V, int STAGES, bool FULL>
cudaError_t phi_ring_chains(const PhiGroup& g, const ChainArgs* all, int p, cudaStream_t st, bool pdl,
                            bool configure) {
  auto kern = k_update_phi_ring_chains<PiT, V, STAGES, FULL>;
  const RingPlan r = ring_plan(g.cfg, g.smem, g.smem_few);
  if (configure) return ammsb_detail::raise_smem_limit(kern, r.smem());
  if (r.single)
    return launch_k(kern, g.map.grid(), 512, r.smem(), st, pdl, all, g.map.d, p, r.few, kPhiFew | kPhiMany);
  if (r.few > 0) {
    cudaError_t e = launch_k(kern, g.map_few.grid(), 512, r.few_bytes, st, pdl, all, g.map_few.d, p, r.few, kPhiFew);
    if (e != cudaSuccess) return e;
  }
  return launch_k(kern, g.map.grid(), r.groups * kPhiGroup, r.groups * r.group_bytes, st, pdl, all, g.map.d, p, r.few,
                  kPhiMany);
}

template <typename PiT, int V>
cudaError_t phi_ring_chains_v(const PhiGroup& g, const ChainArgs* all, int p, cudaStream_t st, bool pdl,
                              bool configure) {
#define RING_CASE(S)                                                                           \
  if (g.cfg.ring_stages == S)                                                                  \
    return g.full ? phi_ring_chains<PiT, V, S, true>(g, all, p, st, pdl, configure)                      \
                  : phi_ring_chains<PiT, V, S, false>(g, all, p, st, pdl, configure);
  AMMSB_PHI_RING_STAGES(RING_CASE)
#undef RING_CASE
  return cudaErrorInvalidConfiguration;
}

template <typename PiT>
cudaError_t phi_chains(const PhiGroup& g, const ChainArgs* all, int p, cudaStream_t st, bool pdl, bool configure) {
  const KernelCfg& c = g.cfg;
  if (c.ring) {
    switch (c.vpl) {
      case 1: return phi_ring_chains_v<PiT, 1>(g, all, p, st, pdl, configure);
      case 2: return phi_ring_chains_v<PiT, 2>(g, all, p, st, pdl, configure);
      case 4: return phi_ring_chains_v<PiT, 4>(g, all, p, st, pdl, configure);
      default: break;
    }
    if constexpr (sizeof(PiT) == 4)
      if (c.vpl == 8) return phi_ring_chains_v<PiT, 8>(g, all, p, st, pdl, configure);
    return cudaErrorInvalidConfiguration;
  }
  if (configure) {
    if (g.smem <= 48 * 1024) return cudaSuccess;
#define REG_CFG(L, V, S)                                                                        \
  if (c.lpn == L && c.vpl == V && c.split == S)                                                 \
    return ammsb_detail::raise_smem_limit(                                                      \
        k_update_phi_chains<PiT, L, V, S, (128 / (L * S) > 0 ? 128 / (L * S) : 1)>, g.smem);
    AMMSB_PHI_REG_SHAPES(REG_CFG)
#undef REG_CFG
    return cudaErrorInvalidConfiguration;
  }
#define REG_CASE(L, V, S) \
  if (c.lpn == L && c.vpl == V && c.split == S) return phi_reg_chains<PiT, L, V, S>(g, all, p, st, pdl);
  AMMSB_PHI_REG_SHAPES(REG_CASE)
#undef REG_CASE
  return cudaErrorInvalidConfiguration;
}

template <typename PiT, int KQ>
cudaError_t commit_chains_k(const CommitGroup& g, const ChainArgs* all, int p, cudaStream_t st, bool pdl,
                            bool configure) {
  auto go = [&](auto* kern, int threads) -> cudaError_t {
    if (configure) return ammsb_detail::raise_smem_limit(kern, g.smem);
    return launch_k(kern, g.map.grid(), threads, g.smem, st, pdl, all, g.map.d, p);
  };
  switch (g.chunk) {
    case 0: return go(k_commit_beta_chains<PiT, KQ>, 128);
    case 1: return go(k_commit_star_chains<PiT, KQ, 1>, 128);
    default: return go(k_commit_star_chains<PiT, KQ, kStarChunk>, 128 * kStarChunk);
  }
}
template <typename PiT>
cudaError_t commit_chains(const CommitGroup& g, const ChainArgs* all, int p, cudaStream_t st, bool pdl,
                          bool configure) {
  switch (g.kq) {
    case 1: return commit_chains_k<PiT, 1>(g, all, p, st, pdl, configure);
    case 2: return commit_chains_k<PiT, 2>(g, all, p, st, pdl, configure);
    case 4: return commit_chains_k<PiT, 4>(g, all, p, st, pdl, configure);
    case 8: return commit_chains_k<PiT, 8>(g, all, p, st, pdl, configure);
    default: return cudaErrorInvalidConfiguration;
  }
}

}  // namespace

struct ammsb_batch {
  int device = 0;
  std::vector<ammsb_handle*> h;
  cudaStream_t stream = nullptr, side = nullptr;
  cudaEvent_t ev_fork = nullptr, ev_join = nullptr, ev_done = nullptr;
  // update_phi groups after the first run side by side on their own streams
  std::vector<cudaStream_t> gstream;
  std::vector<cudaEvent_t> gevent;
  cudaEvent_t ev_groups = nullptr;
  ChainArgs* d_all = nullptr;
  std::vector<void*> allocs;
  std::vector<PhiGroup> phi;
  std::vector<CommitGroup> commit;
  BlockMap theta, nbr;
  int pdl = 0;  // early starts (kPdl* bits), as for one chain
  size_t mb_smem = 0, nbr_smem = 0;
  // captured iterations, as for one chain (ammsb_handle): a block with the
  // other block's draws alongside, both in turn, runs of updates in a block
  cudaGraphExec_t graphB[2] = {}, graphL[2] = {};
  cudaGraphExec_t graphU[kMaxRing][4] = {};
  int block = kMaxBlock;  // iterations per draws launch: the smallest of the chains'
  int slot = 0;           // ring slot of the next iteration, in every chain's ring
  int ahead = 0;          // iterations drawn from `slot` on, as ammsb_handle::ahead
  std::vector<uint64_t> expect_step;  // each chain's step_count after the last batch step
  std::vector<uint64_t> expect_gen;   // and its ring_gen
  std::string err;
};

namespace {

thread_local std::string g_batch_create_error;

#define BK(call)                                                       \
  do {                                                                 \
    cudaError_t e_ = (call);                                           \
    if (e_ != cudaSuccess) {                                           \
      bt->err = std::string(#call) + ": " + cudaGetErrorString(e_);   \
      return AMMSB_E_CUDA;                                             \
    }                                                                  \
  } while (0)

// The update in two parts, as for one chain.  `pdl`: the theta step of the
// iteration before is the kernel ahead in the stream and this iteration's draws
// were complete before that step started.
cudaError_t launch_rows_chains(ammsb_batch* bt, int p, bool pdl) {
  // the update_phi groups touch disjoint chains: they run concurrently
  // (parallel branches of the captured graph), then join before the commits.
  // The first group, the commit and the theta step start early as for one
  // chain; the other groups start when the theta step ahead has completed, and
  // the commit when they have (every chain's update_phi and so its commit
  // follow that step, as the rules for early starts ask).
  const size_t ng = bt->phi.size();
  cudaError_t e = cudaSuccess;
  if (ng > 1 && (e = cudaEventRecord(bt->ev_groups, bt->stream)) != cudaSuccess) return e;
  for (size_t gi = 0; gi < ng; ++gi) {
    const PhiGroup& g = bt->phi[gi];
    cudaStream_t st = gi == 0 ? bt->stream : bt->gstream[gi - 1];
    const bool early = gi == 0 && pdl && (bt->pdl & kPdlPhi);
    if (gi > 0 && (e = cudaStreamWaitEvent(st, bt->ev_groups, 0)) != cudaSuccess) return e;
    e = (g.dtype == AMMSB_PI_BF16) ? phi_chains<__nv_bfloat16>(g, bt->d_all, p, st, early, false)
                                   : phi_chains<float>(g, bt->d_all, p, st, early, false);
    if (e != cudaSuccess) return e;
    if (gi > 0 && (e = cudaEventRecord(bt->gevent[gi - 1], st)) != cudaSuccess) return e;
  }
  for (size_t gi = 1; gi < ng; ++gi)
    if ((e = cudaStreamWaitEvent(bt->stream, bt->gevent[gi - 1], 0)) != cudaSuccess) return e;
  for (size_t ci = 0; ci < bt->commit.size(); ++ci) {
    const CommitGroup& g = bt->commit[ci];
    const bool early = ci == 0 && (bt->pdl & kPdlCommit);
    e = (g.dtype == AMMSB_PI_BF16) ? commit_chains<__nv_bfloat16>(g, bt->d_all, p, bt->stream, early, false)
                                   : commit_chains<float>(g, bt->d_all, p, bt->stream, early, false);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}
cudaError_t launch_theta_chains(ammsb_batch* bt, int p) {
  return launch_k(k_theta_chains, bt->theta.grid(), kThetaThreads, 0, bt->stream, (bt->pdl & kPdlTheta) != 0,
                  bt->d_all, bt->theta.d, p);
}

// Draws of one block of every chain, into the buffer sets from s0 on.
cudaError_t launch_sampling_chains(ammsb_batch* bt, int s0, cudaStream_t st) {
  const unsigned n = (unsigned)bt->h.size(), D = (unsigned)bt->block;
  k_sample_minibatch_chains<<<dim3(D, n), 1024, bt->mb_smem, st>>>(bt->d_all, s0);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  k_sample_neighbors_chains<8><<<dim3(bt->nbr.grid(), D), 256, bt->nbr_smem, st>>>(bt->d_all, bt->nbr.d, s0);
  return cudaGetLastError();
}

cudaError_t launch_updates_chains(ammsb_batch* bt, int s, int count) {
  cudaError_t e = cudaSuccess;
  for (int i = 0; i < count && e == cudaSuccess; ++i) {
    e = launch_rows_chains(bt, s + i, i > 0);
    if (e == cudaSuccess) e = launch_theta_chains(bt, s + i);
  }
  return e;
}

// The draws of block `blk` forked onto the side stream, and their join (as
// fork_draws / join_draws for one chain).
cudaError_t fork_draws_chains(ammsb_batch* bt, int blk) {
  cudaError_t e = cudaEventRecord(bt->ev_fork, bt->stream);
  if (e != cudaSuccess) return e;
  if ((e = cudaStreamWaitEvent(bt->side, bt->ev_fork, 0)) != cudaSuccess) return e;
  if ((e = launch_sampling_chains(bt, blk * bt->block, bt->side)) != cudaSuccess) return e;
  return cudaEventRecord(bt->ev_join, bt->side);
}

cudaError_t launch_block_chains(ammsb_batch* bt, int blk) {
  struct Launches {
    ammsb_batch* bt;
    int blk;
    cudaError_t fork() { return fork_draws_chains(bt, 1 - blk); }
    cudaError_t rows(int i, bool early) { return launch_rows_chains(bt, blk * bt->block + i, early); }
    cudaError_t theta(int i) { return launch_theta_chains(bt, blk * bt->block + i); }
    cudaError_t join() { return cudaStreamWaitEvent(bt->stream, bt->ev_join, 0); }
  };
  return launch_block_order(Launches{bt, blk}, bt->block);
}

// Launches `work` as a captured graph kept in g.
template <typename F>
int launch_graph(ammsb_batch* bt, cudaGraphExec_t& g, F&& work) {
  if (!g) {
    cudaGraph_t graph;
    BK(cudaStreamBeginCapture(bt->stream, cudaStreamCaptureModeThreadLocal));
    cudaError_t e = work();
    cudaError_t e2 = cudaStreamEndCapture(bt->stream, &graph);
    if (e != cudaSuccess || e2 != cudaSuccess) {
      bt->err = std::string("graph capture: ") + cudaGetErrorString(e != cudaSuccess ? e : e2);
      return AMMSB_E_CUDA;
    }
    BK(cudaGraphInstantiate(&g, graph, cudaGraphInstantiateFlagUseNodePriority));
    cudaGraphDestroy(graph);
  }
  BK(cudaGraphLaunch(g, bt->stream));
  return AMMSB_OK;
}

template <typename T>
cudaError_t dev_upload(ammsb_batch* bt, T** out, const std::vector<T>& v) {
  void* p = nullptr;
  cudaError_t e = cudaMalloc(&p, std::max<size_t>(sizeof(T) * v.size(), 16));
  if (e != cudaSuccess) return e;
  bt->allocs.push_back(p);
  *out = static_cast<T*>(p);
  return cudaMemcpy(p, v.data(), sizeof(T) * v.size(), cudaMemcpyHostToDevice);
}

}  // namespace

extern "C" {

const char* ammsb_batch_create_error(void) { return g_batch_create_error.c_str(); }

const char* ammsb_batch_last_error(const ammsb_batch* bt) { return bt ? bt->err.c_str() : "null batch"; }

void ammsb_batch_destroy(ammsb_batch* bt) {
  if (!bt) return;
  cudaSetDevice(bt->device);
  if (bt->stream) cudaStreamSynchronize(bt->stream);
  if (bt->side) cudaStreamSynchronize(bt->side);
  for (int q = 0; q < 2; ++q)
    for (cudaGraphExec_t g : {bt->graphB[q], bt->graphL[q]})
      if (g) cudaGraphExecDestroy(g);
  for (auto& per_slot : bt->graphU)
    for (cudaGraphExec_t g : per_slot)
      if (g) cudaGraphExecDestroy(g);
  for (void* p : bt->allocs) cudaFree(p);
  for (cudaEvent_t ev : {bt->ev_fork, bt->ev_join, bt->ev_done, bt->ev_groups})
    if (ev) cudaEventDestroy(ev);
  for (cudaEvent_t ev : bt->gevent) cudaEventDestroy(ev);
  for (cudaStream_t st : bt->gstream) cudaStreamDestroy(st);
  if (bt->side) cudaStreamDestroy(bt->side);
  if (bt->stream) cudaStreamDestroy(bt->stream);
  delete bt;
}

int ammsb_batch_create(ammsb_handle* const* handles, int32_t n, ammsb_batch** out) {
  g_batch_create_error.clear();
  if (!handles || n < 1 || !out) {
    g_batch_create_error = "need at least one handle";
    return AMMSB_E_ARG;
  }
  *out = nullptr;
  auto* bt = new ammsb_batch();
  auto bail = [&](int code) {
    g_batch_create_error = bt->err;
    ammsb_batch_destroy(bt);
    return code;
  };
  for (int i = 0; i < n; ++i) {
    ammsb_handle* h = handles[i];
    if (!h) {
      bt->err = "null handle";
      return bail(AMMSB_E_ARG);
    }
    for (int j = 0; j < i; ++j)
      if (handles[j] == h) {
        bt->err = "a handle appears twice";
        return bail(AMMSB_E_ARG);
      }
    if (i > 0 && h->device != handles[0]->device) {
      bt->err = "all chains must be on one device";
      return bail(AMMSB_E_ARG);
    }
    bt->h.push_back(h);
  }
  bt->device = handles[0]->device;
  bt->pdl = handles[0]->cfg.pdl;
  if (const char* env = std::getenv("AMMSB_BATCH_GRAPH_ITERS"))  // iterations of both blocks
    bt->block = std::max(1, std::min(kMaxBlock, std::atoi(env) / 2));
  int prio_lo = 0, prio_hi = 0;  // the draws ahead at the higher priority, as for one chain
  if (cudaSetDevice(bt->device) != cudaSuccess ||
      cudaDeviceGetStreamPriorityRange(&prio_lo, &prio_hi) != cudaSuccess ||
      cudaStreamCreateWithFlags(&bt->stream, cudaStreamNonBlocking) != cudaSuccess ||
      cudaStreamCreateWithPriority(&bt->side, cudaStreamNonBlocking, prio_hi) != cudaSuccess ||
      cudaEventCreateWithFlags(&bt->ev_fork, cudaEventDisableTiming) != cudaSuccess ||
      cudaEventCreateWithFlags(&bt->ev_join, cudaEventDisableTiming) != cudaSuccess ||
      cudaEventCreateWithFlags(&bt->ev_done, cudaEventDisableTiming) != cudaSuccess) {
    bt->err = "stream/event creation failed";
    return bail(AMMSB_E_CUDA);
  }
  std::vector<ChainArgs> args(n);
  for (int i = 0; i < n; ++i) {
    ammsb_handle* h = bt->h[i];
    ChainArgs& a = args[i];
    a.m = h->m;
    a.g = h->g;
    a.b = h->b;
    bt->block = std::min(bt->block, h->block);
    a.ncommit = h->ncommit;
    a.star = h->star ? 1 : 0;
    a.smem_hash = h->mb_smem > 0 ? 1 : 0;
    bt->mb_smem = std::max(bt->mb_smem, h->mb_smem);
    bt->nbr_smem = std::max(bt->nbr_smem, h->nbr_smem);
    bt->nbr.add(i, h->nbr_blocks);
    bt->theta.add(i, (h->m.K + 31) / 32);
  }
  if (dev_upload(bt, &bt->d_all, args) != cudaSuccess) {
    bt->err = "upload of the chain table failed";
    return bail(AMMSB_E_CUDA);
  }
  // group the update_phi launches by compiled shape, the commits by K-tile
  std::map<std::tuple<int, int, int, int, int, int, int>, int> pg;
  std::map<std::tuple<int, int, int>, int> cg;
  for (int i = 0; i < n; ++i) {
    ammsb_handle* h = bt->h[i];
    const KernelCfg& c = h->cfg;
    const int ev = (h->opt.pi_dtype == AMMSB_PI_BF16) ? 8 : 4;
    const bool full = (h->m.Kp / ev == 32 * c.vpl);
    auto key = std::make_tuple((int)h->opt.pi_dtype, c.ring, c.lpn, c.vpl, c.split,
                               c.ring ? c.ring_stages : 0, c.ring ? (int)full + 2 * (h->phi_smem_few > 0) : 0);
    auto it = pg.find(key);
    if (it == pg.end()) {
      PhiGroup g;
      g.dtype = h->opt.pi_dtype;
      g.cfg = c;
      g.full = full;
      it = pg.emplace(key, (int)bt->phi.size()).first;
      bt->phi.push_back(g);
    }
    PhiGroup& g = bt->phi[it->second];
    g.chains.push_back(i);
    if (c.ring) {
      g.smem = std::max(g.smem, h->phi_smem);
      g.smem_few = std::max(g.smem_few, h->phi_smem_few);
    } else {
      const int npb = std::max(1, 128 / (c.lpn * c.split));
      g.map.add(i, std::max(1, std::min((h->m.max_nodes + npb - 1) / npb, 152 * 32)));
      const size_t smem = ((size_t)npb * c.split * h->m.Kp + npb * c.split +
                           npb * std::max(1, c.split * c.lpn / 32)) * sizeof(float);
      g.smem = std::max(g.smem, smem);
    }
    const int chunk = h->star ? star_chunk(h->m) : 0;
    auto ck = std::make_tuple((int)h->opt.pi_dtype, c.kq, chunk);
    auto jt = cg.find(ck);
    if (jt == cg.end()) {
      CommitGroup g2;
      g2.dtype = h->opt.pi_dtype;
      g2.kq = c.kq;
      g2.chunk = chunk;
      jt = cg.emplace(ck, (int)bt->commit.size()).first;
      bt->commit.push_back(g2);
    }
    CommitGroup& g2 = bt->commit[jt->second];
    g2.map.add(i, (chunk ? 0 : h->ncommit) + h->m.nbb + (h->m.K + 31) / 32);
    if (chunk)
      g2.smem = std::max(g2.smem, chunk == 1 ? commit_star_smem<1>(h->m.Kp) : commit_star_smem<kStarChunk>(h->m.Kp));
  }
  auto upload = [&](BlockMap& map) { return dev_upload(bt, &map.d, map.blocks) == cudaSuccess; };
  for (PhiGroup& g : bt->phi) {
    if (g.cfg.ring) {  // a node per four-warp group, and a CTA per node of an iteration of few
      const RingPlan r = ring_plan(g.cfg, g.smem, g.smem_few);
      for (int i : g.chains) {
        const int nodes = bt->h[i]->m.max_nodes, many = (nodes + r.groups - 1) / r.groups,
                  few = std::min(r.few, nodes);
        g.map.add(i, r.single ? std::max(many, few) : many);
        if (!r.single && r.few > 0) g.map_few.add(i, few);
      }
    }
    if (!upload(g.map) || !upload(g.map_few)) {
      bt->err = "upload of a group table failed";
      return bail(AMMSB_E_CUDA);
    }
    cudaError_t e = (g.dtype == AMMSB_PI_BF16) ? phi_chains<__nv_bfloat16>(g, bt->d_all, 0, bt->stream, false, true)
                                               : phi_chains<float>(g, bt->d_all, 0, bt->stream, false, true);
    if (e != cudaSuccess) {
      bt->err = std::string("update_phi group configuration: ") + cudaGetErrorString(e);
      return bail(AMMSB_E_CUDA);
    }
  }
  if (cudaEventCreateWithFlags(&bt->ev_groups, cudaEventDisableTiming) != cudaSuccess) {
    bt->err = "event creation failed";
    return bail(AMMSB_E_CUDA);
  }
  for (size_t gi = 1; gi < bt->phi.size(); ++gi) {
    cudaStream_t st = nullptr;
    cudaEvent_t ev = nullptr;
    if (cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess) {
      bt->err = "stream creation failed";
      return bail(AMMSB_E_CUDA);
    }
    bt->gstream.push_back(st);
    if (cudaEventCreateWithFlags(&ev, cudaEventDisableTiming) != cudaSuccess) {
      bt->err = "event creation failed";
      return bail(AMMSB_E_CUDA);
    }
    bt->gevent.push_back(ev);
  }
  for (CommitGroup& g : bt->commit) {
    if (!upload(g.map)) {
      bt->err = "upload of a group table failed";
      return bail(AMMSB_E_CUDA);
    }
    cudaError_t e = (g.dtype == AMMSB_PI_BF16)
                        ? commit_chains<__nv_bfloat16>(g, bt->d_all, 0, bt->stream, false, true)
                        : commit_chains<float>(g, bt->d_all, 0, bt->stream, false, true);
    if (e != cudaSuccess) {
      bt->err = std::string("commit group configuration: ") + cudaGetErrorString(e);
      return bail(AMMSB_E_CUDA);
    }
  }
  if (!upload(bt->theta) || !upload(bt->nbr)) {
    bt->err = "upload of a group table failed";
    return bail(AMMSB_E_CUDA);
  }
  if ((bt->mb_smem > 48 * 1024 &&
       ammsb_detail::raise_smem_limit(k_sample_minibatch_chains, bt->mb_smem) != cudaSuccess) ||
      (bt->nbr_smem > 48 * 1024 &&
       ammsb_detail::raise_smem_limit(k_sample_neighbors_chains<8>, bt->nbr_smem) != cudaSuccess)) {
    bt->err = "sampler shared memory configuration failed";
    return bail(AMMSB_E_CUDA);
  }
  bt->expect_step.assign(n, 0);
  bt->expect_gen.assign(n, 0);
  *out = bt;
  return AMMSB_OK;
}

int32_t ammsb_batch_groups(const ammsb_batch* bt) { return bt ? (int32_t)bt->phi.size() : -1; }

int ammsb_batch_step(ammsb_batch* bt, int64_t n_iters) {
  if (!bt || n_iters < 0) return AMMSB_E_ARG;
  BK(cudaSetDevice(bt->device));
  for (ammsb_handle* h : bt->h)
    if (!h->state_ready) {
      bt->err = "every chain needs a state (ammsb_init_state / ammsb_set_state)";
      return AMMSB_E_STATE;
    }
  if (n_iters == 0) return AMMSB_OK;
  // chains stepped on their own since the last batch step lose the batch's
  // draws made ahead: start from each chain's own step counter again
  bool in_sync = bt->ahead > 0;
  for (size_t i = 0; i < bt->h.size() && in_sync; ++i)
    in_sync = bt->h[i]->ring_gen == bt->expect_gen[i] && bt->h[i]->step_count == bt->expect_step[i];
  for (ammsb_handle* h : bt->h) BK(cudaStreamSynchronize(h->stream));
  const int D = bt->block, R = 2 * D;
  const bool brief = brief_call(D, in_sync ? bt->ahead : 0, n_iters);
  uint32_t drawn = 0;  // iterations drawn by this call
  if (!in_sync) {
    for (size_t i = 0; i < bt->h.size(); ++i) {
      ammsb_handle* h = bt->h[i];
      ammsb_detail::invalidate_prefetch(h);
      bt->expect_gen[i] = h->ring_gen;
      int rc = ammsb_detail::point_draws(h, h->step_count, h->stream);
      if (rc) {
        bt->err = h->err;
        return rc;
      }
      BK(cudaStreamSynchronize(h->stream));
    }
    bt->slot = 0;
    BK(launch_sampling_chains(bt, 0, bt->stream));
    bt->ahead = D;
    drawn += (uint32_t)D;
  }
  bool forked = false;
  int64_t left = n_iters;
  while (left > 0) {  // as ammsb_step
    const int s = bt->slot, blk = s / D;
    const NextLaunch next = next_launch(D, s, bt->ahead, left, brief, true, false);
    const int n = next.n;
    int rc;
    if (next.whole) {
      rc = launch_graph(bt, next.both ? bt->graphL[blk] : bt->graphB[blk], [&] {
        cudaError_t e = launch_block_chains(bt, blk);
        return e == cudaSuccess && next.both ? launch_block_chains(bt, 1 - blk) : e;
      });
      drawn += (uint32_t)n;
    } else {
      if (next.fork) {
        BK(fork_draws_chains(bt, 1 - blk));
        forked = true;
        drawn += (uint32_t)D;
        bt->ahead += D;
      }
      int lg = 0;
      while ((1 << lg) < n) ++lg;
      rc = launch_graph(bt, bt->graphU[s][lg], [&] { return launch_updates_chains(bt, s, n); });
      bt->ahead -= n;
      if (forked && (s + n) % D == 0) {
        BK(cudaStreamWaitEvent(bt->stream, bt->ev_join, 0));
        forked = false;
      }
    }
    if (rc) return rc;
    bt->slot = (s + n) % R;
    left -= n;
  }
  if (forked) BK(cudaStreamWaitEvent(bt->stream, bt->ev_join, 0));
  BK(cudaEventRecord(bt->ev_done, bt->stream));
  for (size_t i = 0; i < bt->h.size(); ++i) {
    ammsb_handle* h = bt->h[i];
    BK(cudaStreamWaitEvent(h->stream, bt->ev_done, 0));  // later work on the chain's own stream
    h->step_count += (uint64_t)n_iters;
    h->dev_next += drawn;
    h->last = (bt->slot + R - 1) % R;
    bt->expect_step[i] = h->step_count;
  }
  BK(cudaStreamSynchronize(bt->stream));
  for (ammsb_handle* h : bt->h) {
    int rc = ammsb_detail::check_device_err(h);
    if (rc) {
      bt->err = h->err;
      return rc;
    }
  }
  return AMMSB_OK;
}

void* ammsb_batch_stream(ammsb_batch* bt) { return bt ? (void*)bt->stream : nullptr; }

}  // extern "C"
