// ammsb_internal.h -- the sampler handle and the helpers shared by the
// host-side translation units (ammsb_gpu.cu: one chain; ammsb_batch.cu:
// many chains per launch).  Not part of the C ABI.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <string>
#include <utility>
#include <vector>

#include "../../include/ammsb_gpu.h"
#include "ammsb_kernels.cuh"

using namespace ammsb;

// The draws of an iteration depend on its step alone, so a launch draws a
// block of iterations at once (ammsb_handle::block of them, a CTA of the minibatch kernel
// and a slice of the neighbour kernel's grid each) while the other block's
// iterations update the state; the ring holds both blocks' buffer sets.
constexpr int kMaxBlock = 16;
constexpr int kMaxRing = 2 * kMaxBlock;
// A ring of at most this many bytes takes the full block (16 sets of the
// 4,096-edge, 128-neighbour minibatch are 35 MB); larger buffer sets
// (random-edge over the whole training set, where an iteration lasts so long
// that its draws' launches do not show) take blocks of two, as does a ring for
// which the device has no room (block_with_room).
constexpr int64_t kRingBytes = 1ll << 30;

// Launches of the iteration that may start before the kernel ahead of them
// has finished (programmatic dependent launch): update_phi after the
// previous iteration's theta step, the commit after update_phi, the theta
// step after the commit.
enum : int { kPdlPhi = 1, kPdlCommit = 2, kPdlTheta = 4 };

struct KernelCfg {
  int lpn, vpl, split, npb;  // update_phi
  int ring;                  // wide rows: the shared-memory ring kernel
  int ring_stages;           // its ring depth
  int ring_few;              // iterations of few nodes take 16 warps per node
  int ring_grid;             // CTAs of the ring launch at most (0: one per node of its groups)
  int pdl;                   // programmatic dependent launches: kPdl* bits
  int ppx_lpn, ppx_vpl;      // perplexity
  int kq;                    // commit: 128-element pieces of a row per lane
};

// The minibatch's shape decides the commit kernel: a star (one source, as the
// default strategies draw) takes k_commit_star, with kStarChunk edges per
// summing warp at once where the minibatch gives a warp more than one (4,096
// edges over 1,024 summing warps: 13 us of an iteration with one edge at a time,
// 5 with four) and one where it does not (the shared memory of four would only
// keep CTAs off the SM).
constexpr int kStarChunk = 4;
inline int star_chunk(const Model& m) { return m.max_edges > 4 * m.nbb ? kStarChunk : 1; }

struct ammsb_handle {
  ammsb_options opt{};
  int device = 0;
  cudaStream_t stream = nullptr;  // the handle's stream: updates, perplexity, copies
  cudaStream_t side = nullptr;    // draws of the next iteration, overlapped with the update
  cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
  Model m{};
  DevGraph g{};
  Buffers b{};        // buffer set 0 and the shared state (slot_buffers gives the other sets)
  DevCounters* gc = nullptr;
  int block = 8;  // iterations per draws launch (half the ring)
  int slot = 0;   // ring slot of the next iteration
  // iterations from `slot` on whose draws are made or queued: none, or the
  // rest of slot's block and, past the block's first iteration, the other
  // block too
  int ahead = 0;
  uint32_t dev_next = 1;    // gc->next_step once the queued work is done
  uint64_t ring_gen = 0;    // raised whenever the ring's draws change hands
  int last = -1;            // buffer set of the last applied iteration
  KernelCfg cfg{};
  int64_t E = 0, H = 0, T = 0;
  int pi_bytes = 4;
  // device allocations
  std::vector<void*> allocs;
  int32_t* d_ha = nullptr;
  int32_t* d_hb = nullptr;
  uint8_t* d_hy = nullptr;
  float* d_ppx = nullptr;
  double* d_ppx_part = nullptr;
  float* d_read = nullptr;  // staging of get_rows, allocated with the first read that needs it
  PpxResult* d_ppx_res = nullptr;
  float* d_fed_phi_noise = nullptr;
  float* d_fed_theta_noise = nullptr;
  int32_t* d_err_init = nullptr;
  GammaTables* d_gamma = nullptr;
  int ncommit = 1;
  bool star = false;  // drawn minibatches are stars
  int nbr_blocks = 1;
  size_t phi_smem = 0, phi_smem_few = 0, nbr_smem = 0, mb_smem = 0;
  // host mirrors
  uint64_t step_count = 1;     // learner.cc:37
  uint64_t average_count = 1;  // learner.cc:30
  std::vector<double> ppx_history;
  bool state_ready = false;
  // captured iterations: whole blocks with the other block's draws made
  // alongside (one block, and both in turn), runs of 1, 2, 4, 8 updates inside
  // a block, and single iterations in the loop's order (pipeline off)
  cudaGraphExec_t graphB[2] = {}, graphL[2] = {};
  cudaGraphExec_t graphU[kMaxRing][4] = {};
  cudaGraphExec_t graphS[kMaxRing] = {};
  // run()'s per-phase timers (mcmc_sampler_stochastic.cc:93-102), printed
  // as PrintStats does (cc:185-198): wall time and ticks per timer
  struct Timer {
    double seconds = 0.0;
    uint64_t ticks = 0;
  };
  enum { kTOuter, kTPerplexity, kTMiniBatch, kTNodes, kTNeighbors, kTPhi, kTPi, kTBeta, kTimers };
  Timer timers[kTimers];
  bool timing = false;  // run() launches the timed captures below
  // the same with CUDA events between the phases: an event set per buffer
  // set for its update (before it and after each of its three phases), and
  // one for the draws launch that starts there (before it and after each of
  // its two kernels)
  cudaGraphExec_t graphBt[2] = {}, graphUt[kMaxRing] = {}, graphSt[kMaxRing] = {};
  cudaEvent_t ev_upd[kMaxRing][4] = {}, ev_drw[kMaxRing][3] = {};
  bool upd_pending[kMaxRing] = {}, drw_pending[kMaxRing] = {};  // event sets not read yet
  uint64_t evals_read = 0;       // edge evaluations counted into the timers' ticks
  // a sharded iteration in progress (ammsb_shard_*): the drawn buffer set
  // and the device arrays of its phases
  int shard_drawn = -1;
  int shard_phase = 0;  // 1 drawn, 2 owned rows updated, 3 committed
  int32_t* d_shard_idx = nullptr;  // max(max_nodes, max_edges) slot / edge indices
  double* d_shard_R = nullptr;     // K x 2 beta-gradient sums
  std::string err;
};

#define CK(call)                                                              \
  do {                                                                        \
    cudaError_t e_ = (call);                                                  \
    if (e_ != cudaSuccess) {                                                  \
      h->err = std::string(#call) + ": " + cudaGetErrorString(e_);            \
      return AMMSB_E_CUDA;                                                    \
    }                                                                         \
  } while (0)

// Shapes of the register-path update_phi kernel that are built: (lanes per
// node, 16-byte vectors per lane, sub-groups splitting the neighbours).  The
// lanes x vectors product is the K-tile a node's row is cut into; lanes x
// split is the number of threads (warps-per-node x 32) that work on a node.
#define AMMSB_PHI_REG_SHAPES(X)                                                         \
  X(1, 1, 1) X(2, 1, 1) X(4, 1, 1) X(8, 1, 1) X(16, 1, 1) X(32, 1, 1) X(32, 1, 2)       \
  X(32, 1, 4) X(32, 2, 1) X(32, 2, 2) X(32, 2, 4) X(32, 4, 1) X(32, 4, 2) X(32, 4, 4)   \
  X(32, 8, 1) X(32, 8, 2) X(32, 8, 4) X(16, 1, 2) X(8, 1, 2) X(8, 1, 4) X(16, 2, 1)     \
  X(8, 2, 1) X(8, 4, 1) X(4, 2, 1) X(4, 4, 1) X(4, 1, 8) X(2, 1, 8) X(1, 1, 8)

// Iterations with at most kRingFewNodes nodes (the link stratum) take the
// ring update_phi kernel's 16 warps per node.
constexpr int kRingFewNodes = 64;

// How the ring update_phi kernel is launched for rows whose four-warp group
// takes group_bytes of shared memory and whose 16-warp node few_bytes: four
// groups to the CTA and both kinds of iteration in one launch where that fits
// an SM's 227 KB, else a launch per kind.
struct RingPlan {
  size_t group_bytes, few_bytes;
  int groups;   // four-warp groups per CTA
  int few;      // most nodes that take 16 warps each (0: none do)
  bool single;  // one launch for both kinds
  size_t smem() const { return few ? std::max((size_t)groups * group_bytes, few_bytes) : groups * group_bytes; }
};
inline RingPlan ring_plan(const KernelCfg& c, size_t group_bytes, size_t few_bytes) {
  constexpr size_t kSmem = 227 * 1024;
  RingPlan r{group_bytes, 0, 1, 0, false};
  r.groups = (int)std::max<size_t>(1, std::min<size_t>(4, kSmem / group_bytes));
  if (c.ring_few && few_bytes <= 200 * 1024) r.few = kRingFewNodes, r.few_bytes = few_bytes;
  r.single = r.groups == 4;
  return r;
}

// Ring depths the ring update_phi kernel is built for.
#define AMMSB_PHI_RING_STAGES(X) X(3) X(4) X(6)

// Launches `k` on stream `s`; with `pdl` as a programmatic dependent launch
// (it may start once every CTA of the kernel ahead of it in the stream has
// triggered, and waits on the device before reading that kernel's results).
template <typename... P, typename... A>
inline cudaError_t launch_k(void (*k)(P...), int grid, int block, size_t smem, cudaStream_t s, bool pdl,
                     A&&... args) {
  cudaLaunchConfig_t lc{};
  lc.gridDim = dim3(grid);
  lc.blockDim = dim3(block);
  lc.dynamicSmemBytes = smem;
  lc.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  lc.attrs = at;
  lc.numAttrs = pdl ? 1 : 0;
  return cudaLaunchKernelEx(&lc, k, std::forward<A>(args)...);
}

namespace ammsb_detail {
// Raises a kernel's dynamic shared memory limit to at least `bytes` and
// never lowers it: the limit belongs to the kernel, not to a handle, and
// handles of different sizes share kernels.
template <typename F>
cudaError_t raise_smem_limit(F* kernel, size_t bytes) {
  static std::mutex mu;
  static std::map<std::pair<int, const void*>, size_t> set;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lock(mu);
  size_t& cur = set[std::make_pair(dev, reinterpret_cast<const void*>(kernel))];
  if (bytes <= cur) return cudaSuccess;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e == cudaSuccess) cur = bytes;
  return e;
}

// Reads the device error word of a handle (synchronises its stream).
int check_device_err(ammsb_handle* h);
// Drops draws made ahead of time: the next ones start from step_count.
void invalidate_prefetch(ammsb_handle* h);
// Points the device's next draws at `step` on stream s, unless queued work
// leaves it there.
int point_draws(ammsb_handle* h, uint64_t step, cudaStream_t s);
}  // namespace ammsb_detail
