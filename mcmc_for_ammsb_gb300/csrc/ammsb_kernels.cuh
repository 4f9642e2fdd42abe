// ammsb_kernels.cuh -- sm_103a kernels of one SG-MCMC iteration.
//
// Phase order of MCMCSamplerStochastic::run (mcmc_sampler_stochastic.cc
// :131-174), one kernel each, all reading the per-iteration scalars from
// DevState so the sequence replays as a CUDA graph:
//   k_sample_minibatch   Network::sample_mini_batch + nodes_in_batch
//   k_sample_neighbors   sample_neighbor_nodes (h:87-108) + y lookups
//   k_update_phi         update_phi (cc:269-313), fused with the noise draw
//                        and the normalisation pi_i = phi_i / sum(phi_i)
//                        into a staging buffer (Jacobi: pi is not touched)
//   k_commit_star        pi[nodes] = staged rows (cc:162-166) and the
//   k_commit_beta        per-edge update_beta gradient (cc:212-240) as a
//                        segmented block reduction: for minibatches of one
//                        source, and for any
//   k_theta              sum of block partials + SGRLD theta step + beta
//                        (cc:244-266), FP64
// The draws (the first two) depend on the step alone, so a launch of either
// makes those of eight iterations: one CTA per iteration's minibatch took 17 us
// of each of a 100,000-node chain's 20 us iterations; eight at once 4.
#pragma once
#include "ammsb_device.cuh"
#include "ammsb_gamma.cuh"
#include "ammsb_plan.h"

namespace ammsb {

// Upper bound of Model::nbb, the blocks of k_commit_beta that write beta
// gradient partials (k_theta reads them back, up to 36 per warp: four chains of 9).
#ifndef AMMSB_MAX_BETA_BLOCKS
#define AMMSB_MAX_BETA_BLOCKS 256
#endif
constexpr int kMaxBetaBlocks = AMMSB_MAX_BETA_BLOCKS;
// k_theta adds the partials in 31 chains of up to 9
constexpr int kThetaChains = 31, kThetaPerChain = 9;
static_assert(kMaxBetaBlocks <= kThetaChains * kThetaPerChain, "k_theta reads the partials in one pass");
constexpr int kThetaThreads = 256;
constexpr int kThetaPre = 10;  // doubles per k of theta_pre_block

struct Model {
  int32_t K;      // communities
  int32_t Kp;     // row stride in elements (K rounded up to 16 bytes)
  int64_t N;
  float alpha, epsilon;
  float Nn;       // N / num_node_sample, as the reference (cc:300)
  float eta0, eta1;
  double a, b, c; // step-size schedule
  uint32_t seed, chain;
  int32_t n_out;  // num_node_sample + 1 neighbours per node
  int32_t max_nodes, max_edges;
  int32_t mini_batch_size;
  int32_t strategy;
  float nonlink_scale, link_scale;
  int32_t nbb;    // beta partial blocks (at most kMaxBetaBlocks)
  int32_t nbr_set_cap;  // per-warp accepted-neighbour set capacity (power of two)
  int32_t max_source;   // sampler.max-source (link stratum)
  int32_t full_set;     // random-edge: the minibatch is the whole training set
  int64_t n_entries;    // 2E: entries of the symmetric CSR
  // the ring of minibatch buffer sets: element strides between consecutive
  // sets (set s of Buffers::nodes starts at s * slot_nodes, and so on), and
  // between the scratch areas of a draws launch's iterations
  int32_t ring;         // buffer sets
  int64_t slot_nodes, slot_edges, slot_nbr, slot_cand;
};

struct Buffers {
  void* pi;            // N x Kp, PiT
  float* phi;          // N x Kp
  float* stage;        // max_nodes x Kp: new pi rows of the minibatch nodes
  float* beta;         // K
  double* theta;       // K x 2
  int32_t* nodes;      // max_nodes
  int32_t* ea;         // max_edges: slot of first endpoint
  int32_t* eb;         // slot of second endpoint
  uint8_t* ey;         // y of each minibatch edge
  uint32_t* nbr;       // max_nodes x n_out: id | y << 31
  int32_t* cand;       // slot_cand: candidate scratch
  uint32_t* htab_key;  // minibatch dedup hash
  uint32_t* htab_idx;
  uint32_t hmask;
  float* beta_part;    // nbb x 2 x Kp
  double* theta_pre;   // kThetaPre x K: the theta step's parts that do not need the sums
  const float* fed_phi_noise;    // max_nodes x K or null
  const float* fed_theta_noise;  // K x 2 or null
  DevState* st;        // this buffer set's per-iteration scalars
  DevCounters* gc;     // sampler-wide counters
};

// Buffer set `slot` of the ring whose set 0 is b0, with scratch area j (a
// draws launch gives each of its iterations an area of its own).
__host__ __device__ __forceinline__ Buffers slot_buffers(const Model& m, const Buffers& b0, int slot,
                                                         int j = 0) {
  Buffers b = b0;
  b.nodes += slot * m.slot_nodes;
  b.ea += slot * m.slot_edges;
  b.eb += slot * m.slot_edges;
  b.ey += slot * m.slot_edges;
  b.nbr += slot * m.slot_nbr;
  b.st += slot;
  b.cand += j * m.slot_cand;
  if (b.htab_key) {
    b.htab_key += (int64_t)j * ((int64_t)b.hmask + 1);
    b.htab_idx += (int64_t)j * ((int64_t)b.hmask + 1);
  }
  return b;
}

// One chain of a multi-chain launch: its model, graph and buffer set 0 of its
// ring, plus the per-chain launch parameters of the single-chain kernels.  The
// launch has the blocks that each chain's own launch would have, one after the
// other, and a map from a block to its chain: with the largest chain's blocks
// for every chain (a grid of chains x blocks) most blocks of a batch of unequal
// chains started only to exit.
struct BlockOf {
  int32_t chain, block, blocks, pad;  // block `block` of the chain's `blocks`
};
struct ChainArgs {
  Model m;
  DevGraph g;
  Buffers b;
  int32_t ncommit;    // k_commit_beta: blocks of the commit part
  int32_t star;       // the commit is k_commit_star (one class of partials)
  int32_t smem_hash;  // k_sample_minibatch: the dedup hash fits shared memory
};

__device__ __forceinline__ uint32_t lanemask_lt() {
  uint32_t m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

// Mask of the aligned group of G lanes (G a power of two <= 32) holding
// `lane`.
template <int G>
__device__ __forceinline__ uint32_t group_mask(int lane) {
  if constexpr (G >= 32) {
    return 0xffffffffu;
  } else {
    return ((1u << G) - 1u) << ((lane / G) * G);
  }
}

// Exclusive prefix sum of per-thread counts over a 1024-thread block, in
// thread order; returns the position and sets *total.  Uses s_warp[33].
__device__ __forceinline__ int block_scan_count_1024(int v, int* s_warp, int* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int n = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += n;
  }
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    const int w = s_warp[lane];
    int winc = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int n = __shfl_up_sync(0xffffffffu, winc, o);
      if (lane >= o) winc += n;
    }
    s_warp[lane] = winc - w;
    if (lane == 31) s_warp[32] = winc;
  }
  __syncthreads();
  const int pos = s_warp[warp] + incl - v;
  *total = s_warp[32];
  __syncthreads();
  return pos;
}

// Exclusive prefix count of `flag` over a 1024-thread block, in thread
// order; returns the position and sets *total.  Uses s_warp[32].
__device__ __forceinline__ int block_scan_1024(bool flag, int* s_warp, int* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t bal = __ballot_sync(0xffffffffu, flag);
  const int in_warp = __popc(bal & lanemask_lt());
  if (lane == 0) s_warp[warp] = __popc(bal);
  __syncthreads();
  if (warp == 0) {
    int v = s_warp[lane];
    int incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int n = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += n;
    }
    s_warp[lane] = incl - v;  // exclusive
    if (lane == 31) s_warp[32] = incl;
  }
  __syncthreads();
  const int pos = s_warp[warp] + in_warp;
  *total = s_warp[32];
  __syncthreads();
  return pos;
}

// Open-addressing insert of key into (hkey, hidx): keeps the smallest
// position per key.  The table is never full (callers keep it at most half
// full), so the probe ends.
__device__ __forceinline__ void hash_insert_min(uint32_t* hkey, uint32_t* hidx, uint32_t hmask,
                                                uint32_t key, uint32_t pos) {
  uint32_t slot = hash32(key) & hmask;
  for (uint32_t probe = 0; probe <= hmask; ++probe) {
    const uint32_t prev = atomicCAS(hkey + slot, 0xffffffffu, key);
    if (prev == 0xffffffffu || prev == key) {
      atomicMin(hidx + slot, pos);
      return;
    }
    slot = (slot + 1) & hmask;
  }
}

// Value stored for key (0xffffffff when absent).
__device__ __forceinline__ uint32_t hash_find(const uint32_t* hkey, const uint32_t* hidx,
                                              uint32_t hmask, uint32_t key) {
  uint32_t slot = hash32(key) & hmask;
  for (uint32_t probe = 0; probe <= hmask; ++probe) {
    const uint32_t k = hkey[slot];
    if (k == key) return hidx[slot];
    if (k == 0xffffffffu) return 0xffffffffu;
    slot = (slot + 1) & hmask;
  }
  return 0xffffffffu;
}

// Row of entry q of the CSR: the last v with row_ptr[v] <= q.
__device__ __forceinline__ int32_t csr_row_of(const int64_t* row_ptr, int64_t n, int64_t q) {
  int64_t lo = 0, hi = n;
  while (hi - lo > 1) {
    const int64_t mid = (lo + hi) >> 1;
    if (__ldg(row_ptr + mid) <= q) lo = mid; else hi = mid;
  }
  return (int32_t)lo;
}

// Node numbering of a general edge list: ea/eb hold the vertex ids of
// `count` edges; the nodes are numbered by first appearance over (a0, b0,
// a1, b1, ...), written to nodes[], and ea/eb are rewritten as slots.
// Returns the node count (or -1 past max_nodes).  Block-wide; uses the
// dedup hash (reset here) and s_warp.
static __device__ int assign_node_slots(const Buffers& b, int count, int max_nodes, uint32_t* hkey,
                                 uint32_t* hidx, int* s_warp) {
  const int tid = threadIdx.x;
  for (uint32_t s = tid; s <= b.hmask; s += blockDim.x) {
    hkey[s] = 0xffffffffu;
    hidx[s] = 0xffffffffu;
  }
  __syncthreads();
  const int np = 2 * count;
  for (int p = tid; p < np; p += blockDim.x) {
    const uint32_t x = (uint32_t)((p & 1) ? b.eb[p >> 1] : b.ea[p >> 1]);
    hash_insert_min(hkey, hidx, b.hmask, x, (uint32_t)p);
  }
  __syncthreads();
  int n = 0;
  for (int base = 0; base < np; base += blockDim.x) {
    const int p = base + tid;
    bool first = false;
    uint32_t x = 0;
    if (p < np) {
      x = (uint32_t)((p & 1) ? b.eb[p >> 1] : b.ea[p >> 1]);
      first = hash_find(hkey, hidx, b.hmask, x) == (uint32_t)p;
    }
    int total;
    const int pos = block_scan_1024(first, s_warp, &total);
    if (first && n + pos < max_nodes) b.nodes[n + pos] = (int32_t)x;
    n += total;
  }
  if (n > max_nodes) return -1;
  __syncthreads();
  // the hash now maps vertex -> slot
  for (int s = tid; s < n; s += blockDim.x) {
    const uint32_t x = (uint32_t)b.nodes[s];
    uint32_t slot = hash32(x) & b.hmask;
    for (uint32_t probe = 0; probe <= b.hmask; ++probe) {
      if (hkey[slot] == x) {
        hidx[slot] = (uint32_t)s;
        break;
      }
      slot = (slot + 1) & b.hmask;
    }
  }
  __syncthreads();
  for (int e = tid; e < count; e += blockDim.x) {
    b.ea[e] = (int32_t)hash_find(hkey, hidx, b.hmask, (uint32_t)b.ea[e]);
    b.eb[e] = (int32_t)hash_find(hkey, hidx, b.hmask, (uint32_t)b.eb[e]);
  }
  __syncthreads();
  return n;
}

// ---------------------------------------------------------------------------
// k_sample_minibatch: one 1024-thread CTA per iteration drawn (CTA j draws
// iteration next_step + j into buffer set (s0 + j) % ring; the draws depend on
// the step alone, so a launch takes as many iterations as half the ring
// holds).  Stratified random node
// (network.cc:410-421): flag = randint(0,1); non-link stratum
// (network.cc:274-349): source v and the first m valid new partners u in
// candidate order (u != v, (v,u) not an edge, not held-out, not test); link
// stratum (network.cc:355-407, max-source 1): all training edges of a random
// v, redrawn while empty.  Candidates are examined in rounds of
// need = m - count; within a round the first occurrence of each u wins
// (atomicMin of its index in a hash), then an ordered block scan appends
// them -- exactly the sequential scan of the oracle.
// ---------------------------------------------------------------------------
static __device__ __forceinline__ void sample_minibatch_body(const Model& m, const DevGraph& g,
                                                             const Buffers& b, int j, int smem_hash) {
  extern __shared__ uint32_t s_htab[];  // dedup hash in shared memory when it fits
  constexpr int kRowCap = 2048;         // the source's row, staged when it fits
  constexpr int kExclCap = 512;         // and its held-out and test partners
  __shared__ int32_t s_row[kRowCap], s_xrow[kExclCap];
  __shared__ int s_warp[33];
  __shared__ int s_flag, s_count, s_nodes;
  __shared__ uint32_t s_step;
  __shared__ int32_t s_v;
  __shared__ int s_brk, s_dup;
  const int tid = threadIdx.x;
  const Stream rs{m.seed, m.chain};
  if (tid == 0) {
    const uint32_t step = b.gc->next_step + (uint32_t)j;
    b.st->step = step;
    int flag;
    if (m.strategy == 0)
      flag = (int)uniform_below(rs.draw_u64(kTagMbFlag, 0, step, 0), 2ull);
    else if (m.strategy == 3)
      flag = 2;  // random-edge
    else
      flag = (m.strategy == 1) ? 1 : 0;
    s_flag = flag;
    s_step = step;
    s_count = 0;
    s_nodes = 0;
  }
  __syncthreads();
  const uint32_t step = s_step;
  const int flag = s_flag;
  int err = 0;
  int rounds = 0;
  if (flag == 0) {
    const int mb = m.mini_batch_size;
    const int32_t v = (int32_t)uniform_below(rs.draw_u64(kTagMbNode, 0, step, 0), (uint64_t)g.n);
    uint32_t* hkey = smem_hash ? s_htab : b.htab_key;
    uint32_t* hidx = smem_hash ? s_htab + (b.hmask + 1) : b.htab_idx;
    for (uint32_t s = tid; s <= b.hmask; s += blockDim.x) {
      hkey[s] = 0xffffffffu;
      hidx[s] = 0xffffffffu;
    }
    if (mb > m.max_edges || mb + 1 > m.max_nodes) err |= kErrCapacity;
    if (tid == 0) b.nodes[0] = v;
    const StagedRow links = stage_row(g.col, g.row_ptr[v], g.row_ptr[v + 1], s_row, kRowCap, tid, blockDim.x);
    const StagedRow excl = stage_row(g.xcol, g.xrow[v], g.xrow[v + 1], s_xrow, kExclCap, tid, blockDim.x);
    __syncthreads();
    int count = 0;
    uint64_t t = 0;
    // the spec scans candidates t = 0, 1, ... until mb are kept, giving up
    // at `cap`; a round examines R >= need of them in parallel and keeps the
    // first new valid ones, in order, up to mb.  R (nonlink_round) follows the
    // acceptance of the rounds so far: a round's cost grows with R
    // (a first round of up to 4,096 whatever the need took the 100k-node
    // workload's non-link minibatch from 16 to 44 us), and small populations
    // with many repeats still finish in two or three rounds.
    const uint64_t cap = 64ull * (uint64_t)mb + 4096ull;
    const int half = (int)((b.hmask + 1u) / 2u);
    int64_t seen = 0, kept = 0;  // candidates examined and kept so far
    while (!err && count < mb) {
      const int need = mb - count;
      if (t >= cap) {
        err |= kErrMinibatchCap;
        break;
      }
      const int R = (int)min((uint64_t)nonlink_round(need, count, half, seen, kept), cap - t);
      const int count0 = count;
      // pass A: validity and first-occurrence index per value; both of the
      // source's rows are in shared memory
      for (int c = tid; c < R; c += blockDim.x) {
        const int32_t u = (int32_t)uniform_below(rs.draw_u64(kTagMbCand, 0, step, t + (uint64_t)c),
                                                 (uint64_t)g.n);
        const bool ok = u != v && !links.contains(u) && !excl.contains(u);
        b.cand[c] = ok ? u : -1;
        if (ok) hash_insert_min(hkey, hidx, b.hmask, (uint32_t)u, (uint32_t)(t + (uint64_t)c));
      }
      __syncthreads();
      // pass B: ordered compaction of first occurrences, one block scan per
      // chunk of up to G * 1,024 (thread-local counts of its g consecutive
      // candidates, g the fewest per thread that cover the chunk); count is
      // block-uniform, so every thread leaves the loop together at mb
      constexpr int G = 4;
      const int chunk = G * (int)blockDim.x;
      for (int c0 = 0; c0 < R && count < mb; c0 += chunk) {
        const int n = min(R - c0, chunk);
        const int gper = (n + (int)blockDim.x - 1) / (int)blockDim.x;
        int32_t u[G];
        bool acc[G];
        int mine = 0;
#pragma unroll
        for (int j = 0; j < G; ++j) {
          const int c = c0 + gper * tid + j;
          u[j] = -1;
          acc[j] = false;
          if (j < gper && c < c0 + n) {
            u[j] = b.cand[c];
            if (u[j] >= 0)
              acc[j] = hash_find(hkey, hidx, b.hmask, (uint32_t)u[j]) == (uint32_t)(t + (uint64_t)c);
          }
          mine += acc[j] ? 1 : 0;
        }
        int total;
        int pos = block_scan_count_1024(mine, s_warp, &total);
#pragma unroll
        for (int j = 0; j < G; ++j) {
          if (acc[j]) {
            const int e = count + pos;
            if (e < mb) {
              b.nodes[e + 1] = u[j];
              b.ea[e] = 0;
              b.eb[e] = e + 1;
              b.ey[e] = 0;
            }
            ++pos;
          }
        }
        count = min(count + total, mb);
      }
      t += (uint64_t)R;
      seen += R;
      kept += count - count0;
      ++rounds;
      __syncthreads();
    }
    if (tid == 0) {
      b.st->scale = m.nonlink_scale;
      s_count = count;
      s_nodes = count + 1;
    }
  } else if (flag == 2) {
    // random_edge_sampling (network.cc:237-268): m distinct training edges,
    // candidates = entries of the symmetric CSR (each edge twice, as the
    // reference's linked_edges), kept when a < b and not held-out/test; the
    // whole training set when m reaches it (network.cc:215-234)
    const int mb = m.mini_batch_size;
    uint32_t* hkey = smem_hash ? s_htab : b.htab_key;
    uint32_t* hidx = smem_hash ? s_htab + (b.hmask + 1) : b.htab_idx;
    int count = 0;
    if (m.full_set) {
      for (int64_t base = 0; base < m.n_entries && !err; base += blockDim.x) {
        const int64_t q = base + tid;
        bool acc = false;
        int32_t a = 0, c = 0;
        if (q < m.n_entries) {
          a = csr_row_of(g.row_ptr, g.n, q);
          c = g.col[q];
          acc = a < c && !is_excluded(g, a, c);
        }
        int total;
        const int pos = block_scan_1024(acc, s_warp, &total);
        if (acc && count + pos < m.max_edges) {
          b.ea[count + pos] = a;
          b.eb[count + pos] = c;
          b.ey[count + pos] = 1;
        }
        count += total;
        if (count > m.max_edges) err |= kErrCapacity;
      }
    } else {
      for (uint32_t sl = tid; sl <= b.hmask; sl += blockDim.x) {
        hkey[sl] = 0xffffffffu;
        hidx[sl] = 0xffffffffu;
      }
      if (mb > m.max_edges) err |= kErrCapacity;
      __syncthreads();
      uint64_t t = 0;
      const uint64_t cap = 64ull * (uint64_t)mb + 4096ull;
      const int half = (int)((b.hmask + 1u) / 2u);
      while (!err && count < mb) {
        const int need = mb - count;
        if (t >= cap) {
          err |= kErrMinibatchCap;
          break;
        }
        const int R = (int)min((uint64_t)edge_round(need, count, half), cap - t);
        for (int c = tid; c < R; c += blockDim.x) {
          const int64_t q = (int64_t)uniform_below(rs.draw_u64(kTagMbCand, 0, step, t + (uint64_t)c),
                                                   (uint64_t)m.n_entries);
          const int32_t a = csr_row_of(g.row_ptr, g.n, q), bb = g.col[q];
          const bool ok = a < bb && !is_excluded(g, a, bb);
          b.cand[c] = ok ? (int32_t)q : -1;
          if (ok) hash_insert_min(hkey, hidx, b.hmask, (uint32_t)q, (uint32_t)(t + (uint64_t)c));
        }
        __syncthreads();
        for (int base = 0; base < R && count < mb; base += blockDim.x) {
          const int c = base + tid;
          int32_t q = -1;
          bool acc = false;
          if (c < R) {
            q = b.cand[c];
            acc = q >= 0 && hash_find(hkey, hidx, b.hmask, (uint32_t)q) == (uint32_t)(t + (uint64_t)c);
          }
          int total;
          const int pos = block_scan_1024(acc, s_warp, &total);
          if (acc && count + pos < mb) {
            b.ea[count + pos] = csr_row_of(g.row_ptr, g.n, q);
            b.eb[count + pos] = g.col[q];
            b.ey[count + pos] = 1;
          }
          count = min(count + total, mb);
        }
        t += (uint64_t)R;
        ++rounds;
        __syncthreads();
      }
    }
    int n = 0;
    if (!err) {
      n = assign_node_slots(b, count, m.max_nodes, hkey, hidx, s_warp);
      if (n < 0) err |= kErrCapacity;
    }
    if (tid == 0) {
      b.st->scale = count > 0 ? (float)((double)(m.N - 1) * (double)m.N / 2.0 / (double)count) : 0.f;
      s_count = count;
      s_nodes = n;
    }
  } else if (m.max_source > 1) {
    // stratified_random_node_sampling_links with sampler.max-source > 1
    // (network.cc:355-407): up to S sources per attempt (draw a*S + s); from
    // the second on, one whose degree would pass m ends the attempt; each
    // source adds its training edges once (an edge to an earlier source was
    // added from it; a repeated source adds none); redrawn while empty
    const int mb = m.mini_batch_size, S = m.max_source;
    uint32_t* hkey = smem_hash ? s_htab : b.htab_key;
    uint32_t* hidx = smem_hash ? s_htab + (b.hmask + 1) : b.htab_idx;
    int32_t* s_src = s_row;  // the attempt's sources (S <= kRowCap)
    int count = 0;
    for (int attempt = 0; attempt < 4096 && count == 0 && !err; ++attempt) {
      count = 0;
      for (int sidx = 0; sidx < S && !err; ++sidx) {
        if (tid == 0) {
          const int32_t v = (int32_t)uniform_below(
              rs.draw_u64(kTagMbNode, 0, step, (uint64_t)attempt * (uint64_t)S + (uint64_t)sidx),
              (uint64_t)g.n);
          const int64_t deg = g.row_ptr[v + 1] - g.row_ptr[v];
          int dup = 0;
          for (int r = 0; r < sidx; ++r) dup |= (s_src[r] == v);
          s_brk = (sidx > 0 && (int64_t)count + deg > (int64_t)mb) ? 1 : 0;
          s_dup = dup;
          s_v = v;
          if (!s_brk) s_src[sidx] = v;
        }
        __syncthreads();
        const int32_t v = s_v;
        const int brk = s_brk, dup = s_dup;
        __syncthreads();
        if (brk) break;
        if (dup) continue;
        const int64_t r0 = g.row_ptr[v];
        const int deg = (int)(g.row_ptr[v + 1] - r0);
        for (int base = 0; base < deg; base += blockDim.x) {
          const int q = base + tid;
          int32_t u = -1;
          bool acc = false;
          if (q < deg) {
            u = g.col[r0 + q];
            acc = !is_excluded(g, v, u);
            for (int r = 0; r < sidx && acc; ++r) acc = (s_src[r] != u);
          }
          int total;
          const int pos = block_scan_1024(acc, s_warp, &total);
          if (acc && count + pos < m.max_edges) {
            b.ea[count + pos] = v;
            b.eb[count + pos] = u;
            b.ey[count + pos] = 1;
          }
          count += total;
          if (count > m.max_edges) err |= kErrCapacity;
        }
      }
      rounds = attempt + 1;
    }
    if (count == 0 && !err) err |= kErrMinibatchCap;
    int n = 0;
    if (!err) {
      n = assign_node_slots(b, count, m.max_nodes, hkey, hidx, s_warp);
      if (n < 0) err |= kErrCapacity;
    }
    if (tid == 0) {
      b.st->scale = count > 0 ? (float)(m.n_entries / 2) / (float)count : 0.f;
      s_count = count;
      s_nodes = n;
    }
  } else {
    int count = 0;
    for (int attempt = 0; attempt < 4096 && count == 0 && !err; ++attempt) {
      const int32_t v =
          (int32_t)uniform_below(rs.draw_u64(kTagMbNode, 0, step, (uint64_t)attempt), (uint64_t)g.n);
      const int64_t r0 = g.row_ptr[v], deg = g.row_ptr[v + 1] - r0;
      if (deg > m.max_edges || deg + 1 > m.max_nodes) {
        err |= kErrCapacity;
        break;
      }
      const int64_t x0 = g.xrow[v], x1 = g.xrow[v + 1];
      for (int64_t base = 0; base < deg; base += blockDim.x) {
        const int64_t q = base + tid;
        int32_t u = -1;
        bool acc = false;
        if (q < deg) {
          u = g.col[r0 + q];
          acc = !span_contains(g.xcol, x0, x1, u);
        }
        int total;
        const int pos = block_scan_1024(acc, s_warp, &total);
        if (acc) {
          const int e = count + pos;
          b.nodes[e + 1] = u;
          b.ea[e] = 0;
          b.eb[e] = e + 1;
          b.ey[e] = 1;
        }
        count += total;
      }
      if (count > 0 && tid == 0) b.nodes[0] = v;
      rounds = attempt + 1;
    }
    if (count == 0 && !err) err |= kErrMinibatchCap;
    if (tid == 0) {
      b.st->scale = m.link_scale;
      s_count = count;
      s_nodes = count + 1;
    }
  }
  __syncthreads();
  if (tid == 0) {
    b.st->flag = flag;
    b.st->n_edges = err ? 0 : s_count;
    b.st->n_nodes = err ? 0 : s_nodes;
    b.st->rounds = rounds;
    b.st->err = err;
  }
}
static __global__ void __launch_bounds__(1024) k_sample_minibatch(Model m, DevGraph g, Buffers b0, int s0,
                                                                  int smem_hash) {
  const int j = blockIdx.x;
  sample_minibatch_body(m, g, slot_buffers(m, b0, (s0 + j) % m.ring, j), j, smem_hash);
}
// a CTA per iteration (blockIdx.x) and chain (blockIdx.y)
static __global__ void __launch_bounds__(1024) k_sample_minibatch_chains(const ChainArgs* __restrict__ c,
                                                                         int s0) {
  const ChainArgs& a = c[blockIdx.y];
  const int j = blockIdx.x;
  sample_minibatch_body(a.m, a.g, slot_buffers(a.m, a.b, s0 + j, j), j, a.smem_hash);
}

// ---------------------------------------------------------------------------
// k_sample_neighbors: one warp per minibatch node of iteration j of a draws
// launch (the grid's last dimension).  n_out distinct ids j,
// j != i, (i,j) neither held-out nor test (h:87-108); 32 candidates per
// round, the first valid new ones in candidate order are kept; y_ij is the
// graph membership the update needs (cc:279-283).
// ---------------------------------------------------------------------------
template <int WARPS>
__device__ __forceinline__ void sample_neighbors_body(const Model& m, const DevGraph& g, const Buffers& b,
                                                      int j0, int count0, int block, int blocks) {
  // per warp: a set of the ids accepted so far (open addressing, capacity a
  // power of two >= 2 n_out, -1 empty) in dynamic shared memory
  extern __shared__ int32_t s_sets[];
  constexpr int kRowCap = 256;  // the node's own row, staged when it fits
  constexpr int kExclCap = 32;  // and its held-out and test partners
  __shared__ int32_t s_rows[WARPS][kRowCap], s_xrows[WARPS][kExclCap];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t smask = (uint32_t)m.nbr_set_cap - 1u;
  int32_t* set = s_sets + (size_t)warp * m.nbr_set_cap;
  const int n_nodes = b.st->n_nodes;
  const uint32_t step = b.st->step;
  const Stream rs{m.seed, m.chain};
  const uint64_t cap = 64ull * (uint64_t)m.n_out + 4096ull;
  // eps_t of the iteration (get_eps_t, cc:143; read by the update kernels alone): an
  // FP64 power, computed by the grid's last warp, which the launch leaves
  // without a node (the grid has a warp more than the nodes) and which no
  // other warp waits for; in the single-CTA minibatch kernel its latency
  // delayed every block barrier (2.8 us of each minibatch)
  if (block == blocks - 1 && warp == WARPS - 1 && lane == 0) {
    b.st->eps = eps_schedule(m.a, m.b, m.c, step);
    // iteration 0 of the launch moves the counter past its `count0`
    // iterations: the minibatch launch ahead has read it, nothing here does
    if (j0 == 0) b.gc->next_step = step + (uint32_t)count0;
  }
  for (int slot = block * WARPS + warp; slot < n_nodes; slot += blocks * WARPS) {
    const int32_t i = b.nodes[slot];
    const int64_t r0 = g.row_ptr[i], r1 = g.row_ptr[i + 1], x0 = g.xrow[i], x1 = g.xrow[i + 1];
    const StagedRow links = stage_row(g.col, r0, r1, s_rows[warp], kRowCap, lane, 32);
    const StagedRow excl = stage_row(g.xcol, x0, x1, s_xrows[warp], kExclCap, lane, 32);
    for (uint32_t q = lane; q <= smask; q += 32) set[q] = -1;
    __syncwarp();
    int count = 0;
    uint64_t t = 0;
    int32_t j0 = 0, j1 = 0;  // candidates 2 lane and 2 lane + 1 of a pair of rounds
    while (count < m.n_out) {
      if (t >= cap) {
        if (lane == 0) atomicOr(&b.st->err, kErrNeighborCap);
        break;
      }
      // a Philox block holds two draws: the lanes form 64 candidates with a
      // block each, and every second round takes the upper half
      const int half = (int)(t >> 5) & 1;
      if (half == 0) {
        const U32x4 o = rs.block(kTagNbr, (uint32_t)i, step, (t >> 1) + lane);
        j0 = (int32_t)uniform_below((uint64_t)o.x | ((uint64_t)o.y << 32), (uint64_t)g.n);
        j1 = (int32_t)uniform_below((uint64_t)o.z | ((uint64_t)o.w << 32), (uint64_t)g.n);
      }
      const int from = half * 16 + (lane >> 1);
      const int32_t ja = __shfl_sync(0xffffffffu, j0, from), jb = __shfl_sync(0xffffffffu, j1, from);
      const int32_t j = (lane & 1) ? jb : ja;
      bool ok = (j != i) && !(excl.deg > 0 && excl.contains(j));
      if (ok) {  // already accepted in an earlier round?
        uint32_t h = hash32((uint32_t)j) & smask;
        for (uint32_t probe = 0; probe <= smask; ++probe) {
          const int32_t e = set[h];
          if (e == j) {
            ok = false;
            break;
          }
          if (e < 0) break;
          h = (h + 1) & smask;
        }
      }
      const uint32_t peers = __match_any_sync(0xffffffffu, j);
      ok = ok && ((peers & lanemask_lt()) == 0);
      const uint32_t bal = __ballot_sync(0xffffffffu, ok);
      const int pos = __popc(bal & lanemask_lt());
      const int need = m.n_out - count;
      __syncwarp();  // every lane has probed the set before it grows
      if (ok && pos < need) {
        const int idx = count + pos;
        uint32_t h = hash32((uint32_t)j) & smask;
        for (uint32_t probe = 0; probe <= smask; ++probe) {
          if (atomicCAS(set + h, -1, j) == -1) break;
          h = (h + 1) & smask;
        }
        const uint32_t y = links.contains(j) ? 1u : 0u;
        b.nbr[(int64_t)slot * m.n_out + idx] = (uint32_t)j | (y << 31);
      }
      count += min(__popc(bal), need);
      t += 32;
      __syncwarp();
    }
    __syncwarp();  // the rows and the set are reused by the warp's next node
  }
}
template <int WARPS>
__global__ void __launch_bounds__(WARPS * 32) k_sample_neighbors(Model m, DevGraph g, Buffers b0, int s0) {
  const int j = blockIdx.y;
  sample_neighbors_body<WARPS>(m, g, slot_buffers(m, b0, (s0 + j) % m.ring), j, (int)gridDim.y, blockIdx.x,
                               gridDim.x);
}
template <int WARPS>
__global__ void __launch_bounds__(WARPS * 32) k_sample_neighbors_chains(const ChainArgs* __restrict__ c,
                                                                      const BlockOf* __restrict__ map, int s0) {
  const BlockOf o = map[blockIdx.x];
  const ChainArgs& a = c[o.chain];
  const int j = blockIdx.y;
  sample_neighbors_body<WARPS>(a.m, a.g, slot_buffers(a.m, a.b, s0 + j), j, (int)gridDim.y, o.block, o.blocks);
}

// ---------------------------------------------------------------------------
// k_update_phi: update_phi (cc:269-313) for NPB minibatch nodes per CTA,
// SPLIT sub-groups of LPN lanes per node, each lane holding VPL 16-byte
// vectors of a pi row.  Sub-group s takes neighbours s, s+SPLIT, ...
//
// A minibatch of narrow rows is too small to hide latency by occupancy (500
// nodes are three warps per SM), so the chain of each node is kept short: U
// rows' warp sums side by side, the next U rows and the words after them in
// flight, and all that beta is not needed for -- ids, words, first rows, phi and
// its sum, the normals -- before the wait for the theta step.  With one row at a
// time and no early start, an iteration of the 5k-node workload (K = 32 FP32)
// took 15.1 us, now 9.0.
//
// Algebra (exact rewrite of the reference's per-k loop).  With
// pi_ik = phi_ik / S, sigma_j = +1 for y=1 else -1, e_j = y ? eps : 1-eps,
// bk = beta_k - epsilon and w_k = pi_ik * bk:
//   probs_jk = pi_ik (sigma_j bk pi_jk + e_j)
//   P_j      = sum_k probs_jk = sigma_j D_j + e_j s_i,
//              D_j = sum_k w_k pi_jk,  s_i = sum_k pi_ik
//   grad_k   = sum_j probs_jk / (P_j phi_ik) - 1/S
//            = (bk A_k + B) / S,  A_k = sum_j (sigma_j / P_j) pi_jk,
//              B = sum_j (e_j (1 - s_i) - sigma_j D_j) / P_j
// so each neighbour row costs two FMAs per element (D_j, then A_k).
// Epilogue: phi_ik <- |phi + eps/2 (alpha - phi + Nn grad) + sqrt(eps phi)
// noise|, clamped to 1e-24; the new row is normalised into the staging
// buffer (pi itself is written after all nodes, by k_commit_beta).
// ---------------------------------------------------------------------------
template <typename PiT, int LPN, int VPL, int SPLIT, int NPB>
__device__ __forceinline__ void update_phi_body(const Model& m, const Buffers& b, int block, int blocks) {
  using TR = PiTraits<PiT>;
  constexpr int EV = TR::kPerVec;
  constexpr int EPL = VPL * EV;
  constexpr int TPN = SPLIT * LPN;
  // rows a sub-group takes together (their dot products' sums overlap), with
  // the next ones in flight: as many as keep a lane at 8 floats of them
  constexpr int U = EPL <= 4 ? 4 : EPL <= 8 ? 2 : 1;
  // a thread's elements of the epilogue: each sub-group covers the whole row,
  // Kp <= LPN * EPL = TPN * EPL / SPLIT; few enough of them draw their normals
  // ahead of the rows
  constexpr int NQ = (EPL + SPLIT - 1) / SPLIT;
  constexpr bool kEarlyNoise = NQ <= 4;
  extern __shared__ float s_dyn[];
  float* s_A = s_dyn;                               // NPB x SPLIT x Kp
  float* s_B = s_A + (size_t)NPB * SPLIT * m.Kp;    // NPB x SPLIT
  float* s_red = s_B + NPB * SPLIT;                 // NPB x (TPN/32 or 1)

  const int tid = threadIdx.x;
  const int ln = tid / TPN;          // node within the CTA
  const int r = tid - ln * TPN;      // thread within the node
  const int sg = r / LPN;            // sub-group
  const int l = r - sg * LPN;        // lane within the sub-group
  const int warp_lane = tid & 31;
  const uint32_t gmask = group_mask<LPN>(warp_lane);
  const int n_nodes = b.st->n_nodes;
  const uint32_t step = b.st->step;
  const float eps_t = b.st->eps;
  const int Kp = m.Kp, K = m.K;
  const int nvec = Kp / EV;
  const PiT* __restrict__ pi = reinterpret_cast<const PiT*>(b.pi);
  const Stream rs{m.seed, m.chain};

  const int first = block * NPB;
  for (int base = first; base < n_nodes; base += blocks * NPB) {
    const int slot = base + ln;
    const bool active = slot < n_nodes;
    float S = 0.f, s_i = 0.f, Bsum = 0.f;
    int32_t i = 0;
    float w[EPL], A[EPL], noise[NQ];
    const uint32_t* nb = b.nbr + (int64_t)slot * m.n_out;
    uint32_t word[U], word_n[U];  // neighbour words of a chunk and the next
    uint4 cur[U][VPL], nxt[U][VPL];
    auto load_words = [&](int q, uint32_t* out) {
#pragma unroll
      for (int u = 0; u < U; ++u) out[u] = q + u * SPLIT < m.n_out ? nb[q + u * SPLIT] : 0u;
    };
    auto load_rows = [&](int q, const uint32_t* words, uint4 (*out)[VPL]) {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const bool on = q + u * SPLIT < m.n_out;
        const PiT* row = pi + (int64_t)(words[u] & 0x7fffffffu) * Kp;
#pragma unroll
        for (int v = 0; v < VPL; ++v) {
          const int vi = l + LPN * v;
          out[u][v] = (on && vi < nvec) ? ldg_nc_v4(row + vi * EV) : make_uint4(0, 0, 0, 0);
        }
      }
    };
    auto noise_at = [&](int k) {
      return b.fed_phi_noise ? b.fed_phi_noise[(int64_t)slot * K + k]
                             : normal_draw(rs, kTagPhiNoise, (uint32_t)i, step, (uint64_t)k);
    };
    if (active) {
      i = b.nodes[slot];
      load_words(sg, word);
      load_words(sg + U * SPLIT, word_n);
      const float* phi_i = b.phi + (int64_t)i * Kp;
      load_rows(sg, word, cur);
      // phi row -> S
#pragma unroll
      for (int v = 0; v < VPL; ++v) {
        const int vi = l + LPN * v;
#pragma unroll
        for (int e = 0; e < EV; ++e) {
          const int k = vi * EV + e;
          w[v * EV + e] = (vi < nvec) ? phi_i[k] : 0.f;
          S += w[v * EV + e];
        }
      }
#pragma unroll
      for (int o = LPN / 2; o > 0; o >>= 1) S += __shfl_xor_sync(gmask, S, o);
      if constexpr (kEarlyNoise) {
#pragma unroll
        for (int qq = 0; qq < NQ; ++qq) noise[qq] = r + TPN * qq < K ? noise_at(r + TPN * qq) : 0.f;
      }
    }
    // beta, read from here on, is written by the theta step ahead of this
    // launch; everything read before was complete before that step started
    grid_dependency_wait();
    grid_launch_dependents();
    if (active) {
      // pi_i = phi_i / S, s_i = sum pi_i, w = pi_i * (beta - epsilon)
#pragma unroll
      for (int v = 0; v < VPL; ++v) {
        const int vi = l + LPN * v;
#pragma unroll
        for (int e = 0; e < EV; ++e) {
          const int k = vi * EV + e;
          const float p = __fdiv_rn(w[v * EV + e], S);
          s_i += p;
          const float bk = (vi < nvec && k < K) ? (b.beta[k] - m.epsilon) : 0.f;
          w[v * EV + e] = p * bk;
          A[v * EV + e] = 0.f;
        }
      }
#pragma unroll
      for (int o = LPN / 2; o > 0; o >>= 1) s_i += __shfl_xor_sync(gmask, s_i, o);
      const float one_m_si = 1.0f - s_i;

      // neighbour loop, U rows at a time, the next U prefetched
      for (int q = sg; q < m.n_out; q += U * SPLIT) {
        const int qn = q + U * SPLIT;
        uint32_t word_f[U];
        load_words(qn + U * SPLIT, word_f);
        load_rows(qn, word_n, nxt);
        float x[U][EPL], D[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
#pragma unroll
          for (int v = 0; v < VPL; ++v) TR::unpack(cur[u][v], x[u] + v * EV);
          float d4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
          for (int e = 0; e < EPL; ++e) d4[e & 3] = fmaf(w[e], x[u][e], d4[e & 3]);
          D[u] = (d4[0] + d4[1]) + (d4[2] + d4[3]);
        }
#pragma unroll
        for (int o = LPN / 2; o > 0; o >>= 1)
#pragma unroll
          for (int u = 0; u < U; ++u) D[u] += __shfl_xor_sync(gmask, D[u], o);
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (u > 0 && q + u * SPLIT >= m.n_out) break;
          const bool y = (word[u] >> 31) != 0;
          const float sg_ = y ? 1.f : -1.f;
          const float ej = y ? m.epsilon : 1.0f - m.epsilon;
          const float P = fmaf(sg_, D[u], ej * s_i);
          const float invP = rcp_approx(P);
          const float cj = sg_ * invP;
          Bsum += (ej * one_m_si - sg_ * D[u]) * invP;
#pragma unroll
          for (int e = 0; e < EPL; ++e) A[e] = fmaf(cj, x[u][e], A[e]);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          word[u] = word_n[u];
          word_n[u] = word_f[u];
#pragma unroll
          for (int v = 0; v < VPL; ++v) cur[u][v] = nxt[u][v];
        }
      }
      // publish A and B of this sub-group
      float* sA = s_A + ((size_t)ln * SPLIT + sg) * Kp;
#pragma unroll
      for (int v = 0; v < VPL; ++v) {
        const int vi = l + LPN * v;
        if (vi < nvec) {
#pragma unroll
          for (int e = 0; e < EV; ++e) sA[vi * EV + e] = A[v * EV + e];
        }
      }
      if (l == 0) s_B[ln * SPLIT + sg] = Bsum;
    }
    __syncthreads();
    // epilogue: TPN threads per node, element k = r + TPN * q
    float pnew[NQ];
    float Snew = 0.f;
    if (active) {
      float Bt = 0.f;
#pragma unroll
      for (int s = 0; s < SPLIT; ++s) Bt += s_B[ln * SPLIT + s];
      float* phi_i = b.phi + (int64_t)i * Kp;
      const float invS = 1.0f / S;
      const float half_eps = eps_t / 2.0f;
#pragma unroll
      for (int qq = 0; qq < NQ; ++qq) {
        const int k = r + TPN * qq;
        float val = 0.f;
        if (k < K) {
          float Ak = 0.f;
#pragma unroll
          for (int s = 0; s < SPLIT; ++s) Ak += s_A[((size_t)ln * SPLIT + s) * Kp + k];
          const float bk = b.beta[k] - m.epsilon;
          const float grad = (bk * Ak + Bt) * invS;
          const float nz = kEarlyNoise ? noise[qq] : noise_at(k);
          const float ph = phi_i[k];
          val = fabsf((ph + half_eps * (m.alpha - ph + m.Nn * grad)) + sqrtf(eps_t * ph) * nz);
          if (val < 1.0e-24f) val = 1.0e-24f;
          phi_i[k] = val;
        }
        pnew[qq] = val;
        Snew += val;
      }
    }
    // sum of the new row over the node's TPN threads
    if constexpr (TPN <= 32) {
#pragma unroll
      for (int o = TPN / 2; o > 0; o >>= 1) Snew += __shfl_xor_sync(group_mask<TPN>(warp_lane), Snew, o);
    } else {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) Snew += __shfl_xor_sync(0xffffffffu, Snew, o);
      if (warp_lane == 0) s_red[ln * (TPN / 32) + (r >> 5)] = Snew;
      __syncthreads();
      Snew = 0.f;
#pragma unroll
      for (int w2 = 0; w2 < TPN / 32; ++w2) Snew += s_red[ln * (TPN / 32) + w2];
    }
    if (active) {
      float* st = b.stage + (int64_t)slot * Kp;
#pragma unroll
      for (int qq = 0; qq < NQ; ++qq) {
        const int k = r + TPN * qq;
        if (k < Kp) st[k] = (k < K) ? __fdiv_rn(pnew[qq], Snew) : 0.f;
      }
    }
    __syncthreads();
  }
  // CTAs with no work wait before they exit
  if (first >= n_nodes) grid_dependency_wait();
}
template <typename PiT, int LPN, int VPL, int SPLIT, int NPB>
__global__ void __launch_bounds__(NPB * SPLIT * LPN) k_update_phi(Model m, Buffers b) {
  update_phi_body<PiT, LPN, VPL, SPLIT, NPB>(m, b, blockIdx.x, gridDim.x);
}
template <typename PiT, int LPN, int VPL, int SPLIT, int NPB>
__global__ void __launch_bounds__(NPB * SPLIT * LPN) k_update_phi_chains(const ChainArgs* __restrict__ c,
                                                                         const BlockOf* __restrict__ map, int p) {
  const BlockOf o = map[blockIdx.x];
  const ChainArgs& a = c[o.chain];
  update_phi_body<PiT, LPN, VPL, SPLIT, NPB>(a.m, slot_buffers(a.m, a.b, p), o.block, o.blocks);
}

// ---------------------------------------------------------------------------
// The parts of k's theta step that do not depend on the sums: theta and beta
// themselves, eta_c - theta_kc, the noise terms sqrt(eps theta_kc) n_kc,
// 1/(theta0+theta1) and the two gradient factors 1/theta_kc - 1/ts -- three FP64
// divisions and two square roots, about 2.5 us at GB300's FP64 rate.  They are
// formed by blocks of one working warp (32 values of k) beside the commit's
// own, because nothing of them waits for update_phi: in the theta kernel they
// were the longest part between the commit's end and the step.  (Folding the
// step into one multiply-add per class and side saves six more dependent FP64
// operations but rounds theta differently: the sum is kept as it was.)
// ---------------------------------------------------------------------------
static __device__ __forceinline__ void theta_pre_block(const Model& m, const Buffers& b, int block) {
  grid_launch_dependents();
  const int k = block * 32 + (int)threadIdx.x;
  if (threadIdx.x < 32 && k < m.K) {
    const double eps_t = (double)b.st->eps;
    const double th0 = b.theta[2 * k], th1 = b.theta[2 * k + 1];
    const double ts_inv = 1.0 / (th0 + th1);
    double n0, n1;
    if (b.fed_theta_noise) {
      n0 = b.fed_theta_noise[2 * k];
      n1 = b.fed_theta_noise[2 * k + 1];
    } else {
      const Stream rs{m.seed, m.chain};
      n0 = normal_draw(rs, kTagThetaNoise, 0, b.st->step, 2ull * k);
      n1 = normal_draw(rs, kTagThetaNoise, 0, b.st->step, 2ull * k + 1);
    }
    double* out = b.theta_pre + k;
    out[0] = th0;
    out[m.K] = th1;
    out[2 * m.K] = (double)m.eta0 - th0;
    out[3 * m.K] = (double)m.eta1 - th1;
    out[4 * m.K] = sqrt(eps_t * th0) * n0;
    out[5 * m.K] = sqrt(eps_t * th1) * n1;
    out[6 * m.K] = ts_inv;
    out[7 * m.K] = 1.0 / th0 - ts_inv;
    out[8 * m.K] = 1.0 / th1 - ts_inv;
    out[9 * m.K] = (double)b.beta[k];
  }
  grid_dependency_wait();
}

// f_k = pi_ak pi_bk of one lane's 4 elements, added to the lane's sums of f
// and of w f (w = beta for a link, 1 - beta otherwise); and 1 / P_e from
// their warp sums.  The roundings are spelled out because k_commit_beta and
// k_commit_star have to give the same bits.
__device__ __forceinline__ float4 edge_terms(const float4& xa, const float4& xb, const float4& w, float& fsum,
                                             float& psum) {
  const float4 f = make_float4(__fmul_rn(xa.x, xb.x), __fmul_rn(xa.y, xb.y), __fmul_rn(xa.z, xb.z),
                               __fmul_rn(xa.w, xb.w));
  fsum = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(fsum, f.x), f.y), f.z), f.w);
  psum = __fmaf_rn(w.w, f.w, __fmaf_rn(w.z, f.z, __fmaf_rn(w.y, f.y, __fmaf_rn(w.x, f.x, psum))));
  return f;
}
__device__ __forceinline__ float edge_inv_prob(float fsum, float psum, bool y, float epsilon) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    fsum += __shfl_xor_sync(0xffffffffu, fsum, o);
    psum += __shfl_xor_sync(0xffffffffu, psum, o);
  }
  return 1.0f / __fmaf_rn(y ? epsilon : 1.0f - epsilon, 1.0f - fsum, psum);
}

// ---------------------------------------------------------------------------
// k_commit_beta: blocks [0, ncommit) copy the staged rows into pi (the
// reference's update_pi loop, cc:162-166); blocks [ncommit, ncommit+nbb)
// evaluate update_beta's per-edge terms (cc:212-240) on the staged (new) pi
// and reduce them per block.  With f_k = pi_ak pi_bk, P_e = sum_k
// (y ? beta_k : 1-beta_k) f_k + (y ? eps : 1-eps)(1 - sum_k f_k) the
// gradient only needs R_yk = sum_{e: y_e = y} f_ek / P_e (k_theta applies the
// theta factors), accumulated per warp in registers, then per block.
// ---------------------------------------------------------------------------
template <typename PiT, int KQ>
__device__ __forceinline__ void commit_beta_body(const Model& m, const Buffers& b, int ncommit, int block) {
  using TR = PiTraits<PiT>;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int Kp = m.Kp, K = m.K;
  if (block >= ncommit + m.nbb) {
    theta_pre_block(m, b, block - ncommit - m.nbb);
    return;
  }
  grid_launch_dependents();
  if (block < ncommit) {
    const int n_nodes = b.st->n_nodes;
    constexpr int EV = TR::kPerVec;
    PiT* pi = reinterpret_cast<PiT*>(b.pi);
    const int nvec = Kp / EV;
    // the staged rows come from update_phi, the launch ahead of this one,
    // which also still reads the pi rows written here
    grid_dependency_wait();
    for (int slot = block * 4 + warp; slot < n_nodes; slot += ncommit * 4) {
      const int32_t i = b.nodes[slot];
      const float* src = b.stage + (int64_t)slot * Kp;
      PiT* dst = pi + (int64_t)i * Kp;
      // a vector's EV floats of the staged row (16-byte aligned: Kp is a
      // multiple of EV) as float4 loads
      for (int vi = lane; vi < nvec; vi += 32) {
        float x[EV];
#pragma unroll
        for (int e = 0; e < EV; e += 4) {
          const float4 q = *reinterpret_cast<const float4*>(src + vi * EV + e);
          x[e] = q.x;
          x[e + 1] = q.y;
          x[e + 2] = q.z;
          x[e + 3] = q.w;
        }
        *reinterpret_cast<uint4*>(dst + vi * EV) = TR::pack(x);
      }
    }
    return;
  }
  __shared__ float s_part[4][2][KQ * 128];
  const int bb = block - ncommit;
  const int n_edges = b.st->n_edges;
  if (bb * 4 >= n_edges) {  // no edges for this block: k_theta skips its partial
    grid_dependency_wait();
    return;
  }
  float R0[KQ * 4], R1[KQ * 4], bt[KQ * 4];
#pragma unroll
  for (int q = 0; q < KQ; ++q)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int k = q * 128 + lane * 4 + e;
      R0[q * 4 + e] = 0.f;
      R1[q * 4 + e] = 0.f;
      bt[q * 4 + e] = (k < K) ? b.beta[k] : 0.f;
    }
  grid_dependency_wait();  // the staged rows (update_phi)
  for (int ed = bb * 4 + warp; ed < n_edges; ed += m.nbb * 4) {
    const float* pa = b.stage + (int64_t)b.ea[ed] * Kp;
    const float* pb = b.stage + (int64_t)b.eb[ed] * Kp;
    const bool y = b.ey[ed] != 0;
    float f[KQ * 4];
    float fsum = 0.f, psum = 0.f;
#pragma unroll
    for (int q = 0; q < KQ; ++q) {
      const int k0 = q * 128 + lane * 4;
      float4 xa = make_float4(0, 0, 0, 0), xb = make_float4(0, 0, 0, 0);
      if (k0 < Kp) {
        xa = *reinterpret_cast<const float4*>(pa + k0);
        xb = *reinterpret_cast<const float4*>(pb + k0);
      }
      const bool in = k0 < K;  // past K the rows hold zeros
      const float4 w = y ? make_float4(bt[q * 4], bt[q * 4 + 1], bt[q * 4 + 2], bt[q * 4 + 3])
                         : make_float4(in ? 1.0f - bt[q * 4] : 0.f, in ? 1.0f - bt[q * 4 + 1] : 0.f,
                                       in ? 1.0f - bt[q * 4 + 2] : 0.f, in ? 1.0f - bt[q * 4 + 3] : 0.f);
      const float4 t = edge_terms(xa, xb, w, fsum, psum);
      f[q * 4 + 0] = t.x;
      f[q * 4 + 1] = t.y;
      f[q * 4 + 2] = t.z;
      f[q * 4 + 3] = t.w;
    }
    const float invP = edge_inv_prob(fsum, psum, y, m.epsilon);
    if (y) {
#pragma unroll
      for (int e = 0; e < KQ * 4; ++e) R1[e] = fmaf(f[e], invP, R1[e]);
    } else {
#pragma unroll
      for (int e = 0; e < KQ * 4; ++e) R0[e] = fmaf(f[e], invP, R0[e]);
    }
  }
#pragma unroll
  for (int q = 0; q < KQ; ++q)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      s_part[warp][0][q * 128 + lane * 4 + e] = R0[q * 4 + e];
      s_part[warp][1][q * 128 + lane * 4 + e] = R1[q * 4 + e];
    }
  __syncthreads();
  float* out = b.beta_part + (int64_t)bb * 2 * Kp;
  for (int k = threadIdx.x; k < Kp; k += 128) {
    out[k] = s_part[0][0][k] + s_part[1][0][k] + s_part[2][0][k] + s_part[3][0][k];
    out[Kp + k] = s_part[0][1][k] + s_part[1][1][k] + s_part[2][1][k] + s_part[3][1][k];
  }
}
template <typename PiT, int KQ>
__global__ void __launch_bounds__(128) k_commit_beta(Model m, Buffers b, int ncommit) {
  commit_beta_body<PiT, KQ>(m, b, ncommit, blockIdx.x);
}
template <typename PiT, int KQ>
__global__ void __launch_bounds__(128) k_commit_beta_chains(const ChainArgs* __restrict__ c,
                                                            const BlockOf* __restrict__ map, int p) {
  const BlockOf o = map[blockIdx.x];
  const ChainArgs& a = c[o.chain];
  commit_beta_body<PiT, KQ>(a.m, slot_buffers(a.m, a.b, p), a.ncommit, o.block);
}

// ---------------------------------------------------------------------------
// k_commit_star: k_commit_beta for a star minibatch (one source: edge e joins
// slot 0 to slot e + 1, one y for all edges), the minibatch of the default
// strategies.  Every staged row is read once, by the warp of its edge, which
// also commits it to pi; the source's row is shared in shared memory; and
// only the R of the minibatch's y is kept and written (the other is zero).
//
// The sums are k_commit_beta's bit for bit: CTA bb stands for its block bb,
// whose warp w adds f_k / P_e of the edges bb*4 + w + j*nbb*4 in the order of
// j.  Here 4*JC warps take JC of those j at once: each forms its edge's f_k
// (kept in shared memory) and 1 / P_e, then the CTA's threads, one float pair
// of k each, add the JC terms of the four w in that order.
// Bound by latency, not bytes: one round of row loads and one warp sum per
// JC*4 edges where k_commit_beta made a round per edge and warp.  4,096 edges of
// K = 1024 BF16: 15.5 and 11.3 us (cold, alone), 13 and 5 us in an iteration; a
// link stratum's few edges 5.2 us alone either way.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void store_pi4(float* dst, const float4& x) {
  *reinterpret_cast<float4*>(dst) = x;
}
__device__ __forceinline__ void store_pi4(__nv_bfloat16* dst, const float4& x) {
  using TR = PiTraits<__nv_bfloat16>;
  *reinterpret_cast<uint2*>(dst) = make_uint2(TR::pack2(x.x, x.y), TR::pack2(x.z, x.w));
}

template <int JC>
constexpr size_t commit_star_smem(int Kp) {  // f, the source's row, w, 1 / P
  return ((size_t)(4 * JC + 2) * Kp + 4 * JC) * sizeof(float);
}

template <typename PiT, int KQ, int JC>
__device__ __forceinline__ void commit_star_body(const Model& m, const Buffers& b, int block) {
  constexpr int NT = 128 * JC;
  constexpr int NIT = (KQ * 64 + NT - 1) / NT;  // float pairs of k per thread
  extern __shared__ __align__(16) float s_star[];
  const int Kp = m.Kp, K = m.K;
  float* s_f = s_star;               // 4*JC rows
  float* s_xa = s_f + 4 * JC * Kp;   // the source's new row
  float* s_w = s_xa + Kp;            // beta or 1 - beta
  float* s_inv = s_w + Kp;           // 4*JC
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int bb = block, n_edges = b.st->n_edges, per = m.nbb * 4;
  if (bb >= m.nbb) {
    theta_pre_block(m, b, bb - m.nbb);
    return;
  }
  grid_launch_dependents();
  if (bb * 4 >= n_edges) {
    grid_dependency_wait();
    return;
  }
  const bool y = b.ey[0] != 0;
  PiT* pi = reinterpret_cast<PiT*>(b.pi);
  for (int k = tid; k < Kp; k += NT) s_w[k] = k < K ? (y ? b.beta[k] : 1.0f - b.beta[k]) : 0.f;
  int ed = bb * 4 + (warp & 3) + per * (warp >> 2);
  int32_t node = ed < n_edges ? b.nodes[ed + 1] : 0;
  const int32_t source = b.nodes[0];
  float2 R[NIT][4];
#pragma unroll
  for (int i = 0; i < NIT; ++i)
#pragma unroll
    for (int w = 0; w < 4; ++w) R[i][w] = make_float2(0.f, 0.f);
  // the staged rows come from update_phi, the launch ahead of this one,
  // which also still reads the pi rows written here
  grid_dependency_wait();
  for (int k = 4 * tid; k < Kp; k += 4 * NT) {
    const float4 x = *reinterpret_cast<const float4*>(b.stage + k);
    *reinterpret_cast<float4*>(s_xa + k) = x;
    if (bb == 0) store_pi4(pi + (int64_t)source * Kp + k, x);
  }
  for (int e0 = bb * 4; e0 < n_edges; e0 += per * JC) {
    const bool on = ed < n_edges;
    float4 x[KQ];
    if (on) {
      const float* row = b.stage + (int64_t)(ed + 1) * Kp;
#pragma unroll
      for (int q = 0; q < KQ; ++q) {
        const int k0 = q * 128 + lane * 4;
        x[q] = k0 < Kp ? *reinterpret_cast<const float4*>(row + k0) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
    __syncthreads();  // s_xa, s_w; the terms of the last round have been added
    if (on) {
      float fsum = 0.f, psum = 0.f;
#pragma unroll
      for (int q = 0; q < KQ; ++q) {
        const int k0 = q * 128 + lane * 4;
        if (k0 < Kp) {
          store_pi4(pi + (int64_t)node * Kp + k0, x[q]);
          const float4 f = edge_terms(*reinterpret_cast<const float4*>(s_xa + k0), x[q],
                                      *reinterpret_cast<const float4*>(s_w + k0), fsum, psum);
          *reinterpret_cast<float4*>(s_f + warp * Kp + k0) = f;
        }
      }
      const float invP = edge_inv_prob(fsum, psum, y, m.epsilon);
      if (lane == 0) s_inv[warp] = invP;
    }
    __syncthreads();
    ed += per * JC;
    if (ed < n_edges) node = b.nodes[ed + 1];
#pragma unroll
    for (int i = 0; i < NIT; ++i) {
      const int k = 2 * (tid + i * NT);
      if (k < Kp) {
#pragma unroll
        for (int w = 0; w < 4; ++w)
#pragma unroll
          for (int j = 0; j < JC; ++j)
            if (e0 + w + j * per < n_edges) {
              const float2 f = *reinterpret_cast<const float2*>(s_f + (w + 4 * j) * Kp + k);
              const float inv = s_inv[w + 4 * j];
              R[i][w].x = fmaf(f.x, inv, R[i][w].x);
              R[i][w].y = fmaf(f.y, inv, R[i][w].y);
            }
      }
    }
  }
  float* out = b.beta_part + ((int64_t)bb * 2 + (y ? 1 : 0)) * Kp;
#pragma unroll
  for (int i = 0; i < NIT; ++i) {
    const int k = 2 * (tid + i * NT);
    if (k < Kp)
      *reinterpret_cast<float2*>(out + k) = make_float2(R[i][0].x + R[i][1].x + R[i][2].x + R[i][3].x,
                                                        R[i][0].y + R[i][1].y + R[i][2].y + R[i][3].y);
  }
}
template <typename PiT, int KQ, int JC>
__global__ void __launch_bounds__(128 * JC, JC == 1 ? 4 : 2) k_commit_star(Model m, Buffers b) {
  commit_star_body<PiT, KQ, JC>(m, b, blockIdx.x);
}
template <typename PiT, int KQ, int JC>
__global__ void __launch_bounds__(128 * JC, JC == 1 ? 4 : 2) k_commit_star_chains(const ChainArgs* __restrict__ c,
                                                                              const BlockOf* __restrict__ map,
                                                                              int p) {
  const BlockOf o = map[blockIdx.x];
  const ChainArgs& a = c[o.chain];
  commit_star_body<PiT, KQ, JC>(a.m, slot_buffers(a.m, a.b, p), o.block);
}

// ---------------------------------------------------------------------------
// k_theta: theta step of update_beta (cc:241-266) in FP64.  With the block
// sums R0_k, R1_k and beta_k the gradients of cc:236-239 are
//   G_k0 = beta R1 (0 - 1/ts) + (1-beta) R0 (1/theta_k0 - 1/ts)
//   G_k1 = beta R1 (1/theta_k1 - 1/ts) + (1-beta) R0 (0 - 1/ts)
// ---------------------------------------------------------------------------
// With R_given the sums are read from it (R0_k, R1_k at 2k, 2k + 1) instead
// of being formed from the partials; with R_out the sums are written there
// and no step is taken (the phases of a sharded iteration).  `star`: the
// partials are k_commit_star's, of the minibatch's y alone.
//
// A latency chain (partial loads, compensated sums, FP64 at 1/64 of the FP32
// rate), so what does not need the partials is done beside the commit
// (theta_pre_block) and two FMA chains and a division are left: 6.6 and 3 us
// behind the commit of a K = 1024 iteration.  256 threads rather than 1,024, so
// that the CTA fits an SM that still holds commit CTAs.
static __device__ __forceinline__ void theta_body(const Model& m, const Buffers& b, int star, int block,
                                                  const double* R_given = nullptr,
                                                  double* R_out = nullptr) {
  // 32 consecutive k per CTA (lane = k).  31 chains add the partials of the
  // active beta blocks c, c+31, ... in FP32 with Kahan compensation, up to 4
  // chains per warp side by side; then warp 0 adds the 31 sums in fixed order
  // (deterministic) and finishes the step: two FMA chains and one division.
  constexpr int C = kThetaChains, P = kThetaPerChain, W = kThetaThreads / 32, CW = (C + W - 1) / W;
  __shared__ float s_r[2][C][33], s_c[2][C][33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int k = block * 32 + lane;
  const int Kp = m.Kp;
  const int active = min(m.nbb, (b.st->n_edges + 3) / 4);  // blocks that saw edges
  const double half_eps = (double)b.st->eps / 2.0, scale = (double)b.st->scale;
  const bool kin = k < m.K;
  const int only = star && active > 0 ? (b.ey[0] ? 1 : 0) : -1;  // the class with partials
  if (block == 0 && threadIdx.x == 32 && !R_out) {
    // the iteration's edge evaluations and errors, counted as it is applied
    if (b.st->err) atomicOr(&b.gc->err, b.st->err);
    b.gc->evals += (unsigned long long)b.st->n_nodes * (unsigned long long)m.n_out;
    b.gc->iters += 1ull;
  }
  grid_dependency_wait();  // the beta partials and theta_pre: the commit, the launch ahead
  grid_launch_dependents();
  double pre[kThetaPre];
#pragma unroll
  for (int i = 0; i < kThetaPre; ++i) pre[i] = (warp == 0 && kin && !R_out) ? b.theta_pre[i * m.K + k] : 0.0;
  double R[2] = {0.0, 0.0};
  if (R_given) {
    if (warp != 0 || !kin) return;
    R[0] = R_given[2 * k];
    R[1] = R_given[2 * k + 1];
  } else {
#pragma unroll
    for (int y = 0; y < 2; ++y) {
      if (only == 1 - y) continue;
      // the warp's partials loaded together, then added in block order
      float v[CW][P];
#pragma unroll
      for (int j = 0; j < CW; ++j)
#pragma unroll
        for (int q = 0; q < P; ++q) {
          const int c = warp + W * j, bb = c + C * q;
          v[j][q] = (kin && c < C && bb < active) ? b.beta_part[((int64_t)bb * 2 + y) * Kp + k] : 0.f;
        }
#pragma unroll
      for (int j = 0; j < CW; ++j) {
        float r = 0.f, e = 0.f;
#pragma unroll
        for (int q = 0; q < P; ++q) {
          if (warp + W * j + C * q < active) {
            const float x = v[j][q] - e, t = r + x;
            e = (t - r) - x;
            r = t;
          }
        }
        if (warp + W * j < C) {
          s_r[y][warp + W * j][lane] = r;
          s_c[y][warp + W * j][lane] = e;
        }
      }
    }
    __syncthreads();
    if (warp != 0 || k >= m.K) return;
#pragma unroll
    for (int y = 0; y < 2; ++y) {
      if (only == 1 - y) continue;
      float r = 0.f, e = 0.f;  // Kahan over the chains' sums
#pragma unroll
      for (int w = 0; w < C; ++w) {
        const float x = (s_r[y][w][lane] - s_c[y][w][lane]) - e;
        const float t = r + x;
        e = (t - r) - x;
        r = t;
      }
      R[y] = (double)r - (double)e;
    }
    if (R_out) {
      R_out[2 * k] = R[0];
      R_out[2 * k + 1] = R[1];
      return;
    }
  }
  const double th0 = pre[0], th1 = pre[1], ts_inv = pre[6], f0 = pre[7], f1 = pre[8], bt = pre[9];
  double G0, G1;
  if (only >= 0) {  // one of the sums is zero, and its products
    const double g = only ? bt * R[1] : (1.0 - bt) * R[0];
    G0 = g * (only ? -ts_inv : f0);
    G1 = g * (only ? f1 : -ts_inv);
  } else {
    G0 = bt * R[1] * (-ts_inv) + (1.0 - bt) * R[0] * f0;
    G1 = bt * R[1] * f1 + (1.0 - bt) * R[0] * (-ts_inv);
  }
  double t0 = fabs(th0 + half_eps * (pre[2] + scale * G0) + pre[4]);
  double t1 = fabs(th1 + half_eps * (pre[3] + scale * G1) + pre[5]);
  if (t0 < 1.0e-24) t0 = 1.0e-24;
  if (t1 < 1.0e-24) t1 = 1.0e-24;
  b.theta[2 * k] = t0;
  b.theta[2 * k + 1] = t1;
  b.beta[k] = (float)(t1 / (t0 + t1));
}
static __global__ void __launch_bounds__(kThetaThreads) k_theta(Model m, Buffers b, int star) {
  theta_body(m, b, star, blockIdx.x);
}
// the per-k sums R0, R1 of the beta partials, without the step
static __global__ void __launch_bounds__(kThetaThreads) k_beta_sums(Model m, Buffers b, double* R_out) {
  theta_body(m, b, 0, blockIdx.x, nullptr, R_out);
}
// the theta step from given sums: a call of its own, so its other parts are
// formed here too, from the theta and beta of now (not those of the commit)
static __global__ void __launch_bounds__(kThetaThreads) k_theta_given(Model m, Buffers b, const double* R) {
  theta_pre_block(m, b, blockIdx.x);
  __syncthreads();
  theta_body(m, b, 0, blockIdx.x, R, nullptr);
}
static __global__ void __launch_bounds__(kThetaThreads) k_theta_chains(const ChainArgs* __restrict__ c,
                                                                       const BlockOf* __restrict__ map, int p) {
  const BlockOf o = map[blockIdx.x];
  const ChainArgs& a = c[o.chain];
  theta_body(a.m, slot_buffers(a.m, a.b, p), a.star, o.block);
}

// ---------------------------------------------------------------------------
// Held-out perplexity (learner.cc:138-183, learner.h:100-139): LPN lanes per
// held-out edge; running average per edge in FP32 as the reference; the log
// sum in FP64.  A block takes PpxPlan::per_block consecutive edges.  A lane
// group keeps its edges' averages a lane each; they meet in shared memory, and
// a warp or two take the logarithms of products of four (an FP64 instruction
// holds the SM's FP64 pipe 16 cycles however few of its lanes are on: 86,246
// pairs of K = 1024 BF16, of which the rows are 53 us, took 262 us with a
// logarithm per edge and warp, 82 with one per warp and 8 edges, 70 with
// one per block and 64).  The product's roundings are within those of the sum
// of four logarithms.  The block that finishes
// last adds the blocks' partials, in a fixed order, so the result does not
// depend on which it is; one thread adding a block's 256 values, and a second
// launch for the partials, were 20 us of a small set's call.
// ---------------------------------------------------------------------------
struct PpxResult {
  double value;
  int32_t err;    // DevCounters::err when the call ran
  uint32_t bad;   // a pair named a row outside pi
  uint32_t done;  // blocks finished: zero between calls
  uint32_t pad;
};

// Edges a lane group takes at a time, eight of them or a lane each; the edges
// and blocks of a call: at most kPpxMaxBlocks partials.
constexpr int kPpxMaxBlocks = 16384;
struct PpxPlan {
  int per_block, blocks;
};
__host__ __device__ constexpr int ppx_edges(int lpn) { return lpn < 8 ? lpn : 8; }
__host__ __device__ constexpr int ppx_chunk(int lpn) { return ppx_edges(lpn) * (256 / lpn); }
inline PpxPlan ppx_plan(int lpn, int64_t H) {
  const int64_t chunk = ppx_chunk(lpn), need = (H + kPpxMaxBlocks - 1) / kPpxMaxBlocks;
  const int64_t per = (need < 1 ? 1 : (need + chunk - 1) / chunk) * chunk;
  return PpxPlan{(int)per, (int)((H + per - 1) / per)};
}

// Sum of one value per thread of a 256-thread block (pairwise, fixed order),
// in thread 0.
__device__ __forceinline__ double block_sum_256(double v, double* s) {
  const int tid = threadIdx.x;
  s[tid] = v;
  __syncthreads();
#pragma unroll
  for (int w = 128; w >= 32; w >>= 1) {
    if (tid < w) s[tid] += s[tid + w];
    __syncthreads();
  }
  if (tid >= 32) return 0.0;
  v = s[tid];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

template <typename PiT, int LPN, int VPL>
__global__ void __launch_bounds__(256, VPL >= 8 ? 2 : VPL >= 4 ? 3 : 4) k_perplexity(Model m, const PiT* __restrict__ pi,
                                                    const float* __restrict__ beta,
                                                    const int32_t* __restrict__ ha,
                                                    const int32_t* __restrict__ hb,
                                                    const uint8_t* __restrict__ hy, int64_t H, int per_block,
                                                    float* __restrict__ ppx, float count,
                                                    double* __restrict__ part, int64_t n_rows,
                                                    const DevCounters* gc, PpxResult* res) {
  using TR = PiTraits<PiT>;
  constexpr int EV = TR::kPerVec;
  constexpr int EPL = VPL * EV;
  constexpr int GPB = 256 / LPN, CH = ppx_chunk(LPN), J = ppx_edges(LPN);
  constexpr int LOGS = CH / 4;  // threads that take logarithms, 16 to 64
  // beta in shared memory, not registers: 32 of them a lane left an SM with two
  // blocks instead of three (four measured no better)
  __shared__ __align__(16) float s_beta[LPN * EPL];
  __shared__ __align__(16) float s_avg[CH];
  __shared__ double s_sum[256];
  __shared__ int s_last;
  const int tid = threadIdx.x, grp = tid / LPN, l = tid % LPN, lane = tid & 31;
  const uint32_t gmask = group_mask<LPN>(lane);
  // rows are Kp apart; only the vectors that hold the K values are read,
  // and elements past K (row padding) take no part in either sum
  const int Kp = m.Kp, K = m.K, nvec = (K + EV - 1) / EV;
  for (int k = tid; k < LPN * EPL; k += 256) s_beta[k] = (k < K) ? beta[k] : 0.f;
  __syncthreads();
  const int64_t e0 = (int64_t)blockIdx.x * per_block;
  const int64_t e1 = e0 + per_block < H ? e0 + per_block : H;
  double sum = 0.0, comp = 0.0;
  for (int64_t c0 = e0; c0 < e1; c0 += CH) {
    float mine = 1.f;  // the average of the lane's edge (logarithm 0: none)
    // lane j reads edge j's words and passes them on
    const int64_t own = c0 + grp + GPB * l;
    const bool on = l < J && own < e1;
    const int32_t own_a = on ? ha[own] : -1, own_b = on ? hb[own] : -1;
    const int own_y = on && hy[own] != 0;
    const float old = on ? ppx[own] : 0.f;
#pragma unroll 2
    for (int j = 0; j < J; ++j) {
      if (c0 + grp + GPB * j >= e1) break;
      const int32_t a = __shfl_sync(gmask, own_a, j, LPN), b = __shfl_sync(gmask, own_b, j, LPN);
      const bool y = __shfl_sync(gmask, own_y, j, LPN) != 0;
      // a pair naming a row outside pi is skipped (no row is read) and flagged
      if ((uint64_t)(int64_t)a >= (uint64_t)n_rows || (uint64_t)(int64_t)b >= (uint64_t)n_rows) {
        if (l == 0) atomicOr(&res->bad, 1u);
        continue;
      }
      const PiT* ra = pi + (int64_t)a * Kp;
      const PiT* rb = pi + (int64_t)b * Kp;
      uint4 va[VPL], vb[VPL];
#pragma unroll
      for (int v = 0; v < VPL; ++v) {
        const int vi = l + LPN * v;
        va[v] = vi < nvec ? ldg_nc_v4(ra + vi * EV) : make_uint4(0, 0, 0, 0);
        vb[v] = vi < nvec ? ldg_nc_v4(rb + vi * EV) : make_uint4(0, 0, 0, 0);
      }
      float s = 0.f, fs = 0.f;
#pragma unroll
      for (int v = 0; v < VPL; ++v) {
        const int vi = l + LPN * v;
        if (vi < nvec) {
          float xa[EV], xb[EV], bt[EV];
          TR::unpack(va[v], xa);
          TR::unpack(vb[v], xb);
#pragma unroll
          for (int e = 0; e < EV; e += 4)
            *reinterpret_cast<float4*>(bt + e) = *reinterpret_cast<const float4*>(s_beta + vi * EV + e);
#pragma unroll
          for (int e = 0; e < EV; ++e) {
            if (vi * EV + e < K) {
              const float f = xa[e] * xb[e];
              fs += f;
              s += f * (y ? bt[e] : 1.0f - bt[e]);
            }
          }
        }
      }
#pragma unroll
      for (int o = LPN / 2; o > 0; o >>= 1) {
        s += __shfl_xor_sync(gmask, s, o);
        fs += __shfl_xor_sync(gmask, fs, o);
      }
      if (l == j) {
        if (!y) s += (1.0f - fs) * (1.0f - m.epsilon);
        if (s < 1.0e-30f) s = 1.0e-30f;
        mine = (old * (count - 1.0f) + s) / count;
        ppx[own] = mine;
      }
    }
    if (l < J) s_avg[grp * J + l] = mine;
    __syncthreads();
    if (tid < LOGS) {
      // NaN for a negative average (of a caller's array), as its logarithm
      // has it; a product of four floats neither overflows nor underflows
      const float4 q = *reinterpret_cast<const float4*>(s_avg + 4 * tid);
      double x = ((double)q.x * q.y) * ((double)q.z * q.w);
      if (fminf(fminf(q.x, q.y), fminf(q.z, q.w)) < 0.f) x = nan("");
      const double term = log(x) - comp;
      const double tsum = sum + term;
      comp = (tsum - sum) - term;
      sum = tsum;
    }
    if (c0 + CH < e1) __syncthreads();  // s_avg is written again
  }
  // the sum over the LOGS threads
  double total = tid < LOGS ? sum - comp : 0.0;
  if (tid < 64) {
#pragma unroll
    for (int o = (LOGS < 32 ? LOGS : 32) / 2; o > 0; o >>= 1) total += __shfl_down_sync(0xffffffffu, total, o);
  }
  if (LOGS > 32) {
    if (tid == 32) s_sum[0] = total;
    __syncthreads();
    if (tid == 0) total += s_sum[0];
  }
  if (tid == 0) {
    part[blockIdx.x] = total;
    __threadfence();
    s_last = atomicAdd(&res->done, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  double t = 0.0, c = 0.0;  // each thread's partials in order (compensated), then a fixed tree
  for (int q = tid; q < (int)gridDim.x; q += 256) {
    const double term = __ldcg(part + q) - c;
    const double ts = t + term;
    c = (ts - t) - term;
    t = ts;
  }
  __syncthreads();
  total = block_sum_256(t - c, s_sum);
  if (tid == 0) {
    res->value = -(total / (double)H);
    res->err = gc ? gc->err : 0;
    res->done = 0;
  }
}

// ---------------------------------------------------------------------------
// init: phi ~ Gamma(1,1) (cc:66), row normalisation into pi (cc:75).  Bound by
// FP32 issue (ammsb_gamma.cuh): 30,000 x 256, 3.28 ms of FP64 draws and 0.2.
// ---------------------------------------------------------------------------
static __global__ void __launch_bounds__(256) k_init_phi(Model m, float* phi, const GammaTables* tables,
                                                         int32_t* err) {
  __shared__ GammaTables s_t;
  static_assert(sizeof(GammaTables) % sizeof(float2) == 0, "copied by pairs");
  for (int i = threadIdx.x; i < (int)(sizeof(GammaTables) / sizeof(float2)); i += 256)
    reinterpret_cast<float2*>(&s_t)[i] = reinterpret_cast<const float2*>(tables)[i];
  __syncthreads();
  const Stream rs{m.seed, m.chain};
  // element x = v Kp + k, the grid's threads side by side: v and k follow
  // without a division each
  const int64_t total = m.N * (int64_t)m.Kp, stride = (int64_t)gridDim.x * 256;
  const int64_t dv = stride / m.Kp;
  const int dk = (int)(stride - dv * m.Kp);
  int64_t x = (int64_t)blockIdx.x * 256 + threadIdx.x;
  int64_t v = x / m.Kp;
  int k = (int)(x - v * m.Kp);
  for (; x < total; x += stride) {
    phi[x] = k < m.K ? gamma_one_draw(rs, kTagPhiInit, (uint32_t)v, (uint64_t)k, s_t, err) : 0.f;
    v += dv;
    k += dk;
    if (k >= m.Kp) {
      k -= m.Kp;
      ++v;
    }
  }
}

// np::row_normalize (np.h:63-75): one warp per row, sum in FP32.
template <typename PiT>
__global__ void k_normalize_rows(Model m, const float* phi, PiT* pi) {
  using TR = PiTraits<PiT>;
  constexpr int EV = TR::kPerVec;
  const int lane = threadIdx.x & 31;
  const int64_t w0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const int Kp = m.Kp, nvec = Kp / EV;
  for (int64_t v = w0; v < m.N; v += nw) {
    const float* src = phi + v * Kp;
    float s = 0.f;
    for (int k = lane; k < Kp; k += 32) s += src[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    PiT* dst = pi + v * Kp;
    for (int vi = lane; vi < nvec; vi += 32) {
      float x[EV];
#pragma unroll
      for (int e = 0; e < EV; ++e) x[e] = __fdiv_rn(src[vi * EV + e], s);
      *reinterpret_cast<uint4*>(dst + vi * EV) = TR::pack(x);
    }
  }
}

// n rows of K elements (stride Kp) as packed floats: a read-out of BF16 pi.
// Bound by the copy to the host behind it (5M values 1,054 us when the host
// widened them one by one, now 235).
template <typename T>
__global__ void __launch_bounds__(256) k_widen_rows(const T* __restrict__ rows, int K, int Kp, int64_t n,
                                                   float* __restrict__ out) {
  const int64_t total = n * K, stride = (int64_t)gridDim.x * 256;
  const int64_t dr = stride / K;
  const int dk = (int)(stride - dr * K);
  int64_t x = (int64_t)blockIdx.x * 256 + threadIdx.x;
  int64_t r = x / K;
  int k = (int)(x - r * K);
  for (; x < total; x += stride) {
    out[x] = (float)rows[r * Kp + k];
    r += dr;
    k += dk;
    if (k >= K) {
      k -= K;
      ++r;
    }
  }
}

}  // namespace ammsb
