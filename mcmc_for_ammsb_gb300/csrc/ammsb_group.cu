// ammsb_group.cu -- a pair list grouped by source and by neighbour: what the
// edge log-likelihood's kernels walk (ammsb_adjoint.cu).
//
// Both groupings are stable sorts of the pairs by a key below 2^31 with few
// significant bits (13 for 4,097 sources, 18 for 200,000 neighbour rows):
// least-significant-digit passes of up to 9 bits over a permutation, each
// counting a tile's digits, scanning the counts of every digit over the tiles
// and placing the tile's pairs behind the earlier ones of their digit.  Within
// a tile each warp takes 128 consecutive pairs in order and ranks them by a
// match among its lanes and a running count per digit, so equal keys keep
// their order.  A list of one tile (2,048 pairs) is grouped by one launch with
// the permutation in shared memory (15 us for 1,600 pairs, where some forty
// launches of sorts, scans and copies took 0.7 ms of host time); sources that
// do not descend, the usual list, skip the first sort on the device.  Bound by
// launches and latency: 528,513 pairs, 10 MB, take 75 us.
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>
#include <string>

#include "../../include/ammsb_gpu.h"

namespace {

constexpr int kThreads = 512, kWarps = kThreads / 32;
constexpr int kRounds = 4;                  // pairs per thread
constexpr int kTile = kThreads * kRounds;   // pairs per block
constexpr int kMaxDigit = 9, kMaxBins = 1 << kMaxDigit;
constexpr int64_t kNamed = 1ll << 31;       // indices that an int32 holds
constexpr int kCheckWords = 4;  // max and ~min of the sources, of the neighbours

__device__ __forceinline__ uint32_t lanes_below() {
  uint32_t m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

struct Digit {
  int shift, bins;
  __device__ __forceinline__ int of(int64_t key) const { return (int)(key >> shift) & (bins - 1); }
};

// Exclusive scan of one value per thread of a kThreads block.
__device__ __forceinline__ int block_scan(int v, int* s_warp) {
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
    const int w = lane < kWarps ? s_warp[lane] : 0;
    int winc = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int n = __shfl_up_sync(0xffffffffu, winc, o);
      if (lane >= o) winc += n;
    }
    if (lane < kWarps) s_warp[lane] = winc - w;
  }
  __syncthreads();
  const int r = s_warp[warp] + incl - v;
  __syncthreads();
  return r;
}

// A tile's pairs by digit: the rank of each of the thread's pairs among the
// warp's of its digit, and per warp and digit the number of pairs in the
// warps before it (s_count, kWarps x bins), and the tile's (s_total, or null).
typedef unsigned short Count;  // at most kTile
__device__ __forceinline__ void rank_tile(const int* digit, int* rank, Count* s_count, int bins, int* s_total) {
  const int tid = threadIdx.x, warp = tid >> 5;
  Count* mine = s_count + warp * bins;
  for (int c = tid; c < kWarps * bins; c += kThreads) s_count[c] = 0;
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kRounds; ++r) {
    const uint32_t peers = __match_any_sync(0xffffffffu, digit[r]);  // -1: no pair
    const int before = digit[r] >= 0 ? mine[digit[r]] : 0;
    __syncwarp();
    rank[r] = before + __popc(peers & lanes_below());
    if (digit[r] >= 0 && (peers & lanes_below()) == 0) mine[digit[r]] = (Count)(before + __popc(peers));
    __syncwarp();
  }
  __syncthreads();
  for (int d = tid; d < bins; d += kThreads) {
    int sum = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const int c = s_count[w * bins + d];
      s_count[w * bins + d] = (Count)sum;
      sum += c;
    }
    if (s_total) s_total[d] = sum;
  }
  __syncthreads();
}

// The position in the tile of the thread's pair of round r.
__device__ __forceinline__ int tile_pos(int r) {
  return (threadIdx.x >> 5) * (32 * kRounds) + 32 * r + (threadIdx.x & 31);
}

// ptr[v] = number of keys below v, by binary search in the sorted keys.
__device__ __forceinline__ int64_t keys_below(const int32_t* keys, int64_t n, int64_t v) {
  int64_t lo = 0, hi = n;
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1;
    if (keys[mid] < v) lo = mid + 1; else hi = mid;
  }
  return lo;
}

struct Lists {
  const int64_t* src;  // n
  const int64_t* nbr;
  const uint8_t* y;
  int64_t src_top, nbr_top;  // indices outside [0, top] are marked: see ammsb_group_pairs
  int64_t n, n_src, n_nbr;
  int64_t* src_ptr;    // n_src + 1
  int32_t* pair_nbr;   // n, in source order
  uint8_t* pair_y;
  int32_t* pair_src;
  int64_t* nbr_ptr;    // n_nbr + 1
  int32_t* nbr_pairs;  // n
};

__device__ __forceinline__ int64_t clamped(int64_t x, int64_t top) { return x < 0 ? 0 : x > top ? top : x; }
// Pair q at place i of the source order.
__device__ __forceinline__ int32_t put_pair(const Lists& g, int64_t i, int64_t q) {
  const int64_t a = g.src[q], b = g.nbr[q], ac = clamped(a, g.src_top), bc = clamped(b, g.nbr_top);
  g.pair_src[i] = (int32_t)ac;
  g.pair_y[i] = g.y[q];
  return g.pair_nbr[i] = (a == ac && b == bc) ? (int32_t)b : -1;
}

// ---- one tile ---------------------------------------------------------------
// Sorts s_order (a permutation of 0 .. n-1, any keys) by key(i) stably.
template <typename Key>
__device__ __forceinline__ void sort_tile(int n, int bits, Count* s_order, Count* s_count, int* s_base, int* s_warp,
                                          Key key) {
  const int passes = (bits + kMaxDigit - 1) / kMaxDigit;
  for (int p = 0, shift = 0; p < passes; ++p) {
    const int w = (bits - shift + passes - p - 1) / (passes - p);
    const Digit dg{shift, 1 << w};
    shift += w;
    int digit[kRounds], rank[kRounds], item[kRounds];
#pragma unroll
    for (int r = 0; r < kRounds; ++r) {
      const int i = tile_pos(r);
      item[r] = i < n ? s_order[i] : 0;
      digit[r] = i < n ? dg.of(key(item[r])) : -1;
    }
    rank_tile(digit, rank, s_count, dg.bins, s_base);
    const int d = threadIdx.x, total = d < dg.bins ? s_base[d] : 0;
    const int base = block_scan(total, s_warp);
    if (d < dg.bins) s_base[d] = base;
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kRounds; ++r)
      if (digit[r] >= 0)
        s_order[s_base[digit[r]] + s_count[(threadIdx.x >> 5) * dg.bins + digit[r]] + rank[r]] = (Count)item[r];
    __syncthreads();
  }
}

__global__ void __launch_bounds__(kThreads) k_group_tile(Lists g, int src_bits, int nbr_bits) {
  __shared__ Count s_order[kTile], s_count[kWarps * kMaxBins];
  __shared__ int s_key[kTile];  // the neighbours in source order, then the sorted keys
  __shared__ int s_base[kMaxBins], s_warp[kWarps];
  const int tid = threadIdx.x, n = (int)g.n;
  bool down = false;
  for (int i = tid; i < n; i += kThreads) {
    s_order[i] = (Count)i;
    down |= i > 0 && clamped(g.src[i - 1], g.src_top) > clamped(g.src[i], g.src_top);
  }
  if (__syncthreads_or(down))
    sort_tile(n, src_bits, s_order, s_count, s_base, s_warp, [&](int i) { return clamped(g.src[i], g.src_top); });
  for (int i = tid; i < n; i += kThreads) s_key[i] = max(0, put_pair(g, i, s_order[i]));
  __syncthreads();
  for (int64_t v = tid; v <= g.n_src; v += kThreads) g.src_ptr[v] = keys_below(g.pair_src, n, v);
  for (int i = tid; i < n; i += kThreads) s_order[i] = (Count)i;
  __syncthreads();
  sort_tile(n, nbr_bits, s_order, s_count, s_base, s_warp, [&](int i) { return (int64_t)s_key[i]; });
  int key[kRounds];
#pragma unroll
  for (int r = 0; r < kRounds; ++r) {
    const int i = tid + r * kThreads;
    key[r] = 0;
    if (i < n) {
      g.nbr_pairs[i] = s_order[i];
      key[r] = s_key[s_order[i]];
    }
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kRounds; ++r)
    if (tid + r * kThreads < n) s_key[tid + r * kThreads] = key[r];
  __syncthreads();
  for (int64_t v = tid; v <= g.n_nbr; v += kThreads) g.nbr_ptr[v] = keys_below(s_key, n, v);
}

// ---- many tiles ---------------------------------------------------------------
// The keys of a pass: an int64 list, or an int32 one already in source order.
// `skip` (null: never): a word that says the list needs no sorting.
struct Keys {
  const int64_t* wide;
  const int32_t* narrow;
  int64_t top;
  const int32_t* skip;
  __device__ __forceinline__ int64_t operator()(int32_t i) const {
    return clamped(wide ? wide[i] : (int64_t)narrow[i], top);
  }
  __device__ __forceinline__ bool skipped() const { return skip && *skip == 0; }
};

// hist[d * tiles + tile]: pairs of digit d in the tile
__global__ void __launch_bounds__(kThreads) k_group_count(Keys key, const int32_t* order, int64_t n, Digit dg,
                                                          int32_t* hist) {
  __shared__ int s_hist[kMaxBins];
  if (key.skipped()) return;
  for (int d = threadIdx.x; d < dg.bins; d += kThreads) s_hist[d] = 0;
  __syncthreads();
  const int64_t t0 = (int64_t)blockIdx.x * kTile;
#pragma unroll
  for (int r = 0; r < kRounds; ++r) {
    const int64_t i = t0 + threadIdx.x + r * kThreads;
    if (i < n) atomicAdd(s_hist + dg.of(key(order ? order[i] : (int32_t)i)), 1);
  }
  __syncthreads();
  for (int d = threadIdx.x; d < dg.bins; d += kThreads) hist[(int64_t)d * gridDim.x + blockIdx.x] = s_hist[d];
}

// Block d: the exclusive scan of digit d's counts over the tiles, and its total.
__global__ void __launch_bounds__(kThreads) k_group_scan(Keys key, int32_t* hist, int tiles, int32_t* total) {
  __shared__ int s_warp[kWarps];
  __shared__ int s_sum;
  if (key.skipped()) return;
  int32_t* row = hist + (int64_t)blockIdx.x * tiles;
  int carry = 0;
  for (int t0 = 0; t0 < tiles; t0 += kThreads) {
    const int t = t0 + threadIdx.x;
    const int v = t < tiles ? row[t] : 0;
    const int before = block_scan(v, s_warp);
    if (t < tiles) row[t] = carry + before;
    if (threadIdx.x == kThreads - 1) s_sum = before + v;
    __syncthreads();
    carry += s_sum;
    __syncthreads();
  }
  if (threadIdx.x == 0) total[blockIdx.x] = carry;
}

// Places the tile's pairs behind the earlier ones of their digit.
__global__ void __launch_bounds__(kThreads) k_group_place(Keys key, const int32_t* order, int64_t n, Digit dg,
                                                          const int32_t* hist, const int32_t* total,
                                                          int32_t* to) {
  __shared__ Count s_count[kWarps * kMaxBins];
  __shared__ int s_base[kMaxBins], s_warp[kWarps];
  if (key.skipped()) return;
  const int64_t t0 = (int64_t)blockIdx.x * kTile;
  int digit[kRounds], rank[kRounds], item[kRounds];
#pragma unroll
  for (int r = 0; r < kRounds; ++r) {
    const int64_t i = t0 + tile_pos(r);
    item[r] = i < n ? (order ? order[i] : (int32_t)i) : 0;
    digit[r] = i < n ? dg.of(key(item[r])) : -1;
  }
  const int d = threadIdx.x;
  const int base = block_scan(d < dg.bins ? total[d] : 0, s_warp);
  if (d < dg.bins) s_base[d] = base + hist[(int64_t)d * gridDim.x + blockIdx.x];
  rank_tile(digit, rank, s_count, dg.bins, nullptr);  // synchronises
#pragma unroll
  for (int r = 0; r < kRounds; ++r)
    if (digit[r] >= 0)
      to[s_base[digit[r]] + s_count[(threadIdx.x >> 5) * dg.bins + digit[r]] + rank[r]] = item[r];
}

// Whether the sources descend anywhere (*unsorted starts at zero).
__global__ void __launch_bounds__(256) k_group_check(Lists g, int32_t* unsorted) {
  bool down = false;
  for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < g.n; i += (int64_t)gridDim.x * 256)
    down |= i > 0 && clamped(g.src[i - 1], g.src_top) > clamped(g.src[i], g.src_top);
  if (__syncthreads_or(down) && threadIdx.x == 0) *unsorted = 1;
}
// The pair arrays in source order.
__global__ void __launch_bounds__(256) k_group_gather(Lists g, const int32_t* order, const int32_t* unsorted) {
  const bool permuted = *unsorted != 0;
  for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < g.n; i += (int64_t)gridDim.x * 256)
    put_pair(g, i, permuted ? order[i] : i);
}
// The sorted neighbour keys.
__global__ void __launch_bounds__(256) k_group_keys(const int32_t* pair_nbr, const int32_t* order, int64_t n,
                                                    int32_t* keys) {
  for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (int64_t)gridDim.x * 256)
    keys[i] = max(0, pair_nbr[order[i]]);
}
__global__ void __launch_bounds__(256) k_group_ptr(const int32_t* keys, int64_t n, int64_t n_keys, int64_t* ptr) {
  for (int64_t v = (int64_t)blockIdx.x * 256 + threadIdx.x; v <= n_keys; v += (int64_t)gridDim.x * 256)
    ptr[v] = keys_below(keys, n, v);
}

// Largest and smallest index of both lists, as atomics on words that start
// at zero: the order-preserving map of an int64 to unsigned, and its
// complement for the smallest.
__global__ void __launch_bounds__(256) k_pairs_check(const int64_t* src, const int64_t* nbr, int64_t n,
                                                     unsigned long long* words) {
  unsigned long long m[kCheckWords] = {0, 0, 0, 0};
  for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (int64_t)gridDim.x * 256) {
    const unsigned long long s = (unsigned long long)src[i] ^ (1ull << 63), b = (unsigned long long)nbr[i] ^ (1ull << 63);
    m[0] = s > m[0] ? s : m[0];
    m[1] = ~s > m[1] ? ~s : m[1];
    m[2] = b > m[2] ? b : m[2];
    m[3] = ~b > m[3] ? ~b : m[3];
  }
#pragma unroll
  for (int w = 0; w < kCheckWords; ++w) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long x = __shfl_xor_sync(0xffffffffu, m[w], o);
      m[w] = x > m[w] ? x : m[w];
    }
    if ((threadIdx.x & 31) == 0) atomicMax(words + w, m[w]);
  }
}

int bits_below(int64_t n) {  // bits of the keys 0 .. n - 1
  int b = 1;
  while (b < 31 && (1ll << b) < n) ++b;
  return b;
}

size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

struct Work {
  size_t off_a, off_b, off_hist, off_total, bytes;
};
int64_t tiles_of(int64_t n) { return (n + kTile - 1) / kTile; }
Work work_of(int64_t n) {
  Work w{};
  w.off_a = align256(sizeof(unsigned long long) * kCheckWords);
  w.off_b = w.off_a + align256(sizeof(int32_t) * (size_t)n);
  w.off_hist = w.off_b + align256(sizeof(int32_t) * (size_t)n);
  w.off_total = w.off_hist + align256(sizeof(int32_t) * (size_t)tiles_of(n) * kMaxBins);
  w.bytes = w.off_total + align256(sizeof(int32_t) * kMaxBins);
  return w;
}

unsigned grid_of(int64_t n) {
  const int64_t b = (n + 255) / 256;
  return (unsigned)(b < 1 ? 1 : b > 152 * 8 ? 152 * 8 : b);
}

// Stable order of 0 .. n - 1 by key, into one of the two buffers (returned).
cudaError_t sort_tiles(Keys key, int64_t n, int bits, char* ws, const Work& w, cudaStream_t s, int32_t** out) {
  int32_t* buf[2] = {reinterpret_cast<int32_t*>(ws + w.off_a), reinterpret_cast<int32_t*>(ws + w.off_b)};
  int32_t* hist = reinterpret_cast<int32_t*>(ws + w.off_hist);
  int32_t* total = reinterpret_cast<int32_t*>(ws + w.off_total);
  const int tiles = (int)tiles_of(n), passes = (bits + kMaxDigit - 1) / kMaxDigit;
  const int32_t* from = nullptr;
  for (int p = 0, shift = 0; p < passes; ++p) {
    const int wd = (bits - shift + passes - p - 1) / (passes - p);
    const Digit dg{shift, 1 << wd};
    shift += wd;
    k_group_count<<<tiles, kThreads, 0, s>>>(key, from, n, dg, hist);
    k_group_scan<<<dg.bins, kThreads, 0, s>>>(key, hist, tiles, total);
    k_group_place<<<tiles, kThreads, 0, s>>>(key, from, n, dg, hist, total, buf[p & 1]);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    from = buf[p & 1];
  }
  *out = buf[(passes - 1) & 1];
  return cudaSuccess;
}

int fail(const char* fn, const std::string& msg, int code) {
  std::fprintf(stderr, "%s: %s\n", fn, msg.c_str());
  return code;
}

}  // namespace

extern "C" {

size_t ammsb_group_pairs_workspace_size(int64_t n_pairs) {
  return n_pairs < 0 ? 0 : work_of(n_pairs).bytes;
}

int ammsb_check_pairs(const int64_t* src, const int64_t* nbr, int64_t n_pairs, void* workspace, void* stream,
                      int64_t* bounds) {
  const char* fn = "ammsb_check_pairs";
  if (n_pairs < 1 || !src || !nbr || !workspace || !bounds) return fail(fn, "null argument or no pairs", AMMSB_E_ARG);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  unsigned long long* words = static_cast<unsigned long long*>(workspace);
  unsigned long long host[kCheckWords];
  cudaError_t e = cudaMemsetAsync(words, 0, sizeof(host), s);
  if (e == cudaSuccess) {
    k_pairs_check<<<grid_of((n_pairs + 3) / 4), 256, 0, s>>>(src, nbr, n_pairs, words);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(host, words, sizeof(host), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return fail(fn, cudaGetErrorString(e), AMMSB_E_CUDA);
  const unsigned long long top = 1ull << 63;
  bounds[0] = (int64_t)(~host[1] ^ top);
  bounds[1] = (int64_t)(host[0] ^ top);
  bounds[2] = (int64_t)(~host[3] ^ top);
  bounds[3] = (int64_t)(host[2] ^ top);
  return AMMSB_OK;
}

int ammsb_group_pairs(const int64_t* src, const int64_t* nbr, const uint8_t* y, int64_t n_pairs, int64_t n_src,
                      int64_t n_nbr, int64_t src_keys, int64_t nbr_keys, int64_t* src_ptr, int32_t* pair_nbr,
                      uint8_t* pair_y, int32_t* pair_src, int64_t* nbr_ptr, int32_t* nbr_pairs, void* workspace,
                      void* stream) {
  const char* fn = "ammsb_group_pairs";
  if (n_pairs < 0 || n_pairs > INT32_MAX || n_src < 0 || n_nbr < 0 || src_keys < n_src || nbr_keys < n_nbr ||
      (n_pairs > 0 && (src_keys < 1 || nbr_keys < 1)))
    return fail(fn, "sizes out of range", AMMSB_E_ARG);
  // there may be more rows than the int32 arrays can name: pairs of those are marked
  src_keys = src_keys < kNamed ? src_keys : kNamed;
  nbr_keys = nbr_keys < kNamed ? nbr_keys : kNamed;
  if (!src_ptr || !nbr_ptr || !workspace ||
      (n_pairs > 0 && (!src || !nbr || !y || !pair_nbr || !pair_y || !pair_src || !nbr_pairs)))
    return fail(fn, "null argument", AMMSB_E_ARG);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const Lists g{src,     nbr,      y,      src_keys - 1, nbr_keys - 1, n_pairs, n_src,
                n_nbr,   src_ptr,  pair_nbr, pair_y,     pair_src,     nbr_ptr, nbr_pairs};
  const int src_bits = bits_below(src_keys), nbr_bits = bits_below(nbr_keys);
  cudaError_t e = cudaSuccess;
  // one block also fills the pointers, a binary search each: 512 a few times
  // (1,600 pairs 15 us; the general path's launches are some 40 us of host time)
  if (n_pairs <= kTile && n_src + n_nbr <= 16384) {
    k_group_tile<<<1, kThreads, 0, s>>>(g, src_bits, nbr_bits);
    e = cudaGetLastError();
  } else if (n_pairs == 0) {
    e = cudaMemsetAsync(src_ptr, 0, sizeof(int64_t) * (size_t)(n_src + 1), s);
    if (e == cudaSuccess) e = cudaMemsetAsync(nbr_ptr, 0, sizeof(int64_t) * (size_t)(n_nbr + 1), s);
  } else {
    const Work w = work_of(n_pairs);
    char* ws = static_cast<char*>(workspace);
    int32_t* unsorted = static_cast<int32_t*>(workspace);
    int32_t* order = nullptr;
    e = cudaMemsetAsync(unsorted, 0, sizeof(int32_t), s);
    if (e == cudaSuccess) {
      k_group_check<<<grid_of((n_pairs + 3) / 4), 256, 0, s>>>(g, unsorted);
      e = sort_tiles(Keys{src, nullptr, g.src_top, unsorted}, n_pairs, src_bits, ws, w, s, &order);
    }
    if (e == cudaSuccess) {
      k_group_gather<<<grid_of(n_pairs), 256, 0, s>>>(g, order, unsorted);
      k_group_ptr<<<grid_of(n_src + 1), 256, 0, s>>>(pair_src, n_pairs, n_src, src_ptr);
      e = sort_tiles(Keys{nullptr, pair_nbr, g.nbr_top, nullptr}, n_pairs, nbr_bits, ws, w, s, &order);
    }
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(nbr_pairs, order, sizeof(int32_t) * (size_t)n_pairs, cudaMemcpyDeviceToDevice, s);
    if (e == cudaSuccess) {
      // the sorted keys go where the permutation is not
      int32_t* keys = reinterpret_cast<int32_t*>(ws + w.off_a);
      if (order == keys) keys = reinterpret_cast<int32_t*>(ws + w.off_b);
      k_group_keys<<<grid_of(n_pairs), 256, 0, s>>>(pair_nbr, order, n_pairs, keys);
      k_group_ptr<<<grid_of(n_nbr + 1), 256, 0, s>>>(keys, n_pairs, n_nbr, nbr_ptr);
      e = cudaGetLastError();
    }
  }
  if (e != cudaSuccess) return fail(fn, cudaGetErrorString(e), AMMSB_E_CUDA);
  return AMMSB_OK;
}

}  // extern "C"
