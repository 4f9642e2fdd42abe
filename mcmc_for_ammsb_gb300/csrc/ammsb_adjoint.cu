// ammsb_adjoint.cu -- the minibatch edge log-likelihood and its hand-written
// adjoint: the SGRLD drift of phi and theta.
//
// The reference never forms this function; it differentiates it by hand:
//   L(phi, theta) = sum over pairs q = (a, b, y) of log p_q,
//   p_q = sum_k pi_ak pi_bk (f_qk - e_q) + e_q,          pi_a = phi_a / S_a,
//   f_qk = y ? beta_k : 1 - beta_k,  e_q = y ? eps : 1 - eps,
//   beta_k = theta_k1 / (theta_k0 + theta_k1),
// p_q is the normaliser prob_sum of update_beta (mcmc_sampler_stochastic.cc
// :212-240) and, as sum_k pi_ak = 1, of update_phi (cc:279-290).
// cal_edge_likelihood (learner.h:100-139) equals it for a non-link and leaves
// out the term eps * (1 - sum_k pi_ak pi_bk) for a link.
// Its gradients are the reference's hand-derived terms:
//   dL/dphi_ak = sum_q (probs_qk / (p_q phi_ak) - 1/S_a)  -- update_phi
//                (mcmc_sampler_stochastic.cc:274-296, pi_b held fixed)
//   dL/dtheta  = the update_beta gradient (cc:212-240).
// With sigma_q = +-1 for y = 1/0, f - e = sigma (beta - eps), so
//   p_q = sigma_q D_q + e_q,  D_q = sum_k w_ak pi_bk,  w_ak = pi_ak (beta_k - eps),
//   dL/dphi_ak  = ((beta_k - eps) A_ak - B_a) / S_a,
//       A_ak = sum_{q of a} sigma_q pi_bk / p_q,  B_a = sum_{q of a} (p_q - e_q) / p_q,
//   dL/dbeta_k  = sum_a pi_ak A_ak,
//   dL/dpi_bk   = (beta_k - eps) sum_{q of b} sigma_q pi_ak / p_q,
// and beta's chain rule: dbeta/dtheta_k0 = -beta_k / T_k,
// dbeta/dtheta_k1 = (1 - beta_k) / T_k, T_k = theta_k0 + theta_k1.
//
// The forward forms D_q, p_q and, from the same row in registers, the terms
// that the source's gradient needs: A_a and B_a stay in the workspace beside
// S_a and p_q, so each neighbour row is gathered once for L, dL/dphi and
// dL/dtheta (the gather is what bounds it: K elements for two FMAs each).  The
// backward is then a pass over n_src rows, and for dL/dpi a gather of phi rows
// per neighbour.  All sums are in a fixed order (a CTA per source, a group of
// lanes per neighbour row, fixed partials for theta), so repeated calls give
// identical bits.
//
// A row is held by LPR lanes of VPL 16-byte vectors each (one element per
// vector where a pointer, a stride or K is no multiple of 16 bytes); a CTA's
// 128 / LPR groups take a source's pairs in turn.  Measured on GB300 (4,097
// sources x 129 pairs, K = 1000, FP32, 200,000 neighbour rows), before and
// after: forward 1,012 and 333 us (2.1 GB of gathered rows at 6.4 TB/s),
// backward 1,226 (430 for dphi, 286 for dtheta, 510 for dpi) and 312 us (23, 8
// and 280: 2.1 GB of phi rows from L2, 0.8 GB written).
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>
#include <string>

#include "../../include/ammsb_gpu.h"

namespace {

constexpr int kThreads = 128;
constexpr int kMaxParts = 304;  // theta partials: two blocks per SM
constexpr int kErrIndex = 1;    // a pair or CSR index out of range
constexpr int kErrNonPos = 2;   // a row sum S_a or a probability p_q <= 0

// Sum over an aligned group of G lanes.
template <int G, typename T>
__device__ __forceinline__ T group_sum(T v, uint32_t mask) {
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(mask, v, o);
  return v;
}
template <int G>
__device__ __forceinline__ uint32_t lane_group_mask() {
  if constexpr (G >= 32)
    return 0xffffffffu;
  else
    return ((1u << G) - 1u) << ((threadIdx.x & 31) / G * G);
}

// workspace: [err word | beta - eps (K) | S, B, ll (n_src) | p (n_pairs) |
// A (n_src x K) | theta partials]
struct Workspace {
  size_t off_bm, off_S, off_B, off_ll, off_p, off_A, off_part, bytes;
};

size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

int parts_of(int64_t n_src) { return (int)(n_src < kMaxParts ? n_src : kMaxParts); }

Workspace layout(size_t es, int64_t K, int64_t n_src, int64_t n_pairs) {
  Workspace w{};
  const size_t rows = align256(es * (size_t)n_src);
  w.off_bm = 256;
  w.off_S = w.off_bm + align256(es * (size_t)K);
  w.off_B = w.off_S + rows;
  w.off_ll = w.off_B + rows;
  w.off_p = w.off_ll + rows;
  w.off_A = w.off_p + align256(es * (size_t)n_pairs);
  w.off_part = w.off_A + align256(es * (size_t)n_src * (size_t)K);
  w.bytes = w.off_part + align256(es * (size_t)parts_of(n_src) * (size_t)K);
  return w;
}

struct Args {
  int32_t K;
  const void* phi;   // n_src x ld_phi
  int64_t ld_phi;
  const void* pin;   // n_nbr x ld_pi
  int64_t ld_pi;
  int64_t n_nbr;
  const void* theta; // K x 2
  double eps;
  const int64_t* src_ptr;  // n_src + 1: pairs of source a are [src_ptr[a], src_ptr[a+1])
  int64_t n_src;
  const int32_t* pair_nbr; // n_pairs: row of pin
  const uint8_t* pair_y;
  int64_t n_pairs;
  // backward only
  const int32_t* pair_src; // n_pairs: source row of each pair
  const int64_t* nbr_ptr;  // n_nbr + 1 over nbr_pairs
  const int32_t* nbr_pairs;
  const void* gout;        // device scalar dL
  void* gphi;              // n_src x ld_phi
  void* gpin;              // n_nbr x ld_pi (or null)
  void* gtheta;            // K x 2
  char* ws;
  Workspace w;
  int parts, rows_per_part;  // theta partials and the source rows of each
  template <typename T>
  __host__ __device__ T* at(size_t off) const { return reinterpret_cast<T*>(ws + off); }
};

// A grid of any number of blocks: in rows of 2^30 where they are more than its
// x dimension holds (kernels return from blocks past their rows).
constexpr int64_t kGridRow = 1ll << 30;
dim3 grid_of(int64_t blocks) {
  return blocks <= kGridRow ? dim3((unsigned)blocks) : dim3((unsigned)kGridRow, (unsigned)((blocks - 1) / kGridRow + 1));
}
__device__ __forceinline__ int64_t block_of_grid() { return blockIdx.x + (int64_t)blockIdx.y * kGridRow; }

// VEC elements of a row as one load or store (VEC * sizeof(T) bytes, aligned).
template <typename T, int VEC>
struct alignas(sizeof(T) * VEC) Vec {
  T v[VEC];
};
// A lane's VPL vectors (vectors l + LPR v) of a row of nvec vectors, zero
// past its end.
template <typename T, int VEC, int LPR, int VPL>
__device__ __forceinline__ void load_row(const T* row, int l, int nvec, T* x) {
#pragma unroll
  for (int v = 0; v < VPL; ++v) {
    const int vi = l + LPR * v;
    Vec<T, VEC> r{};
    if (vi < nvec) r = reinterpret_cast<const Vec<T, VEC>*>(row)[vi];
#pragma unroll
    for (int e = 0; e < VEC; ++e) x[v * VEC + e] = r.v[e];
  }
}
// Rows in flight per group: as many as keep a lane at 16 elements of them.
template <int EPL>
__host__ __device__ constexpr int rows_ahead() { return EPL <= 4 ? 4 : EPL <= 8 ? 2 : 1; }

// beta_k - eps, and a clear status word
template <typename T>
__global__ void __launch_bounds__(256) k_ll_prepare(Args g) {
  const int k = blockIdx.x * 256 + threadIdx.x;
  if (k == 0) *reinterpret_cast<int32_t*>(g.ws) = 0;
  if (k >= g.K) return;
  const T* theta = static_cast<const T*>(g.theta);
  const T t0 = theta[2 * k], t1 = theta[2 * k + 1];
  g.at<T>(g.w.off_bm)[k] = t1 / (t0 + t1) - (T)g.eps;
}

template <typename T, int VEC, int LPR, int VPL>
__global__ void __launch_bounds__(kThreads) k_ll_forward(Args g) {
  constexpr int EPL = VPL * VEC, NG = kThreads / LPR, U = rows_ahead<EPL>();
  __shared__ T s_A[kThreads * EPL];  // a row per group
  __shared__ T s_B[NG], s_ll[kThreads / 32];
  const int tid = threadIdx.x, l = tid % LPR, grp = tid / LPR;
  const uint32_t mask = lane_group_mask<LPR>();
  const int64_t a = block_of_grid();
  if (a >= g.n_src) return;
  const int K = g.K, nvec = K / VEC;
  const T eps = (T)g.eps;
  const T* pin = static_cast<const T*>(g.pin);
  T* p_out = g.at<T>(g.w.off_p);
  int32_t* err = reinterpret_cast<int32_t*>(g.ws);

  int64_t q0 = g.src_ptr[a], q1 = g.src_ptr[a + 1];
  if (q0 < 0 || q1 < q0 || q1 > g.n_pairs) {
    if (tid == 0) atomicOr(err, kErrIndex);
    q0 = q1 = 0;
  }
  T w[EPL], A[EPL], S = 0;
  load_row<T, VEC, LPR, VPL>(static_cast<const T*>(g.phi) + a * g.ld_phi, l, nvec, w);
#pragma unroll
  for (int e = 0; e < EPL; ++e) S += w[e];
  S = group_sum<LPR>(S, mask);
  {
    T bm[EPL];
    load_row<T, VEC, LPR, VPL>(g.at<T>(g.w.off_bm), l, nvec, bm);
#pragma unroll
    for (int e = 0; e < EPL; ++e) {
      w[e] = w[e] / S * bm[e];
      A[e] = T(0);
    }
  }
  T B = 0;
  for (int64_t qb = q0 + grp; qb < q1; qb += NG * U) {
    T x[U][EPL], D[U];
    int32_t nb[U];
    bool on[U], y[U];  // on: not past the source's pairs
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t q = qb + (int64_t)u * NG;
      on[u] = q < q1;
      nb[u] = on[u] ? g.pair_nbr[q] : -1;
      y[u] = on[u] && g.pair_y[q] != 0;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const bool in = nb[u] >= 0 && nb[u] < g.n_nbr;
      load_row<T, VEC, LPR, VPL>(pin + (in ? (int64_t)nb[u] * g.ld_pi : 0), l, in ? nvec : 0, x[u]);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      D[u] = T(0);
#pragma unroll
      for (int e = 0; e < EPL; ++e) D[u] += w[e] * x[u][e];
    }
#pragma unroll
    for (int o = LPR / 2; o > 0; o >>= 1)
#pragma unroll
      for (int u = 0; u < U; ++u) D[u] += __shfl_xor_sync(mask, D[u], o);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (!on[u]) continue;
      const int64_t q = qb + (int64_t)u * NG;
      if (nb[u] < 0 || nb[u] >= g.n_nbr) {
        if (l == 0) {
          atomicOr(err, kErrIndex);
          p_out[q] = T(1);
        }
        continue;
      }
      const T e_q = y[u] ? eps : T(1) - eps;
      const T p = (y[u] ? D[u] : -D[u]) + e_q;
      const T inv = T(1) / p;
      const T c = y[u] ? inv : -inv;
      B += (p - e_q) * inv;
      if (l == 0) {
        p_out[q] = p;
        if (!(p > T(0))) atomicOr(err, kErrNonPos);
      }
#pragma unroll
      for (int e = 0; e < EPL; ++e) A[e] += c * x[u][e];
    }
  }
  // the groups' A and B, added in group order
#pragma unroll
  for (int v = 0; v < VPL; ++v)
#pragma unroll
    for (int e = 0; e < VEC; ++e) {
      const int k = (l + LPR * v) * VEC + e;
      if (k < K) s_A[grp * K + k] = A[v * VEC + e];
    }
  if (l == 0) s_B[grp] = B;
  __syncthreads();  // also makes the CTA's p visible to its threads
  T* A_out = g.at<T>(g.w.off_A) + a * K;
  for (int k = tid; k < K; k += kThreads) {
    T sum = 0;
#pragma unroll 4
    for (int r = 0; r < NG; ++r) sum += s_A[r * K + k];
    A_out[k] = sum;
  }
  T ll = 0;
  for (int64_t q = q0 + tid; q < q1; q += kThreads) ll += log(p_out[q]);
  ll = group_sum<32>(ll, 0xffffffffu);
  if ((tid & 31) == 0) s_ll[tid >> 5] = ll;
  __syncthreads();
  if (tid == 0) {
    T b = 0, sum = 0;
    for (int r = 0; r < NG; ++r) b += s_B[r];
    for (int r = 0; r < kThreads / 32; ++r) sum += s_ll[r];
    if (!(S > T(0))) atomicOr(err, kErrNonPos);
    g.at<T>(g.w.off_S)[a] = S;
    g.at<T>(g.w.off_B)[a] = b;
    g.at<T>(g.w.off_ll)[a] = sum;
  }
}

// loss = sum_a ll[a], one block, fixed order
template <typename T>
__global__ void __launch_bounds__(512) k_ll_sum(Args g, T* loss) {
  __shared__ T part[16];
  const T* ll = g.at<T>(g.w.off_ll);
  T s = 0;
#pragma unroll 4
  for (int64_t a = threadIdx.x; a < g.n_src; a += 512) s += ll[a];
  s = group_sum<32>(s, 0xffffffffu);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    T t = 0;
    for (int r = 0; r < 16; ++r) t += part[r];
    *loss = t;
  }
}

// dL/dphi rows, and the sums of pi_ak A_ak over the block's source rows
// (blockIdx.x) for its KT values of k (blockIdx.y); 256 / KT rows side by side.
template <typename T>
__global__ void __launch_bounds__(256) k_ll_backward_src(Args g, int KT) {
  __shared__ T s_U[256];
  const int K = g.K, tid = threadIdx.x, kt = tid % KT, rg = tid / KT, RG = 256 / KT;
  const int k = blockIdx.y * KT + kt;
  const T gout = *static_cast<const T*>(g.gout);
  const T* phi = static_cast<const T*>(g.phi);
  T* gphi = static_cast<T*>(g.gphi);
  const T *S_in = g.at<T>(g.w.off_S), *B_in = g.at<T>(g.w.off_B), *A_in = g.at<T>(g.w.off_A);
  const int64_t a0 = (int64_t)blockIdx.x * g.rows_per_part;
  const int64_t a1 = a0 + g.rows_per_part < g.n_src ? a0 + g.rows_per_part : g.n_src;
  T U = 0;
  if (k < K) {
    const T b = g.at<T>(g.w.off_bm)[k];
#pragma unroll 4
    for (int64_t a = a0 + rg; a < a1; a += RG) {
      const T S = S_in[a], A = A_in[a * K + k], x = phi[a * g.ld_phi + k];
      gphi[a * g.ld_phi + k] = gout * (b * A - B_in[a]) / S;
      U += x / S * A;
    }
  }
  if (RG > 1) {
    s_U[tid] = U;
    __syncthreads();
    if (rg == 0) {
      U = 0;
      for (int r = 0; r < RG; ++r) U += s_U[r * KT + kt];
    }
  }
  if (rg == 0 && k < K) g.at<T>(g.w.off_part)[(int64_t)blockIdx.x * K + k] = U;
}

// dL/dtheta from the partials: 32 k per block, eight warps over the partials
template <typename T>
__global__ void __launch_bounds__(256) k_ll_backward_theta(Args g) {
  __shared__ T s_U[8][33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, k = blockIdx.x * 32 + lane;
  const T* part = g.at<T>(g.w.off_part);
  T U = 0;
  if (k < g.K) {
#pragma unroll 8
    for (int r = warp; r < g.parts; r += 8) U += part[(int64_t)r * g.K + k];
  }
  s_U[warp][lane] = U;
  __syncthreads();
  if (warp != 0 || k >= g.K) return;
  U = 0;
#pragma unroll
  for (int r = 0; r < 8; ++r) U += s_U[r][lane];
  const T gout = *static_cast<const T*>(g.gout);
  const T* theta = static_cast<const T*>(g.theta);
  const T t0 = theta[2 * k], t1 = theta[2 * k + 1];
  const T Tk = t0 + t1;
  const T bk = t1 / Tk;
  T* gt = static_cast<T*>(g.gtheta);
  gt[2 * k] = gout * U * (-bk / Tk);
  gt[2 * k + 1] = gout * U * ((T(1) - bk) / Tk);
}

// dL/dpi_nbr rows: LPR lanes per neighbour row over its pairs (nbr CSR).  The
// lanes read the pairs' words (pair -> source -> S) side by side, LPR pairs at
// a time, so that their chain of loads is paid once.
template <typename T, int VEC, int LPR, int VPL>
__global__ void __launch_bounds__(kThreads) k_ll_backward_nbr(Args g) {
  constexpr int EPL = VPL * VEC, U = rows_ahead<EPL>();
  const int l = threadIdx.x % LPR;
  const uint32_t mask = lane_group_mask<LPR>();
  const int64_t b = (block_of_grid() * kThreads + threadIdx.x) / LPR;
  if (b >= g.n_nbr) return;
  const int K = g.K, nvec = K / VEC;
  const T* phi = static_cast<const T*>(g.phi);
  const T gout = *static_cast<const T*>(g.gout);
  const T *p_in = g.at<T>(g.w.off_p), *S_in = g.at<T>(g.w.off_S);
  int32_t* err = reinterpret_cast<int32_t*>(g.ws);

  T acc[EPL];
#pragma unroll
  for (int e = 0; e < EPL; ++e) acc[e] = T(0);
  int64_t r0 = g.nbr_ptr[b], r1 = g.nbr_ptr[b + 1];
  if (r0 < 0 || r1 < r0 || r1 > g.n_pairs) {
    if (l == 0) atomicOr(err, kErrIndex);
    r0 = r1 = 0;
  }
  for (int64_t rb = r0; rb < r1; rb += LPR) {
    // this lane's pair: its source (-1: none) and sigma / (p S)
    int32_t src = -1;
    T coef = 0;
    if (rb + l < r1) {
      const int32_t q = g.nbr_pairs[rb + l];
      const bool in = q >= 0 && q < g.n_pairs;
      const int32_t a = in ? g.pair_src[q] : -1;
      if (!in || a < 0 || a >= g.n_src || g.pair_nbr[q] != b) {
        atomicOr(err, kErrIndex);
      } else {
        src = a;
        coef = (g.pair_y[q] != 0 ? T(1) : T(-1)) / (p_in[q] * S_in[a]);
      }
    }
    const int n = r1 - rb < LPR ? (int)(r1 - rb) : LPR;
    for (int i = 0; i < n; i += U) {
      T x[U][EPL], c[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int from = i + u < n ? i + u : i;
        const int32_t a = __shfl_sync(mask, src, from, LPR);
        c[u] = __shfl_sync(mask, coef, from, LPR);
        const bool in = i + u < n && a >= 0;
        if (!in) c[u] = T(0);
        load_row<T, VEC, LPR, VPL>(phi + (in ? (int64_t)a * g.ld_phi : 0), l, in ? nvec : 0, x[u]);
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int e = 0; e < EPL; ++e) acc[e] += c[u] * x[u][e];
    }
  }
  const Vec<T, VEC>* bm = reinterpret_cast<const Vec<T, VEC>*>(g.at<T>(g.w.off_bm));
  Vec<T, VEC>* gp = reinterpret_cast<Vec<T, VEC>*>(static_cast<T*>(g.gpin) + b * g.ld_pi);
#pragma unroll
  for (int v = 0; v < VPL; ++v) {
    const int vi = l + LPR * v;
    if (vi < nvec) {
      const Vec<T, VEC> f = bm[vi];
      Vec<T, VEC> r;
#pragma unroll
      for (int e = 0; e < VEC; ++e) r.v[e] = gout * f.v[e] * acc[v * VEC + e];
      gp[vi] = r;
    }
  }
}

unsigned blocks_of(int64_t n, int64_t per) { return (unsigned)((n + per - 1) / per); }

template <typename T, int VEC, int LPR, int VPL>
cudaError_t launch_rows(bool fwd, const Args& g, cudaStream_t s) {
  if (fwd) {
    if (g.n_src) k_ll_forward<T, VEC, LPR, VPL><<<grid_of(g.n_src), kThreads, 0, s>>>(g);
  } else if (g.n_nbr) {
    k_ll_backward_nbr<T, VEC, LPR, VPL><<<grid_of((g.n_nbr - 1) / (kThreads / LPR) + 1), kThreads, 0, s>>>(g);
  }
  return cudaGetLastError();
}

// Lanes and vectors for a row of K elements: the fewest lanes (a power of two
// up to a warp) that hold it at one vector each, then more vectors per lane.
// Whole 16-byte vectors need 16-byte rows; any other row goes element by
// element, a warp to the row.
template <typename T>
cudaError_t dispatch_rows(bool fwd, const Args& g, cudaStream_t s) {
  constexpr int EV = 16 / sizeof(T);
  auto whole = [&](const void* p, int64_t ld) {
    return reinterpret_cast<uintptr_t>(p) % 16 == 0 && ld % EV == 0;
  };
  const bool vec = g.K % EV == 0 && whole(g.phi, g.ld_phi) && whole(g.pin, g.ld_pi) && whole(g.ws, 0) &&
                   (fwd || whole(g.gpin, g.ld_pi));
  const int nvec = vec ? g.K / EV : g.K;
  int lpr = 32, vpl = 1;
  if (vec)
    for (lpr = 1; lpr < 32 && lpr < nvec;) lpr <<= 1;
  while (lpr * vpl < nvec) vpl <<= 1;
#define ROWS(V, L, P) \
  if (lpr == L && vpl == P) return launch_rows<T, V, L, P>(fwd, g, s);
  if (vec) {
    ROWS(EV, 1, 1) ROWS(EV, 2, 1) ROWS(EV, 4, 1) ROWS(EV, 8, 1) ROWS(EV, 16, 1) ROWS(EV, 32, 1) ROWS(EV, 32, 2)
    ROWS(EV, 32, 4) ROWS(EV, 32, 8)
    if constexpr (EV == 2) { ROWS(EV, 32, 16) }
  } else {
    ROWS(1, 32, 1) ROWS(1, 32, 2) ROWS(1, 32, 4) ROWS(1, 32, 8) ROWS(1, 32, 16) ROWS(1, 32, 32)
  }
#undef ROWS
  return cudaErrorInvalidConfiguration;
}

template <typename T>
cudaError_t forward(const Args& g, void* loss, cudaStream_t s) {
  k_ll_prepare<T><<<blocks_of(g.K, 256), 256, 0, s>>>(g);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = dispatch_rows<T>(true, g, s);
  if (e != cudaSuccess) return e;
  k_ll_sum<T><<<1, 512, 0, s>>>(g, static_cast<T*>(loss));
  return cudaGetLastError();
}

template <typename T>
cudaError_t backward(const Args& g, cudaStream_t s) {
  int kt = 1;
  while (kt < 256 && kt < g.K) kt <<= 1;
  if (g.parts) k_ll_backward_src<T><<<dim3(g.parts, blocks_of(g.K, kt)), 256, 0, s>>>(g, kt);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  k_ll_backward_theta<T><<<blocks_of(g.K, 32), 256, 0, s>>>(g);
  e = cudaGetLastError();
  if (e != cudaSuccess || !g.gpin) return e;
  return dispatch_rows<T>(false, g, s);
}

void set_parts(Args* g) {
  g->parts = parts_of(g->n_src);
  g->rows_per_part = g->parts ? (int)((g->n_src + g->parts - 1) / g->parts) : 0;
  if (g->rows_per_part) g->parts = (int)((g->n_src + g->rows_per_part - 1) / g->rows_per_part);
}

int fail(const char* fn, const std::string& msg, int code) {
  std::fprintf(stderr, "%s: %s\n", fn, msg.c_str());
  return code;
}

int check_common(const char* fn, int32_t dtype, int64_t K, const void* phi, int64_t ld_phi,
                 const void* pin, int64_t ld_pi, int64_t n_nbr, const void* theta,
                 const int64_t* src_ptr, int64_t n_src, const int32_t* pair_nbr,
                 const uint8_t* pair_y, int64_t n_pairs, const void* ws) {
  if (dtype != AMMSB_REAL_F32 && dtype != AMMSB_REAL_F64)
    return fail(fn, "dtype must be AMMSB_REAL_F32 or AMMSB_REAL_F64", AMMSB_E_ARG);
  if (K < 1 || K > 1024) return fail(fn, "need 1 <= K <= 1024", AMMSB_E_ARG);
  if (ld_phi < K || ld_pi < K) return fail(fn, "row strides must be >= K", AMMSB_E_ARG);
  if (n_src < 0 || n_nbr < 0 || n_pairs < 0 || n_pairs > INT32_MAX)
    return fail(fn, "negative size, or more than 2^31 - 1 pairs", AMMSB_E_ARG);
  if (!theta || !src_ptr || !ws || (n_src > 0 && !phi) || (n_nbr > 0 && !pin) ||
      (n_pairs > 0 && (!pair_nbr || !pair_y)))
    return fail(fn, "null argument", AMMSB_E_ARG);
  return AMMSB_OK;
}

}  // namespace

extern "C" {

size_t ammsb_edge_loglik_workspace_size(int32_t dtype, int64_t K, int64_t n_src,
                                        int64_t n_pairs) {
  if (K < 1 || n_src < 0 || n_pairs < 0) return 0;
  const size_t es = (dtype == AMMSB_REAL_F64) ? 8 : 4;
  return layout(es, K, n_src, n_pairs).bytes;
}

int ammsb_edge_loglik_forward(int32_t dtype, int64_t K, const void* phi_src, int64_t ld_phi,
                              const void* pi_nbr, int64_t ld_pi, int64_t n_nbr,
                              const void* theta, double epsilon, const int64_t* src_ptr,
                              int64_t n_src, const int32_t* pair_nbr, const uint8_t* pair_y,
                              int64_t n_pairs, void* loss, void* workspace, void* stream) {
  const char* fn = "ammsb_edge_loglik_forward";
  int rc = check_common(fn, dtype, K, phi_src, ld_phi, pi_nbr, ld_pi, n_nbr, theta, src_ptr,
                        n_src, pair_nbr, pair_y, n_pairs, workspace);
  if (rc) return rc;
  if (!loss) return fail(fn, "null loss", AMMSB_E_ARG);
  const size_t es = (dtype == AMMSB_REAL_F64) ? 8 : 4;
  Args g{};
  g.K = (int32_t)K;
  g.phi = phi_src; g.ld_phi = ld_phi;
  g.pin = pi_nbr; g.ld_pi = ld_pi; g.n_nbr = n_nbr;
  g.theta = theta; g.eps = epsilon;
  g.src_ptr = src_ptr; g.n_src = n_src;
  g.pair_nbr = pair_nbr; g.pair_y = pair_y; g.n_pairs = n_pairs;
  g.ws = static_cast<char*>(workspace);
  g.w = layout(es, K, n_src, n_pairs);
  set_parts(&g);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  cudaError_t e = (dtype == AMMSB_REAL_F64) ? forward<double>(g, loss, s) : forward<float>(g, loss, s);
  if (e != cudaSuccess) return fail(fn, cudaGetErrorString(e), AMMSB_E_CUDA);
  return AMMSB_OK;
}

int ammsb_edge_loglik_backward(int32_t dtype, int64_t K, const void* phi_src, int64_t ld_phi,
                               const void* pi_nbr, int64_t ld_pi, int64_t n_nbr,
                               const void* theta, double epsilon, const int64_t* src_ptr,
                               int64_t n_src, const int32_t* pair_nbr, const uint8_t* pair_y,
                               int64_t n_pairs, const int32_t* pair_src, const int64_t* nbr_ptr,
                               const int32_t* nbr_pairs, const void* grad_loss,
                               void* grad_phi_src, void* grad_pi_nbr, void* grad_theta,
                               void* workspace, void* stream) {
  const char* fn = "ammsb_edge_loglik_backward";
  int rc = check_common(fn, dtype, K, phi_src, ld_phi, pi_nbr, ld_pi, n_nbr, theta, src_ptr,
                        n_src, pair_nbr, pair_y, n_pairs, workspace);
  if (rc) return rc;
  if (!grad_loss || !grad_theta || (n_src > 0 && !grad_phi_src))
    return fail(fn, "null gradient argument", AMMSB_E_ARG);
  if (grad_pi_nbr && (!nbr_ptr || (n_pairs > 0 && (!pair_src || !nbr_pairs))))
    return fail(fn, "grad_pi_nbr needs pair_src, nbr_ptr and nbr_pairs", AMMSB_E_ARG);
  const size_t es = (dtype == AMMSB_REAL_F64) ? 8 : 4;
  Args g{};
  g.K = (int32_t)K;
  g.phi = phi_src; g.ld_phi = ld_phi;
  g.pin = pi_nbr; g.ld_pi = ld_pi; g.n_nbr = n_nbr;
  g.theta = theta; g.eps = epsilon;
  g.src_ptr = src_ptr; g.n_src = n_src;
  g.pair_nbr = pair_nbr; g.pair_y = pair_y; g.n_pairs = n_pairs;
  g.pair_src = pair_src; g.nbr_ptr = nbr_ptr; g.nbr_pairs = nbr_pairs;
  g.gout = grad_loss; g.gphi = grad_phi_src; g.gpin = grad_pi_nbr; g.gtheta = grad_theta;
  g.ws = static_cast<char*>(workspace);
  g.w = layout(es, K, n_src, n_pairs);
  set_parts(&g);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  cudaError_t e = (dtype == AMMSB_REAL_F64) ? backward<double>(g, s) : backward<float>(g, s);
  if (e != cudaSuccess) return fail(fn, cudaGetErrorString(e), AMMSB_E_CUDA);
  return AMMSB_OK;
}

int ammsb_edge_loglik_status(const void* workspace, void* stream, int32_t* flags) {
  if (!workspace || !flags) return AMMSB_E_ARG;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  cudaError_t e = cudaMemcpyAsync(flags, workspace, sizeof(int32_t), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return fail("ammsb_edge_loglik_status", cudaGetErrorString(e), AMMSB_E_CUDA);
  return AMMSB_OK;
}

}  // extern "C"
