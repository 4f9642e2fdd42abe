// ammsb_phi_ring.cuh -- update_phi for wide pi rows (>= 512 bytes), with the
// neighbour rows staged in shared memory through a per-warp ring.
//
// SPLIT warps per minibatch node.  Warp g handles neighbours g, g+SPLIT, ...:
// each of its lanes keeps its own 16-byte pieces of the next rows in flight
// (cp.async global -> shared, one commit group per chunk of U rows), waits
// for the chunk's group, reads back exactly the pieces it copied and does the
// two FMA passes of the factored gradient (see k_update_phi in
// ammsb_kernels.cuh for the algebra).  A lane never reads another lane's
// pieces of a row, so the ring needs no barrier; the waits are on the lane's
// own copies, which always complete.  (A variant with one cp.async.bulk copy
// per row and an mbarrier per slot measured 5% slower: its per-row barrier
// wait, warp vote, __syncwarp and single-lane issue cost more than four
// 16-byte copies per lane.)
#pragma once
#include "ammsb_kernels.cuh"

namespace ammsb {

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

// Packed FP32 pairs (Blackwell fma.rn.f32x2): two IEEE round-to-nearest
// FMAs per instruction, element-wise identical to two scalar fmaf.
typedef unsigned long long f32x2;

__device__ __forceinline__ f32x2 pack_f32x2(float lo, float hi) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}

__device__ __forceinline__ void unpack_f32x2(f32x2 v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}

__device__ __forceinline__ f32x2 fma_f32x2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

__device__ __forceinline__ f32x2 add_f32x2(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// The 16 bytes of a row vector as EV/2 float pairs.
template <typename PiT>
struct PairLoad;

template <>
struct PairLoad<float> {
  __device__ __forceinline__ static void get(const uint4& v, f32x2* out) {
    out[0] = pack_f32x2(__uint_as_float(v.x), __uint_as_float(v.y));
    out[1] = pack_f32x2(__uint_as_float(v.z), __uint_as_float(v.w));
  }
};

template <>
struct PairLoad<__nv_bfloat16> {
  __device__ __forceinline__ static f32x2 word(uint32_t w) {
    return pack_f32x2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
  }
  __device__ __forceinline__ static void get(const uint4& v, f32x2* out) {
    out[0] = word(v.x);
    out[1] = word(v.y);
    out[2] = word(v.z);
    out[3] = word(v.w);
  }
};

// Rows taken together by a warp: their dot products' warp sums (five dependent
// shuffles each, some 150 cycles) then overlap.  As many as keep a lane at 32
// floats of rows or fewer beside its w and A; rows of 32 floats a lane (K =
// 1024 BF16) are bound by HBM with 16 warps per SM and take one at a time.
// 100,000 x 256 BF16, 32 neighbours: 6.66 ms per 500 iterations with one row at
// a time and a launch per kind, now 5.60; 400,000 x 1024 BF16 10.30 and 10.12 per 100.
template <typename PiT, int VPL>
__host__ __device__ constexpr int ring_rows() {
  constexpr int EPL = VPL * PiTraits<PiT>::kPerVec;
  return EPL <= 8 ? 4 : EPL <= 16 ? 2 : 1;
}

template <typename PiT, int VPL, int SPLIT, int STAGES>
struct PhiRingSmem {
  static constexpr int kRows = STAGES * ring_rows<PiT, VPL>();  // ring slots per warp
  // BF16 rows keep the node's phi row and normals in shared memory across
  // the rows (two more rows of floats)
  static constexpr bool kStash = sizeof(PiT) == 2;
  // the per-warp A vectors of the epilogue reuse the warp's own ring slice
  static_assert(kRows * sizeof(PiT) >= sizeof(float), "ring slice must hold a row of floats");
  __host__ __device__ static size_t bytes(int Kp, int n_out) {
    size_t ring = (size_t)SPLIT * kRows * Kp * sizeof(PiT);
    size_t w = (size_t)(kStash ? 3 : 1) * Kp * sizeof(float);
    size_t misc = (size_t)(4 * SPLIT + 8) * sizeof(float) + (size_t)n_out * sizeof(uint32_t);
    return (ring + w + misc + 127) / 128 * 128;
  }
};

// One row of the ring as the lane's float pairs (FULL: every lane's vectors
// lie inside the row).
template <typename PiT, int VPL, bool FULL>
__device__ __forceinline__ void load_row_pairs(const PiT* row, int lane, int nvec, f32x2* x2) {
  constexpr int EV = PiTraits<PiT>::kPerVec;
#pragma unroll
  for (int v = 0; v < VPL; ++v) {
    const int vi = lane + 32 * v;
    const uint4 raw = (FULL || vi < nvec) ? *reinterpret_cast<const uint4*>(row + vi * EV)
                                          : make_uint4(0, 0, 0, 0);
    PairLoad<PiT>::get(raw, x2 + v * (EV / 2));
  }
}

// The four normals of elements k0 .. k0+3 of node i's phi update (one
// Philox block), or the fed values when the caller supplies them.
__device__ __forceinline__ float4 phi_normals(const Buffers& b, const Stream& rs, int slot, int32_t i,
                                              uint32_t step, int k0, int K) {
  float4 nz = make_float4(0.f, 0.f, 0.f, 0.f);
  if (b.fed_phi_noise) {
    const float* f = b.fed_phi_noise + (int64_t)slot * K + k0;
    nz.x = (k0 + 0 < K) ? f[0] : 0.f;
    nz.y = (k0 + 1 < K) ? f[1] : 0.f;
    nz.z = (k0 + 2 < K) ? f[2] : 0.f;
    nz.w = (k0 + 3 < K) ? f[3] : 0.f;
  } else {
    const U32x4 o = rs.block(kTagPhiNoise, (uint32_t)i, step, (uint64_t)k0 >> 2);
    float s0, c0, s1, c1;
    const float r0 = sqrtf(-2.0f * logf(u24_open(o.x)));
    const float r1 = sqrtf(-2.0f * logf(u24_open(o.z)));
    sincospif(2.0f * u24(o.y), &s0, &c0);
    sincospif(2.0f * u24(o.w), &s1, &c1);
    nz.x = r0 * c0;
    nz.y = r0 * s0;
    nz.z = r1 * c1;
    nz.w = r1 * s1;
  }
  return nz;
}

// The lane's 16-byte pieces of a row (vectors lane + 32 v), copied into the
// same places of a ring slot by cp.async: a lane only ever reads back the
// pieces it copied itself.
template <typename PiT, int VPL, bool FULL>
__device__ __forceinline__ void copy_row_lane(PiT* dst, const PiT* src, int lane, int nvec) {
  constexpr int EV = PiTraits<PiT>::kPerVec;
#pragma unroll
  for (int v = 0; v < VPL; ++v) {
    const int vi = lane + 32 * v;
    if (FULL || vi < nvec)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst + vi * EV)), "l"(src + vi * EV)
                   : "memory");
  }
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// The threads of one node: a whole CTA of 16 warps, or one of its groups of
// four warps (named barrier 1 + group).
template <int SPLIT>
__device__ __forceinline__ void node_sync(int group) {
  if constexpr (SPLIT * 32 == 512)
    __syncthreads();
  else
    asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "n"(SPLIT * 32) : "memory");
}

// Each warp walks its rows in chunks of U with the ring slots of every chunk
// compile-time constants, refilling a chunk's slots with the rows STAGES
// chunks ahead as soon as its dot products have taken it into registers; every
// chunk commits one group (empty past the node's last row), so
// cp.async.wait_group STAGES-1 always means "this chunk is in".  When FULL the
// row length is the compile-time 32 * VPL * EV, so row offsets and sizes are
// constants.  A node's first STAGES chunks are sent before its prologue, which
// they overlap.  With BF16 rows (STASH) the node's phi row and its normals are
// read and drawn in the prologue and kept in shared memory for the epilogue.
// The first node of the `group` (of `groups` in the grid) is its own number;
// with DYNAMIC it takes the next ones from the buffer set's counter, one fetch
// per node, the last of which brings the counter back to zero: the SMs then
// share the nodes as they finish, without a wave of short CTAs.
template <typename PiT, int VPL, int SPLIT, int STAGES, bool FULL, bool DYNAMIC>
__device__ __forceinline__ void update_phi_ring_body(const Model& m, const Buffers& b, unsigned char* s_raw,
                                                     int group, int first, int groups) {
  using TR = PiTraits<PiT>;
  using Smem = PhiRingSmem<PiT, VPL, SPLIT, STAGES>;
  constexpr int U = ring_rows<PiT, VPL>(), ROWS = Smem::kRows;
  constexpr int EV = TR::kPerVec;
  constexpr int EPL = VPL * EV;
  constexpr int NT = SPLIT * 32;
  constexpr int NP = EPL / 2;  // float pairs per lane
  constexpr bool STASH = Smem::kStash;
  // thread's elements of a row: k0 = 4 * (tid + NT * g) .. k0 + 3, g < NG
  constexpr int NG = (EPL * 32 + 4 * NT - 1) / (4 * NT);
  const int Kp = FULL ? 32 * EPL : m.Kp;
  const int K = m.K, n_out = m.n_out;
  PiT* ring = reinterpret_cast<PiT*>(s_raw);
  float* s_w = reinterpret_cast<float*>(ring + (size_t)SPLIT * ROWS * Kp);
  float* s_phi = s_w + Kp;                    // STASH: the node's phi row
  float* s_nz = s_phi + Kp;                   // STASH: its normals
  float* s_red = s_w + (STASH ? 3 : 1) * Kp;  // 4*SPLIT + 8 floats
  uint32_t* s_nb = reinterpret_cast<uint32_t*>(s_red + 4 * SPLIT + 8);

  const int tid = threadIdx.x & (NT - 1), lane = tid & 31, warp = tid >> 5;
  const int n_nodes = b.st->n_nodes;
  const uint32_t step = b.st->step;
  const float eps_t = b.st->eps;
  const PiT* __restrict__ pi = reinterpret_cast<const PiT*>(b.pi);
  const int nvec = Kp / EV;
  int* s_next = reinterpret_cast<int*>(s_red + 4 * SPLIT);
  const Stream rs{m.seed, m.chain};

  PiT* my_ring = ring + (size_t)warp * ROWS * Kp;
  float* my_A = reinterpret_cast<float*>(my_ring);  // epilogue: this warp's A (Kp floats)

  int next = 0;
  for (int slot = first; slot < n_nodes; slot = DYNAMIC ? next : slot + groups) {
    if (DYNAMIC && tid == 0) next = groups + (int)atomicInc(&b.st->next_node, (unsigned)n_nodes - 1u);
    const int32_t i = b.nodes[slot];
    const float* phi_i = b.phi + (int64_t)i * Kp;
    const uint32_t* nbr_g = b.nbr + (int64_t)slot * n_out;
    // rows of this warp: q = warp + SPLIT * t, t < T
    const int T = (n_out > warp) ? (n_out - warp + SPLIT - 1) / SPLIT : 0;
    // the first chunks: ids read first, then every lane sends its pieces,
    // one commit group per chunk (empty past T), before the node prologue,
    // which they overlap
    uint32_t j0[ROWS];
#pragma unroll
    for (int t = 0; t < ROWS; ++t) j0[t] = (t < T) ? (nbr_g[warp + SPLIT * t] & 0x7fffffffu) : 0u;
    // (BF16) the thread's phi elements, loaded before the copies are sent
    float4 ph[STASH ? NG : 1];
    if constexpr (STASH) {
#pragma unroll
      for (int g = 0; g < NG; ++g) {
        const int k0 = 4 * (tid + NT * g);
        ph[g] = (k0 < Kp) ? *reinterpret_cast<const float4*>(phi_i + k0) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
#pragma unroll
    for (int t = 0; t < ROWS; ++t) {
      if (t < T) copy_row_lane<PiT, VPL, FULL>(my_ring + (size_t)t * Kp, pi + (int64_t)j0[t] * Kp, lane, nvec);
      if (t % U == U - 1) cp_async_commit();
    }
    float S, si;
    f32x2 w2[NP], A2[NP];
    // ---- node prologue: S = sum phi, s_i = sum pi, w = pi * (beta - eps)
    S = 0.f;
    if constexpr (STASH) {
      for (int q = tid; q < n_out; q += NT) s_nb[q] = nbr_g[q];
#pragma unroll
      for (int g = 0; g < NG; ++g) {
        const int k0 = 4 * (tid + NT * g);
        if (k0 < K) *reinterpret_cast<float4*>(s_nz + k0) = phi_normals(b, rs, slot, i, step, k0, K);
      }
#pragma unroll
      for (int g = 0; g < NG; ++g) S += (ph[g].x + ph[g].y) + (ph[g].z + ph[g].w);
    } else {
      for (int k = tid; k < Kp; k += NT) S += phi_i[k];
      for (int q = tid; q < n_out; q += NT) s_nb[q] = nbr_g[q];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) S += __shfl_xor_sync(0xffffffffu, S, o);
    if (lane == 0) s_red[warp] = S;
    node_sync<SPLIT>(group);
    // beta, read from here on, is written by the theta step ahead of this
    // launch; everything read before (node ids, neighbour words and rows,
    // phi) was complete before that step started
    grid_dependency_wait();
    grid_launch_dependents();
    S = 0.f;
#pragma unroll
    for (int w = 0; w < SPLIT; ++w) S += s_red[w];
    si = 0.f;
    if constexpr (STASH) {
      const float rS = 1.0f / S;  // pi = phi / S as phi * (1/S): within 1 ulp
#pragma unroll
      for (int g = 0; g < NG; ++g) {
        const int k0 = 4 * (tid + NT * g);
        if (k0 < Kp) {
          const float4 bt = *reinterpret_cast<const float4*>(b.beta + k0);
          float4 p, wv;
          p.x = ph[g].x * rS;
          p.y = ph[g].y * rS;
          p.z = ph[g].z * rS;
          p.w = ph[g].w * rS;
          si += p.x;
          si += p.y;
          si += p.z;
          si += p.w;
          wv.x = (k0 + 0 < K) ? p.x * (bt.x - m.epsilon) : 0.f;
          wv.y = (k0 + 1 < K) ? p.y * (bt.y - m.epsilon) : 0.f;
          wv.z = (k0 + 2 < K) ? p.z * (bt.z - m.epsilon) : 0.f;
          wv.w = (k0 + 3 < K) ? p.w * (bt.w - m.epsilon) : 0.f;
          *reinterpret_cast<float4*>(s_w + k0) = wv;
          *reinterpret_cast<float4*>(s_phi + k0) = ph[g];
        }
      }
    } else {
      for (int k = tid; k < Kp; k += NT) {
        const float p = __fdiv_rn(phi_i[k], S);
        si += p;
        s_w[k] = (k < K) ? p * (b.beta[k] - m.epsilon) : 0.f;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) si += __shfl_xor_sync(0xffffffffu, si, o);
    if (lane == 0) s_red[SPLIT + warp] = si;
    node_sync<SPLIT>(group);
    si = 0.f;
#pragma unroll
    for (int w = 0; w < SPLIT; ++w) si += s_red[SPLIT + w];
#pragma unroll
    for (int v = 0; v < VPL; ++v) {
      const int vi = lane + 32 * v;
#pragma unroll
      for (int e = 0; e < EV; e += 4) {
        float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
        if (FULL || vi < nvec) q = *reinterpret_cast<const float4*>(s_w + vi * EV + e);
        w2[(v * EV + e) / 2] = pack_f32x2(q.x, q.y);
        w2[(v * EV + e) / 2 + 1] = pack_f32x2(q.z, q.w);
        A2[(v * EV + e) / 2] = 0ull;
        A2[(v * EV + e) / 2 + 1] = 0ull;
      }
    }
    // the per-row constants of y = 1 and y = 0
    const float one_m_si = 1.0f - si;
    const float e1si = m.epsilon * si, e0si = (1.0f - m.epsilon) * si;
    const float e1o = m.epsilon * one_m_si, e0o = (1.0f - m.epsilon) * one_m_si;
    float Bsum = 0.f;
    for (int t0 = 0; t0 < T; t0 += ROWS) {
#pragma unroll
      for (int u = 0; u < STAGES; ++u) {
        const int t = t0 + u * U;  // rows t .. t + U - 1, in slots u * U ..
        if (t >= T) break;
        // one group per chunk, so the lane's pieces of it are in once no
        // more than the STAGES - 1 later groups are pending
        cp_async_wait<STAGES - 1>();
        // neighbour words of the rows, and of those that refill their slots
        uint32_t nbw[U], nxt[U];
        f32x2 x2[U][NP], d2[U][4];
#pragma unroll
        for (int r = 0; r < U; ++r) {
          const int tn = t + r + ROWS;
          nbw[r] = (r == 0 || t + r < T) ? s_nb[warp + SPLIT * (t + r)] : 0u;
          nxt[r] = (tn < T) ? s_nb[warp + SPLIT * tn] : 0u;
        }
#pragma unroll
        for (int r = 0; r < U; ++r) {
          if (r > 0 && t + r >= T) break;
          load_row_pairs<PiT, VPL, FULL>(my_ring + (size_t)(u * U + r) * Kp, lane, nvec, x2[r]);
          // four independent pair accumulators break the FMA dependency chain
#pragma unroll
          for (int e = 0; e < 4; ++e) d2[r][e] = 0ull;
#pragma unroll
          for (int e = 0; e < NP; ++e) d2[r][e & 3] = fma_f32x2(w2[e], x2[r][e], d2[r][e & 3]);
        }
        // refill the lane's pieces of the chunk's slots (read above, now in
        // registers)
#pragma unroll
        for (int r = 0; r < U; ++r)
          if (t + r + ROWS < T)
            copy_row_lane<PiT, VPL, FULL>(my_ring + (size_t)(u * U + r) * Kp,
                                          pi + (int64_t)(nxt[r] & 0x7fffffffu) * Kp, lane, nvec);
        cp_async_commit();
        float D[U];
#pragma unroll
        for (int r = 0; r < U; ++r) {
          float lo = 0.f, hi = 0.f;
          if (r == 0 || t + r < T)
            unpack_f32x2(add_f32x2(add_f32x2(d2[r][0], d2[r][1]), add_f32x2(d2[r][2], d2[r][3])), lo, hi);
          D[r] = lo + hi;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
          for (int r = 0; r < U; ++r) D[r] += __shfl_xor_sync(0xffffffffu, D[r], o);
#pragma unroll
        for (int r = 0; r < U; ++r) {
          if (r > 0 && t + r >= T) break;
          const bool y = (nbw[r] >> 31) != 0;
          const float Ds = y ? D[r] : -D[r];
          const float P = Ds + (y ? e1si : e0si);
          const float invP = rcp_approx(P);
          const float cj = y ? invP : -invP;
          Bsum += ((y ? e1o : e0o) - Ds) * invP;
          const f32x2 c2 = pack_f32x2(cj, cj);
#pragma unroll
          for (int e = 0; e < NP; ++e) A2[e] = fma_f32x2(c2, x2[r][e], A2[e]);
        }
      }
    }
    // every copy of the node is in (the groups after the last row are
    // empty); the A vectors below reuse the ring
    __syncwarp();
    // ---- publish A (into this warp's own ring slice, now idle) and B
#pragma unroll
    for (int v = 0; v < VPL; ++v) {
      const int vi = lane + 32 * v;
      if (FULL || vi < nvec) {
#pragma unroll
        for (int e = 0; e < EV; e += 4) {
          float4 q;
          unpack_f32x2(A2[(v * EV + e) / 2], q.x, q.y);
          unpack_f32x2(A2[(v * EV + e) / 2 + 1], q.z, q.w);
          *reinterpret_cast<float4*>(my_A + vi * EV + e) = q;
        }
      }
    }
    if (lane == 0) s_red[2 * SPLIT + warp] = Bsum;
    if (DYNAMIC && tid == 0) *s_next = next;
    node_sync<SPLIT>(group);
    if (DYNAMIC) next = *s_next;
    float Bt = 0.f;
#pragma unroll
    for (int w2i = 0; w2i < SPLIT; ++w2i) Bt += s_red[2 * SPLIT + w2i];
    const float invS = 1.0f / S;
    const float half_eps = eps_t / 2.0f;
    float* phi_w = b.phi + (int64_t)i * Kp;
    float pn[NG][4];
    float Snew = 0.f;
#pragma unroll
    for (int g = 0; g < NG; ++g) {
      const int k0 = 4 * (tid + NT * g);
      float nz[4] = {0.f, 0.f, 0.f, 0.f};
      float Ak[4] = {0.f, 0.f, 0.f, 0.f};
      float phk[4] = {0.f, 0.f, 0.f, 0.f};
      float btk[4] = {0.f, 0.f, 0.f, 0.f};
      if (k0 < K) {
        if constexpr (STASH) {
          const float4 q = *reinterpret_cast<const float4*>(s_nz + k0);
          const float4 r = *reinterpret_cast<const float4*>(s_phi + k0);
          nz[0] = q.x, nz[1] = q.y, nz[2] = q.z, nz[3] = q.w;
          phk[0] = r.x, phk[1] = r.y, phk[2] = r.z, phk[3] = r.w;
        } else {
          const float4 q = phi_normals(b, rs, slot, i, step, k0, K);
          nz[0] = q.x, nz[1] = q.y, nz[2] = q.z, nz[3] = q.w;
#pragma unroll
          for (int e = 0; e < 4; ++e) phk[e] = (k0 + e < K) ? phi_i[k0 + e] : 0.f;
        }
        const float4 bt = *reinterpret_cast<const float4*>(b.beta + k0);
        btk[0] = bt.x, btk[1] = bt.y, btk[2] = bt.z, btk[3] = bt.w;
        // A_k: the warps' partial sums, added in warp order (Kp is a
        // multiple of 4, so the four elements lie inside the row)
#pragma unroll
        for (int s = 0; s < SPLIT; ++s) {
          const float4 a = *reinterpret_cast<const float4*>(
              reinterpret_cast<const float*>(ring + (size_t)s * ROWS * Kp) + k0);
          Ak[0] += a.x;
          Ak[1] += a.y;
          Ak[2] += a.z;
          Ak[3] += a.w;
        }
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int k = k0 + e;
        float val = 0.f;
        if (k < K) {
          const float bk = btk[e] - m.epsilon;
          const float grad = (bk * Ak[e] + Bt) * invS;
          const float ph = phk[e];
          val = fabsf((ph + half_eps * (m.alpha - ph + m.Nn * grad)) + sqrtf(eps_t * ph) * nz[e]);
          if (val < 1.0e-24f) val = 1.0e-24f;
        }
        pn[g][e] = val;
        Snew += val;
      }
      if (k0 < K) {
        if (k0 + 3 < K) {
          *reinterpret_cast<float4*>(phi_w + k0) = make_float4(pn[g][0], pn[g][1], pn[g][2], pn[g][3]);
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (k0 + e < K) phi_w[k0 + e] = pn[g][e];
        }
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) Snew += __shfl_xor_sync(0xffffffffu, Snew, o);
    if (lane == 0) s_red[3 * SPLIT + warp] = Snew;
    node_sync<SPLIT>(group);
    Snew = 0.f;
#pragma unroll
    for (int w2i = 0; w2i < SPLIT; ++w2i) Snew += s_red[3 * SPLIT + w2i];
    float* st = b.stage + (int64_t)slot * Kp;
    const float rSnew = 1.0f / Snew;  // the new pi row as phi * (1/S'): within 1 ulp
#pragma unroll
    for (int g = 0; g < NG; ++g) {
      const int k0 = 4 * (tid + NT * g);
      if (k0 < Kp) {
        float4 o;
        o.x = (k0 + 0 < K) ? pn[g][0] * rSnew : 0.f;
        o.y = (k0 + 1 < K) ? pn[g][1] * rSnew : 0.f;
        o.z = (k0 + 2 < K) ? pn[g][2] * rSnew : 0.f;
        o.w = (k0 + 3 < K) ? pn[g][3] * rSnew : 0.f;
        *reinterpret_cast<float4*>(st + k0) = o;
      }
    }
    node_sync<SPLIT>(group);  // smem reuse by the next node
  }
}
// One launch for both kinds of iteration, which the node count picks: up to
// `few` nodes (the link stratum: one vertex and its edges) take 16 warps each,
// a node per CTA, so that a node's rows are in flight together; more take
// four warps each, four nodes to the CTA.  (With a launch per kind, the one
// without work stood between the theta step and the update: 5 us of a
// link-stratum iteration.)  A CTA of 16 warps at up to 128 registers fills an
// SM.  `parts`: the kinds this launch may do (kPhiFew, kPhiMany); ring depths
// of which four groups do not fit shared memory take a launch per kind, the
// second with as many groups per CTA as fit.
constexpr int kPhiFew = 1, kPhiMany = 2;
constexpr int kPhiGroup = 4 * 32;  // threads of a four-warp node
template <typename PiT>
__host__ __device__ constexpr int ring_few_stages() { return sizeof(PiT) == 2 ? 4 : 2; }

template <typename PiT, int VPL, int STAGES, bool FULL>
__device__ __forceinline__ void update_phi_ring_any(const Model& m, const Buffers& b, int few, int parts, int block,
                                                    int blocks) {
  extern __shared__ __align__(128) unsigned char s_ring[];
  const int n_nodes = b.st->n_nodes;
  if (n_nodes <= few) {
    if (parts & kPhiFew)
      update_phi_ring_body<PiT, VPL, 16, ring_few_stages<PiT>(), FULL, false>(m, b, s_ring, 0, block, blocks);
  } else if (parts & kPhiMany) {
    const int per = blockDim.x / kPhiGroup, group = threadIdx.x / kPhiGroup;
    const int Kp = FULL ? 32 * VPL * PiTraits<PiT>::kPerVec : m.Kp;
    update_phi_ring_body<PiT, VPL, 4, STAGES, FULL, true>(
        m, b, s_ring + group * PhiRingSmem<PiT, VPL, 4, STAGES>::bytes(Kp, m.n_out), group,
        block * per + group, blocks * per);
  }
  // CTAs with no work wait for the kernel ahead before they exit, so that
  // this launch completes after it
  grid_dependency_wait();
}
template <typename PiT, int VPL, int STAGES, bool FULL>
__global__ void __launch_bounds__(512, 1) k_update_phi_ring(Model m, Buffers b, int few, int parts) {
  update_phi_ring_any<PiT, VPL, STAGES, FULL>(m, b, few, parts, blockIdx.x, gridDim.x);
}
template <typename PiT, int VPL, int STAGES, bool FULL>
__global__ void __launch_bounds__(512, 1) k_update_phi_ring_chains(const ChainArgs* __restrict__ c,
                                                                   const BlockOf* __restrict__ map, int p, int few,
                                                                   int parts) {
  const BlockOf o = map[blockIdx.x];
  const ChainArgs& a = c[o.chain];
  update_phi_ring_any<PiT, VPL, STAGES, FULL>(a.m, slot_buffers(a.m, a.b, p), few, parts, o.block, o.blocks);
}

}  // namespace ammsb
