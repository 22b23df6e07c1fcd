// The MeshProcessor sweep steps for one primitive (dual) and one vertex
// (primal), shared by the whole-mesh kernels (bmf_process.cu, bmf_extract.cu)
// and the chunk-by-chunk kernel (bmf_extract.cu).  MeshProcessor.cpp:130-306.
//
// A primitive's dual point and normal are kept as ((float4*)dual_p)[t] = (p, n.x)
// and ((float2*)dual_n)[t] = (n.y, n.z): one 16-byte and one 8-byte gather per
// primitive in the primal step instead of six 4-byte ones.
#pragma once

#include "bmf_device.cuh"
#include "bmf_internal.h"

namespace bmf {

// Threads of the chunk-by-chunk sweep kernel's CTA and CTAs per SM (1024 x 2 at
// 32 registers: full occupancy).
constexpr int kSweepThreads = 1024, kSweepCtas = 2;

// Thread-block clusters: this CTA's rank, the cluster's size, a barrier over
// it (release / acquire at cluster scope: what its CTAs wrote to global memory
// before is visible to all of them after), and a store into the same shared
// variable of another CTA.
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_size() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_barrier() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_store(uint32_t* p, uint32_t rank, uint32_t v) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
  asm volatile(
      "{\n\t.reg .u32 ra;\n\tmapa.shared::cluster.u32 ra, %0, %1;\n\tst.shared::cluster.u32 [ra], %2;\n\t}" ::"r"(a),
      "r"(rank), "r"(v)
      : "memory");
}

constexpr int kTeamThreads = 512;
// Vertices per CTA that make the team one CTA larger.  Whole calls, us, at 128 / 256 / 512 /
// 1024: 33^3 75 / 75 / 79 / 91, 65^3 76 / 77 / 81 / 98, 129^3 110 / 110 / 112 / 128, Mode Q
// 65^3 with eight sweeps 92 / 94 / 97 / 116, fit step 65^3 167 / 165 / 171 / 202.
constexpr int kTeamVerts = 256;
constexpr int kTeamRegs = 6;     // list entries gathered at once (and kept for a thread's first vertex)

// Barrier over the team's CTAs (all resident: a cooperative launch).  The wait
// is bounded: after `limit` polls (a second or so) or once another CTA has
// given up, the CTA marks the team failed and no longer waits anywhere, so that
// every CTA comes to team_leave; the host finds the object's mark.  Thread 0 releases the CTA's
// stores with its arrival and acquires the others' with its polls, and the block
// barriers carry both to the other threads; sequentially consistent fences around
// a relaxed arrival cost 0.3 us more a meeting (129^3 chunk: 117.8 against 113.8 us).
constexpr unsigned kTeamSpins = 1u << 22;
__device__ __forceinline__ void team_barrier(TeamSync* y, unsigned* host_failed, unsigned& target, unsigned team,
                                             bool& dead, unsigned limit = kTeamSpins) {
  __syncthreads();
  target += team;
  if (threadIdx.x == 0 && team > 1 && !dead) {
    // release: the CTA's stores (ordered before by the block barrier) come before the arrival
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&y->arrived) : "memory");
    unsigned v = 0;
    for (unsigned spins = 0;; ++spins) {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(&y->arrived) : "memory");
      if (v >= target) break;
      if (spins >= limit || ((spins & 1023u) == 1023u && *(volatile unsigned*)&y->failed)) {
        *(volatile unsigned*)&y->failed = 1u;
        *(volatile unsigned*)host_failed = 1u;
        __threadfence();  // before this CTA leaves
        dead = true;  // this CTA waits nowhere any more
        break;
      }
    }
  }
  __syncthreads();
}
// The team's last CTA leaves the barrier as the first launch found it, also after a
// wait that ran out: nothing of a failed launch is left for the next one.
__device__ __forceinline__ void team_leave(TeamSync* y, unsigned team) {
  __syncthreads();
  if (threadIdx.x == 0 && atomicAdd(&y->left, 1u) == team - 1u) {
    __threadfence();  // behind the others' last words
    y->arrived = y->left = y->failed = 0u;
  }
}

// COH selects the load for data that the same kernel also writes (positions,
// normals and dual values where one launch runs every sweep, and its
// adjacency): a plain L1-cached load, which barriers order.  Otherwise the
// read-only path.
template <bool COH, typename T>
__device__ __forceinline__ T sweep_ld(const T* p) {
  if (COH) return __ldca(p);
  return __ldg(p);
}

__device__ __forceinline__ void nrm3(const float v[3], float o[3]) {
  const float l2 = (v[0] * v[0] + v[1] * v[1]) + v[2] * v[2];
  const float inv = 1.0f / sqrtf(l2);
  o[0] = v[0] * inv;
  o[1] = v[1] * inv;
  o[2] = v[2] * inv;
}
__device__ __forceinline__ void cross3(const float a[3], const float b[3], float o[3]) {
  o[0] = a[1] * b[2] - b[1] * a[2];
  o[1] = a[2] * b[0] - b[2] * a[0];
  o[2] = a[0] * b[1] - b[0] * a[1];
}

template <int N, typename I>
__device__ __forceinline__ void prim_corners(I t, I nvb, const uint32_t* __restrict__ idx, uint32_t v[N]) {
#pragma unroll
  for (int k = 0; k < N; ++k) {
    v[k] = __ldg(idx + N * t + k);
    if ((I)v[k] >= nvb) v[k] = 0;  // an index outside the mesh reads vertex 0 instead of faulting
  }
}

// Face normal of a primitive from its corner positions.
template <int N>
__device__ __forceinline__ void face_normal(const uint32_t v[N], const float P[N][3], float o[3]) {
  if (N == 3) {
    float a[3] = {0.0f, 0.0f, 0.0f}, b[3] = {0.0f, 0.0f, 0.0f}, na[3], nb[3];
    if (v[0] != v[1] && v[1] != v[2] && v[0] != v[2]) {
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        a[c] = P[0][c] - P[1][c];
        b[c] = P[0][c] - P[2][c];
      }
    }
    nrm3(a, na);
    nrm3(b, nb);
    cross3(na, nb, o);
#pragma unroll
    for (int c = 0; c < 3; ++c) o[c] = -o[c];
  } else {
    float a[3], b[3], na[3], nb[3], n1[3], n2[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      a[c] = P[0][c] - P[1][c];
      b[c] = P[0][c] - P[2][c];
    }
    nrm3(a, na);
    nrm3(b, nb);
    cross3(na, nb, n1);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      a[c] = P[2][c] - P[N - 1][c];
      b[c] = P[2][c] - P[0][c];
    }
    nrm3(a, na);
    nrm3(b, nb);
    cross3(na, nb, n2);
    if (isnan(n1[0])) {
      n1[0] = n2[0]; n1[1] = n2[1]; n1[2] = n2[2];
      if (isnan(n1[0])) { n1[0] = 0.0f; n1[1] = 1.0f; n1[2] = 0.0f; }
    }
    if (isnan(n2[0])) { n2[0] = n1[0]; n2[1] = n1[1]; n2[2] = n1[2]; }
    const float h[3] = {(n1[0] + n2[0]) * 0.5f, (n1[1] + n2[1]) * 0.5f, (n1[2] + n2[2]) * 0.5f};
    nrm3(h, o);
#pragma unroll
    for (int c = 0; c < 3; ++c) o[c] = -o[c];
  }
}

// optimize_dual_grid body (MeshProcessor.cpp:142-227) of primitive t with
// corners v.  I: the index type of t -- int64_t over a whole mesh, or uint32_t
// within one chunk (the arrays then start at the chunk).
template <int N, bool COH, typename I>
__device__ __forceinline__ void dual_corners(I t, const uint32_t v[N], const float* __restrict__ pos,
                                             const float* __restrict__ nrm, float* __restrict__ dual_p,
                                             float* __restrict__ dual_n, int normals) {
  // each corner position is loaded once; the centroid and the face normal
  // read the same registers
  float P[N][3];
#pragma unroll
  for (int k = 0; k < N; ++k)
#pragma unroll
    for (int c = 0; c < 3; ++c) P[k][c] = sweep_ld<COH>(pos + 3 * v[k] + c);
  float p[3] = {0.0f, 0.0f, 0.0f};
#pragma unroll
  for (int k = 0; k < N; ++k) {
#pragma unroll
    for (int c = 0; c < 3; ++c) p[c] = p[c] + P[k][c];
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) p[c] = p[c] / (float)N;
  if (normals == 0) {
    reinterpret_cast<float4*>(dual_p)[t] = make_float4(p[0], p[1], p[2], 0.0f);
    return;
  }
  float o[3] = {0.0f, 0.0f, 0.0f};
  if (normals == 1) {
    face_normal<N>(v, P, o);
  } else {
#pragma unroll
    for (int k = 0; k < N; ++k) {
#pragma unroll
      for (int c = 0; c < 3; ++c) o[c] = o[c] + sweep_ld<COH>(nrm + 3 * v[k] + c);
    }
  }
  reinterpret_cast<float4*>(dual_p)[t] = make_float4(p[0], p[1], p[2], o[0]);
  reinterpret_cast<float2*>(dual_n)[t] = make_float2(o[1], o[2]);
}
template <int N, bool COH = false, typename I = int64_t>
__device__ __forceinline__ void dual_prim(I t, I nvb, const uint32_t* __restrict__ idx,
                                          const float* __restrict__ pos, const float* __restrict__ nrm,
                                          float* __restrict__ dual_p, float* __restrict__ dual_n, int normals) {
  uint32_t v[N];
  prim_corners<N, I>(t, nvb, idx, v);
  dual_corners<N, COH, I>(t, v, pos, nrm, dual_p, dual_n, normals);
}

// A vertex that no primal step moves (no primitives, or a frozen boundary vertex).
template <bool COH>
__device__ __forceinline__ void primal_frozen(uint32_t v, const SweepStep& s, float* __restrict__ nrm) {
  if (s.dst != s.src) {
#pragma unroll
    for (int c = 0; c < 3; ++c) s.dst[3 * (size_t)v + c] = sweep_ld<COH>(s.src + 3 * (size_t)v + c);
  }
  if (s.skipped && nrm) nrm[3 * v] = nrm[3 * v + 1] = nrm[3 * v + 2] = 0.0f;
}

// The normal of vertex v whose n.y was 0 in the last face sweep: that of the
// last left-out face sweep whose n.y is not 0, from the positions before it
// (the sums in list order, as that sweep would have made them); it stays 0
// when none has.  Rare (walls exactly along y).  rel: the primitive that the
// list's ids count from.
template <int N, bool COH, typename AT>
__device__ __noinline__ void primal_older_normal(int64_t v, const AT* __restrict__ list, uint32_t n, uint32_t np_lim,
                                                 uint32_t rel, const uint32_t* __restrict__ idx, uint32_t nvb,
                                                 int skipped, const float* __restrict__ x0,
                                                 const float* __restrict__ x1, int iters, float* __restrict__ nrm) {
#pragma unroll 1
  for (int j = skipped - 1; j >= 0; --j) {
    const float* x = j == 1 ? x1 : x0;
    float nn[3] = {0.0f, 0.0f, 0.0f};
#pragma unroll 1
    for (uint32_t k = 0; k < n; ++k) {
      const uint32_t t = sweep_ld<COH>(list + k);
      if (t >= np_lim) continue;
      uint32_t w[N];
      float P[N][3], o[3];
      prim_corners<N, uint32_t>(rel + t, nvb, idx, w);
      for (int q = 0; q < N; ++q)
        for (int c = 0; c < 3; ++c) P[q][c] = sweep_ld<COH>(x + 3 * (int64_t)w[q] + c);
      face_normal<N>(w, P, o);
      for (int c = 0; c < 3; ++c) nn[c] = nn[c] + o[c];
    }
    for (int c = 0; c < 3; ++c) nn[c] = nn[c] / (float)n;
    if (sweep_colors(j, iters)) {
      float o[3];
      nrm3(nn, o);
      nn[0] = o[0]; nn[1] = o[1]; nn[2] = o[2];
    }
    if (nn[1] != 0.0f) {
      nrm[3 * v] = nn[0];
      nrm[3 * v + 1] = nn[1];
      nrm[3 * v + 2] = nn[2];
      return;
    }
  }
}

// optimize_primal_grid body (MeshProcessor.cpp:238-306) of vertex v in two
// parts.  The sums over the vertex's list of n entries, G of them gathered at
// once (first: the first G of them, where the caller keeps them), added in list
// order (the same rounding).  AT: the list's entry type; its ids count from
// primitive rel.  All lanes of the warp call it (n = 0: nothing to sum) and
// leave it together: without the barrier the lanes with short lists ran ahead
// into the divisions by themselves (19 instead of 27 lanes per instruction).
template <int G, bool NORMALS, bool COH, typename AT>
__device__ __forceinline__ void primal_sums(const AT* __restrict__ list, uint32_t n, uint32_t np_lim, uint32_t rel,
                                            const float* __restrict__ dual_p, const float* __restrict__ dual_n,
                                            float p[3], float nn[3], const uint32_t* first = nullptr) {
#pragma unroll
  for (int c = 0; c < 3; ++c) p[c] = nn[c] = 0.0f;
#pragma unroll 1
  for (uint32_t k0 = 0; k0 < n; k0 += G) {
    uint32_t t[G];
    float4 q[G];
    float2 r[G];
#pragma unroll
    for (int k = 0; k < G; ++k)
      t[k] = first && k0 == 0 ? first[k] : (k0 + k < n ? (uint32_t)sweep_ld<COH>(list + k0 + k) : 0xffffffffu);
#pragma unroll
    for (int k = 0; k < G; ++k) {
      q[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      r[k] = make_float2(0.0f, 0.0f);
      if (t[k] < np_lim) {  // never read past the dual points
        q[k] = sweep_ld<COH>(reinterpret_cast<const float4*>(dual_p) + (rel + t[k]));
        if (NORMALS) r[k] = sweep_ld<COH>(reinterpret_cast<const float2*>(dual_n) + (rel + t[k]));
      }
    }
#pragma unroll
    for (int k = 0; k < G; ++k) {
      if (t[k] < np_lim) {
        p[0] = p[0] + q[k].x; p[1] = p[1] + q[k].y; p[2] = p[2] + q[k].z;
        if (NORMALS) { nn[0] = nn[0] + q[k].w; nn[1] = nn[1] + r[k].x; nn[2] = nn[2] + r[k].y; }
      }
    }
  }
  __syncwarp();
}

// The vertex's new position and normal from the sums.  Returns whether it
// needs primal_older_normal (its normal is 0 until then).
template <bool NORMALS>
__device__ __forceinline__ bool primal_store(uint32_t v, uint32_t n, float p[3], float nn[3], float* __restrict__ dst,
                                             float* __restrict__ nrm, int set_colors, int skipped) {
  const float cnt = (float)n;
#pragma unroll
  for (int c = 0; c < 3; ++c) dst[3 * (size_t)v + c] = p[c] / cnt;
  // (without smoothed normals the colour step normalises a zero vector, and
  // the NaN it gives is written, MeshProcessor.cpp:276-290)
  if (!nrm || (!NORMALS && !set_colors)) return false;
  if (NORMALS) {
#pragma unroll
    for (int c = 0; c < 3; ++c) nn[c] = nn[c] / cnt;
  }
  if (set_colors) {
    float o[3];
    nrm3(nn, o);
    nn[0] = o[0]; nn[1] = o[1]; nn[2] = o[2];
  }
  const bool keep = nn[1] == 0.0f;  // (a NaN is written)
  if (keep && skipped) nn[0] = nn[2] = 0.0f;
  if (!keep || skipped) {
#pragma unroll
    for (int c = 0; c < 3; ++c) nrm[3 * (size_t)v + c] = nn[c];
  }
  return keep && skipped;
}

}  // namespace bmf
