// Stage 5: MeshProcessor<N> dual / primal smoothing and normals
// (MeshProcessor.cpp:26-306), in the order ChunkGenerator::extract_chunk runs
// it (ChunkGenerator.cpp:112-124): iters dual steps, a primal step after each
// but the last inside optimize_dual_grid, then one more primal step.
//
// The reference's sweeps are Jacobi-style (a dual step reads only vertex
// positions, a primal step reads only dual points), so every primitive and
// every vertex is independent: one thread each.  The one order that matters
// for bit-exact sums is the adjacency order: init_primitives appends prims to
// each vertex in ascending prim id (MeshProcessor.cpp:114-127).  The CSR
// fill uses atomic cursors and then sorts each (short) list.
#include "bmf_device.cuh"
#include "bmf_internal.h"
#include "bmf_sweep.cuh"

namespace bmf {

constexpr int kScanBlock = 1024;
constexpr int kScanPer = 4;

// Block-level exclusive scan of u8 counts -> u32 offsets; writes block totals.
__global__ void __launch_bounds__(kScanBlock) k_scan_u8_local(const uint8_t* __restrict__ in, uint32_t* __restrict__ out,
                                                             int64_t n, const int64_t* __restrict__ d_n,
                                                             uint32_t* __restrict__ block_tot) {
  __shared__ uint32_t warp_tot[kScanBlock / 32];
  const int64_t n_valid = d_n ? min(n, *d_n) : n;
  const int64_t i0 = ((int64_t)blockIdx.x * kScanBlock + threadIdx.x) * kScanPer;
  uint32_t v[kScanPer], s = 0;
#pragma unroll
  for (int k = 0; k < kScanPer; ++k) {
    v[k] = (i0 + k < n_valid) ? in[i0 + k] : 0u;
    s += v[k];
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t inc = s;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(kFull, inc, o);
    if (lane >= o) inc += t;
  }
  if (lane == 31) warp_tot[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    uint32_t w = warp_tot[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(kFull, w, o);
      if (lane >= o) w += t;
    }
    warp_tot[lane] = w;
  }
  __syncthreads();
  uint32_t e = (warp ? warp_tot[warp - 1] : 0u) + inc - s;
#pragma unroll
  for (int k = 0; k < kScanPer; ++k) {
    if (i0 + k < n) out[i0 + k] = e;
    e += v[k];
  }
  if (threadIdx.x == kScanBlock - 1) block_tot[blockIdx.x] = warp_tot[31];
}

// Scans the block totals in place (single CTA) and stores the grand total at [nb].
__global__ void __launch_bounds__(1024) k_scan_totals(uint32_t* __restrict__ t, int nb) {
  __shared__ uint32_t s[1024];
  uint32_t carry = 0;
  for (int base = 0; base < nb; base += 1024) {
    const int i = base + threadIdx.x;
    const uint32_t v = i < nb ? t[i] : 0u;
    s[threadIdx.x] = v;
    __syncthreads();
    for (int o = 1; o < 1024; o <<= 1) {
      const uint32_t a = threadIdx.x >= o ? s[threadIdx.x - o] : 0u;
      __syncthreads();
      s[threadIdx.x] += a;
      __syncthreads();
    }
    if (i < nb) t[i] = carry + s[threadIdx.x] - v;
    carry += s[1023];
    __syncthreads();
  }
  if (threadIdx.x == 0) t[nb] = carry;
}

__global__ void k_scan_add(uint32_t* __restrict__ out, int64_t n, const uint32_t* __restrict__ block_off) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] += block_off[i / ((int64_t)kScanBlock * kScanPer)];
}

void launch_exclusive_scan_u8_to_u32(const uint8_t* in, uint32_t* out, int64_t n, const int64_t* d_n,
                                     uint32_t* block_tmp, cudaStream_t st) {
  const int64_t per = (int64_t)kScanBlock * kScanPer;
  const int nb = (int)((n + per - 1) / per);
  if (nb == 0) return;
  k_scan_u8_local<<<nb, kScanBlock, 0, st>>>(in, out, n, d_n, block_tmp);
  k_scan_totals<<<1, 1024, 0, st>>>(block_tmp, nb);
  k_scan_add<<<(int)((n + 255) / 256), 256, 0, st>>>(out, n, block_tmp);
  // off[n] = total
  cudaMemcpyAsync(out + n, block_tmp + nb, sizeof(uint32_t), cudaMemcpyDeviceToDevice, st);
}

// set_adj (MeshRecursion.hpp:173-190): adj[off[v] + k] = prim.
__global__ void k_fill_adj(int N, int64_t n_slots, int64_t nv, const int64_t* __restrict__ d_counts,
                           const uint32_t* __restrict__ idx, const uint32_t* __restrict__ off,
                           const uint8_t* __restrict__ valence, uint32_t* __restrict__ cursor,
                           uint32_t* __restrict__ adj) {
  const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= (d_counts ? min(n_slots, d_counts[1] / N * N) : n_slots)) return;
  const uint32_t v = idx[j];
  if ((int64_t)v >= (d_counts ? min(nv, d_counts[0]) : nv)) return;  // an index outside the mesh is ignored
  const uint32_t k = atomicAdd(cursor + v, 1u);
  // a caller's valence may not sum to more than the index slots: stay inside adj
  if (k < valence[v] && (int64_t)off[v] + k < n_slots) adj[off[v] + k] = (uint32_t)(j / N);
}

// Restores ascending prim order in each vertex's list (insertion sort; the
// lists hold at most a few dozen entries).
__global__ void k_sort_adj(int64_t nv, int64_t adj_cap, const int64_t* __restrict__ d_counts,
                           const uint32_t* __restrict__ off, const uint32_t* __restrict__ cursor,
                           const uint8_t* __restrict__ valence, uint32_t* __restrict__ adj) {
  const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= (d_counts ? min(nv, d_counts[0]) : nv)) return;
  const int64_t room = adj_cap - (int64_t)off[v];
  const uint32_t n = (uint32_t)max((int64_t)0, min((int64_t)min(cursor[v], (uint32_t)valence[v]), room));
  uint32_t* a = adj + off[v];
  for (uint32_t i = 1; i < n; ++i) {
    const uint32_t key = a[i];
    int j = (int)i - 1;
    while (j >= 0 && a[j] > key) {
      a[j + 1] = a[j];
      --j;
    }
    a[j + 1] = key;
  }
}

template <int N>
__global__ void k_dual(int64_t n_prims, int64_t nv, const int64_t* __restrict__ d_counts,
                       const uint32_t* __restrict__ idx, const float* __restrict__ pos, const float* __restrict__ nrm,
                       float* __restrict__ dual_p, float* __restrict__ dual_n, int normals) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (d_counts ? min(n_prims, d_counts[1] / N) : n_prims)) return;
  dual_prim<N>(t, d_counts ? min(nv, d_counts[0]) : nv, idx, pos, nrm, dual_p, dual_n, normals);
}

// optimize_primal_grid (MeshProcessor.cpp:238-306).  cursor (nullable): list
// lengths where the lists were filled from the indices.
template <int N>
__global__ void k_primal(int64_t nv, int64_t n_prims, int64_t adj_cap, const int64_t* __restrict__ d_counts,
                         const uint32_t* __restrict__ off, const uint32_t* __restrict__ cursor,
                         const uint8_t* __restrict__ valence, const uint32_t* __restrict__ adj,
                         const uint8_t* __restrict__ boundary, const float* __restrict__ dual_p,
                         const float* __restrict__ dual_n, const uint32_t* __restrict__ idx, SweepStep st, SweepBufs b,
                         int iters, int process_boundary) {
  const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t nvb = d_counts ? min(nv, d_counts[0]) : nv;
  uint32_t o = 0u, n = 0u;
  if (v < nvb) {
    // list length: adj_next (MeshProcessor.cpp:247); with a prebuilt adjacency it equals init_valence
    const uint32_t val = valence[v];
    const bool frozen = !process_boundary && boundary[v];
    o = __ldg(off + v);
    n = (uint32_t)max((int64_t)0, min((int64_t)(cursor ? min(cursor[v], val) : val), adj_cap - (int64_t)o));
    if (frozen) n = 0u;
  }
  const uint32_t np_lim = (uint32_t)min(n_prims, (int64_t)UINT32_MAX);
  float p[3], nn[3];
  if (st.normals == 0)
    primal_sums<4, false, false>(adj + o, n, np_lim, 0u, dual_p, dual_n, p, nn);
  else
    primal_sums<4, true, false>(adj + o, n, np_lim, 0u, dual_p, dual_n, p, nn);
  if (n == 0u) {
    if (v < nvb) primal_frozen<false>((uint32_t)v, st, b.nrm);
  } else if (st.normals == 0) {
    primal_store<false>((uint32_t)v, n, p, nn, st.dst, b.nrm, st.set_colors, 0);
  } else if (primal_store<true>((uint32_t)v, n, p, nn, st.dst, b.nrm, st.set_colors, st.skipped)) {
    primal_older_normal<N, false>(v, adj + o, n, np_lim, 0u, idx, (uint32_t)min(nvb, (int64_t)UINT32_MAX),
                                  st.skipped, b.x[0], b.x[1], iters, b.nrm);
  }
}

// ---------------------------------------------------------------------------
// Draw layout (GLChunk::format_data, GLChunk.cpp:278-335): per-vertex p/n/c,
// or quads unwound to 4 vertices sharing one normal.  Colours are white: the
// vertex colour is (1, 1, 1) at creation (DMCChunk.cpp:681) and the sweeps
// only average it.  Counts come from d_counts (vertices, indices) when given.
// ---------------------------------------------------------------------------
__global__ void k_format_verts(int64_t nv, const int64_t* __restrict__ d_counts, int64_t cap,
                               const float* __restrict__ pos, const float* __restrict__ nrm, float* __restrict__ p,
                               float* __restrict__ n, float* __restrict__ c) {
  const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= min(cap, d_counts ? min(nv, d_counts[0]) : nv)) return;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    p[3 * v + k] = __ldg(pos + 3 * v + k);
    n[3 * v + k] = nrm ? __ldg(nrm + 3 * v + k) : 0.0f;
    c[3 * v + k] = 1.0f;
  }
}

// chunks (nullable): quad slots are arena positions and indices chunk-local;
// a quad's chunk is the last one whose index offset is <= its first slot.
__global__ void k_format_quads(const ChunkDev* __restrict__ chunks, int n_chunks, int64_t ni,
                               const int64_t* __restrict__ d_counts, int64_t cap, const float* __restrict__ pos,
                               const float* __restrict__ nrm, const uint32_t* __restrict__ idx, int smooth,
                               float* __restrict__ p, float* __restrict__ n, float* __restrict__ c) {
  const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t nidx = d_counts ? min(ni, d_counts[1]) : ni;
  const int64_t i = 4 * q;
  if (i + 3 >= nidx || i + 3 >= cap) return;
  int64_t vo = 0, nvb = d_counts ? d_counts[0] : INT64_MAX;
  if (chunks) {
    int lo = 0, hi = n_chunks - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (chunks[mid].iout <= i) lo = mid; else hi = mid - 1;
    }
    vo = chunks[lo].vout;
  }
  int64_t v[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    v[k] = vo + (int64_t)__ldg(idx + i + k);
    if (v[k] >= nvb) v[k] = 0;  // an index outside the mesh reads vertex 0 instead of faulting
  }
  float P[4][3];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
#pragma unroll
    for (int d = 0; d < 3; ++d) P[k][d] = __ldg(pos + 3 * v[k] + d);
  }
  float m[3];
  if (smooth) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      float s = __ldg(nrm + 3 * v[0] + d) + __ldg(nrm + 3 * v[1] + d);
      s = s + __ldg(nrm + 3 * v[2] + d);
      s = s + __ldg(nrm + 3 * v[3] + d);
      m[d] = s * 0.25f;
    }
  } else {
    float a[3], b[3], na[3], nb[3], m0[3], m1[3], h[3], o[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      a[d] = P[0][d] - P[1][d];
      b[d] = P[0][d] - P[2][d];
    }
    nrm3(a, na);
    nrm3(b, nb);
    cross3(na, nb, m0);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      a[d] = P[2][d] - P[3][d];
      b[d] = P[2][d] - P[0][d];
    }
    nrm3(a, na);
    nrm3(b, nb);
    cross3(na, nb, m1);
    if (isnan(m0[0])) { m0[0] = m1[0]; m0[1] = m1[1]; m0[2] = m1[2]; }
    if (isnan(m1[0])) { m1[0] = m0[0]; m1[1] = m0[1]; m1[2] = m0[2]; }
#pragma unroll
    for (int d = 0; d < 3; ++d) h[d] = (m0[d] + m1[d]) * 0.5f;
    nrm3(h, o);
#pragma unroll
    for (int d = 0; d < 3; ++d) m[d] = -o[d];
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      p[3 * (i + k) + d] = P[k][d];
      n[3 * (i + k) + d] = m[d];
      c[3 * (i + k) + d] = 1.0f;
    }
  }
}

int launch_format(const ChunkDev* d_chunks, int n_chunks, int64_t nv, int64_t ni, const int64_t* d_counts,
                  const float* pos, const float* nrm, const uint32_t* idx, int unwind, int smooth, float* p, float* n,
                  float* c, int64_t cap, cudaStream_t st) {
  if (!unwind) {
    if (nv <= 0) return 0;
    k_format_verts<<<(int)((nv + 255) / 256), 256, 0, st>>>(nv, d_counts, cap, pos, nrm, p, n, c);
  } else {
    const int64_t nq = ni / 4;
    if (nq <= 0) return 0;
    k_format_quads<<<(int)((nq + 255) / 256), 256, 0, st>>>(d_chunks, n_chunks, ni, d_counts, cap, pos, nrm, idx,
                                                            smooth, p, n, c);
  }
  return 1;
}

// ---------------------------------------------------------------------------
// Adjoint of the position sweeps.  A dual step averages each primitive's N
// vertices; a primal step replaces every updated vertex (adjacency non-empty,
// not a frozen boundary vertex) by the mean of its primitives' dual points and
// leaves the others unchanged.  Both are linear in the positions and do not
// depend on them, so the backward needs no stored iterates: it applies the
// transposes, last sweep first.  Both transposes are gathers (per primitive /
// per vertex through the CSR), so they need no atomics.
// ---------------------------------------------------------------------------
//
// What the gathers read is stored ready for them, as float4: h[v] = g[v] / count(v)
// (0 for a vertex that is not updated) and g_dual[t] / N.  A primitive then
// sums four 16-byte gathers and a vertex its list's, instead of three 4-byte
// gathers, a valence, a boundary flag and a division per corner; the products
// and the order of the sums are the same.  Quads only (Mode Q).  Eight sweeps of
// 512 x 65^3: 780 -> 613 us chunk by chunk, bound by the L1's wavefronts; of one 65^3
// grid: sixteen launches of 4 us and the gaps between them -> 27 us as a team.
struct BwdArgs {
  int64_t nv, n_prims;
  const int64_t* __restrict__ d_counts;
  const uint32_t* __restrict__ off;
  const uint8_t *__restrict__ valence, *__restrict__ boundary;
  const uint32_t* __restrict__ adj;
  const uint32_t* __restrict__ idx;  // mesh-wide
  const float* __restrict__ grad;    // dL/d(final positions) of the first n_grad vertices (0 for the others)
  int64_t n_grad;
  float* g;       // dL/d(initial positions), and between the steps g of the vertices that are not updated
  float4* h;      // g / count of the updated ones
  float4* gd;     // g_dual / N
  int iters, process_boundary;
};

// Vertex v's list: its length on return; updated: whether the primal step moves it.
__device__ __forceinline__ uint32_t bwd_list(const BwdArgs& A, uint32_t v, uint32_t cap, uint32_t& o, uint32_t& val,
                                             bool& updated) {
  o = __ldg(A.off + v);
  val = __ldg(A.valence + v);
  updated = val != 0u && (A.process_boundary || !__ldg(A.boundary + v));
  return o < cap ? min(val, cap - o) : 0u;
}
__device__ __forceinline__ void bwd_put(const BwdArgs& A, uint32_t v, const float s[3], uint32_t val, bool updated,
                                        bool last) {
  if (updated && !last) {
    const float inv = 1.0f / (float)val;
    A.h[v] = make_float4(s[0] * inv, s[1] * inv, s[2] * inv, 0.0f);
  } else {
#pragma unroll
    for (int c = 0; c < 3; ++c) A.g[3 * (size_t)v + c] = s[c];
  }
}
// Before the first step.
__device__ __forceinline__ void bwd_begin(const BwdArgs& A, uint32_t v) {
  float s[3] = {0.0f, 0.0f, 0.0f};
  if ((int64_t)v < A.n_grad) {
#pragma unroll
    for (int c = 0; c < 3; ++c) s[c] = __ldg(A.grad + 3 * (size_t)v + c);
  }
  const uint32_t val = __ldg(A.valence + v);
  const bool updated = val != 0u && (A.process_boundary || !__ldg(A.boundary + v));
  if (!updated) A.h[v] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  bwd_put(A, v, s, val, updated, false);
}
// g_dual[t] / N from the sum over its corners.
__device__ __forceinline__ void bwd_prim(const BwdArgs& A, uint32_t t, const uint4 v, uint32_t nv) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
  float4 q[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) q[k] = w[k] < nv ? __ldca(A.h + w[k]) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  float s[3] = {0.0f, 0.0f, 0.0f};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    s[0] += q[k].x;
    s[1] += q[k].y;
    s[2] += q[k].z;
  }
  A.gd[t] = make_float4(s[0] * 0.25f, s[1] * 0.25f, s[2] * 0.25f, 0.0f);
}
// s += the list's g_dual / N, kBwdGather at once, in list order; all lanes of the warp call it.
constexpr int kBwdGather = 4;
template <int G>
__device__ __forceinline__ void bwd_sums(const BwdArgs& A, uint32_t o, uint32_t n, uint32_t np, float s[3],
                                         const uint32_t* first = nullptr) {
#pragma unroll 1
  for (uint32_t k0 = 0; k0 < n; k0 += G) {
    uint32_t t[G];
    float4 q[G];
#pragma unroll
    for (int k = 0; k < G; ++k)
      t[k] = first && k0 == 0 ? first[k] : (k0 + k < n ? __ldg(A.adj + o + k0 + k) : 0xffffffffu);
#pragma unroll
    for (int k = 0; k < G; ++k) q[k] = t[k] < np ? __ldca(A.gd + t[k]) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
    for (int k = 0; k < G; ++k)
      if (t[k] < np) {
        s[0] += q[k].x;
        s[1] += q[k].y;
        s[2] += q[k].z;
      }
  }
  __syncwarp();
}
// A backward primal step's vertex (whole warps; in: v is one).
__device__ __forceinline__ void bwd_vert(const BwdArgs& A, uint32_t v, bool in, uint32_t cap, uint32_t np, bool last) {
  uint32_t o = 0u, n = 0u, val = 0u;
  bool updated = true;
  float s[3] = {0.0f, 0.0f, 0.0f};
  if (in) {
    n = bwd_list(A, v, cap, o, val, updated);
    if (!updated) {
#pragma unroll
      for (int c = 0; c < 3; ++c) s[c] = A.g[3 * (size_t)v + c];
    }
  }
  bwd_sums<kBwdGather>(A, o, n, np, s);
  if (in) bwd_put(A, v, s, val, updated, last);
}

__device__ __forceinline__ void bwd_extent(const BwdArgs& A, uint32_t& nv, uint32_t& np) {
  nv = (uint32_t)(A.d_counts ? min(A.nv, A.d_counts[0]) : A.nv);
  np = (uint32_t)(A.d_counts ? min(A.n_prims, A.d_counts[1] / 4) : A.n_prims);
}

// The steps one launch each.
__global__ void k_bwd_begin(BwdArgs A) {
  uint32_t nv, np;
  bwd_extent(A, nv, np);
  const uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v < nv) bwd_begin(A, v);
}
__global__ void k_primal_bwd(BwdArgs A) {
  uint32_t nv, np;
  bwd_extent(A, nv, np);
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < np) bwd_prim(A, t, __ldg(reinterpret_cast<const uint4*>(A.idx) + t), nv);
}
__global__ void k_dual_bwd(BwdArgs A, bool last) {
  uint32_t nv, np;
  bwd_extent(A, nv, np);
  const uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
  bwd_vert(A, v, v < nv, (uint32_t)min(4 * A.n_prims, (int64_t)UINT32_MAX), np, last);
}

// Chunk by chunk: one CTA per chunk (from the queue) runs every backward step
// of its chunk with block barriers in between -- a chunk's primitives only
// read its own vertices and the reverse.  1024 threads, two CTAs per SM (fit steps, us,
// against 512 threads, four: 256 x 33^3 934 / 1004, 300 x 65^3 2497 / 2680, 512 x 65^3
// 3978 / 4016): fewer chunks at a time, and the last ones end sooner.
constexpr int kBwdChunkThreads = 1024;

__global__ void __launch_bounds__(kBwdChunkThreads, 2) k_sweep_bwd_chunks(const ChunkDev* __restrict__ chunks,
                                                                         const uint32_t* __restrict__ tot,
                                                                         const int* __restrict__ order,
                                                                         const int* __restrict__ head,
                                                                         int* __restrict__ queue,
                                                                         const __grid_constant__ BwdArgs A) {
  __shared__ int s_item;
  uint32_t nv, np;
  bwd_extent(A, nv, np);
  const uint32_t cap = (uint32_t)min(4 * A.n_prims, (int64_t)UINT32_MAX);
  const int n_list = head[1];
  for (;;) {
    if (threadIdx.x == 0) s_item = atomicAdd(queue, 1);
    __syncthreads();
    const int it = s_item;
    __syncthreads();  // everyone has read s_item before thread 0 takes the next
    if (it >= n_list) break;
    const int c = order[it];
    const int64_t vo = chunks[c].vout, po = chunks[c].iout / 4;
    const uint32_t v0 = (uint32_t)vo, v1 = (uint32_t)min(vo + (int64_t)tot[2 * c], (int64_t)nv);
    const uint32_t p0 = (uint32_t)po, p1 = (uint32_t)min(po + (int64_t)(tot[2 * c + 1] / 4), (int64_t)np);
    for (uint32_t v = v0 + threadIdx.x; v < v1; v += kBwdChunkThreads) bwd_begin(A, v);
    __syncthreads();
    for (int m = A.iters - 1; m >= 0; --m) {
      for (uint32_t t = p0 + threadIdx.x; t < p1; t += kBwdChunkThreads)
        bwd_prim(A, t, __ldg(reinterpret_cast<const uint4*>(A.idx) + t), nv);
      __syncthreads();
      for (uint32_t v = v0 + threadIdx.x; v - (threadIdx.x & 31u) < v1; v += kBwdChunkThreads)
        bwd_vert(A, v, v < v1, cap, np, m == 0);
      __syncthreads();
    }
  }
}

// The whole mesh in one cooperative launch (as the forward's team, which also
// says when): the team's CTAs keep their vertices and primitives, a thread its
// first vertex's list and its first primitive's corners.
__global__ void __launch_bounds__(kTeamThreads, 1) k_sweep_bwd_team(const __grid_constant__ BwdArgs A, TeamSync* sync,
                                                                   unsigned* host_failed) {
  uint32_t nv, np;
  bwd_extent(A, nv, np);
  const uint32_t cap = (uint32_t)min(4 * A.n_prims, (int64_t)UINT32_MAX);
  const unsigned team = min(gridDim.x, max(1u, (nv + kTeamVerts - 1u) / kTeamVerts)), rank = blockIdx.x;
  if (rank >= team || nv == 0u) return;
  const uint32_t tid = threadIdx.x, lane = tid & 31u;
  unsigned target = 0;
  bool dead = false;
  const uint32_t vs = (nv + team - 1u) / team, ps = (np + team - 1u) / team;
  const uint32_t va = min(rank * vs, nv), ve = min(va + vs, nv), pa = min(rank * ps, np), pe = min(pa + ps, np);
  for (uint32_t v = va + tid; v < ve; v += kTeamThreads) bwd_begin(A, v);
  const uint4* quads = reinterpret_cast<const uint4*>(A.idx);
  const uint32_t v_own = va + tid, p_own = pa + tid;
  const uint4 c_own = p_own < pe ? __ldg(quads + p_own) : make_uint4(0u, 0u, 0u, 0u);
  uint32_t o_own = 0u, n_own = 0u, val_own = 0u, ids[kTeamRegs] = {};
  bool upd_own = true;
  if (v_own < ve) {
    n_own = bwd_list(A, v_own, cap, o_own, val_own, upd_own);
#pragma unroll
    for (int k = 0; k < kTeamRegs; ++k) ids[k] = k < (int)n_own ? __ldg(A.adj + o_own + k) : 0xffffffffu;
  }
  team_barrier(sync, host_failed, target, team, dead);
  for (int m = A.iters - 1; m >= 0; --m) {
    for (uint32_t t = p_own; t < pe; t += kTeamThreads) bwd_prim(A, t, t == p_own ? c_own : __ldg(quads + t), nv);
    team_barrier(sync, host_failed, target, team, dead);
    float s[3] = {0.0f, 0.0f, 0.0f};
    if (v_own < ve && !upd_own) {
#pragma unroll
      for (int c = 0; c < 3; ++c) s[c] = A.g[3 * (size_t)v_own + c];
    }
    bwd_sums<kTeamRegs>(A, o_own, n_own, np, s, ids);
    if (v_own < ve) bwd_put(A, v_own, s, val_own, upd_own, m == 0);
    for (uint32_t v = v_own + kTeamThreads; v - lane < ve; v += kTeamThreads) bwd_vert(A, v, v < ve, cap, np, m == 0);
    if (m > 0) team_barrier(sync, host_failed, target, team, dead);
  }
  team_leave(sync, team);
}

// One CTA of a team of two: its wait runs out after `limit` polls, and it leaves.
__global__ void __launch_bounds__(32) k_team_timeout(TeamSync* sync, unsigned* host_failed, unsigned limit) {
  unsigned target = 0;
  bool dead = false;
  team_barrier(sync, host_failed, target, 2u, dead, limit);
  team_leave(sync, 1u);
}
void launch_team_timeout(TeamSync* sync, unsigned* host_failed, cudaStream_t st) {
  k_team_timeout<<<1, 32, 0, st>>>(sync, host_failed, 1024u);
}

int launch_process_bwd(int64_t nv, int64_t n_prims, const int64_t* d_counts, const uint8_t* boundary,
                       const uint8_t* valence, const uint32_t* idx, int iters, int process_boundary,
                       const ProcessScratch& s, const float* grad, int64_t n_grad, float* g, float* h,
                       const StructuredAdj* sa, cudaStream_t st) {
  BwdArgs A{nv,  n_prims, d_counts, s.off, valence, boundary, s.adj, idx, grad, n_grad, g, reinterpret_cast<float4*>(h),
            reinterpret_cast<float4*>(s.dual_p), iters, process_boundary};
  if (sa->tot && sa->bwd_queue) {
    static std::atomic<int> slots[64] = {};
    const int grid = per_device_once(slots, [](int dev) {
      int sms = 0, per_sm = 0;
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_sweep_bwd_chunks, kBwdChunkThreads, 0);
      return (sms > 0 ? sms : 1) * (per_sm > 0 ? per_sm : 1);
    });
    cudaMemsetAsync(sa->bwd_queue, 0, sizeof(int), st);
    k_sweep_bwd_chunks<<<grid, kBwdChunkThreads, 0, st>>>(sa->chunks, sa->tot, sa->lists.order, sa->lists.head,
                                                         sa->bwd_queue, A);
    return 1;
  }
  if (sa->team) {
    static std::atomic<int> slots[64] = {};
    const int grid = per_device_once(slots, [](int dev) {
      int sms = 0, per_sm = 0;
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_sweep_bwd_team, kTeamThreads, 0);
      return per_sm > 0 ? min(sms, kTeamMax) : -1;
    });
    if (grid > 0) {
      cudaLaunchConfig_t cfg{};
      cudaLaunchAttribute at{};
      at.id = cudaLaunchAttributeCooperative;
      at.val.cooperative = 1;
      cfg.gridDim = dim3(grid);
      cfg.blockDim = dim3(kTeamThreads);
      cfg.stream = st;
      cfg.attrs = &at;
      cfg.numAttrs = 1;
      cudaLaunchKernelEx(&cfg, k_sweep_bwd_team, A, sa->team, sa->team_failed);
      return 1;
    }
  }
  const int vb = (int)((nv + 255) / 256), pb = (int)((n_prims + 255) / 256);
  k_bwd_begin<<<vb, 256, 0, st>>>(A);
  for (int m = iters - 1; m >= 0; --m) {
    k_primal_bwd<<<pb, 256, 0, st>>>(A);
    k_dual_bwd<<<vb, 256, 0, st>>>(A, m == 0);
  }
  return 2 * iters + 1;
}

int launch_process(int N, int64_t nv, int64_t n_prims, const int64_t* d_counts, float* pos, float* nrm,
                   const uint8_t* boundary, const uint8_t* valence, const uint32_t* idx, int iters,
                   int process_boundary, int smooth_normals, ProcessScratch s, const StructuredAdj* sa,
                   cudaStream_t st) {
  if (nv == 0 || iters <= 0 || (n_prims == 0 && !s.x[0])) return 0;
  const int64_t n_slots = n_prims * N;
  const bool sn = smooth_normals != 0 && nrm != nullptr;
  if (sa && sa->tot && sa->lists.order) {
    launch_sweep_chunks(*sa, N, nv, n_prims, d_counts, pos, nrm, boundary, valence, idx, iters, process_boundary,
                        sn ? 1 : 0, s, st);
    return 1;
  }
  if (sa && sa->team) {
    launch_sweep_team(*sa, N, nv, n_prims, d_counts, pos, nrm, boundary, valence, idx, iters, process_boundary,
                      sn ? 1 : 0, s, st);
    return 1;
  }
  int launched = 3;
  // CSR offsets: exclusive scan of init_valence (MeshProcessor.cpp:32-40)
  launch_exclusive_scan_u8_to_u32(valence, s.off, nv, d_counts, s.tmp, st);
  const int tb = s.block > 0 ? s.block : 256;
  const int vb = (int)((nv + 255) / 256);
  const int vbt = (int)((nv + tb - 1) / tb), pbt = (int)((n_prims + tb - 1) / tb);
  const uint32_t* cursor = nullptr;
  if (sa) {
    launch_adj_build(sa->mode, sa->chunks, sa->n_chunks, sa->ws, sa->vkey, sa->vadj, s.off, d_counts, nv, n_slots, s.adj,
                     st);
    launched += 1;
  } else {
    cudaMemsetAsync(s.cursor, 0, (size_t)nv * sizeof(uint32_t), st);
    k_fill_adj<<<(int)((n_slots + 255) / 256), 256, 0, st>>>(N, n_slots, nv, d_counts, idx, s.off, valence,
                                                             s.cursor, s.adj);
    k_sort_adj<<<vb, 256, 0, st>>>(nv, n_slots, d_counts, s.off, s.cursor, valence, s.adj);
    cursor = s.cursor;
    launched += 2;
  }
  const SweepBufs b{{s.x[0], s.x[1]}, pos, nrm};
  for (int m = 0; m < iters; ++m) {
    const SweepStep step = sweep_step(m, iters, sn ? 1 : 0, b.keep(), b);
    if (pbt == 0) {
      // no primitives: nothing but kept positions to hand on
    } else if (N == 3)
      k_dual<3><<<pbt, tb, 0, st>>>(n_prims, nv, d_counts, idx, step.src, nrm, s.dual_p, s.dual_n, step.normals);
    else
      k_dual<4><<<pbt, tb, 0, st>>>(n_prims, nv, d_counts, idx, step.src, nrm, s.dual_p, s.dual_n, step.normals);
    // primal after every dual step but the last (MeshProcessor.cpp:229-232),
    // and once more after the loop with set_colors false (ChunkGenerator.cpp:120)
    if (N == 3)
      k_primal<3><<<vbt, tb, 0, st>>>(nv, n_prims, n_slots, d_counts, s.off, cursor, valence, s.adj, boundary, s.dual_p,
                                      s.dual_n, idx, step, b, iters, process_boundary);
    else
      k_primal<4><<<vbt, tb, 0, st>>>(nv, n_prims, n_slots, d_counts, s.off, cursor, valence, s.adj, boundary, s.dual_p,
                                      s.dual_n, idx, step, b, iters, process_boundary);
    launched += 2;
  }
  return launched;
}

}  // namespace bmf
