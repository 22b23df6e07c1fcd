// Hermite data, the reference's FP32 QEF and its adjoint, shared by the
// extraction TU and the FP64 adjoint TU (compiled with FMA contraction).
#pragma once

#include "bmf_device.cuh"
#include "bmf_df.cuh"
#include "bmf_internal.h"

namespace bmf {

// Chunk of vertex v: the last chunk whose vertex offset is <= v (empty
// chunks share the next one's offset).
__device__ __forceinline__ int find_chunk_by_vertex(const ChunkDev* __restrict__ chunks, int n, int64_t v) {
  int lo = 0, hi = n - 1;  // last chunk whose vout <= v (empty chunks share the next one's offset)
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (chunks[mid].vout <= v) lo = mid; else hi = mid - 1;
  }
  return lo;
}

__device__ __forceinline__ float dens_at(const float* D, int dim, int x, int y, int z) {
  return __ldg(D + ((int64_t)x * dim + y) * dim + z);
}

// Central-difference grid gradient at sample (x, y, z), at offset o of the
// chunk's densities (at most 2^27 of them), one-sided at the chunk faces.
__device__ __forceinline__ void grid_gradient(const float* __restrict__ D, int dim, int x, int y, int z, int o,
                                              float g[3]) {
  const int c[3] = {x, y, z}, st[3] = {dim * dim, dim, 1};
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const bool lo = c[a] > 0, hi = c[a] < dim - 1;
    const float h = lo && hi ? 0.5f : 1.0f;
    g[a] = (__ldg(D + (o + (hi ? st[a] : 0))) - __ldg(D + (o - (lo ? st[a] : 0)))) * h;
  }
}

// The edges of a cell in the order of their quads' ids (by owner sample, then
// axis): 0, 4, 8, 1, 5, 2, 9, 3, 6, 10, 7, 11 from the low nibble; and a set of
// edges with its bits in that order.
constexpr uint64_t kQuadOrder = 0xB7A639251840ull;
constexpr uint32_t in_quad_order(uint32_t edges) {
  uint32_t r = 0u;
  for (int i = 0; i < 12; ++i)
    if ((edges >> ((kQuadOrder >> (4 * i)) & 0xF)) & 1u) r |= 1u << i;
  return r;
}

// The edges on a side of the cell (each has a quad only if the cell across it
// exists): y-edges 4, 5 and z-edges 8, 9 at dx = 0, and so on.
constexpr uint32_t kQuadDx0 = in_quad_order(0x330u), kQuadDx1 = in_quad_order(0xCC0u),
                   kQuadDy0 = in_quad_order(0x503u), kQuadDy1 = in_quad_order(0xA0Cu),
                   kQuadDz0 = in_quad_order(0x055u), kQuadDz1 = in_quad_order(0x0AAu);

// Per corner mask and vertex group (four per mask): the group's edges as a
// 12-bit set, and the same in quad order.
struct GroupEdges {
  uint16_t w[1024], q[1024];
};
constexpr GroupEdges make_group_edges() {
  constexpr uint64_t grp[256] = BMF_GROUP_CASES_INIT;
  GroupEdges r{};
  for (int m = 0; m < 256; ++m)
    for (int e = 0; e < 12; ++e) {
      const int g = (int)((grp[m] >> (4 * e)) & 0xFu);
      if (g < 4) r.w[4 * m + g] |= (uint16_t)(1u << e);
    }
  for (int i = 0; i < 1024; ++i) r.q[i] = (uint16_t)in_quad_order(r.w[i]);
  return r;
}
static __device__ const GroupEdges g_group_edges = make_group_edges();
__device__ __forceinline__ uint32_t group_edges(int mask, int g) { return __ldg(&g_group_edges.w[4 * mask + g]); }
__device__ __forceinline__ uint32_t group_edges_q(int mask, int g) { return __ldg(&g_group_edges.q[4 * mask + g]); }

// QEF solve, restating qef_simd.h:150-579 lane by lane in FP32 with the exact
// 1/sqrt in place of _mm_rsqrt_ps.
__device__ __forceinline__ float dot4(const float a[4], const float b[4]) {
  const float m0 = a[0] * b[0], m1 = a[1] * b[1], m2 = a[2] * b[2], m3 = a[3] * b[3];
  return (m0 + m1) + (m3 + m2);
}
__device__ __forceinline__ void vec_mul_m4(const float a[4], const float B[4][4], float out[4]) {
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    float r = a[0] * B[0][k];
    r = r + a[1] * B[1][k];
    r = r + a[2] * B[2][k];
    r = r + a[3] * B[3][k];
    out[k] = r;
  }
}

// What the QEF adjoint needs from a solve: the eigen decomposition the
// Jacobi sweeps produced, the kept reciprocals, the mass point and the
// centred right-hand side r = ATb - ATA * masspoint.
struct QefSolveInfo {
  float V[3][3];
  float sigma[3];
  float inv[3];
  float mp[3];
  float r[3];
};

struct QefAccum {
  float ata[4][4];
  float atb[4];
  float acc[4];
  int count;
  __device__ __forceinline__ void init() {
#pragma unroll
    for (int r = 0; r < 4; ++r) {
#pragma unroll
      for (int k = 0; k < 4; ++k) ata[r][k] = 0.0f;
      atb[r] = 0.0f;
      acc[r] = 0.0f;
    }
    count = 0;
  }
  // qef_simd_add, qef_simd.h:411-430
  __device__ __forceinline__ void add(const float pp[3], const float nn[3]) {
    const float p[4] = {pp[0], pp[1], pp[2], 1.0f};
    const float n[4] = {nn[0], nn[1], nn[2], 0.0f};
#pragma unroll
    for (int r = 0; r < 3; ++r) {
#pragma unroll
      for (int k = 0; k < 4; ++k) ata[r][k] = ata[r][k] + n[r] * n[k];
    }
    const float d = dot4(p, n);
    const float dd[4] = {d, d, d, 0.0f};
#pragma unroll
    for (int k = 0; k < 4; ++k) atb[k] = atb[k] + dd[k] * n[k];
#pragma unroll
    for (int k = 0; k < 4; ++k) acc[k] = acc[k] + p[k];
    ++count;
  }
  // qef_simd_solve + svd_solve_ATA_ATb (qef_simd.h:304-461); returns false
  // for fewer than 2 or more than 12 inputs (qef_simd.h:556-560).
  __device__ bool solve(float out[3], QefSolveInfo* info = nullptr) const {
    if (count < 2 || count > 12) {
      out[0] = out[1] = out[2] = 0.0f;
      return false;
    }
    float mp[4], pr[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) mp[k] = acc[k] / acc[3];
    vec_mul_m4(mp, ata, pr);
#pragma unroll
    for (int k = 0; k < 4; ++k) pr[k] = atb[k] - pr[k];
    float V[4][4] = {{1, 0, 0, 0}, {0, 1, 0, 0}, {0, 0, 1, 0}, {0, 0, 0, 0}};
    float vt[4][4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
#pragma unroll
      for (int k = 0; k < 4; ++k) vt[r][k] = ata[r][k];
    }
#pragma unroll 1
    for (int sweep = 0; sweep < 5; ++sweep) {
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        const int a = q == 2 ? 1 : 0, b = q == 0 ? 1 : 2;
        if (vt[a][b] != 0.0f) {
          // givens_coeffs_sym
          const float pp = vt[a][a], pq = vt[a][b], qq = vt[b][b];
          const float tau = (qq - pp) / (pq * 2.0f);
          const float stt = sqrtf(tau * tau + 1.0f);
          const float tn = 1.0f / ((tau >= 0.0f) ? (tau + stt) : (tau - stt));
          float cc = 1.0f / sqrtf(1.0f + tn * tn);
          float ss = tn * cc;
          if (pq == 0.0f) { cc = 1.0f; ss = 0.0f; }
          // rotateq_xy
          const float c2 = cc * cc, s2 = ss * ss;
          const float mx = ((2.0f * cc) * ss) * pq;
          const float nx = (c2 * pp - mx) + s2 * qq;
          const float ny = (s2 * pp + mx) + c2 * qq;
          vt[a][a] = nx;
          vt[b][b] = ny;
          // rotate_xy
          const float u3 = vt[0][3 - b], v3 = vt[1 - a][2];
#pragma unroll
          for (int r = 0; r < 3; ++r) {
            const float uu = V[r][a], vv = V[r][b];
            V[r][a] = cc * uu - ss * vv;
            V[r][b] = ss * uu + cc * vv;
          }
          vt[0][3 - b] = cc * u3 - ss * v3;
          vt[1 - a][2] = ss * u3 + cc * v3;
          vt[a][b] = 0.0f;
        }
      }
    }
    const float sigma[4] = {vt[0][0], vt[1][1], vt[2][2], 0.0f};
    float invdet[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {  // svd_invdet
      const float oo = 1.0f / sigma[k];
      const float a1 = fabsf(sigma[k]), a2 = fabsf(oo);
      const float mn = (a1 < a2) ? a1 : a2;
      invdet[k] = (mn >= 0.001f) ? oo : 0.0f;
    }
    float mm[3][4], o[4][4];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
#pragma unroll
      for (int k = 0; k < 4; ++k) mm[r][k] = V[r][k] * invdet[k];
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
#pragma unroll
      for (int k = 0; k < 4; ++k) o[r][k] = (r < 3 && k < 3) ? dot4(mm[k], V[r]) : 0.0f;
    }
    float xq[4];
    vec_mul_m4(pr, o, xq);
    out[0] = xq[0] + mp[0];
    out[1] = xq[1] + mp[1];
    out[2] = xq[2] + mp[2];
    if (info) {
#pragma unroll
      for (int r = 0; r < 3; ++r) {
#pragma unroll
        for (int k = 0; k < 3; ++k) info->V[r][k] = V[r][k];
        info->sigma[r] = sigma[r];
        info->inv[r] = invdet[r];
        info->mp[r] = mp[r];
        info->r[r] = pr[r];
      }
    }
    return true;
  }
};

// Crossing point (and hermite normal) of edge e of cell (x, y, z).
__device__ __forceinline__ void hermite(const float* __restrict__ D, int dim, int x, int y, int z, int e, bool want_n,
                                        float p[3], float n[3]) {
  const int ca = edge_c0(e), ax = e >> 2;
  const int a0[3] = {x + ((ca >> 2) & 1), y + ((ca >> 1) & 1), z + (ca & 1)};
  const int a1[3] = {a0[0] + (ax == 0), a0[1] + (ax == 1), a0[2] + (ax == 2)};
  const int o0 = (a0[0] * dim + a0[1]) * dim + a0[2], o1 = o0 + (ax == 0 ? dim * dim : (ax == 1 ? dim : 1));
  const float s0 = __ldg(D + o0), s1 = __ldg(D + o1);
  float g0[3], g1[3];
  if (want_n) {  // (loads in flight together with the samples')
    grid_gradient(D, dim, a0[0], a0[1], a0[2], o0, g0);
    grid_gradient(D, dim, a1[0], a1[1], a1[2], o1, g1);
  }
  const float mu = (0.0f - s0) / (s1 - s0);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float dv = ((float)a1[k] - (float)a0[k]) * mu;
    p[k] = dv + (float)a0[k];
  }
  if (want_n) {
    float g[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) g[k] = g0[k] + (g1[k] - g0[k]) * mu;
    const float l2 = (g[0] * g[0] + g[1] * g[1]) + g[2] * g[2];
    const float inv = 1.0f / sqrtf(l2);
#pragma unroll
    for (int k = 0; k < 3; ++k) n[k] = g[k] * inv;
  }
}

// Position of the vertex of the cell's edges `edges` (group_edges), taken in
// ascending order: each lane walks its own set, so that a warp runs as many
// rounds as its longest list, not the union of the lists over twelve edges.
// WARP: all lanes of the warp call it (edges = 0: nothing is placed) and leave
// the walk together.
// info / qef_used (optional, QEF placement): the solve's eigen data and
// whether the vertex took the QEF branch (a successful solve inside the cell)
// -- what the QEF adjoint needs from the forward.
template <int PLACE, bool WARP>
__device__ __forceinline__ void q_place(const float* __restrict__ D, int dim, int x, int y, int z, uint32_t edges,
                                        float out[3], QefSolveInfo* info = nullptr, bool* qef_used = nullptr) {
  if (PLACE == 0) {
    out[0] = (float)x + 0.5f;
    out[1] = (float)y + 0.5f;
    out[2] = (float)z + 0.5f;
    return;
  }
  float mp[3] = {0.0f, 0.0f, 0.0f};
  const int cnt = __popc(edges);
  QefAccum q;
  if (PLACE == 2) q.init();
#pragma unroll 1
  for (uint32_t em = edges; em; em &= em - 1u) {
    float p[3], n[3];
    hermite(D, dim, x, y, z, __ffs(em) - 1, PLACE == 2, p, n);
#pragma unroll
    for (int k = 0; k < 3; ++k) mp[k] = mp[k] + p[k];
    if (PLACE == 2) q.add(p, n);
  }
  if (WARP) {
    __syncwarp();
    if (!edges) return;
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) mp[k] = mp[k] / (float)cnt;
  if (PLACE == 2) {
    float s[3];
    const bool solved = q.solve(s, info);
    const bool ok = s[0] >= (float)x && s[0] <= (float)(x + 1) && s[1] >= (float)y && s[1] <= (float)(y + 1) &&
                    s[2] >= (float)z && s[2] <= (float)(z + 1);
    if (qef_used) *qef_used = solved && ok;
    if (ok) {
      out[0] = s[0]; out[1] = s[1]; out[2] = s[2];
      return;
    }
  }
  out[0] = mp[0]; out[1] = mp[1]; out[2] = mp[2];
}

// ---------------------------------------------------------------------------
// Adjoint of the Mode Q vertex placement with respect to the density, in FP32.
// The incoming position gradient goes through the QEF -- x = m + V f(S) V^T r,
// r = ATb - ATA m, differentiated with the truncation pattern held fixed
// (Daleckii-Krein: F_ij = (f_i - f_j)/(s_i - s_j), F_ii = f'(s_i)) -- or
// through the mass point, then through every hermite pair: the normal n =
// G/|G| of the lerped central-difference gradients and the crossing p = a0 +
// (a1 - a0) mu, mu = -s0 / (s1 - s0), into the density samples (float atomics).
// The wide adjoint of QEF-placed vertices is k_qef_bwd (bmf_adjoint64.cu).
// ---------------------------------------------------------------------------
struct QefAdj {
  float A[3][3];    // ATA
  float V[3][3];    // eigenvectors (columns)
  float sigma[3];   // eigenvalues
  float inv[3];     // kept reciprocals (0 = truncated)
  float mp[3];      // mass point
  float r[3];       // ATb - ATA mp
};

// Hermite pair of edge e (the crossing, the lerped gradient, its length and
// the unit normal).
struct HermitePair {
  int a0[3], a1[3];
  float s0, s1, mu, p[3], g0[3], g1[3], n[3], iglen;
};

__device__ __forceinline__ void hermite_pair(const float* __restrict__ D, int dim, int x, int y, int z, int e,
                                             bool want_n, HermitePair& h) {
  const int ca = edge_c0(e), cb = edge_c1(e);
  h.a0[0] = x + ((ca >> 2) & 1); h.a0[1] = y + ((ca >> 1) & 1); h.a0[2] = z + (ca & 1);
  h.a1[0] = x + ((cb >> 2) & 1); h.a1[1] = y + ((cb >> 1) & 1); h.a1[2] = z + (cb & 1);
  const int o0 = (h.a0[0] * dim + h.a0[1]) * dim + h.a0[2], o1 = (h.a1[0] * dim + h.a1[1]) * dim + h.a1[2];
  h.s0 = __ldg(D + o0);
  h.s1 = __ldg(D + o1);
  h.mu = (0.0f - h.s0) / (h.s1 - h.s0);
#pragma unroll
  for (int k = 0; k < 3; ++k) h.p[k] = ((float)h.a1[k] - (float)h.a0[k]) * h.mu + (float)h.a0[k];
  h.iglen = 1.0f;
  if (want_n) {
    grid_gradient(D, dim, h.a0[0], h.a0[1], h.a0[2], o0, h.g0);
    grid_gradient(D, dim, h.a1[0], h.a1[1], h.a1[2], o1, h.g1);
    float G[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) G[k] = h.g0[k] + (h.g1[k] - h.g0[k]) * h.mu;
    h.iglen = 1.0f / sqrtf((G[0] * G[0] + G[1] * G[1]) + G[2] * G[2]);
#pragma unroll
    for (int k = 0; k < 3; ++k) h.n[k] = G[k] * h.iglen;
  }
}

// ALL: every vertex, the forward's branch replayed in FP32 (same hermite data,
// same FP32 QEF) and differentiated with its own eigen pairs; else the vertices
// the forward did not flag in qflag (mass-point placed; the others are
// k_qef_bwd's).
template <int PLACE, bool ALL>
__global__ void __launch_bounds__(128) k_place_bwd(const ChunkDev* __restrict__ chunks, int n_chunks,
                                                   const uint32_t* __restrict__ words, const float* __restrict__ dens,
                                                   const uint32_t* __restrict__ vkey,
                                                   const int64_t* __restrict__ d_counts, int64_t vcap,
                                                   const float* __restrict__ grad_pos, float* __restrict__ grad_dens,
                                                   const uint8_t* __restrict__ qflag) {
  const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= (d_counts ? min(vcap, d_counts[0]) : vcap)) return;
  if (!ALL && qflag[v]) return;
  const int c = find_chunk_by_vertex(chunks, n_chunks, v);
  const ChunkDev ch = chunks[c];
  const int dim = ch.dim, zc = ch.zc;
  const uint32_t* W = words + ch.words;
  const float* D = dens + ch.dens;
  float* GD = grad_dens + ch.dens;
  int x, y, z, g;
  vertex_key_decode(vkey[v], x, y, z, g);
  const int mask = cell_mask_at(W, dim, zc, x, y, z);
  const uint32_t edges = group_edges(mask, g);
  const float gx[3] = {grad_pos[3 * v], grad_pos[3 * v + 1], grad_pos[3 * v + 2]};
  int cnt = 0;
  bool use_qef = false;
  QefAdj Q;
  QefAccum q;
  QefSolveInfo info;
  if constexpr (!ALL) {
    // the forward recorded the branch: a vertex left to this pass took the mass point
    cnt = __popc(edges);
    if (cnt == 0) return;
  } else {
    // the forward's branch: replay of q_place in FP32
    if (PLACE == 2) q.init();
    for (uint32_t em = edges; em; em &= em - 1u) {
      const int e = __ffs(em) - 1;
      float p[3], n[3];
      hermite(D, dim, x, y, z, e, PLACE == 2, p, n);
      ++cnt;
      if (PLACE == 2) q.add(p, n);
    }
    if (cnt == 0) return;
    if (PLACE == 2) {
      float s[3];
      if (q.solve(s, &info))
        use_qef = s[0] >= (float)x && s[0] <= (float)(x + 1) && s[1] >= (float)y && s[1] <= (float)(y + 1) &&
                  s[2] >= (float)z && s[2] <= (float)(z + 1);
    }
  }
  if (PLACE == 2) {
    if (use_qef) {
#pragma unroll
      for (int r = 0; r < 3; ++r) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          Q.A[r][k] = q.ata[r][k];
          Q.V[r][k] = info.V[r][k];
        }
        Q.sigma[r] = info.sigma[r];
        Q.inv[r] = info.inv[r];
        Q.mp[r] = info.mp[r];
        Q.r[r] = info.r[r];
      }
    }
  }
  // QEF adjoint down to gA (symmetric), gr, gm
  float gA[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}}, gr[3] = {0, 0, 0}, gm[3] = {gx[0], gx[1], gx[2]};
  if (use_qef) {
    float Pm[3][3];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
#pragma unroll
      for (int k = 0; k < 3; ++k)
        Pm[r][k] = Q.V[r][0] * Q.inv[0] * Q.V[k][0] + Q.V[r][1] * Q.inv[1] * Q.V[k][1] + Q.V[r][2] * Q.inv[2] * Q.V[k][2];
    }
#pragma unroll
    for (int r = 0; r < 3; ++r) gr[r] = Pm[r][0] * gx[0] + Pm[r][1] * gx[1] + Pm[r][2] * gx[2];
    float Gs[3][3], M[3][3], F[3][3], W[3][3];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
#pragma unroll
      for (int k = 0; k < 3; ++k) Gs[r][k] = 0.5f * (gx[r] * Q.r[k] + gx[k] * Q.r[r]);
    }
    // M = V^T Gs V as two 3x3 products (W = Gs V, then V^T W)
#pragma unroll
    for (int r = 0; r < 3; ++r) {
#pragma unroll
      for (int b = 0; b < 3; ++b) W[r][b] = Gs[r][0] * Q.V[0][b] + Gs[r][1] * Q.V[1][b] + Gs[r][2] * Q.V[2][b];
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        M[a][b] = Q.V[0][a] * W[0][b] + Q.V[1][a] * W[1][b] + Q.V[2][a] * W[2][b];
        // f(s) = 1/s: (f_a - f_b) / (s_a - s_b) = -f_a f_b (no cancellation for
        // close eigenvalues) and f'(s) = -f^2; a truncated eigenvalue (f = 0)
        // beside a kept one takes the quotient
        const float fa = Q.inv[a], fb = Q.inv[b], sa = Q.sigma[a], sb = Q.sigma[b];
        if (fa != 0.0f && fb != 0.0f)
          F[a][b] = -fa * fb;
        else if (a == b || fabs(sa - sb) <= 1e-6f * (fabs(sa) + fabs(sb)))
          F[a][b] = 0.0f;
        else
          F[a][b] = (fa - fb) / (sa - sb);
        F[a][b] = F[a][b] * M[a][b];
      }
    }
    // gA = V (F o M) V^T - sym(gr mp^T), again as two products
#pragma unroll
    for (int r = 0; r < 3; ++r) {
#pragma unroll
      for (int b = 0; b < 3; ++b) W[r][b] = Q.V[r][0] * F[0][b] + Q.V[r][1] * F[1][b] + Q.V[r][2] * F[2][b];
    }
#pragma unroll
    for (int r = 0; r < 3; ++r) {
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const float s = W[r][0] * Q.V[k][0] + W[r][1] * Q.V[k][1] + W[r][2] * Q.V[k][2];
        gA[r][k] = s - 0.5f * (gr[r] * Q.mp[k] + gr[k] * Q.mp[r]);
      }
    }
#pragma unroll
    for (int r = 0; r < 3; ++r) gm[r] -= Q.A[r][0] * gr[0] + Q.A[r][1] * gr[1] + Q.A[r][2] * gr[2];
  }
  const float inv_cnt = 1.0f / (float)cnt;
  // per hermite pair: g_p, g_n, then into the density
  for (uint32_t em = edges; em; em &= em - 1u) {
    const int e = __ffs(em) - 1;
    HermitePair h;
    hermite_pair(D, dim, x, y, z, e, PLACE == 2 && use_qef, h);  // the mass point needs no normals
    const int ax = e >> 2;
    float gp[3], gn[3] = {0.0f, 0.0f, 0.0f};
    if (!use_qef) {
#pragma unroll
      for (int k = 0; k < 3; ++k) gp[k] = gx[k] * inv_cnt;
    } else {
      const float d = h.n[0] * h.p[0] + h.n[1] * h.p[1] + h.n[2] * h.p[2];
      const float gd = gr[0] * h.n[0] + gr[1] * h.n[1] + gr[2] * h.n[2];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        gn[k] = 2.0f * (gA[k][0] * h.n[0] + gA[k][1] * h.n[1] + gA[k][2] * h.n[2]) + d * gr[k] + gd * h.p[k];
        gp[k] = gd * h.n[k] + gm[k] * inv_cnt;
      }
    }
    float gmu = gp[ax];
    if (use_qef) {
      const float nd = h.n[0] * gn[0] + h.n[1] * gn[1] + h.n[2] * gn[2];
      float gG[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        gG[k] = (gn[k] - h.n[k] * nd) * h.iglen;
        gmu += gG[k] * (h.g1[k] - h.g0[k]);
      }
      // central differences at both endpoints: g[a] = (s[hi] - s[lo]) * h
#pragma unroll
      for (int a = 0; a < 3; ++a) {
#pragma unroll
        for (int end = 0; end < 2; ++end) {
          const int* q0 = end ? h.a1 : h.a0;
          const float w = gG[a] * (end ? h.mu : 1.0f - h.mu);
          int lo[3] = {q0[0], q0[1], q0[2]}, hi[3] = {q0[0], q0[1], q0[2]};
          float hh = 0.5f;
          if (q0[a] > 0) lo[a]--; else hh = 1.0f;
          if (q0[a] < dim - 1) hi[a]++; else hh = 1.0f;
          atomicAdd(GD + ((int64_t)hi[0] * dim + hi[1]) * dim + hi[2], w * hh);
          atomicAdd(GD + ((int64_t)lo[0] * dim + lo[1]) * dim + lo[2], -w * hh);
        }
      }
    }
    const float iden = 1.0f / ((h.s1 - h.s0) * (h.s1 - h.s0));
    atomicAdd(GD + ((int64_t)h.a0[0] * dim + h.a0[1]) * dim + h.a0[2], gmu * (-h.s1 * iden));
    atomicAdd(GD + ((int64_t)h.a1[0] * dim + h.a1[1]) * dim + h.a1[2], gmu * (h.s0 * iden));
  }
}

}  // namespace bmf
