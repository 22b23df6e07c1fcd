// The QEF adjoint of the vertices that the forward placed by QEF (its list, with
// their FP32 eigenvectors), in a wide type W -- double-float or FP64 -- where
// it has to be: its own translation unit, built with FMA contraction, since
// nothing here has to reproduce the reference's float rounding and the
// double-float product needs fmaf.
//
// The placement is x = m + V f(S) V^T r with A = sum n n^T, r = sum (n.p) n - A m
// and f(s) = 1/s or 0; 1/s^2 amplifies the ~1e-6 absolute error of a small kept
// FP32 eigenvalue, so A, r, the eigen pairs and the derivative of the
// pseudo-inverse are wide.  What remains, the chain rule into the density, is
// a product of well-conditioned factors in FP32 on the forward's own hermite data.
//
// In the wide part points are taken relative to the cell (A and r do not change
// with the origin, and p stays below 1); dL/dA and the chain rule use the chunk's
// coordinates, as the FP32 adjoint does.
// The wide part is written for few wide operations (a double-float product is 4
// instructions, a sum 20, a division a call):
//   - n n^T = G G^T / (G.G): one reciprocal per hermite pair, no root;
//   - Jacobi rotations by FP32 angles with a wide (c, s) on the unit circle: each
//     rotation leaves 1e-7 of the entry it is for, so the sweeps converge as
//     fast as with exact angles from 1e-6 entries (two sweeps), without wide
//     divisions and roots; B = V^T A V is kept as its six entries;
//   - M = V^T sym(gx r^T) V = sym((V^T gx) (V^T r)^T): two vectors, not four
//     3x3 products.
// A vertex's contributions meet in shared memory first: its four or five
// hermite pairs touch 32 samples around the cell about 63 times.
//
// Bound by issue and by instruction fetch: the code is larger than the
// instruction caches, and warps at different places of it stall on fetches (8 of
// 12.6 cycles per issue with free-running warps).  So the parts are kept small
// (the rotation's code exists once) and a CTA's warps go through them together,
// with a block barrier between parts.  3.9 M vertices (512 x 65^3), whole fitting
// step: 5.76 ms with the previous kernel (2.40 ms of it here), 5.62 with this
// algebra and free-running 128-thread CTAs, 4.54 with barriers, 4.33 at 256
// threads x 2 CTAs (4.42 at 512 x 1).
#include "bmf_qef.cuh"

namespace bmf {
namespace {

__device__ __forceinline__ double w_diff(float a, float b, double) { return (double)a - (double)b; }
__device__ __forceinline__ DF w_diff(float a, float b, DF) { return dfl::df_two_sum(a, -b); }
__device__ __forceinline__ double w_scale(double a, float b) { return a * (double)b; }
__device__ __forceinline__ DF w_scale(DF a, float b) {
  const float p = a.hi * b;
  return dfl::df_fast_two_sum(p, fmaf(a.lo, b, fmaf(a.hi, b, -p)));
}
__device__ __forceinline__ double w_square(float a, double) { return (double)a * (double)a; }
__device__ __forceinline__ DF w_square(float a, DF) {
  const float p = a * a;
  return DF(p, fmaf(a, a, -p));
}
// 1/a and 1/sqrt(a) (a > 0): the float result and a correction from its exact
// residual, second order included.
__device__ __forceinline__ double w_recip(double a) { return 1.0 / a; }
__device__ __forceinline__ DF w_recip(DF a) {
  const float q = 1.0f / a.hi;
  const float e = fmaf(-a.lo, q, fmaf(-a.hi, q, 1.0f));
  return dfl::df_fast_two_sum(q, q * fmaf(e, e, e));
}
__device__ __forceinline__ double w_rsqrt(double a) { return 1.0 / sqrt(a); }
__device__ __forceinline__ DF w_rsqrt(DF a) {
  const float y = rsqrtf(a.hi);
  const DF u = a * w_square(y, a);
  const float e = (1.0f - u.hi) - u.lo;
  return dfl::df_fast_two_sum(y, y * fmaf(0.375f * e, e, 0.5f * e));
}
__device__ __forceinline__ float w_abs(double a) { return (float)fabs(a); }
__device__ __forceinline__ float w_abs(DF a) { return fabsf(a.hi); }

// Where the rotations stop, in units of |A|.
__device__ __forceinline__ float w_tol(double) { return 1e-17f; }
__device__ __forceinline__ float w_tol(DF) { return 3e-14f; }

// Entry (i, j) of a symmetric 3x3 matrix kept as {00, 01, 02, 11, 12, 22}.
__device__ __forceinline__ constexpr int sym(int i, int j) {
  return i <= j ? (i == 0 ? j : (i == 1 ? 2 + j : 5)) : (j == 0 ? i : (j == 1 ? 2 + i : 5));
}

// Central differences of the densities at offset o, exact but for the scale's
// power of two.
template <typename W>
__device__ __forceinline__ void gradient_w(const float* __restrict__ D, int dim, const int c[3], int o, W g[3]) {
  const int st[3] = {dim * dim, dim, 1};
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const bool lo = c[a] > 0, hi = c[a] < dim - 1;
    g[a] = w_scale(w_diff(__ldg(D + (o + (hi ? st[a] : 0))), __ldg(D + (o - (lo ? st[a] : 0))), W()), lo && hi ? 0.5f : 1.0f);
  }
}

// (two resident CTAs keep 128 registers: no spills)
constexpr int kQefBwdThreads = 256;
constexpr int kStencil = 32;  // samples a vertex's hermite pairs touch
constexpr size_t kQefBwdSmem = sizeof(float) * kStencil * kQefBwdThreads;

template <typename W>
__global__ void __launch_bounds__(kQefBwdThreads, 2) k_qef_bwd(
    const ChunkDev* __restrict__ chunks, int n_chunks, const uint32_t* __restrict__ words,
    const float* __restrict__ dens, const uint32_t* __restrict__ vkey, const float* __restrict__ grad_pos,
    float* __restrict__ grad_dens, const uint32_t* __restrict__ qlist, const uint32_t* __restrict__ qcount,
    const float* __restrict__ qseed) {
  // contributions to the samples around each thread's cell: corner c at c;
  // beyond it along axis a on side s at 8 + 8 a + 4 s + (the two other offsets)
  extern __shared__ float s_acc_[];
  float(*s_acc)[kQefBwdThreads] = reinterpret_cast<float(*)[kQefBwdThreads]>(s_acc_);
  const int64_t n = *qcount;
  for (int64_t s0 = (int64_t)blockIdx.x * kQefBwdThreads; s0 < n; s0 += (int64_t)gridDim.x * kQefBwdThreads) {
    const int64_t slot = s0 + threadIdx.x;
    const bool in = slot < n;
    const uint32_t v = in ? qlist[slot] : 0u;
    const ChunkDev& ch = chunks[find_chunk_by_vertex(chunks, n_chunks, v)];
    const int dim = ch.dim;
    const float* __restrict__ D = dens + ch.dens;
    int x, y, z, g;
    vertex_key_decode(vkey[v], x, y, z, g);
    const uint32_t edges = in ? group_edges(cell_mask_at(words + ch.words, dim, ch.zc, x, y, z), g) : 0u;
    const int ocell = (x * dim + y) * dim + z, st[3] = {dim * dim, dim, 1};
    float fA[6], fr[3], fm[3];
    const float inv_cnt = 1.0f / (float)max(1, __popc(edges));
    {
      // A, sum (n.p) n and the mass point
      W A[6], b[3], m[3];
#pragma unroll
      for (int k = 0; k < 6; ++k) A[k] = W(0.0f);
#pragma unroll
      for (int k = 0; k < 3; ++k) b[k] = m[k] = W(0.0f);
#pragma unroll 1
      for (uint32_t em = edges; em; em &= em - 1u) {
        const int e = __ffs(em) - 1, ca = edge_c0(e), ax = e >> 2;
        const int d0[3] = {(ca >> 2) & 1, (ca >> 1) & 1, ca & 1};
        const int a0[3] = {x + d0[0], y + d0[1], z + d0[2]};
        const int a1[3] = {a0[0] + (ax == 0), a0[1] + (ax == 1), a0[2] + (ax == 2)};
        const int o0 = ocell + d0[0] * st[0] + d0[1] * st[1] + d0[2], o1 = o0 + (ax == 0 ? st[0] : (ax == 1 ? dim : 1));
        const float s0d = __ldg(D + o0), s1d = __ldg(D + o1);
        W g0[3], G[3];
        gradient_w<W>(D, dim, a0, o0, g0);
        gradient_w<W>(D, dim, a1, o1, G);
        const W mu = w_scale(w_recip(w_diff(s1d, s0d, W())), -s0d);
#pragma unroll
        for (int k = 0; k < 3; ++k) G[k] = g0[k] + (G[k] - g0[k]) * mu;
        const W iw = w_recip(G[0] * G[0] + G[1] * G[1] + G[2] * G[2]);
        // G.p with p = d0 + mu along the axis
        W d = (ax == 0 ? G[0] : (ax == 1 ? G[1] : G[2])) * mu;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          if (d0[k]) {
            d += G[k];
            m[k] += W(1.0f);
          }
          if (k == ax) m[k] += mu;
        }
        const W Gw[3] = {G[0] * iw, G[1] * iw, G[2] * iw};
#pragma unroll
        for (int i = 0; i < 3; ++i) {
#pragma unroll
          for (int j = i; j < 3; ++j) A[sym(i, j)] += Gw[i] * G[j];
          b[i] += Gw[i] * d;
        }
      }
      __syncthreads();  // the CTA's warps run each part's code together
      const W ic = w_recip(W((float)max(1, __popc(edges))));
#pragma unroll
      for (int k = 0; k < 3; ++k) m[k] = m[k] * ic;
      W r[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) r[k] = b[k] - (A[sym(k, 0)] * m[0] + A[sym(k, 1)] * m[1] + A[sym(k, 2)] * m[2]);
      // eigen pairs of A, refined from the forward's FP32 eigenvectors
      W V[3][3], B[6];  // V[c]: column c
      {
        float c0[3], c1[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          c0[k] = in ? qseed[9 * slot + 3 * k] : (k == 0 ? 1.0f : 0.0f);
          c1[k] = in ? qseed[9 * slot + 3 * k + 1] : (k == 1 ? 1.0f : 0.0f);
        }
        W il = w_rsqrt(w_square(c0[0], W()) + w_square(c0[1], W()) + w_square(c0[2], W()));
#pragma unroll
        for (int k = 0; k < 3; ++k) V[0][k] = w_scale(il, c0[k]);
        const W dt = w_scale(V[0][0], c1[0]) + w_scale(V[0][1], c1[1]) + w_scale(V[0][2], c1[2]);
#pragma unroll
        for (int k = 0; k < 3; ++k) V[1][k] = W(c1[k]) - dt * V[0][k];
        il = w_rsqrt(V[1][0] * V[1][0] + V[1][1] * V[1][1] + V[1][2] * V[1][2]);
#pragma unroll
        for (int k = 0; k < 3; ++k) V[1][k] = V[1][k] * il;
#pragma unroll
        for (int k = 0; k < 3; ++k)
          V[2][k] = V[0][(k + 1) % 3] * V[1][(k + 2) % 3] - V[0][(k + 2) % 3] * V[1][(k + 1) % 3];
      }
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        W t[3];  // A V[j]
#pragma unroll
        for (int k = 0; k < 3; ++k) t[k] = A[sym(k, 0)] * V[j][0] + A[sym(k, 1)] * V[j][1] + A[sym(k, 2)] * V[j][2];
#pragma unroll
        for (int i = 0; i <= j; ++i) B[sym(i, j)] = V[i][0] * t[0] + V[i][1] * t[1] + V[i][2] * t[2];
      }
      const float tol = w_tol(W()) * (w_abs(B[0]) + w_abs(B[3]) + w_abs(B[5]));
      // cyclic rotations of axes 0 and 1, the axes relabelled after each
      // (one copy of the rotation's code)
#pragma unroll 1
      for (int rot = 0; rot < 48; ++rot) {
        const bool more = w_abs(B[1]) + w_abs(B[2]) + w_abs(B[4]) > tol;
        if (!__syncthreads_or(more)) break;
        if (more && w_abs(B[1]) > tol) {
          const W app = B[0], ass = B[3], aps = B[1];
          const float tau = (float)(ass - app) / (2.0f * (float)aps);
          const float t = copysignf(1.0f, tau) / (fabsf(tau) + sqrtf(1.0f + tau * tau));
          const W c = w_rsqrt(W(1.0f) + w_square(t, W())), sn = w_scale(c, t);
          const W c2 = c * c, s2 = sn * sn, cs = c * sn;
          const W x2 = w_scale(cs * aps, 2.0f);
          B[0] = c2 * app - x2 + s2 * ass;
          B[3] = s2 * app + x2 + c2 * ass;
          B[1] = (c2 - s2) * aps + cs * (app - ass);
          const W bkp = B[2], bks = B[4];
          B[2] = c * bkp - sn * bks;
          B[4] = sn * bkp + c * bks;
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            const W vp = V[0][i], vs = V[1][i];
            V[0][i] = c * vp - sn * vs;
            V[1][i] = sn * vp + c * vs;
          }
        }
        // axes (0, 1, 2) <- (1, 2, 0)
        const W b00 = B[0], b01 = B[1], b02 = B[2];
        B[0] = B[3];
        B[1] = B[4];
        B[2] = b01;
        B[3] = B[5];
        B[4] = b02;
        B[5] = b00;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          const W v0 = V[0][i];
          V[0][i] = V[1][i];
          V[1][i] = V[2][i];
          V[2][i] = v0;
        }
      }
      // f(s) = 1/s kept where min(|s|, |1/s|) >= 0.001 (qef_simd.h:346-368)
      W sg[3] = {B[0], B[3], B[5]}, f[3];
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        f[i] = W(0.0f);
        if (fabs(sg[i]) >= W(0.001f)) {
          const W oo = w_recip(sg[i]);
          if (fabs(oo) >= W(0.001f)) f[i] = oo;
        }
      }
      // dL/d(A, r, m): gr = V f V^T gx, gm = gx - A gr, and gA = V (F o M) V^T -
      // sym(gr m^T) with M = V^T sym(gx r^T) V (Daleckii-Krein)
      const float gx[3] = {in ? grad_pos[3 * (int64_t)v] : 0.0f, in ? grad_pos[3 * (int64_t)v + 1] : 0.0f,
                           in ? grad_pos[3 * (int64_t)v + 2] : 0.0f};
      W u[3], w[3], gr[3], H[6];
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        u[i] = w_scale(V[i][0], gx[0]) + w_scale(V[i][1], gx[1]) + w_scale(V[i][2], gx[2]);
        w[i] = V[i][0] * r[0] + V[i][1] * r[1] + V[i][2] * r[2];
      }
      const W fu[3] = {f[0] * u[0], f[1] * u[1], f[2] * u[2]};
#pragma unroll
      for (int k = 0; k < 3; ++k) gr[k] = V[0][k] * fu[0] + V[1][k] * fu[1] + V[2][k] * fu[2];
#pragma unroll
      for (int i = 0; i < 3; ++i) {
#pragma unroll
        for (int j = i; j < 3; ++j) {
          // (f_i - f_j) / (s_i - s_j): -f_i f_j for two kept eigenvalues (no
          // cancellation for close ones), the quotient for a kept and a truncated one
          W F = -(f[i] * f[j]);
          if (i != j && (f[i] != W(0.0f)) != (f[j] != W(0.0f))) {
            const W ds = sg[i] - sg[j];
            F = fabs(ds) <= W(1e-6f) * (fabs(sg[i]) + fabs(sg[j])) ? W(0.0f) : (f[i] - f[j]) * w_recip(ds);
          }
          H[sym(i, j)] = F * w_scale(u[i] * w[j] + u[j] * w[i], 0.5f);
        }
      }
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        W t[3];  // row j of H V^T
#pragma unroll
        for (int k = 0; k < 3; ++k) t[k] = H[sym(j, 0)] * V[0][k] + H[sym(j, 1)] * V[1][k] + H[sym(j, 2)] * V[2][k];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
#pragma unroll
          for (int k = i; k < 3; ++k) {
            const W p = V[j][i] * t[k];
            B[sym(i, k)] = j == 0 ? p : B[sym(i, k)] + p;
          }
        }
      }
      const int org[3] = {x, y, z};
#pragma unroll
      for (int k = 0; k < 3; ++k) m[k] += W((float)org[k]);
#pragma unroll
      for (int i = 0; i < 3; ++i) {
#pragma unroll
        for (int k = i; k < 3; ++k)
          fA[sym(i, k)] = (float)(B[sym(i, k)] - w_scale(gr[i] * m[k] + gr[k] * m[i], 0.5f));
        fr[i] = (float)gr[i];
        fm[i] = (float)(W(gx[i]) - (A[sym(i, 0)] * gr[0] + A[sym(i, 1)] * gr[1] + A[sym(i, 2)] * gr[2]));
      }
    }
    __syncthreads();
    // the chain rule through every hermite pair (FP32)
    uint32_t touched = 0u;
    const auto add = [&](int at, float val) {
      float* a = &s_acc[at][threadIdx.x];
      *a = (touched >> at) & 1u ? *a + val : val;
      touched |= 1u << at;
    };
#pragma unroll 1
    for (uint32_t em = edges; em; em &= em - 1u) {
      const int e = __ffs(em) - 1, ca = edge_c0(e), ax = e >> 2;
      HermitePair h;
      hermite_pair(D, dim, x, y, z, e, true, h);
      float gp[3], gn[3];
      const float d = h.n[0] * h.p[0] + h.n[1] * h.p[1] + h.n[2] * h.p[2];
      const float gd = fr[0] * h.n[0] + fr[1] * h.n[1] + fr[2] * h.n[2];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        gn[k] = 2.0f * (fA[sym(k, 0)] * h.n[0] + fA[sym(k, 1)] * h.n[1] + fA[sym(k, 2)] * h.n[2]) + d * fr[k] + gd * h.p[k];
        gp[k] = gd * h.n[k] + fm[k] * inv_cnt;
      }
      float gmu = ax == 0 ? gp[0] : (ax == 1 ? gp[1] : gp[2]);
      const float nd = h.n[0] * gn[0] + h.n[1] * gn[1] + h.n[2] * gn[2];
      float gG[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        gG[k] = (gn[k] - h.n[k] * nd) * h.iglen;
        gmu += gG[k] * (h.g1[k] - h.g0[k]);
      }
      // central differences at both ends: g[a] = (s[hi] - s[lo]) * h
#pragma unroll
      for (int end = 0; end < 2; ++end) {
        const int* q0 = end ? h.a1 : h.a0;
        const int cq = end ? ca | (4 >> ax) : ca;  // the end as a corner of the cell
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          const float wgt = gG[a] * (end ? h.mu : 1.0f - h.mu);
          const bool lo = q0[a] > 0, hi = q0[a] < dim - 1, far = (cq >> (2 - a)) & 1;
          const float hh = lo && hi ? wgt * 0.5f : wgt;
          // the two other offsets of the corner, and the samples beyond it along the axis
          const int rest = a == 0 ? cq & 3 : (a == 1 ? ((cq >> 1) & 2) | (cq & 1) : (cq >> 1) & 3);
          const int out_at = 8 + 8 * a + 4 * (far ? 1 : 0) + rest, in_at = cq ^ (4 >> a);
          add(hi ? (far ? out_at : in_at) : cq, hh);
          add(lo ? (far ? in_at : out_at) : cq, -hh);
        }
      }
      const float iden = 1.0f / ((h.s1 - h.s0) * (h.s1 - h.s0));
      add(ca, gmu * (-h.s1 * iden));
      add(ca | (4 >> ax), gmu * (h.s0 * iden));
    }
    __syncthreads();
    float* __restrict__ GD = grad_dens + ch.dens;
#pragma unroll 1
    for (uint32_t tm = touched; tm; tm &= tm - 1u) {
      const int at = __ffs(tm) - 1;
      int dx, dy, dz;
      if (at < 8) {
        dx = at >> 2, dy = (at >> 1) & 1, dz = at & 1;
      } else {
        const int a = (at - 8) >> 3, side = (at >> 2) & 1 ? 2 : -1, h = (at >> 1) & 1, l = at & 1;
        dx = a == 0 ? side : h;
        dy = a == 1 ? side : (a == 0 ? h : l);
        dz = a == 2 ? side : l;
      }
      atomicAdd(GD + (ocell + dx * st[0] + dy * st[1] + dz), s_acc[at][threadIdx.x]);
    }
    __syncwarp();
  }
}

template <typename W>
int qef_bwd_grid() {
  static std::atomic<int> grid[64] = {};
  return per_device_once(grid, [](int dev) {
    int sms = 0, per_sm = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaFuncSetAttribute(k_qef_bwd<W>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kQefBwdSmem);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_qef_bwd<W>, kQefBwdThreads, kQefBwdSmem);
    return (sms > 0 ? sms : 1) * (per_sm > 0 ? per_sm : 1);
  });
}

}  // namespace

void launch_qef_bwd(int wide, const ChunkDev* d_chunks, int n_chunks, const uint32_t* words, const float* dens,
                    const uint32_t* vkey, int64_t vcap, const float* grad_pos, float* grad_dens, const uint32_t* qlist,
                    const uint32_t* qcount, const float* qseed, cudaStream_t st) {
  const int64_t need = (vcap + kQefBwdThreads - 1) / kQefBwdThreads;
  if (need == 0) return;
#define BMF_QEF_BWD(W)                                                                                              \
  k_qef_bwd<W><<<(int)(need < qef_bwd_grid<W>() ? need : qef_bwd_grid<W>()), kQefBwdThreads, kQefBwdSmem, st>>>(    \
      d_chunks, n_chunks, words, dens, vkey, grad_pos, grad_dens, qlist, qcount, qseed)
  if (wide == 2) BMF_QEF_BWD(DF); else BMF_QEF_BWD(double);
#undef BMF_QEF_BWD
}

}  // namespace bmf
