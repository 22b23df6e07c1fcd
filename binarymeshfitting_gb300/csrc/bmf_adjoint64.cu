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
// Bound by what 16 warps per SM leave uncovered of the latencies (0.59 of the issue
// slots, the FMA pipe half busy).  The double-float code is larger than the
// instruction caches, and free-running warps, at different places of it, stall on
// fetches instead (8 of 12.6 cycles per issue; now 0.9).  So a CTA's warps go through
// the parts together, with a block barrier between them and between the sweeps,
// the three rotations of a sweep share one copy of the code (the axes change
// places), and 128 registers keep the matrices out of local memory.  512 x 65^3
// (3.9 M vertices): 2.40 -> 1.35 ms against one free-running thread per vertex at
// 8 x 128 threads; one 65^3 grid 85 -> 76 us.
//
// The wide operations and their order are what they were there: with the largest
// gradients 1000 times the rms, a last bit of dL/dA is 1e-3 of the rms after the
// chain rule's cancellations.  (With n n^T = G G^T / (G.G), rotations by FP32
// angles and cell-relative points the step is 0.42 ms shorter and as near to
// FP64, but single samples move by up to 2e-3 of the rms.)
#include "bmf_qef.cuh"

namespace bmf {
namespace {

// Stopping point of the eigen refinement, in units of |A|: 1e-17 in FP64, 3e-14
// (about its resolution) in double-float.
__device__ __forceinline__ double eig_tol(double) { return 1e-17; }
__device__ __forceinline__ DF eig_tol(DF) { return DF(3e-14); }

template <typename W>
__device__ __forceinline__ void grid_gradient_w(const float* __restrict__ D, int dim, const int c[3], int o, W g[3]) {
  const int st[3] = {dim * dim, dim, 1};
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const bool lo = c[a] > 0, hi = c[a] < dim - 1;
    g[a] = (W(__ldg(D + (o + (hi ? st[a] : 0)))) - W(__ldg(D + (o - (lo ? st[a] : 0))))) * W(lo && hi ? 0.5f : 1.0f);
  }
}

// axes i and j of the rotated matrix and its basis change places
template <typename W>
__device__ __forceinline__ void swap_axes(W B[3][3], W V[3][3], int i, int j) {
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const W b = B[k][i], v = V[k][i];
    B[k][i] = B[k][j];
    B[k][j] = b;
    V[k][i] = V[k][j];
    V[k][j] = v;
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const W b = B[i][k];
    B[i][k] = B[j][k];
    B[j][k] = b;
  }
}

template <typename W, int THREADS>
__global__ void __launch_bounds__(THREADS, 512 / THREADS) k_qef_bwd(
    const ChunkDev* __restrict__ chunks, int n_chunks, const uint32_t* __restrict__ words,
    const float* __restrict__ dens, const uint32_t* __restrict__ vkey, const float* __restrict__ grad_pos,
    float* __restrict__ grad_dens, const uint32_t* __restrict__ qlist, const uint32_t* __restrict__ qcount,
    const float* __restrict__ qseed) {
  const int64_t n = *qcount;
  for (int64_t s0 = (int64_t)blockIdx.x * THREADS; s0 < n; s0 += (int64_t)gridDim.x * THREADS) {
    const int64_t slot = s0 + threadIdx.x;
    const bool in = slot < n;
    const uint32_t v = in ? qlist[slot] : 0u;
    const ChunkDev& ch = chunks[find_chunk_by_vertex(chunks, n_chunks, v)];
    const int dim = ch.dim;
    const float* __restrict__ D = dens + ch.dens;
    int x, y, z, g;
    vertex_key_decode(vkey[v], x, y, z, g);
    const uint32_t edges = in ? group_edges(cell_mask_at(words + ch.words, dim, ch.zc, x, y, z), g) : 0u;
    const int ocell = (x * dim + y) * dim + z, st[3] = {dim * dim, dim, 1}, cnt = max(1, __popc(edges));
    float fA[3][3], fr[3], fm[3];
    {
      // A, sum (n.p) n and the mass point in the wide type
      W A[3][3], b[3], m[3];
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        b[r] = m[r] = W(0.0f);
#pragma unroll
        for (int k = 0; k < 3; ++k) A[r][k] = W(0.0f);
      }
#pragma unroll 1
      for (uint32_t em = edges; em; em &= em - 1u) {
        const int e = __ffs(em) - 1, ca = edge_c0(e), ax = e >> 2;
        const int a0[3] = {x + ((ca >> 2) & 1), y + ((ca >> 1) & 1), z + (ca & 1)};
        const int a1[3] = {a0[0] + (ax == 0), a0[1] + (ax == 1), a0[2] + (ax == 2)};
        const int o0 = ocell + ((ca >> 2) & 1) * st[0] + ((ca >> 1) & 1) * st[1] + (ca & 1);
        const int o1 = o0 + (ax == 0 ? st[0] : (ax == 1 ? st[1] : 1));
        const W s0d(__ldg(D + o0)), s1d(__ldg(D + o1));
        const W mu = (W(0.0f) - s0d) / (s1d - s0d);
        W g0[3], nn[3], pp[3];
        grid_gradient_w<W>(D, dim, a0, o0, g0);
        grid_gradient_w<W>(D, dim, a1, o1, nn);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          pp[k] = (W((float)a1[k]) - W((float)a0[k])) * mu + W((float)a0[k]);
          nn[k] = g0[k] + (nn[k] - g0[k]) * mu;
        }
        const W il = W(1.0f) / sqrt((nn[0] * nn[0] + nn[1] * nn[1]) + nn[2] * nn[2]);
#pragma unroll
        for (int k = 0; k < 3; ++k) nn[k] = nn[k] * il;
        const W d = nn[0] * pp[0] + nn[1] * pp[1] + nn[2] * pp[2];
#pragma unroll
        for (int r = 0; r < 3; ++r) {
#pragma unroll
          for (int k = 0; k < 3; ++k) A[r][k] += nn[r] * nn[k];
          b[r] += d * nn[r];
          m[r] += pp[r];
        }
      }
      __syncthreads();  // the CTA's warps run each part's code together
#pragma unroll
      for (int r = 0; r < 3; ++r) m[r] /= W(cnt);
#pragma unroll
      for (int r = 0; r < 3; ++r) b[r] = b[r] - (A[r][0] * m[0] + A[r][1] * m[1] + A[r][2] * m[2]);  // r
      // eigen pairs of A: the forward's FP32 eigenvectors, orthonormalised; B = V^T A V
      W V[3][3], B[3][3];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        W t[3];
#pragma unroll
        for (int r = 0; r < 3; ++r) t[r] = W(in ? qseed[9 * slot + 3 * r + c] : (r == c ? 1.0f : 0.0f));
#pragma unroll
        for (int k = 0; k < c; ++k) {
          const W d = t[0] * V[0][k] + t[1] * V[1][k] + t[2] * V[2][k];
#pragma unroll
          for (int r = 0; r < 3; ++r) t[r] -= d * V[r][k];
        }
        const W il = W(1.0f) / sqrt(t[0] * t[0] + t[1] * t[1] + t[2] * t[2]);
#pragma unroll
        for (int r = 0; r < 3; ++r) V[r][c] = t[r] * il;
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        W t[3];  // column c of A V
#pragma unroll
        for (int r = 0; r < 3; ++r) t[r] = A[r][0] * V[0][c] + A[r][1] * V[1][c] + A[r][2] * V[2][c];
#pragma unroll
        for (int r = 0; r < 3; ++r) B[r][c] = V[0][r] * t[0] + V[1][r] * t[1] + V[2][r] * t[2];
      }
#pragma unroll
      for (int r = 0; r < 3; ++r) {
#pragma unroll
        for (int c = 0; c < r; ++c) B[r][c] = B[c][r] = W(0.5f) * (B[r][c] + B[c][r]);
      }
      const W tol = eig_tol(W()) * (fabs(B[0][0]) + fabs(B[1][1]) + fabs(B[2][2]));
#pragma unroll 1
      for (int sweep = 0; sweep < 16; ++sweep) {
        const bool more = !(fabs(B[0][1]) + fabs(B[0][2]) + fabs(B[1][2]) <= tol);
        if (!__syncthreads_or(more)) break;
        // axes (0, 1), (0, 2), (1, 2) in turn, each brought to places 0 and 1:
        // one copy of the rotation's code
#pragma unroll 1
        for (int q = 0; q < 3; ++q) {
          if (more && !(fabs(B[0][1]) <= tol)) {
            const W tau = (B[1][1] - B[0][0]) / (W(2.0f) * B[0][1]);
            const W t = (tau >= W(0.0f) ? W(1.0f) : W(-1.0f)) / (fabs(tau) + sqrt(W(1.0f) + tau * tau));
            const W c = W(1.0f) / sqrt(W(1.0f) + t * t), s = t * c;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
              const W bp = B[k][0], br = B[k][1];
              B[k][0] = c * bp - s * br;
              B[k][1] = s * bp + c * br;
            }
#pragma unroll
            for (int k = 0; k < 3; ++k) {
              const W bp = B[0][k], br = B[1][k];
              B[0][k] = c * bp - s * br;
              B[1][k] = s * bp + c * br;
            }
#pragma unroll
            for (int k = 0; k < 3; ++k) {
              const W vp = V[k][0], vr = V[k][1];
              V[k][0] = c * vp - s * vr;
              V[k][1] = s * vp + c * vr;
            }
          }
          if (q == 0) {
            swap_axes(B, V, 1, 2);  // 0 2 1
          } else if (q == 1) {
            swap_axes(B, V, 0, 2);  // 1 2 0
          } else {
            swap_axes(B, V, 0, 2);  // 0 2 1
            swap_axes(B, V, 1, 2);  // 0 1 2
          }
        }
      }
      // f(s) = 1/s kept where min(|s|, |1/s|) >= 0.001 (qef_simd.h:346-368)
      W sg[3], f[3];
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        sg[i] = B[i][i];
        const W oo = W(1.0f) / sg[i];
        const W mn = fabs(sg[i]) < fabs(oo) ? fabs(sg[i]) : fabs(oo);
        f[i] = mn >= W(0.001f) ? oo : W(0.0f);
      }
      __syncthreads();
      // dL/d(A, r, m): gr = V f V^T gx, gm = gx - A gr, and gA = V (F o M) V^T -
      // sym(gr m^T) with M = V^T sym(gx r^T) V (Daleckii-Krein)
      W gx[3], gr[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) gx[k] = W(in ? grad_pos[3 * (int64_t)v + k] : 0.0f);
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        W pm[3];
#pragma unroll
        for (int k = 0; k < 3; ++k)
          pm[k] = V[r][0] * f[0] * V[k][0] + V[r][1] * f[1] * V[k][1] + V[r][2] * f[2] * V[k][2];
        gr[r] = pm[0] * gx[0] + pm[1] * gx[1] + pm[2] * gx[2];
      }
      W U[3][3];  // sym(gx r^T) V, then V (F o M)
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        W gs[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) gs[k] = W(0.5f) * (gx[r] * b[k] + gx[k] * b[r]);
#pragma unroll
        for (int c = 0; c < 3; ++c) U[r][c] = gs[0] * V[0][c] + gs[1] * V[1][c] + gs[2] * V[2][c];
      }
#pragma unroll
      for (int a = 0; a < 3; ++a) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const W M = V[0][a] * U[0][c] + V[1][a] * U[1][c] + V[2][a] * U[2][c];
          // (f_a - f_c) / (s_a - s_c): -f_a f_c for two kept eigenvalues (no
          // cancellation for close ones), the quotient for a kept and a truncated one
          W F;
          if (f[a] != W(0.0f) && f[c] != W(0.0f))
            F = -f[a] * f[c];
          else if (a == c || fabs(sg[a] - sg[c]) <= W(1e-6) * (fabs(sg[a]) + fabs(sg[c])))
            F = W(0.0f);
          else
            F = (f[a] - f[c]) / (sg[a] - sg[c]);
          B[a][c] = F * M;
        }
      }
#pragma unroll
      for (int r = 0; r < 3; ++r) {
#pragma unroll
        for (int c = 0; c < 3; ++c) U[r][c] = V[r][0] * B[0][c] + V[r][1] * B[1][c] + V[r][2] * B[2][c];
      }
#pragma unroll
      for (int r = 0; r < 3; ++r) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const W s = U[r][0] * V[k][0] + U[r][1] * V[k][1] + U[r][2] * V[k][2];
          fA[r][k] = (float)(s - W(0.5f) * (gr[r] * m[k] + gr[k] * m[r]));
        }
        fr[r] = (float)gr[r];
        fm[r] = (float)(gx[r] - (A[r][0] * gr[0] + A[r][1] * gr[1] + A[r][2] * gr[2]));
      }
    }
    __syncthreads();
    // The chain rule through every hermite pair runs in FP32 on the forward's own
    // hermite data: what remains is a product of well-conditioned factors.
    float* __restrict__ GD = grad_dens + ch.dens;
    const float inv_cnt = 1.0f / (float)cnt;
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
        gn[k] = 2.0f * (fA[k][0] * h.n[0] + fA[k][1] * h.n[1] + fA[k][2] * h.n[2]) + d * fr[k] + gd * h.p[k];
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
      const int oa = ocell + ((ca >> 2) & 1) * st[0] + ((ca >> 1) & 1) * st[1] + (ca & 1);
      const int ob = oa + (ax == 0 ? st[0] : (ax == 1 ? st[1] : 1));
#pragma unroll
      for (int a = 0; a < 3; ++a) {
#pragma unroll
        for (int end = 0; end < 2; ++end) {
          const int* q0 = end ? h.a1 : h.a0;
          const int o = end ? ob : oa;
          const float wgt = gG[a] * (end ? h.mu : 1.0f - h.mu);
          const bool lo = q0[a] > 0, hi = q0[a] < dim - 1;
          const float hh = lo && hi ? wgt * 0.5f : wgt;
          atomicAdd(GD + (o + (hi ? st[a] : 0)), hh);
          atomicAdd(GD + (o - (lo ? st[a] : 0)), -hh);
        }
      }
      const float iden = 1.0f / ((h.s1 - h.s0) * (h.s1 - h.s0));
      atomicAdd(GD + oa, gmu * (-h.s1 * iden));
      atomicAdd(GD + ob, gmu * (h.s0 * iden));
    }
    __syncwarp();
  }
}

// The resident CTAs, and the launch.
template <typename W, int THREADS>
int qef_bwd_grid() {
  static std::atomic<int> grid[64] = {};
  return per_device_once(grid, [](int dev) {
    int sms = 0, per_sm = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_qef_bwd<W, THREADS>, THREADS, 0);
    return (sms > 0 ? sms : 1) * (per_sm > 0 ? per_sm : 1);
  });
}
template <typename W, int THREADS, typename... A>
void qef_bwd_run(int64_t vcap, cudaStream_t st, A... args) {
  const int64_t need = (vcap + THREADS - 1) / THREADS, grid = qef_bwd_grid<W, THREADS>();
  if (need > 0) k_qef_bwd<W, THREADS><<<(int)(need < grid ? need : grid), THREADS, 0, st>>>(args...);
}

}  // namespace

// Double-float: lists that one or two waves of 128-thread CTAs take go out in those, spread over more SMs with half the warps per
// barrier (fit steps, us, 128 / 256 threads: 1 x 65^3 173 / 181, 4 x 192 / 201, 16 x
// 284 / 291); longer ones in 256-thread CTAs, whose warps share more of the code's
// fetches (512 x 4310 / 4020).  The host knows the arena's capacity, not the list (which is
// about half of it in the usual arena): a small list in a far larger arena takes the
// longer lists' form, and its 8 us.
void launch_qef_bwd(int wide, const ChunkDev* d_chunks, int n_chunks, const uint32_t* words, const float* dens,
                    const uint32_t* vkey, int64_t vcap, const float* grad_pos, float* grad_dens, const uint32_t* qlist,
                    const uint32_t* qcount, const float* qseed, cudaStream_t st) {
  const auto run = [&](auto go) {
    go(vcap, st, d_chunks, n_chunks, words, dens, vkey, grad_pos, grad_dens, qlist, qcount, qseed);
  };
  if (wide != 2)
    run([](auto... a) { qef_bwd_run<double, 256>(a...); });
  else if (vcap <= 4ll * 128 * qef_bwd_grid<DF, 128>())
    run([](auto... a) { qef_bwd_run<DF, 128>(a...); });
  else
    run([](auto... a) { qef_bwd_run<DF, 256>(a...); });
}

}  // namespace bmf
