// Stage 3 + 4: surface-cell enumeration, vertex / primitive compaction and
// emission (DMCChunk::label_edges enumeration + calculate_cell +
// calculate_isovertex + polygonize, DMCChunk.cpp:440-674), and the DMC quad
// emitter with mass-point / QEF placement (qef_simd.h).
//
// The reference numbers vertices in one sequential scan: cells in linear
// (x, y, z) order, and inside a cell its x-, y-, z-edge crossings
// (DMCChunk.cpp:449-474, 599-654).  Here every 32-bit occupancy word W[x][y][zb]
// stands for the 32 cells (x, y, 32zb..32zb+31), and the crossings those cells
// own are three bit words:
//     X = W[x][y] ^ W[x+1][y],  Y = W[x][y] ^ W[x][y+1],  Z = W ^ (W >> 1 | next << 31)
// so a word hosts popc(X)+popc(Y)+popc(Z) vertices, and the vertex id of cell z's
// axis-a crossing is   base(word) + popc((X|Y|Z bits of cells < z)) + (own earlier axes).
// base(word) is the exclusive sum of the per-word counts in (x, y, zb) order --
// of the planes before x (ws.pb) plus of the plane's words before it (ws.vcnt)
// -- which is exactly the reference's sequential order.  Triangles are counted
// and placed the same way, so vertex and index buffers come out bit-identical
// to the reference without any per-cell index volume (IndexesBlock) or cell
// list (DMC_CellsBlock).
#include "bmf_device.cuh"
#include "bmf_internal.h"
#include "bmf_qef.cuh"
#include "bmf_sweep.cuh"

namespace bmf {

// Chunk of x-plane u, by a whole warp: 32 candidates per step (a dependent load
// per factor of 32 in the chunk count, not per factor of 2).
__device__ __forceinline__ int find_chunk_e(const int* __restrict__ unit_start, int n_chunks, int u) {
  const int lane = threadIdx.x & 31;
  int lo = 0, n = n_chunks;
  while (n > 1) {
    const int step = (n + 31) >> 5, cand = lane * step;
    const uint32_t le = __ballot_sync(kFull, cand < n && __ldg(unit_start + lo + cand) <= u);
    const int at = (__popc(le) - 1) * step;  // unit_start ascends: le is a prefix of the lanes, lane 0 in it
    lo += at;
    n = min(step, n - at);
  }
  return lo;
}

template <typename T>
__device__ __forceinline__ T warp_incl_sum(T v, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const T n = __shfl_up_sync(kFull, v, o);
    if (lane >= o) v += n;
  }
  return v;
}

// EDGE_V offsets (DMCChunk.cpp:32, 543-565): edge e of a cell is the axis-a
// crossing owned by the cell at offset (ox, oy, oz).
static __constant__ int8_t c_edge_owner[12][4] = {{0, 0, 0, 0}, {0, 0, 1, 0}, {0, 1, 0, 0}, {0, 1, 1, 0},
                                                  {0, 0, 0, 1}, {0, 0, 1, 1}, {1, 0, 0, 1}, {1, 0, 1, 1},
                                                  {0, 0, 0, 2}, {0, 1, 0, 2}, {1, 0, 0, 2}, {1, 1, 0, 2}};

// Mask of cell (x, y, 32zb + lane) from the four line words around it and the
// four next-block words (for corner z + 1 of the block's last cell).
__device__ __forceinline__ int mask_from_lines(uint32_t w00, uint32_t w01, uint32_t w10, uint32_t w11, uint32_t n00,
                                               uint32_t n01, uint32_t n10, uint32_t n11, int lane) {
  const uint64_t q00 = ((uint64_t)n00 << 32) | w00, q01 = ((uint64_t)n01 << 32) | w01;
  const uint64_t q10 = ((uint64_t)n10 << 32) | w10, q11 = ((uint64_t)n11 << 32) | w11;
  return (int)(((q00 >> lane) & 3u) | (((q01 >> lane) & 3u) << 2) | (((q10 >> lane) & 3u) << 4) |
               (((q11 >> lane) & 3u) << 6));
}

struct LineWords {
  uint32_t w00, w01, w10, w11, n00, n01, n10, n11;
  __device__ __forceinline__ void load(const uint32_t* W, int dim, int zc, int x, int y, int zb) {
    w00 = word_at(W, dim, zc, x, y, zb);
    w01 = word_at(W, dim, zc, x, y + 1, zb);
    w10 = word_at(W, dim, zc, x + 1, y, zb);
    w11 = word_at(W, dim, zc, x + 1, y + 1, zb);
    n00 = word_at(W, dim, zc, x, y, zb + 1);
    n01 = word_at(W, dim, zc, x, y + 1, zb + 1);
    n10 = word_at(W, dim, zc, x + 1, y, zb + 1);
    n11 = word_at(W, dim, zc, x + 1, y + 1, zb + 1);
  }
  __device__ __forceinline__ int mask(int lane) const {
    return mask_from_lines(w00, w01, w10, w11, n00, n01, n10, n11, lane);
  }
};

constexpr int kWordBlock = 256;  // threads per CTA of the count / emit kernels

// A word is quiet when its 32 cells can neither own a crossing nor have a
// mixed corner mask: the four line words around it are identical, so are the
// four next-block words, and the line has no z-crossing.  Then X = Y = Z = 0
// and every cell with all corners inside the chunk has mask 0 or 255, so the
// word contributes no vertex, triangle or quad in either mode.
__device__ __forceinline__ bool word_is_quiet(const uint32_t* W, int dim, int zc, int x, int y, int zb) {
  const uint32_t w = word_at(W, dim, zc, x, y, zb);
  if (word_at(W, dim, zc, x, y + 1, zb) != w || word_at(W, dim, zc, x + 1, y, zb) != w ||
      word_at(W, dim, zc, x + 1, y + 1, zb) != w)
    return false;
  const uint32_t n = word_at(W, dim, zc, x, y, zb + 1);
  if (word_at(W, dim, zc, x, y + 1, zb + 1) != n || word_at(W, dim, zc, x + 1, y, zb + 1) != n ||
      word_at(W, dim, zc, x + 1, y + 1, zb + 1) != n)
    return false;
  return zcross_word(W, dim, zc, x, y, zb) == 0u;
}

// Interior-edge test of Mode Q: the grid edge from sample s along axis a has
// all four surrounding cells.
__device__ __forceinline__ bool q_edge_interior(int dim, int sx, int sy, int sz, int a) {
  const int s[3] = {sx, sy, sz};
  const int b = (a + 1) % 3, c = (a + 2) % 3;
  return s[a] <= dim - 2 && s[b] >= 1 && s[b] <= dim - 2 && s[c] >= 1 && s[c] <= dim - 2;
}

// Interior crossing words of Mode Q (quads) for line (x, y) block zb.
__device__ __forceinline__ void q_quad_words(const uint32_t* W, int dim, int zc, int x, int y, int zb, uint32_t& Xi,
                                             uint32_t& Yi, uint32_t& Zi) {
  // z in [1, dim-2]
  uint32_t zint = kFull;
  const int lo = 1 - 32 * zb, hi = dim - 2 - 32 * zb;  // valid bit range [lo, hi]
  if (hi < 0 || lo > 31) zint = 0u;
  else {
    if (hi < 31) zint &= (2u << hi) - 1u;
    if (lo > 0) zint &= ~((1u << lo) - 1u);
  }
  Xi = (y >= 1 && y <= dim - 2) ? (xcross_word(W, dim, zc, x, y, zb) & zint) : 0u;
  Yi = (x >= 1 && x <= dim - 2) ? (ycross_word(W, dim, zc, x, y, zb) & zint) : 0u;
  Zi = (x >= 1 && x <= dim - 2 && y >= 1 && y <= dim - 2) ? zcross_word(W, dim, zc, x, y, zb) : 0u;
}

// ---------------------------------------------------------------------------
// K2: per-word counts, one thread per occupancy word, a CTA or a warp per x-plane.
//
// It walks its plane's words in order and keeps the running sums, so a
// word's count leaves as the sum of the plane's words before it, and the
// plane's totals go to ws.pb: a scan over a chunk's planes (k_chunk_scan, at
// most 512 pairs) then replaces a pass over all words (read and written back:
// 0.28 ms of a 4096-chunk update, 65 us of one 129^3 chunk, whose words one
// CTA scanned).  Quiet words write nothing.
//
// Everything a word contributes is bit arithmetic on the eight line words
// around it (lines (x..x+1, y..y+1), blocks zb and zb + 1): its owned
// crossings X / Y / Z (vertex count by popc, Mode R), its interior quad edges
// (Mode Q), and the set of its cells whose corner mask is mixed (neither 0 nor
// 255).  Only mixed cells can emit triangles or hold vertex groups, so the
// per-cell table lookup runs over the set bits of that mask alone; the
// counts go into three bit-planes (a cell's first primitive / vertex is
// base + popc(p0 & lt) + 2 popc(p1 & lt) + 4 popc(p2 & lt)).
// ---------------------------------------------------------------------------

// Per corner mask: Mode R triangle count (low nibble) and Mode Q vertex-group
// count (high nibble), four masks per word.
struct CaseCounts {
  uint32_t w[64];
};
constexpr CaseCounts make_case_counts() {
  constexpr uint64_t tri[256] = BMF_TRI_CASES_INIT;
  constexpr uint64_t grp[256] = BMF_GROUP_CASES_INIT;
  CaseCounts c{};
  for (int m = 0; m < 256; ++m)
    c.w[m >> 2] |= (uint32_t)((tri[m] >> 60) | (((grp[m] >> 48) & 0xF) << 4)) << (8 * (m & 3));
  return c;
}
static __device__ const CaseCounts g_case_counts = make_case_counts();

// Per corner mask and edge e: which of the case's triangles (bit t, t < 5)
// use edge e, at bits [5 e, 5 e + 5) -- derived from the triangle table.
struct EdgeTris {
  uint64_t w[256];
};
constexpr EdgeTris make_edge_tris() {
  constexpr uint64_t tri[256] = BMF_TRI_CASES_INIT;
  EdgeTris r{};
  for (int m = 0; m < 256; ++m) {
    const int nt = (int)(tri[m] >> 60);
    for (int t = 0; t < nt; ++t)
      for (int i = 0; i < 3; ++i) r.w[m] |= 1ull << (5 * (int)((tri[m] >> (4 * (3 * t + i))) & 0xFu) + t);
  }
  return r;
}
static __device__ const EdgeTris g_edge_tris = make_edge_tris();

// With few planes (a chunk or a small batch) a CTA of 256 threads per plane shortens
// the walk over its words (129^3: 645 words); a whole update's planes fill the GPU
// with a warp each, which leaves out the block's barriers and the quiet words.  Mixed
// updates without sweeps, us, a warp / a CTA per plane: 20 chunks (1.3 k planes) 183 /
// 175, 32 (2.0 k) 192 / 189, 48 (2.9 k) 174 / 177, 96 243 / 259, 400 625 / 714.
constexpr int kCountThreads = 256;
constexpr int kCountFewUnits = 2048;

// What one word contributes: its vertices and indices, the count planes, whether it
// is busy, and (Mode R band fill) the samples to make exact -- in its own line
// (f00), lines x + 1 and y + 1, and bit 0 of the next word.
struct WordCounts {
  uint32_t vc = 0u, ic = 0u, p0 = 0u, p1 = 0u, p2 = 0u, act = 0u;
  uint32_t f00 = 0u, f10 = 0u, f01 = 0u, fnx = 0u;
};

// Word wi = (y, zb) of plane x, whose words start at Wx (cw: the chunk's first word).
template <int MODE>
__device__ __forceinline__ WordCounts count_word(const uint32_t* s_cnt, const WordScratch& ws,
                                                 const uint32_t* __restrict__ Wx, int64_t cw, int dim, int zc, int x,
                                                 int wi, int y, int zb, uint32_t& fl) {
  WordCounts r;
  const int nw = dim * zc;
  const bool xin = x + 1 < dim;  // line x + 1 exists (cells and x-crossings of this plane)
  const bool yin = y + 1 < dim, nin = zb + 1 < zc;
  const uint32_t* L00 = Wx + wi;  // the word (x, y, zb)
  const uint32_t w00 = __ldg(L00), n00 = nin ? __ldg(L00 + 1) : 0u;
  const uint32_t w01 = yin ? __ldg(L00 + zc) : 0u, n01 = (yin && nin) ? __ldg(L00 + zc + 1) : 0u;
  const uint32_t* L10 = L00 + nw;
  const uint32_t w10 = xin ? __ldg(L10) : 0u, n10 = (xin && nin) ? __ldg(L10 + 1) : 0u;
  const uint32_t w11 = (xin && yin) ? __ldg(L10 + zc) : 0u, n11 = (xin && yin && nin) ? __ldg(L10 + zc + 1) : 0u;
  fl |= (w00 != 0u && w00 != kFull) ? 1u : (w00 == kFull ? 2u : 4u);
  // corner words: bit l = corner (dx, dy, dz) of cell 32 zb + l
  const uint32_t a0 = w00, a1 = (w00 >> 1) | (n00 << 31), b0 = w01, b1 = (w01 >> 1) | (n01 << 31);
  const uint32_t c0 = w10, c1 = (w10 >> 1) | (n10 << 31), d0 = w11, d1 = (w11 >> 1) | (n11 << 31);
  const uint32_t any = a0 | a1 | b0 | b1 | c0 | c1 | d0 | d1, all = a0 & a1 & b0 & b1 & c0 & c1 & d0 & d1;
  const uint32_t zint = zbits_upto(dim - 2, zb);  // cells z <= dim - 2
  const uint32_t interior = (xin && yin) ? zint : 0u;
  const uint32_t mixed = interior & any & ~all;
  uint32_t t = 0u;
  for (uint32_t m = mixed; m; m &= m - 1u) {
    const int l = __ffs(m) - 1;
    const int mask = (int)(((w00 >> l) & 1u) | (((a1 >> l) & 1u) << 1) | (((w01 >> l) & 1u) << 2) |
                           (((b1 >> l) & 1u) << 3) | (((w10 >> l) & 1u) << 4) | (((c1 >> l) & 1u) << 5) |
                           (((w11 >> l) & 1u) << 6) | (((d1 >> l) & 1u) << 7));
    const uint32_t k = (s_cnt[mask >> 2] >> (8 * (mask & 3))) >> (MODE == 0 ? 0 : 4);
    const uint32_t n = k & 0xFu;
    t += n;
    r.p0 |= (n & 1u) << l;
    r.p1 |= ((n >> 1) & 1u) << l;
    r.p2 |= ((n >> 2) & 1u) << l;
  }
  const uint32_t planes = r.p0 | r.p1 | r.p2;
  if (MODE == 0) {
    const uint32_t X = xin ? (w00 ^ w10) : 0u;
    const uint32_t Y = yin ? (w00 ^ w01) : 0u;
    const uint32_t Z = (w00 ^ a1) & zint;
    r.vc = __popc(X) + __popc(Y) + __popc(Z);
    r.ic = 3u * t;
    r.act = planes | X | Y | Z;
    if (ws.exact && (X | Y | Z)) {
      // own samples (X, Y, Z starts, Z ends), line x + 1 (X), line y + 1 (Y),
      // and bit 0 of the next word (the end of a crossing from bit 31)
      const uint32_t* E = ws.exact + cw + (int64_t)x * nw + wi;
      r.f00 = (X | Y | Z | (Z << 1)) & ~__ldg(E);
      r.f10 = X ? (X & ~__ldg(E + nw)) : 0u;
      r.f01 = Y ? (Y & ~__ldg(E + zc)) : 0u;
      r.fnx = (Z >> 31) ? (~__ldg(E + 1) & 1u) : 0u;
    }
  } else {
    // interior quad edges: the four cells around the edge exist
    const bool yi = y >= 1 && y <= dim - 2, xi = x >= 1 && x <= dim - 2;
    const uint32_t zlo = zb == 0 ? ~1u : kFull;  // with zint: z in [1, dim - 2]
    const uint32_t Z = (w00 ^ a1) & zint;
    const uint32_t Xi = (yi && xin) ? ((w00 ^ w10) & zint & zlo) : 0u;
    const uint32_t Yi = (xi && yin) ? ((w00 ^ w01) & zint & zlo) : 0u;
    const uint32_t Zi = (xi && yi) ? Z : 0u;
    r.vc = t;
    r.ic = 4u * (__popc(Xi) + __popc(Yi) + __popc(Zi));
    r.act = planes | Xi | Yi | Zi;
    if (ws.ends) {
      // samples with a neighbour of the other sign, along each axis and way
      uint32_t e = Z | (Z << 1) | (xin ? w00 ^ w10 : 0u) | (yin ? w00 ^ w01 : 0u);
      if (zb > 0) e |= (w00 ^ (__ldg(L00 - 1) >> 31)) & 1u;
      if (x > 0) e |= w00 ^ __ldg(L00 - nw);
      if (y > 0) e |= w00 ^ __ldg(L00 - zc);
      ws.ends[cw + (int64_t)x * nw + wi] = e;
    }
  }
  return r;
}

// The warp's entries of the fix-up list and of the work list, one global
// reservation each (word index wp in the chunk, plane x, line y).
template <int MODE>
__device__ __forceinline__ void count_lists(const WordScratch& ws, const WordCounts& r, int c, int dim, int x, int y,
                                            int zb, int wp, int lane) {
  if (MODE == 0 && ws.exact && __any_sync(kFull, (r.f00 | r.f10 | r.f01 | r.fnx) != 0u)) {
    const int nf = __popc(r.f00) + __popc(r.f10) + __popc(r.f01) + __popc(r.fnx);
    int incl = nf;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int v = __shfl_up_sync(kFull, incl, off);
      if (lane >= off) incl += v;
    }
    uint32_t fbase = 0u;
    if (lane == 31) fbase = atomicAdd(ws.fcount, (uint32_t)incl);
    fbase = __shfl_sync(kFull, fbase, 31);
    if (nf) {
      int64_t slot = (int64_t)fbase + incl - nf;
      const uint32_t s00 = (uint32_t)((((int64_t)x * dim + y) * dim) + 32 * zb);
      auto put = [&](uint32_t m, uint32_t sbase) {
        for (; m; m &= m - 1u, ++slot)
          if (slot < ws.fix_cap) ws.fix[slot] = make_uint2((uint32_t)c, sbase + (uint32_t)(__ffs(m) - 1));
      };
      put(r.f00, s00);
      put(r.f10, s00 + (uint32_t)dim * (uint32_t)dim);
      put(r.f01, s00 + (uint32_t)dim);
      put(r.fnx, s00 + 32u);
    }
  }
  if (ws.clist) {
    const uint32_t busy = __ballot_sync(kFull, r.act != 0u);
    if (busy == 0u) return;
    uint32_t wbase = 0u;
    if (lane == 0) wbase = atomicAdd(ws.ccount, (uint32_t)__popc(busy));
    wbase = __shfl_sync(kFull, wbase, 0);
    const int64_t slot = (int64_t)wbase + __popc(busy & lane_lt(lane));
    if (r.act && slot < ws.clist_cap) ws.clist[slot] = make_uint2((uint32_t)c, (uint32_t)wp);
  }
}

// One CTA per plane.
template <int MODE>
__global__ void __launch_bounds__(kCountThreads) k_count(const ChunkDev* __restrict__ chunks, int n_chunks,
                                                         const int* __restrict__ unit_start,
                                                         const uint32_t* __restrict__ words,
                                                         const uint32_t* __restrict__ flags,
                                                         uint32_t* __restrict__ flags_out, WordScratch ws) {
  constexpr int kWarps = kCountThreads / 32;
  __shared__ uint32_t s_cnt[64];
  __shared__ uint2 s_sum[2][kWarps];  // per warp {vertices, indices} of this step's words, two steps in turn
  const int u = blockIdx.x;
  const int c = find_chunk_e(unit_start, n_chunks, u);
  // a chunk without a mesh has equal words everywhere: nothing to count
  if (flags && !contains_mesh(__ldg(flags + c))) {
    if (threadIdx.x == 0) ws.pb[u] = make_uint2(0u, 0u);
    return;
  }
  for (int i = threadIdx.x; i < 64; i += kCountThreads) s_cnt[i] = g_case_counts.w[i];
  __syncthreads();
  const ChunkDev ch = chunks[c];
  const int x = u - __ldg(unit_start + c);
  const int dim = ch.dim, zc = ch.zc, nw = dim * zc;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t carry_v = 0u, carry_i = 0u, fl = 0u;
  // a word's y is its index times the rounded-up 2^32 / zc, high half: exact
  // while index * zc < 2^32
  const uint64_t zmagic = ((1ull << 32) + (uint64_t)zc - 1u) / (uint64_t)zc;
  const uint32_t* Wx = words + ch.words + (int64_t)x * nw;  // the plane's words
  for (int base = 0, step = 0; base < nw; base += kCountThreads, step ^= 1) {
    const int wi = base + threadIdx.x;
    const int y = (int)(((uint64_t)(uint32_t)wi * zmagic) >> 32), zb = wi - y * zc;
    WordCounts r;
    if (wi < nw) r = count_word<MODE>(s_cnt, ws, Wx, ch.words, dim, zc, x, wi, y, zb, fl);
    // the plane's running sums; indices per plane stay below 2^32 (at most
    // 15 per cell, 2^18 cells)
    uint32_t iv = r.vc, ii = r.ic;
    if (__any_sync(kFull, r.act != 0u)) {
      iv = warp_incl_sum(iv, lane);
      ii = warp_incl_sum(ii, lane);
    }
    if (lane == 31) s_sum[step][warp] = make_uint2(iv, ii);
    __syncthreads();
    uint32_t bv = carry_v, bi = carry_i;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const uint2 t = s_sum[step][w];
      if (w < warp) { bv += t.x; bi += t.y; }
      carry_v += t.x;
      carry_i += t.y;
    }
    if (r.act) {
      const int64_t o = ch.words + (int64_t)x * nw + wi;
      ws.vcnt[o] = bv + iv - r.vc;
      ws.rec[o] = make_uint4(r.p0, r.p1, r.p2, bi + ii - r.ic);
    }
    count_lists<MODE>(ws, r, c, dim, x, y, zb, x * nw + wi, lane);
  }
  if (threadIdx.x == 0) ws.pb[u] = make_uint2(carry_v, carry_i);
  if (flags_out) {
    fl = __reduce_or_sync(kFull, fl);
    if (lane == 0 && fl) atomicOr(flags_out + c, fl);
  }
}

// One warp per plane, 31 words a step (lane 31 only looks ahead).  In a whole update
// most words are quiet: a word whose four lines are equal, all inside or all
// outside, and go on so in the next word has no crossing and no mixed cell, which
// four loads and a shuffle show.  The others are gathered in order, and the counts'
// several hundred instructions run on 32 of them at a time.  flags: the chunks'
// (from the fill).  4096-chunk update 951 -> 598 us (counting a step's 31 words as they
// come, whenever one of them is busy: 693), 1024 2D chunks 237 -> 160, 512 x 65^3 101 -> 70.
constexpr int kCountPlanes = 8;  // warps per CTA

template <int MODE>
__global__ void __launch_bounds__(32 * kCountPlanes) k_count_planes(const ChunkDev* __restrict__ chunks, int n_chunks,
                                                                   const int* __restrict__ unit_start, int n_units,
                                                                   const uint32_t* __restrict__ words,
                                                                   const uint32_t* __restrict__ flags,
                                                                   WordScratch ws) {
  __shared__ uint32_t s_cnt[64];
  __shared__ uint16_t s_busy[kCountPlanes][64];  // (a plane has at most 8192 words)
  if (threadIdx.x < 64) s_cnt[threadIdx.x] = g_case_counts.w[threadIdx.x];
  __syncthreads();
  const int u = blockIdx.x * kCountPlanes + (int)(threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (u >= n_units) return;
  const int c = find_chunk_e(unit_start, n_chunks, u);
  if (!contains_mesh(__ldg(flags + c))) {
    if (lane == 0) ws.pb[u] = make_uint2(0u, 0u);
    return;
  }
  uint16_t* list = s_busy[threadIdx.x >> 5];
  const ChunkDev& ch = chunks[c];
  const int64_t cw = ch.words;
  const int dim = ch.dim, zc = ch.zc, nw = dim * zc, x = u - __ldg(unit_start + c);
  const int xo = x + 1 < dim ? nw : 0;  // to the next plane (to itself from the last)
  const uint32_t magic = zc > 1 ? 0xFFFFFFFFu / (uint32_t)zc + 1u : 0u;  // y = high half of index * magic
  const uint32_t* Wx = words + cw + (int64_t)x * nw;
  uint32_t carry_v = 0u, carry_i = 0u, fl = 0u;
  int held = 0;
  // the four lines' words at wi (past the plane's last line and word: its own again)
  const auto load = [&](int wi, uint32_t q[4]) {
    const uint32_t* L = Wx + min(wi, nw - 1);
    const int yo = wi + zc < nw ? zc : 0;
    q[0] = __ldg(L);
    q[1] = __ldg(L + yo);
    q[2] = __ldg(L + xo);
    q[3] = __ldg(L + xo + yo);
  };
  uint32_t q[4];
  load(lane, q);
  for (int base = 0; base < nw; base += 31) {
    const int wi = base + lane;
    const bool in = wi < nw;
    const int y = zc > 1 ? (int)__umulhi((uint32_t)wi, magic) : wi, zb = wi - y * zc;
    const uint32_t w = q[0], s = (w & 1u) ? zbits_upto(dim - 1, zb) : 0u;
    // 1, 2: the four lines are all outside, all inside
    const uint32_t code = ((w ^ s) | (q[1] ^ s) | (q[2] ^ s) | (q[3] ^ s)) == 0u ? 1u + (w & 1u) : 0u;
    load(base + 31 + lane, q);  // the next step's
    const uint32_t next = __shfl_down_sync(kFull, code, 1);
    const bool own = in && lane < 31, quiet = code != 0u && (zb == zc - 1 || next == code);
    if (MODE == 1 && ws.ends) {  // crossings that end in a quiet word come from the words before it
      const uint32_t up = __shfl_up_sync(kFull, w, 1);
      if (own && quiet) {
        uint32_t e = 0u;
        if (zb > 0) e |= (w ^ ((lane ? up : __ldg(Wx + wi - 1)) >> 31)) & 1u;
        if (x > 0) e |= w ^ __ldg(Wx + wi - nw);
        if (y > 0) e |= w ^ __ldg(Wx + wi - zc);
        ws.ends[cw + (int64_t)x * nw + wi] = e;
      }
    }
    const uint32_t busy = __ballot_sync(kFull, own && !quiet);
    if (own && !quiet) list[held + __popc(busy & lane_lt(lane))] = (uint16_t)wi;
    held += __popc(busy);
    // a full round, or what is left after the last step
    while (held >= 32 || (base + 31 >= nw && held > 0)) {
      const int n = min(held, 32);
      __syncwarp();
      const int bw = lane < n ? list[lane] : 0;
      const int more = lane < held - n ? list[32 + lane] : 0;
      __syncwarp();
      if (lane < held - n) list[lane] = (uint16_t)more;
      held -= n;
      const int by = zc > 1 ? (int)__umulhi((uint32_t)bw, magic) : bw, bz = bw - by * zc;
      WordCounts r;
      if (lane < n) r = count_word<MODE>(s_cnt, ws, Wx, cw, dim, zc, x, bw, by, bz, fl);
      __syncwarp();
      // the plane's running sums (as k_count)
      const uint32_t iv = warp_incl_sum(r.vc, lane), ii = warp_incl_sum(r.ic, lane);
      if (r.act) {
        const int64_t o = cw + (int64_t)x * nw + bw;
        ws.vcnt[o] = carry_v + iv - r.vc;
        ws.rec[o] = make_uint4(r.p0, r.p1, r.p2, carry_i + ii - r.ic);
      }
      carry_v += __shfl_sync(kFull, iv, 31);
      carry_i += __shfl_sync(kFull, ii, 31);
      count_lists<MODE>(ws, r, c, dim, x, by, bz, x * nw + bw, lane);
    }
  }
  if (lane == 0) ws.pb[u] = make_uint2(carry_v, carry_i);
}

// ---------------------------------------------------------------------------
// K3: plane totals -> plane bases per chunk (one warp per chunk), then chunk
// totals -> arena offsets, info table and totals, by the CTA that finishes
// last (one for up to 32 chunks).  Latency only: a few KB per chunk.  As one
// CTA with a shared-memory scan after a separate word scan the offsets of 4096
// chunks took 28 us.
// ---------------------------------------------------------------------------
constexpr int kScanThreads = 1024, kScanWarps = kScanThreads / 32;

// Size class of v >= 1 items: two per power of two.
__device__ __forceinline__ int size_bin(uint32_t v) {
  const int l = 31 - __clz(v);
  return 2 * l + (l > 0 ? (int)((v >> (l - 1)) & 1u) : 0);
}

__global__ void __launch_bounds__(kScanThreads) k_chunk_scan(ChunkDev* __restrict__ chunks, int n, uint2* __restrict__ pb,
                                                             uint32_t* tot, const uint32_t* __restrict__ flags,
                                                             int64_t vcap, int64_t icap, int64_t* __restrict__ info,
                                                             int64_t* __restrict__ totals,
                                                             int64_t* __restrict__ h_totals, int* __restrict__ ticket,
                                                             SweepLists sweep) {
  __shared__ int64_t s_v[kScanWarps], s_i[kScanWarps];
  __shared__ bool s_last;
  __shared__ int s_bin[64];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int mine = blockIdx.x * kScanWarps + warp;
  if (n == 1) {
    // one chunk: a thread per plane (at most 512), all of them loaded at once
    // (129 planes: 4.0 us; by one warp's steps, and with the fences, 5.2)
    const int dim = chunks[0].dim, at = threadIdx.x;
    uint2* p = pb + chunks[0].unit0;
    const uint2 t = at < dim ? p[at] : make_uint2(0u, 0u);
    const uint32_t iv = warp_incl_sum(t.x, lane), ii = warp_incl_sum(t.y, lane);
    if (lane == 31) {
      s_v[warp] = iv;
      s_i[warp] = ii;
    }
    __syncthreads();
    const uint32_t bv = __reduce_add_sync(kFull, lane < warp ? (uint32_t)s_v[lane] : 0u);
    const uint32_t bi = __reduce_add_sync(kFull, lane < warp ? (uint32_t)s_i[lane] : 0u);
    if (at < dim) p[at] = make_uint2(bv + iv - t.x, bi + ii - t.y);
    if (at == kScanThreads - 1) {
      tot[0] = bv + iv;
      tot[1] = bi + ii;
    }
  } else if (mine < n) {
    const int dim = chunks[mine].dim;
    uint2* p = pb + chunks[mine].unit0;
    uint32_t cv = 0u, ci = 0u;
    for (int b = 0; b < dim; b += 32) {
      const bool in = b + lane < dim;
      const uint2 t = in ? p[b + lane] : make_uint2(0u, 0u);
      const uint32_t iv = warp_incl_sum(t.x, lane), ii = warp_incl_sum(t.y, lane);
      if (in) p[b + lane] = make_uint2(cv + iv - t.x, ci + ii - t.y);
      cv += __shfl_sync(kFull, iv, 31);
      ci += __shfl_sync(kFull, ii, 31);
    }
    if (lane == 0) {
      tot[2 * mine] = cv;
      tot[2 * mine + 1] = ci;
    }
  }
  if (gridDim.x > 1) __threadfence();  // this CTA's totals before its ticket
  __syncthreads();
  if (threadIdx.x == 0) s_last = gridDim.x == 1 || atomicAdd(ticket, 1) == (int)gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  if (gridDim.x > 1) __threadfence();  // the other CTAs' totals after their tickets
  int64_t carry_v = 0, carry_i = 0;
  for (int base = 0; base < n; base += kScanThreads) {
    const int c = base + threadIdx.x;
    const int64_t v = c < n ? (int64_t)__ldcg(tot + 2 * c) : 0, i = c < n ? (int64_t)__ldcg(tot + 2 * c + 1) : 0;
    const int64_t iv = warp_incl_sum(v, lane), ii = warp_incl_sum(i, lane);
    if (lane == 31) {
      s_v[warp] = iv;
      s_i[warp] = ii;
    }
    __syncthreads();
    if (warp == 0) {
      s_v[lane] = warp_incl_sum(s_v[lane], lane);
      s_i[lane] = warp_incl_sum(s_i[lane], lane);
    }
    __syncthreads();
    if (c < n) {
      const int64_t vo = carry_v + (warp ? s_v[warp - 1] : 0) + iv - v, io = carry_i + (warp ? s_i[warp - 1] : 0) + ii - i;
      chunks[c].vout = vo;
      chunks[c].iout = io;
      if (info) {
        info[6 * c + 0] = vo;
        info[6 * c + 1] = v;
        info[6 * c + 2] = io;
        info[6 * c + 3] = i;
        info[6 * c + 4] = contains_mesh(flags[c]) ? 1 : 0;
        info[6 * c + 5] = (vo + v > vcap || io + i > icap) ? 3 : 0;
      }
    }
    carry_v += s_v[kScanWarps - 1];
    carry_i += s_i[kScanWarps - 1];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    totals[0] = carry_v;
    totals[1] = carry_i;
    totals[2] = contains_mesh(flags[0]) ? 1 : 0;
    if (h_totals)
      for (int k = 0; k < kTotals; ++k) h_totals[k] = totals[k];
    if (gridDim.x > 1) *ticket = 0;
  }
  if (!sweep.order) return;
  // the sweeps' work lists: a counting sort by size, largest first, without
  // the empty chunks.  A chunk goes to a whole cluster when it holds more than
  // a CTA's even share of the vertices: alone it would end after all others.
  if (threadIdx.x < 64) s_bin[threadIdx.x] = 0;
  __syncthreads();
  for (int c = threadIdx.x; c < n; c += kScanThreads) {
    const uint32_t v = __ldcg(tot + 2 * c);
    if (v) atomicAdd(&s_bin[63 - size_bin(v)], 1);
  }
  __syncthreads();
  if (warp == 0) {
    const int a = s_bin[2 * lane], b = s_bin[2 * lane + 1], incl = warp_incl_sum(a + b, lane);
    const int64_t share = carry_v / sweep.ctas;
    const int cut = sweep.cluster > 1 ? 63 - size_bin((uint32_t)max(min(share, (int64_t)0x7fffffff), (int64_t)512)) : 0;
    const int big = __reduce_add_sync(kFull, (2 * lane < cut ? a : 0) + (2 * lane + 1 < cut ? b : 0));
    s_bin[2 * lane] = incl - a - b;
    s_bin[2 * lane + 1] = incl - b;
    if (lane == 31) {
      sweep.head[0] = big;
      sweep.head[1] = incl;
    }
  }
  __syncthreads();
  for (int c = threadIdx.x; c < n; c += kScanThreads) {
    const uint32_t v = __ldcg(tot + 2 * c);
    if (v) sweep.order[atomicAdd(&s_bin[63 - size_bin(v)], 1)] = c;
  }
}

// ---------------------------------------------------------------------------
// K4: emission
// ---------------------------------------------------------------------------

// Per-warp staging of a busy word's neighbourhood (Mode R emit): the
// occupancy words of lines (x-1+i, y-1+j), i, j in 0..3, for blocks zb-1, zb,
// zb+1, and the scanned vertex bases of lines (x+i, y+j), i, j in 0..1, for
// blocks zb, zb+1.  Every valence and every neighbour vertex id of the word's
// 32 cells is then computed from shared memory.
struct NbCache {
  uint32_t w[48];  // [i][j][b], b = block - (zb - 1)
  uint32_t vb[8];  // [i][j][b], b = block - zb
};

__device__ __forceinline__ void nb_load(NbCache& c, const uint32_t* W, const uint32_t* vbase, const uint2* pb, int dim,
                                        int zc, int x, int y, int zb, int lane) {
  __syncwarp();  // every lane is done with the previous word's cache
  for (int k = lane; k < 48; k += 32) {
    const int i = k / 12, j = (k / 3) & 3, b = k % 3;
    c.w[k] = word_at(W, dim, zc, x - 1 + i, y - 1 + j, zb - 1 + b);
  }
  if (lane < 8) {
    const int xx = x + (lane >> 2), yy = y + ((lane >> 1) & 1), bb = zb + (lane & 1);
    c.vb[lane] = (xx < dim && yy < dim && bb < zc) ? __ldg(vbase + ((int64_t)xx * dim + yy) * zc + bb) + pb[xx].x : 0u;
  }
  __syncwarp();
}

// Inside bit of sample (x-1+i, y-1+j, 32*(zb-1) + zr), zr in [0, 96).
__device__ __forceinline__ int nb_bit(const NbCache& c, int i, int j, int zr) {
  return (int)((c.w[(i * 4 + j) * 3 + (zr >> 5)] >> (zr & 31)) & 1u);
}

// Reference mask of cell (x-1+ci, y-1+cj, 32*(zb-1) + zr).
__device__ __forceinline__ int nb_mask(const NbCache& c, int ci, int cj, int zr) {
  int m = 0;
#pragma unroll
  for (int k = 0; k < 8; ++k) m |= nb_bit(c, ci + ((k >> 2) & 1), cj + ((k >> 1) & 1), zr + (k & 1)) << k;
  return m;
}

// Vertex id (chunk-local) of the axis-a crossing owned by sample
// (x+i, y+j, zabs), i, j in {0, 1}, zabs in [32zb, 32zb+32].
__device__ __forceinline__ uint32_t nb_vertex_id(const NbCache& c, int dim, int x, int y, int zb, int i, int j,
                                                 int zabs, int a) {
  const int b = (zabs >> 5) - zb, l = zabs & 31;
  const uint32_t wc = c.w[((i + 1) * 4 + (j + 1)) * 3 + b + 1];
  const uint32_t X = (x + i + 1 < dim) ? wc ^ c.w[((i + 2) * 4 + (j + 1)) * 3 + b + 1] : 0u;
  const uint32_t Y = (y + j + 1 < dim) ? wc ^ c.w[((i + 1) * 4 + (j + 2)) * 3 + b + 1] : 0u;
  const uint32_t lt = lane_lt(l);
  uint32_t id = c.vb[i * 4 + j * 2 + b] + __popc(X & lt) + __popc(Y & lt);
  if (l > 0) {  // then b == 0 and the next block is cached
    uint32_t Z = wc ^ ((wc >> 1) | (c.w[((i + 1) * 4 + (j + 1)) * 3 + 2] << 31));
    const int valid = dim - 1 - 32 * zb;
    if (valid < 32) Z &= valid <= 0 ? 0u : ((1u << valid) - 1u);
    id += __popc(Z & lt);
  }
  if (a >= 1) id += (X >> l) & 1u;
  if (a >= 2) id += (Y >> l) & 1u;
  return id;
}

// Mode Q vertex base of cell (x, y, z).
__device__ __forceinline__ uint32_t q_vertex_base(const uint32_t* vbase, const uint4* rec, const uint2* pb, int dim,
                                                  int zc, int x, int y, int z) {
  const int64_t wi = ((int64_t)x * dim + y) * zc + (z >> 5);
  const uint32_t lt = lane_lt(z & 31);
  const uint4 r = __ldg(rec + wi);
  return __ldg(&pb[x].x) + __ldg(vbase + wi) + __popc(r.x & lt) + 2 * __popc(r.y & lt) + 4 * __popc(r.z & lt);
}

// Without a work list (the allocation-free call, which keeps no vertex keys either): a
// CTA per x-plane, a warp per busy word.
template <int MODE, int PLACE>
__global__ void __launch_bounds__(256) k_emit(const ChunkDev* __restrict__ chunks, int n_chunks,
                                              const int* __restrict__ unit_start, const uint32_t* __restrict__ words,
                                              const float* __restrict__ dens, const uint32_t* __restrict__ flags,
                                              WordScratch ws, MeshOut out) {
  const int u = blockIdx.x;
  const int c = find_chunk_e(unit_start, n_chunks, u);
  if (!contains_mesh(__ldg(flags + c))) return;
  const ChunkDev ch = chunks[c];
  const int x = u - __ldg(unit_start + c);
  const int dim = ch.dim, zc = ch.zc, nw = dim * zc;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const uint32_t* W = words + ch.words;
  const uint32_t* vbase = ws.vcnt + ch.words;
  const uint4* rec = ws.rec + ch.words;
  const uint2* pb = ws.pb + ch.unit0;
  const uint2 pbx = pb[x];
  const float* D = dens + ch.dens;
  const uint32_t lt = lane_lt(lane);
  __shared__ int s_busy[kWordBlock];
  __shared__ int s_nbusy;
  __shared__ NbCache s_nb[kWordBlock / 32];
  for (int base = 0; base < nw; base += kWordBlock) {
    // level 1: one thread per word; quiet words emit nothing
    if (threadIdx.x == 0) s_nbusy = 0;
    __syncthreads();
    if (base + (int)threadIdx.x < nw) {
      const int wi = base + threadIdx.x;
      const int y = wi / zc, zb = wi - y * zc;
      if (!word_is_quiet(W, dim, zc, x, y, zb)) s_busy[atomicAdd(&s_nbusy, 1)] = wi;
    }
    __syncthreads();
    // level 2: one warp per busy word, one lane per cell
    const int nbusy = s_nbusy;
    for (int li = warp; li < nbusy; li += nwarps) {
    const int wi = s_busy[li];
    const int y = wi / zc, zb = wi - y * zc;
    const int z = 32 * zb + lane;
    const int64_t wo = (int64_t)x * nw + wi;
    LineWords lw;
    lw.load(W, dim, zc, x, y, zb);
    if (MODE == 0) {
      NbCache& nb = s_nb[warp];
      nb_load(nb, W, vbase, pb, dim, zc, x, y, zb, lane);
      // ---- vertices: calculate_cell / calculate_isovertex order ----
      const uint32_t X = (x + 1 < dim) ? (lw.w00 ^ lw.w10) : 0u;
      const uint32_t Y = (y + 1 < dim) ? (lw.w00 ^ lw.w01) : 0u;
      const uint32_t Z = zcross_word(W, dim, zc, x, y, zb);
      if ((X | Y | Z) != 0u) {
        uint32_t vid = pbx.x + __ldg(vbase + wo) + __popc(X & lt) + __popc(Y & lt) + __popc(Z & lt);
        const uint32_t own = ((X >> lane) & 1u) | (((Y >> lane) & 1u) << 1) | (((Z >> lane) & 1u) << 2);
        for (int a = 0; a < 3; ++a) {
          if (!((own >> a) & 1u)) continue;
          const int x1 = x + (a == 0), y1 = y + (a == 1), z1 = z + (a == 2);
          const int64_t gv = ch.vout + vid;
          ++vid;
          if (gv >= out.vcap) continue;
          const float s0 = dens_at(D, dim, x, y, z), s1 = dens_at(D, dim, x1, y1, z1);
          const float mu = (0.0f - s0) / (s1 - s0);
          const float q0[3] = {(float)x, (float)y, (float)z};
          const float dl[3] = {(float)(x1 - x), (float)(y1 - y), (float)(z1 - z)};
          float* P = out.pos + 3 * gv;
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            const float dv = dl[k] * mu;
            P[k] = dv + q0[k];
          }
          if (out.boundary)
            out.boundary[gv] = (x == 0 || y == 0 || z == 0 || x == dim - 1 || y == dim - 1 || z == dim - 1 ||
                                x1 == dim - 1 || y1 == dim - 1 || z1 == dim - 1);
          if (out.nrm) { out.nrm[3 * gv] = 0.0f; out.nrm[3 * gv + 1] = 0.0f; out.nrm[3 * gv + 2] = 0.0f; }
          if (out.valence) {
            // init_valence: uses of this edge by the (up to) four interior
            // cells around it (polygonize skips far-face cells, DMCChunk.cpp:528).
            int val = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const int d1 = k >> 1, d2 = k & 1;
              int cx = x, cy = y, cz = z, e;
              if (a == 0) { cy -= d1; cz -= d2; e = 2 * d1 + d2; }
              else if (a == 1) { cx -= d1; cz -= d2; e = 4 + 2 * d1 + d2; }
              else { cx -= d1; cy -= d2; e = 8 + 2 * d1 + d2; }
              if (cx < 0 || cy < 0 || cz < 0 || cx > dim - 2 || cy > dim - 2 || cz > dim - 2) continue;
              val += edge_uses(nb_mask(nb, cx - x + 1, cy - y + 1, cz - 32 * (zb - 1)), e);
            }
            out.valence[gv] = (uint8_t)val;
          }
        }
      }
      // ---- triangles: polygonize_cell order ----
      const bool interior = x < dim - 1 && y < dim - 1 && z < dim - 1;
      const int mask = interior ? lw.mask(lane) : 0;
      const uint64_t tw = c_tri_cases[mask];
      const int t3 = 3 * (int)(tw >> 60);
      if (__ballot_sync(kFull, t3 != 0) == 0u) continue;
      const int incl = warp_incl_scan(t3);
      int64_t gi = ch.iout + (int64_t)(pbx.y + __ldg(&rec[wo].w)) + (incl - t3);
      for (int i = 0; i < t3; ++i, ++gi) {
        const int e = tri_edge(tw, i);
        const uint32_t vid = nb_vertex_id(nb, dim, x, y, zb, c_edge_owner[e][0], c_edge_owner[e][1],
                                          z + c_edge_owner[e][2], c_edge_owner[e][3]);
        if (gi < out.icap) out.idx[gi] = vid;
      }
    } else {
      // ---- Mode Q vertices: one per vertex group of each interior surface cell ----
      const bool interior = x <= dim - 2 && y <= dim - 2 && z <= dim - 2;
      const int mask = interior ? lw.mask(lane) : 0;
      const int ng = group_count(mask);
      if (ng) {
        const uint4 r = __ldg(rec + wo);
        uint32_t vid = pbx.x + __ldg(vbase + wo) + __popc(r.x & lt) + 2 * __popc(r.y & lt) + 4 * __popc(r.z & lt);
        const int nc = dim - 1;
        const uint8_t bnd = (x == 0 || y == 0 || z == 0 || x == nc - 1 || y == nc - 1 || z == nc - 1);
        for (int g = 0; g < ng; ++g, ++vid) {
          const int64_t gv = ch.vout + vid;
          if (gv >= out.vcap) continue;
          float P[3];
          q_place<PLACE, false>(D, dim, x, y, z, group_edges(mask, g), P);
          out.pos[3 * gv] = P[0];
          out.pos[3 * gv + 1] = P[1];
          out.pos[3 * gv + 2] = P[2];
          if (out.nrm) { out.nrm[3 * gv] = 0.0f; out.nrm[3 * gv + 1] = 0.0f; out.nrm[3 * gv + 2] = 0.0f; }
          if (out.boundary) out.boundary[gv] = bnd;
          if (out.valence) {
            int val = 0;
            for (int e = 0; e < 12; ++e) {
              if (group_of(mask, e) != g) continue;
              const int c0 = edge_c0(e);
              val += q_edge_interior(dim, x + ((c0 >> 2) & 1), y + ((c0 >> 1) & 1), z + (c0 & 1), e >> 2);
            }
            out.valence[gv] = (uint8_t)val;
          }
        }
      }
      // ---- quads: one per interior sign-changing grid edge ----
      uint32_t Xi, Yi, Zi;
      q_quad_words(W, dim, zc, x, y, zb, Xi, Yi, Zi);
      const int own = (int)(((Xi >> lane) & 1u) | (((Yi >> lane) & 1u) << 1) | (((Zi >> lane) & 1u) << 2));
      const int nq = __popc(own);
      if (__ballot_sync(kFull, nq != 0) == 0u) continue;
      const int incl = warp_incl_scan(4 * nq);
      int64_t gi = ch.iout + (int64_t)(pbx.y + __ldg(&rec[wo].w)) + (incl - 4 * nq);
      const bool in0 = ((lw.w00 >> lane) & 1u) != 0u;
      for (int a = 0; a < 3; ++a) {
        if (!((own >> a) & 1)) continue;
        const int b = (a + 1) % 3, cax = (a + 2) % 3;
        uint32_t q[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int ob = (k == 0 || k == 3) ? -1 : 0, oc = (k < 2) ? -1 : 0;
          int cc[3] = {x, y, z};
          cc[b] += ob;
          cc[cax] += oc;
          int lo[3] = {0, 0, 0};
          lo[b] = -ob;
          lo[cax] = -oc;
          const int e = a == 0 ? 2 * lo[1] + lo[2] : (a == 1 ? 4 + 2 * lo[0] + lo[2] : 8 + 2 * lo[0] + lo[1]);
          const int cm = cell_mask_at(W, dim, zc, cc[0], cc[1], cc[2]);
          q[k] = q_vertex_base(vbase, rec, pb, dim, zc, cc[0], cc[1], cc[2]) +
                 (uint32_t)group_of(cm, e);
        }
        if (!in0) {
          const uint32_t t = q[1];
          q[1] = q[3];
          q[3] = t;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k, ++gi)
          if (gi < out.icap) out.idx[gi] = q[k];
      }
    }
    }
    __syncthreads();
  }
}

int launch_place_bwd(int placement, int wide, const ChunkDev* d_chunks, int n_chunks, const uint32_t* words,
                     const float* dens, const uint32_t* vkey, const int64_t* d_counts, int64_t vcap,
                     const float* grad_pos, float* grad_dens, const uint32_t* qlist, const uint32_t* qcount,
                     const float* qseed, const uint8_t* qflag, cudaStream_t st) {
  const int blocks = (int)((vcap + 127) / 128);
  if (blocks == 0) return 0;
#define BMF_PLACE_BWD(P, A)                                                                                        \
  k_place_bwd<P, A><<<blocks, 128, 0, st>>>(d_chunks, n_chunks, words, dens, vkey, d_counts, vcap, grad_pos,        \
                                            grad_dens, qflag)
  if (placement == 2 && wide) {
    // the forward recorded the branch and built the list: float pass over the
    // mass-point vertices, then the wide QEF adjoint over the list
    BMF_PLACE_BWD(2, false);
    launch_qef_bwd(wide, d_chunks, n_chunks, words, dens, vkey, vcap, grad_pos, grad_dens, qlist, qcount, qseed, st);
    return 2;
  }
  if (placement == 2) BMF_PLACE_BWD(2, true); else BMF_PLACE_BWD(1, true);
#undef BMF_PLACE_BWD
  return 1;
}

// ---------------------------------------------------------------------------
// K5: vertex -> primitive adjacency (the CSR of MeshProcessor::init /
// init_primitives, MeshProcessor.cpp:26-128), built per vertex from the grid
// structure instead of by scattering primitives: a Mode R vertex on the axis-a
// edge of sample s is used by the (up to) four interior cells around that
// edge, whose primitive ids are ascending in linear cell order and, inside a
// cell, in triangle-list order -- exactly the ascending-prim order
// init_primitives produces.  A Mode Q vertex is used by one quad per interior
// crossing edge of its group, walked in ascending quad order.  No atomics, no
// sort, deterministic.
// ---------------------------------------------------------------------------

// The adjacency list of one vertex (key: its packed grid position; bits: its
// MeshOut::vadj) of chunk ch, at most room entries, into out.  An entry is its
// word's first primitive plus its rank in the word: one 16-byte record of the emit
// per cell (Mode R) or quad (Mode Q).
// OUT = uint16_t with rel = the chunk's first primitive: the list holds
// chunk-relative ids (the chunk-by-chunk sweeps, for chunks of at most 65535
// primitives: half the bytes in the gathers' working set).
// Rebuilding the crossings around the vertex from the occupancy words instead was
// 80% of the instructions of a Mode Q mesh's sweeps, at 18 lanes each: k_sweep_chunks
// on 512 x 65^3, eight sweeps, 1090 us against 689, a 512-chunk QEF update, four, 750
// against 402; in Mode R (23 words against 4 records) a 4096-chunk update, four sweeps,
// 4250 against 4090.
template <int MODE, typename OUT = uint32_t>
__device__ __forceinline__ void adj_vertex(const ChunkDev& ch, const WordScratch& ws, uint32_t key, uint32_t bits,
                                           OUT* __restrict__ out, int room, int64_t rel = 0) {
  const int dim = ch.dim, zc = ch.zc;
  int x, y, z, k;
  vertex_key_decode(key, x, y, z, k);
  // the chunk's first primitive (its index offset and word bases are
  // multiples of the primitive size)
  const int64_t pbase = ch.iout / (MODE == 0 ? 3 : 4) - rel;
  int n = 0;
  if (MODE == 0) {
    const uint4* P = ws.rec + ch.words;
#pragma unroll
    for (int q = 0; q < 4; ++q) {  // cells around the edge, ascending linear order
      uint32_t tm = (bits >> (5 * q)) & 31u;  // the cell's triangles that use the edge, ascending
      const int d1 = (q >> 1) ^ 1, d2 = (q & 1) ^ 1;
      const int cx = x - (k == 0 ? 0 : d1), cy = y - (k == 0 ? d1 : (k == 1 ? 0 : d2)), cz = z - (k == 2 ? 0 : d2);
      if (tm == 0u || (cx | cy | cz) < 0) continue;
      const uint4 r = __ldg(P + ((cx * dim + cy) * zc + (cz >> 5)));
      const uint32_t lt = lane_lt(cz & 31);
      const int64_t first = pbase + r.w + __popc(r.x & lt) + 2 * __popc(r.y & lt) + 4 * __popc(r.z & lt);
      for (; tm && n < room; tm &= tm - 1u) out[n++] = (OUT)(first + __ffs(tm) - 1);
    }
  } else {
    constexpr uint64_t kCorner = 0x654432211000ull;  // owner sample 4 dx + 2 dy + dz per edge in quad order
    constexpr uint32_t kAxis = 0x992124u;            // and axis
    const uint4* Q = ws.quads + ch.words;
#pragma unroll 1
    for (uint32_t set = bits & 0xFFFu; set; set &= set - 1u) {
      const int i = __ffs(set) - 1, c0 = (int)(kCorner >> (4 * i)) & 7, a = (int)(kAxis >> (2 * i)) & 3;
      const int sz = z + (c0 & 1);
      const uint4 q = __ldg(Q + (((x + (c0 >> 2)) * dim + (y + ((c0 >> 1) & 1))) * zc + (sz >> 5)));
      const int l = sz & 31;
      const uint32_t bit = 1u << l, lt = bit - 1u, lx = a >= 1 ? lt | bit : lt, ly = a >= 2 ? lt | bit : lt;
      const uint32_t pre = __popc(q.x & lx) + __popc(q.y & ly) + __popc(q.z & lt);
      if (n < room) out[n++] = (OUT)(pbase + q.w + pre);
    }
  }
}

template <int MODE>
__global__ void __launch_bounds__(256) k_adj_build(const ChunkDev* __restrict__ chunks, int n_chunks, WordScratch ws,
                                                   const uint32_t* __restrict__ vkey,
                                                   const uint32_t* __restrict__ vadj, const uint32_t* __restrict__ off,
                                                   const int64_t* __restrict__ d_counts, int64_t vcap,
                                                   int64_t adj_cap, uint32_t* __restrict__ adj) {
  const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= (d_counts ? min(vcap, d_counts[0]) : vcap)) return;
  const int c = find_chunk_by_vertex(chunks, n_chunks, v);
  // the vertex's CSR range (the exclusive scan of init_valence), and of that what
  // the slots hold (an index arena that is too small has fewer): never write past it
  const int64_t o = off[v], room = min((int64_t)off[v + 1], adj_cap) - o;
  if (room > 0) adj_vertex<MODE>(chunks[c], ws, vkey[v], vadj[v], adj + o, (int)room);
}

void launch_adj_build(int mode, const ChunkDev* d_chunks, int n_chunks, WordScratch ws, const uint32_t* vkey,
                      const uint32_t* vadj, const uint32_t* off, const int64_t* d_counts,
                      int64_t vcap, int64_t adj_cap, uint32_t* adj, cudaStream_t st) {
  const int blocks = (int)((vcap + 255) / 256);
  if (blocks == 0) return;
  const auto kernel = mode == 0 ? k_adj_build<0> : k_adj_build<1>;
  kernel<<<blocks, 256, 0, st>>>(d_chunks, n_chunks, ws, vkey, vadj, off, d_counts, vcap, adj_cap, adj);
}

// ---------------------------------------------------------------------------
// K5+K6 chunk by chunk: a cluster of CTAs (a chunk that is large beside the
// work of one CTA) or one CTA (the others) runs a chunk's CSR offsets, its
// adjacency and every dual / primal sweep with barriers in between.  A chunk's
// vertices only touch its own primitives, and the sum of its vertices'
// valences is its index count, so the chunk's offsets are its index offset plus
// the exclusive scan of its own valences -- the global scan's values.  Per
// primitive and vertex the operations are those of k_adj_build, k_dual and
// k_primal, so the results are identical.  In a cluster each CTA keeps a fixed
// range of the chunk's vertices (its offsets and lists are then its own) and
// of its primitives; dual and primal steps meet at cluster barriers.
//
// Bound by the latency of dependent gathers.  One launch instead of 4 + 2 iters
// dependent small ones, and the update's largest chunks no longer run on one
// CTA each at the end of a small or middle-sized update.
// ---------------------------------------------------------------------------
struct SweepArgs {
  const ChunkDev* __restrict__ chunks;
  const uint32_t* __restrict__ tot;
  SweepLists lists;
  WordScratch ws;
  const uint32_t* __restrict__ vkey;
  const uint32_t* __restrict__ vadj;
  int64_t nv, n_prims, adj_cap;
  const int64_t* __restrict__ d_counts;
  uint32_t* __restrict__ off;
  const uint8_t* __restrict__ valence;
  uint32_t* __restrict__ adj;
  const uint8_t* __restrict__ boundary;
  const uint32_t* __restrict__ idx;  // mesh-wide
  SweepBufs b;
  float *__restrict__ dual_p, *__restrict__ dual_n;
  int iters, process_boundary, sn, wide_adj;
};

// One chunk (or a cluster CTA's part of it) in mesh-wide 32-bit ids: every
// address is a kernel parameter plus a 32-bit index, so the loops below keep
// few registers (the kernel has 32).
struct ChunkPart {
  uint32_t v0, p0, io;  // the chunk's first vertex, primitive and index
  uint32_t nv, np;      // its vertices and primitives, of those the arena holds
  uint32_t nvb;         // the mesh's vertices, of those the arena holds
  uint32_t va, ve, pa, pe;  // this CTA's (from v0 / p0)
};

// Length of vertex v's list from offset o on: adj_next (MeshProcessor.cpp:247),
// with a prebuilt adjacency init_valence; 0 for a vertex that is not moved.
__device__ __forceinline__ uint32_t sweep_list_len(const SweepArgs& A, uint32_t v, uint32_t o) {
  const uint32_t n = __ldg(A.valence + v), fz = __ldg(A.boundary + v);
  const uint32_t m = (int64_t)o + n <= A.adj_cap ? n : (uint32_t)max((int64_t)0, A.adj_cap - (int64_t)o);
  return !A.process_boundary && fz ? 0u : m;
}

// AT = uint16_t: lists of 16-bit ids relative to the chunk's first primitive,
// in the first half of the chunk's own span of adj.
template <typename AT>
__device__ __forceinline__ const AT* sweep_list(const SweepArgs& A, const ChunkPart& c, uint32_t o) {
  if (sizeof(AT) == 2) return reinterpret_cast<const AT*>(A.adj) + ((int64_t)o + c.io);
  return reinterpret_cast<const AT*>(A.adj) + o;
}

template <int N>
__device__ __forceinline__ void sweep_dual(const SweepArgs& A, const ChunkPart& c, const float* __restrict__ src,
                                           int normals) {
  for (uint32_t t = c.pa + threadIdx.x; t < c.pe; t += kSweepThreads) {
    uint32_t v[N];
    prim_corners<N, uint32_t>(c.p0 + t, c.nvb, A.idx, v);
    dual_corners<N, true, uint32_t>(c.p0 + t, v, src, A.b.nrm, A.dual_p, A.dual_n, normals);
  }
}

template <bool NORMALS, typename AT>
__device__ __forceinline__ bool sweep_primal(const SweepArgs& A, const ChunkPart& c, const SweepStep& st) {
  bool older = false;
  const uint32_t rel = sizeof(AT) == 2 ? c.p0 : 0u;
  const uint32_t lim = sizeof(AT) == 2 ? c.np : (uint32_t)min(A.n_prims, (int64_t)UINT32_MAX);
  const uint32_t end = c.v0 + c.ve;
  // whole warps: v - lane is the same for all lanes
  for (uint32_t v = c.v0 + c.va + threadIdx.x; v - (threadIdx.x & 31u) < end; v += kSweepThreads) {
    uint32_t o = 0u, n = 0u;
    if (v < end) {
      o = __ldca(A.off + v);
      n = sweep_list_len(A, v, o);
    }
    float p[3], nn[3];
    primal_sums<2, NORMALS, true>(sweep_list<AT>(A, c, o), n, lim, rel, A.dual_p, A.dual_n, p, nn);
    if (n != 0u)
      older |= primal_store<NORMALS>(v, n, p, nn, st.dst, A.b.nrm, st.set_colors, st.skipped);
    else if (v < end)
      primal_frozen<true>(v, st, A.b.nrm);
  }
  return older;
}

template <int N, typename AT>
__device__ __forceinline__ void sweep_older(const SweepArgs& A, ChunkPart c, int skipped) {
  const uint32_t rel = sizeof(AT) == 2 ? c.p0 : 0u;
  const uint32_t lim = sizeof(AT) == 2 ? c.np : (uint32_t)min(A.n_prims, (int64_t)UINT32_MAX);
  for (uint32_t v = c.v0 + c.va + threadIdx.x; v < c.v0 + c.ve; v += kSweepThreads) {
    const uint32_t o = A.off[v], n = sweep_list_len(A, v, o);
    const float* q = A.b.nrm + 3 * (int64_t)v;
    if (n == 0 || q[0] != 0.0f || q[1] != 0.0f || q[2] != 0.0f) continue;
    primal_older_normal<N, true>(v, sweep_list<AT>(A, c, o), n, lim, rel, A.idx, c.nvb, skipped, A.b.x[0],
                                 A.b.x[1], A.iters, A.b.nrm);
  }
}

template <int MODE, int N>
__global__ void __launch_bounds__(kSweepThreads, kSweepCtas) k_sweep_chunks(
    const ChunkDev* __restrict__ chunks, const uint32_t* __restrict__ tot, SweepLists lists,
    WordScratch ws, const uint32_t* __restrict__ vkey, const uint32_t* __restrict__ vadj, int64_t nv, int64_t n_prims,
    int64_t adj_cap, const int64_t* __restrict__ d_counts, uint32_t* __restrict__ off,
    const uint8_t* __restrict__ valence, uint32_t* __restrict__ adj, const uint8_t* __restrict__ boundary,
    const uint32_t* __restrict__ idx, SweepBufs b_, float* __restrict__ dual_p, float* __restrict__ dual_n, int iters,
    int process_boundary, int sn, int wide_adj) {
  const SweepArgs A{chunks, tot, lists, ws, vkey, vadj, nv, n_prims, adj_cap, d_counts, off, valence, adj, boundary,
                    idx, b_, dual_p, dual_n, iters, process_boundary, sn, wide_adj};
  constexpr int kThreads = kSweepThreads, kWarps = kThreads / 32;
  __shared__ uint32_t s_warp[32];
  __shared__ uint32_t s_total;
  __shared__ uint32_t s_item;
  __shared__ uint32_t s_seg[8];  // valence sum of each CTA's vertices
  cluster_barrier();  // every CTA of the cluster has started before its shared memory is written
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n_big = A.lists.head[0], n_list = A.lists.head[1];
  bool wide = true;  // the cluster's items first, then single CTAs
  for (;;) {
    int it;
    if (wide) {
      if (cluster_rank() == 0 && threadIdx.x == 0) {
        const uint32_t k = (uint32_t)atomicAdd(A.lists.head + 2, 1);
        for (uint32_t r = 0; r < cluster_size(); ++r) cluster_store(&s_item, r, k);
      }
      // everyone has read s_item before the next item's store: the item's own
      // cluster barriers are in between
      cluster_barrier();
      it = (int)s_item;
      if (it >= n_big) {
        wide = false;
        __syncthreads();  // s_item is read
        continue;
      }
    } else {
      if (threadIdx.x == 0) s_item = (uint32_t)atomicAdd(A.lists.head + 3, 1);
      __syncthreads();
      it = n_big + (int)s_item;
      __syncthreads();  // everyone has read s_item before thread 0 takes the next
      if (it >= n_list) break;
    }
    const int ci = A.lists.order[it];
    const ChunkDev& ch = A.chunks[ci];
    ChunkPart c;
    {
      const int64_t nvb = A.d_counts ? min(A.nv, A.d_counts[0]) : A.nv;
      const int64_t npb = A.d_counts ? min(A.n_prims, A.d_counts[1] / N) : A.n_prims;
      const int64_t v0 = ch.vout, p0 = ch.iout / N;
      c.nvb = (uint32_t)nvb;
      c.v0 = (uint32_t)v0;
      c.p0 = (uint32_t)p0;
      c.io = (uint32_t)ch.iout;
      c.nv = (uint32_t)max((int64_t)0, min((int64_t)A.tot[2 * ci], nvb - v0));
      c.np = (uint32_t)max((int64_t)0, min((ch.iout + (int64_t)A.tot[2 * ci + 1]) / N, npb) - p0);
    }
    // this CTA's vertices and primitives of the chunk (all of them for one CTA)
    c.va = c.pa = 0u;
    c.ve = c.nv;
    c.pe = c.np;
    // CSR offsets (MeshProcessor.cpp:32-40), blockDim vertices per pass;
    // vertex v is always handled by the same thread below
    uint32_t carry = c.io;
    if (wide) {
      const uint32_t csize = cluster_size(), rank = cluster_rank();
      const uint32_t vs = (c.nv + csize - 1u) / csize, ps = (c.np + csize - 1u) / csize;
      c.va = min(rank * vs, c.nv);
      c.ve = min(c.va + vs, c.nv);
      c.pa = min(rank * ps, c.np);
      c.pe = min(c.pa + ps, c.np);
      uint32_t sum = 0u;
      for (uint32_t v = c.va + threadIdx.x; v < c.ve; v += kThreads) sum += __ldg(A.valence + c.v0 + v);
      sum = __reduce_add_sync(kFull, sum);
      if (lane == 0) s_warp[warp] = sum;
      __syncthreads();
      if (warp == 0) {
        sum = __reduce_add_sync(kFull, lane < kWarps ? s_warp[lane] : 0u);
        if (lane < (int)csize) cluster_store(&s_seg[rank], lane, sum);
      }
      cluster_barrier();
      for (uint32_t r = 0; r < rank; ++r) carry += s_seg[r];
    }
    for (uint32_t b = c.va; b < c.ve; b += kThreads) {
      const uint32_t v = b + threadIdx.x;
      const uint32_t x = v < c.ve ? (uint32_t)__ldg(A.valence + c.v0 + v) : 0u;
      uint32_t incl = x;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += y;
      }
      if (lane == 31) s_warp[warp] = incl;
      __syncthreads();
      if (warp == 0) {
        const uint32_t w = lane < kWarps ? s_warp[lane] : 0u;
        uint32_t wi = w;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const uint32_t y = __shfl_up_sync(0xffffffffu, wi, d);
          if (lane >= d) wi += y;
        }
        s_warp[lane] = wi - w;  // exclusive over warps
        if (lane == kWarps - 1) s_total = wi;
      }
      __syncthreads();
      if (v < c.ve) A.off[c.v0 + v] = carry + s_warp[warp] + incl - x;
      carry += s_total;
      __syncthreads();
    }
    // adjacency, in each vertex's own CSR range and inside adj; a chunk of at
    // most 65535 primitives keeps 16-bit ids
    const bool compact = !A.wide_adj && c.np <= 65535u;
    for (uint32_t v = c.v0 + c.va + threadIdx.x; v < c.v0 + c.ve; v += kThreads) {
      const uint32_t o = A.off[v];
      const int room = (int)max((int64_t)0, min((int64_t)__ldg(A.valence + v), A.adj_cap - (int64_t)o));
      if (compact)
        adj_vertex<MODE, uint16_t>(ch, A.ws, __ldg(A.vkey + v), __ldg(A.vadj + v),
                                   const_cast<uint16_t*>(sweep_list<uint16_t>(A, c, o)), room, (int64_t)c.p0);
      else
        adj_vertex<MODE>(ch, A.ws, __ldg(A.vkey + v), __ldg(A.vadj + v), A.adj + o, room);
    }
    for (int m = 0; m < A.iters; ++m) {
      const SweepStep st = sweep_step(m, A.iters, A.sn, A.b.keep(), A.b);
      sweep_dual<N>(A, c, st.src, st.normals);
      if (wide) cluster_barrier(); else __syncthreads();
      bool older = false;
      if (st.normals == 0) {
        if (compact) sweep_primal<false, uint16_t>(A, c, st); else sweep_primal<false, uint32_t>(A, c, st);
      } else {
        older = compact ? sweep_primal<true, uint16_t>(A, c, st) : sweep_primal<true, uint32_t>(A, c, st);
      }
      if (st.skipped && __syncthreads_or(older)) {
        if (compact) sweep_older<N, uint16_t>(A, c, st.skipped); else sweep_older<N, uint32_t>(A, c, st.skipped);
      }
      if (wide) cluster_barrier(); else __syncthreads();
    }
  }
}

// ---------------------------------------------------------------------------
// K5+K6 over the whole mesh in one cooperative launch, for meshes whose steps
// are too short to be launched one by one (a chunk, a small update): CSR
// offsets, adjacency and every dual / primal step, with a barrier over the
// team's CTAs in between.  The team is as many of the launch's CTAs as the
// mesh can use (kTeamVerts vertices each): fewer CTAs meet faster.  Every CTA
// keeps a fixed range of the vertices and of the primitives; each thread keeps
// its first vertex's list and its first two primitives' corners in registers,
// so a step is one round of independent gathers from L2 (what the other SMs
// wrote), the sums in list order, and the barrier.  Values and order of the
// sums are those of k_adj_build, k_dual and k_primal.
// ---------------------------------------------------------------------------
struct TeamArgs {
  const ChunkDev* chunks;
  int n_chunks;
  WordScratch ws;
  const uint32_t* vkey;
  const uint32_t* vadj;
  int64_t nv, n_prims;
  const int64_t* d_counts;
  uint32_t* off;
  uint32_t* cursor;  // MODE 2: entries of each vertex's list so far
  const uint8_t* valence;
  uint32_t* adj;
  const uint8_t* boundary;
  const uint32_t* idx;
  SweepBufs b;
  float *dual_p, *dual_n;
  int iters, process_boundary, sn;
  TeamSync* sync;
  unsigned* host_failed;  // pinned host memory
};

// Ascending order of a list of n entries: by rank in registers, or (long
// lists) by insertion in place.
__device__ __forceinline__ void sort_list(uint32_t* a, uint32_t n) {
  constexpr int kRegs = 10;
  if (n <= kRegs) {
    uint32_t e[kRegs];
#pragma unroll
    for (int k = 0; k < kRegs; ++k) e[k] = k < (int)n ? a[k] : 0xffffffffu;
#pragma unroll
    for (int k = 0; k < kRegs; ++k) {
      int rank = 0;
#pragma unroll
      for (int j = 0; j < kRegs; ++j) rank += j < k ? e[j] <= e[k] : (j > k ? e[j] < e[k] : 0);
      if (k < (int)n) a[rank] = e[k];
    }
    return;
  }
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

// MODE 2: any mesh, its lists filled from the indices through cursors and put in
// ascending order (set_adj, MeshRecursion.hpp:173-190).
template <int MODE, int N>
__global__ void __launch_bounds__(kTeamThreads, 1) k_sweep_team(const __grid_constant__ TeamArgs A) {
  constexpr int kWarps = kTeamThreads / 32;
  __shared__ uint32_t s_warp[kWarps], s_total;
  const uint32_t nv = (uint32_t)(A.d_counts ? min(A.nv, A.d_counts[0]) : A.nv);
  const uint32_t np = (uint32_t)(A.d_counts ? min(A.n_prims, A.d_counts[1] / N) : A.n_prims);
  const unsigned team = min(gridDim.x, max(1u, (nv + kTeamVerts - 1u) / kTeamVerts));
  const unsigned rank = blockIdx.x;
  if (rank >= team || nv == 0) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, tid = threadIdx.x;
  const int iters = A.iters;
  unsigned target = 0;
  bool dead = false;
  const uint32_t vs = (nv + team - 1u) / team, ps = (np + team - 1u) / team;
  const uint32_t va = min(rank * vs, nv), ve = min(va + vs, nv), pa = min(rank * ps, np), pe = min(pa + ps, np);
  const uint32_t cap = np * N;  // slots of adj
  // CSR offsets (MeshProcessor.cpp:32-40): the CTAs' valence sums, then a scan of the own range
  uint32_t sum = 0u;
  for (uint32_t v = va + tid; v < ve; v += kTeamThreads) {
    sum += __ldg(A.valence + v);
    if (MODE == 2) A.cursor[v] = 0u;
  }
  sum = __reduce_add_sync(kFull, sum);
  if (lane == 0) s_warp[warp] = sum;
  __syncthreads();
  if (warp == 0) {
    sum = __reduce_add_sync(kFull, lane < kWarps ? s_warp[lane] : 0u);
    if (lane == 0) A.sync->seg[rank] = sum;
  }
  team_barrier(A.sync, A.host_failed, target, team, dead);
  if (warp == 0) {
    uint32_t c = 0u;
    for (unsigned r = lane; r < rank; r += 32) c += __ldcg(A.sync->seg + r);
    c = __reduce_add_sync(kFull, c);
    if (lane == 0) s_total = c;
  }
  __syncthreads();
  uint32_t carry = s_total;
  __syncthreads();
  for (uint32_t b = va; b < ve; b += kTeamThreads) {
    const uint32_t v = b + tid, x = v < ve ? (uint32_t)__ldg(A.valence + v) : 0u;
    const uint32_t incl = warp_incl_sum(x, lane);
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    if (warp == 0) {
      const uint32_t w = lane < kWarps ? s_warp[lane] : 0u, wi = warp_incl_sum(w, lane);
      if (lane < kWarps) s_warp[lane] = wi - w;
      if (lane == kWarps - 1) s_total = wi;
    }
    __syncthreads();
    if (v < ve) {
      const uint32_t o = carry + s_warp[warp] + incl - x;
      A.off[v] = o;
      if (MODE != 2) {
        const int room = o < cap ? (int)min(x, cap - o) : 0;
        adj_vertex<MODE>(A.chunks[find_chunk_by_vertex(A.chunks, A.n_chunks, v)], A.ws, __ldg(A.vkey + v),
                         __ldg(A.vadj + v), A.adj + o, room);
      }
    }
    carry += s_total;
    __syncthreads();
  }
  if (MODE == 2) {
    team_barrier(A.sync, A.host_failed, target, team, dead);  // every offset and cursor
    for (uint32_t j = pa * N + tid; j < pe * N; j += kTeamThreads) {
      const uint32_t v = __ldg(A.idx + j);
      if (v >= nv) continue;  // an index outside the mesh is ignored
      const uint32_t k = atomicAdd(A.cursor + v, 1u), o = A.off[v] + k;
      if (k < __ldg(A.valence + v) && o < cap) A.adj[o] = j / N;  // a caller's valences may not add up
    }
    team_barrier(A.sync, A.host_failed, target, team, dead);
    for (uint32_t v = va + tid; v < ve; v += kTeamThreads) {
      const uint32_t o = A.off[v];
      if (o < cap) sort_list(A.adj + o, min(min(A.cursor[v], (uint32_t)__ldg(A.valence + v)), cap - o));
    }
  }
  // what a thread keeps over all steps: its first vertex's list and its first two primitives' corners
  const auto list_of = [&](uint32_t v, uint32_t& n, uint32_t& o) {
    o = A.off[v];
    n = o < cap ? min((uint32_t)__ldg(A.valence + v), cap - o) : 0u;
    if (MODE == 2) n = min(n, A.cursor[v]);
    if (!A.process_boundary && __ldg(A.boundary + v)) n = 0u;
  };
  const auto load_ids = [&](uint32_t o, uint32_t n, uint32_t ids[kTeamRegs]) {
#pragma unroll
    for (int k = 0; k < kTeamRegs; ++k) ids[k] = k < (int)n ? A.adj[o + k] : 0xffffffffu;
  };
  uint32_t n0 = 0u, o0 = 0u, ids0[kTeamRegs] = {}, c0[2][N];
  const uint32_t v_own = va + tid, p_own = pa + tid;
  if (v_own < ve) {
    list_of(v_own, n0, o0);
    load_ids(o0, n0, ids0);
  }
#pragma unroll
  for (int k = 0; k < 2; ++k)
    if (p_own + k * kTeamThreads < pe) prim_corners<N, uint32_t>(p_own + k * kTeamThreads, nv, A.idx, c0[k]);
  const bool keep = A.b.keep();
  for (int m = 0; m < iters; ++m) {
    const SweepStep st = sweep_step(m, iters, A.sn, keep, A.b);
#pragma unroll
    for (int k = 0; k < 2; ++k)
      if (p_own + k * kTeamThreads < pe)
        dual_corners<N, true, uint32_t>(p_own + k * kTeamThreads, c0[k], st.src, A.b.nrm, A.dual_p, A.dual_n,
                                        st.normals);
    for (uint32_t t = p_own + 2 * kTeamThreads; t < pe; t += kTeamThreads)
      dual_prim<N, true, uint32_t>(t, nv, A.idx, st.src, A.b.nrm, A.dual_p, A.dual_n, st.normals);
    team_barrier(A.sync, A.host_failed, target, team, dead);
    bool older = false;
    for (uint32_t v = v_own; v - lane < ve; v += kTeamThreads) {
      uint32_t n = n0, o = o0;
      if (v != v_own) {
        n = o = 0u;
        if (v < ve) list_of(v, n, o);
      }
      const uint32_t* first = v == v_own ? ids0 : nullptr;
      float p[3], nn[3];
      if (st.normals == 0)
        primal_sums<kTeamRegs, false, true>(A.adj + o, n, np, 0u, A.dual_p, A.dual_n, p, nn, first);
      else
        primal_sums<kTeamRegs, true, true>(A.adj + o, n, np, 0u, A.dual_p, A.dual_n, p, nn, first);
      if (n == 0u) {
        if (v < ve) primal_frozen<true>(v, st, A.b.nrm);
      } else if (st.normals == 0) {
        primal_store<false>(v, n, p, nn, st.dst, A.b.nrm, st.set_colors, 0);
      } else {
        older |= primal_store<true>(v, n, p, nn, st.dst, A.b.nrm, st.set_colors, st.skipped);
      }
    }
    if (st.skipped && __syncthreads_or(older)) {
      for (uint32_t v = v_own; v < ve; v += kTeamThreads) {
        uint32_t n, o;
        list_of(v, n, o);
        const float* nv3 = A.b.nrm + 3 * (int64_t)v;
        if (n == 0u || nv3[0] != 0.0f || nv3[1] != 0.0f || nv3[2] != 0.0f) continue;
        primal_older_normal<N, true>(v, A.adj + o, n, np, 0u, A.idx, nv, st.skipped, A.b.x[0], A.b.x[1], iters, A.b.nrm);
      }
    }
    if (m + 1 < iters) team_barrier(A.sync, A.host_failed, target, team, dead);
  }
  team_leave(A.sync, team);
}

template <int MODE, int N>
static int team_grid() {
  static std::atomic<int> grid[64] = {};
  return per_device_once(grid, [](int dev) {
    int sms = 0, coop = 0, per_sm = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_sweep_team<MODE, N>, kTeamThreads, 0);
    return coop && per_sm > 0 ? min(sms, kTeamMax) : -1;
  });
}

static int sweep_team_grid(int mode, int N) {
  if (mode == 0) return team_grid<0, 3>();
  if (mode == 1) return team_grid<1, 4>();
  return N == 3 ? team_grid<2, 3>() : team_grid<2, 4>();
}

// Any mesh (the lists filled from its indices): one launch instead of 7 + 2 iters
// small ones, up to kTeamMeshVerts vertices.  Polygonize + smoothing + layout, us,
// launches / team: 33^3 121 / 91, 100^3 137 / 104, 160^3 178 / 136, 256^3 (~195 k
// vertices) 221 / 186; Mode Q, 65^3 188 / 136, 320^3 270 / 239.
constexpr int64_t kTeamMeshVerts = 200000;
bool sweep_team_mesh(int N, int64_t nv, int64_t n_prims) {
  return nv <= kTeamMeshVerts && n_prims <= 3 * kTeamMeshVerts && sweep_team_grid(2, N) > 0;
}

void launch_sweep_team(const StructuredAdj& sa, int N, int64_t nv, int64_t n_prims, const int64_t* d_counts,
                       float* pos, float* nrm, const uint8_t* boundary, const uint8_t* valence, const uint32_t* idx,
                       int iters, int process_boundary, int smooth_normals, const ProcessScratch& s,
                       cudaStream_t st) {
  TeamArgs A{sa.chunks, sa.n_chunks, sa.ws, sa.vkey, sa.vadj, nv, n_prims, d_counts, s.off, s.cursor, valence, s.adj, boundary,
             idx, SweepBufs{{s.x[0], s.x[1]}, pos, nrm}, s.dual_p, s.dual_n, iters, process_boundary,
             smooth_normals, sa.team, sa.team_failed};
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeCooperative;
  at.val.cooperative = 1;
  cfg.gridDim = dim3(sweep_team_grid(sa.mode, N));
  cfg.blockDim = dim3(kTeamThreads);
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  if (sa.mode == 0) cudaLaunchKernelEx(&cfg, k_sweep_team<0, 3>, A);
  else if (sa.mode == 1) cudaLaunchKernelEx(&cfg, k_sweep_team<1, 4>, A);
  else if (N == 3) cudaLaunchKernelEx(&cfg, k_sweep_team<2, 3>, A);
  else cudaLaunchKernelEx(&cfg, k_sweep_team<2, 4>, A);
}

// Clusters of `size` (1, 2 or 4) CTAs that can be resident at once (negative: none).
template <int MODE, int N>
static int sweep_max_clusters(int size) {
  static std::atomic<int> slots[3][64] = {};
  int lg = 0;
  while ((1 << lg) < size) ++lg;
  return per_device_once(slots[lg], [size](int dev) {
    (void)dev;
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = size;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.gridDim = dim3(size);
    cfg.blockDim = dim3(kSweepThreads);
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, k_sweep_chunks<MODE, N>, &cfg) != cudaSuccess) n = 0;
    cudaGetLastError();
    return n > 0 ? n : -1;
  });
}

void launch_sweep_chunks(const StructuredAdj& sa, int N, int64_t nv, int64_t n_prims, const int64_t* d_counts,
                         float* pos, float* nrm, const uint8_t* boundary, const uint8_t* valence,
                         const uint32_t* idx, int iters, int process_boundary, int smooth_normals,
                         const ProcessScratch& s, cudaStream_t st) {
  SweepArgs A{sa.chunks, sa.tot, sa.lists, sa.ws, sa.vkey, sa.vadj, nv, n_prims, n_prims * N, d_counts, s.off,
              valence, s.adj, boundary, idx, SweepBufs{{s.x[0], s.x[1]}, pos, nrm}, s.dual_p, s.dual_n, iters,
              process_boundary, smooth_normals, sa.wide_adj ? 1 : 0};
  cudaMemsetAsync(sa.lists.head + 2, 0, 2 * sizeof(int), st);  // the queues: each launch takes the whole lists
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = sa.lists.cluster;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.gridDim = dim3(sa.lists.ctas);
  cfg.blockDim = dim3(kSweepThreads);
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  const auto go = [&](auto kernel) {
    cudaLaunchKernelEx(&cfg, kernel, A.chunks, A.tot, A.lists, A.ws, A.vkey, A.vadj, A.nv, A.n_prims,
                       A.adj_cap,
                       A.d_counts, A.off, A.valence, A.adj, A.boundary, A.idx, A.b, A.dual_p, A.dual_n, A.iters,
                       A.process_boundary, A.sn, A.wide_adj);
  };
  if (sa.mode == 0) go(k_sweep_chunks<0, 3>);
  else go(k_sweep_chunks<1, 4>);
}

// Where the lines lie (whole passes, us; launches / team / chunks with the
// cluster size chosen here):
//   one 33^3 chunk, Mode R            110 /   74 /    -
//   one 257^3 chunk, Mode R           244 /  213 /    -       (66 k columns)
//   fit, 8 x 65^3 (adjoint in all)    290 /  214 /  279
//   fit, 32 x 65^3                    526 /  473 /  476       (135 k columns)
//   fit, 64 x 65^3                    771 /  721 /  701
//   mixed update, 48 chunks           272 /  296 /  426       (214 k columns)
//   128 chunks Mode R / Q        464 / 541   552 / 588   618 / 632
//   256                         918 / 1082 1223 / 1298  898 / 1068
//   384                        1275 / 1546 1728 / 1877 1209 / 1475
//   512                        1604 / 1954 2181 / 2368 1518 / 1837
//   1024                       3086 / 3819 4256 / 4635 2630 / 3465
//   300, 2D heightmap, two sweeps     710 /    - /  739
//   fit, 64 x 97^3, 128 x 65^3 (four sweeps), 200 x 33^3  923, 1044, 866 / - / 815, 1009, 860
// A team pays off while a step is shorter than a launch; its 16 warps per SM
// carry fewer gathers than full occupancy once steps are long.  A chunk per CTA
// or cluster needs several chunks per resident CTA to balance, or equal ones (a
// fit plan's) that fill the GPU as clusters.  Between 256 and 384 mixed chunks the two
// forms are within 5 % of each other, and which is ahead depends on the field and
// the number of sweeps as well: 320 is the middle.  Clusters of 4 against 2 and 1 (taken with the adjacency built from
// the occupancy words): 512 chunks 1643 / 1802 / 2434 us, 1024 chunks 2996 / 2954 /
// 3456, 2048 chunks 5805 / 5764 / 5781.
constexpr int64_t kTeamColumns = 140000;
constexpr int kChunkSweepMin = 320, kChunkSweepEqual = 64, kChunkSweepPairs = 1024;

SweepForm sweep_form(int mode, int n_chunks, int64_t columns, bool equal, SweepLists* s) {
  if (columns <= kTeamColumns && sweep_team_grid(mode, mode == 0 ? 3 : 4) > 0) return kSweepTeam;
  if (n_chunks >= (equal ? kChunkSweepEqual : kChunkSweepMin)) {
    for (int size = n_chunks >= kChunkSweepPairs ? 2 : 4; size >= 1; size >>= 1) {
      const int clusters = mode == 0 ? sweep_max_clusters<0, 3>(size) : sweep_max_clusters<1, 4>(size);
      if (clusters <= 0) continue;
      s->cluster = size;
      s->ctas = size * min(clusters, n_chunks);
      return kSweepChunks;
    }
  }
  return kSweepLaunches;
}

__global__ void k_setup_chunk(const ChunkDev c, ChunkDev* d_c, int* units, uint32_t* flags, uint32_t* ccount) {
  *d_c = c;
  units[0] = 0;
  units[1] = c.dim;
  *flags = 0u;
  if (ccount) *ccount = 0u;
}

void launch_setup_chunk(const ChunkDev& c, ChunkDev* d_c, int* d_units, uint32_t* d_flags, uint32_t* d_ccount,
                        cudaStream_t st) {
  k_setup_chunk<<<1, 1, 0, st>>>(c, d_c, d_units, d_flags, d_ccount);
}

void launch_count(int mode, const ChunkDev* d_chunks, int n_chunks, const int* d_unit_start, int n_units,
                  const uint32_t* words, const uint32_t* flags, WordScratch ws, cudaStream_t st,
                  uint32_t* flags_out) {
  if (n_units < kCountFewUnits || flags_out) {
    const auto kernel = mode == 0 ? k_count<0> : k_count<1>;
    kernel<<<n_units, kCountThreads, 0, st>>>(d_chunks, n_chunks, d_unit_start, words, flags, flags_out, ws);
  } else {
    const auto kernel = mode == 0 ? k_count_planes<0> : k_count_planes<1>;
    kernel<<<(n_units + kCountPlanes - 1) / kCountPlanes, 32 * kCountPlanes, 0, st>>>(d_chunks, n_chunks, d_unit_start,
                                                                                      n_units, words, flags, ws);
  }
}

void launch_chunk_scan(ChunkDev* d_chunks, int n_chunks, WordScratch ws, uint32_t* d_tot, const uint32_t* flags,
                       int64_t vcap, int64_t icap, int64_t* d_info, int64_t* d_totals, int64_t* h_totals, int* d_ticket,
                       cudaStream_t st, const SweepLists* sweep) {
  k_chunk_scan<<<(n_chunks + kScanWarps - 1) / kScanWarps, kScanThreads, 0, st>>>(
      d_chunks, n_chunks, ws.pb, d_tot, flags, vcap, icap, d_info, d_totals, h_totals, d_ticket,
      sweep ? *sweep : SweepLists{});
}

// Corner mask of the cell at offset (ox, oy, oz) in {-1, 0} from sample
// (x, y, z), from the inside bits of lines (x-1+i, y-1+j) at samples z-1..z+1
// packed 3 bits per line at bit 3 (3i + j): corner (dx, dy, dz) is bit
// 3 (3 (1 + ox + dx) + 1 + oy + dy) + 1 + oz + dz.
__device__ __forceinline__ int packed_mask(uint32_t nbits, int ox, int oy, int oz) {
  const uint32_t b = nbits >> (3 * (3 * (1 + ox) + (1 + oy)) + 1 + oz);
  return (int)((b & 3u) | (((b >> 3) & 3u) << 2) | (((b >> 9) & 3u) << 4) | (((b >> 12) & 3u) << 6));
}

// Mode R emission over the busy-word list.  Each warp takes kTileWords list
// entries at a time and stages, per word, its neighbourhood (NbCache: the
// occupancy words of lines (x-1..x+2, y-1..y+2) in blocks zb-1..zb+1 and the
// scanned vertex bases of lines (x..x+1, y..y+1) in blocks zb..zb+1), its
// index base and its triangle-count planes in shared memory.  Then the tile's
// output is written in two flattened lists, so that every lane does the same
// work: one lane per vertex (the k-th vertex of a word is found from the
// popcounts of its crossing words; calculate_isovertex position, boundary,
// key, init_valence), then one lane per triangle (the k-th triangle of a word
// from its count planes; the cell's Marching-Cubes case and its three vertex
// ids, polygonize_cell order).  Ids and slots come from the scanned counts, so
// the output is exactly the reference's.  Every mask, valence and neighbour
// vertex id is read from shared memory; only the two endpoint densities of a
// vertex come from global memory.  Warps work on their own tiles with no
// block-wide barrier, so one warp's staging loads overlap the others' work.
constexpr int kTileWords = 16;
constexpr int kEmitWarps = 8;

// One 4-byte global -> shared copy in flight (cp.async; the staged pieces are
// 4-byte words of scattered lines, below the 16-byte unit of bulk copies), and
// the wait for all of a thread's copies.  BMF_EMIT_ASYNC 0 keeps plain loads.
#ifndef BMF_EMIT_ASYNC
#define BMF_EMIT_ASYNC 1
#endif
__device__ __forceinline__ void stage_async(uint32_t* dst, const uint32_t* src) {
#if BMF_EMIT_ASYNC
  const unsigned sa = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(sa), "l"(src) : "memory");
#else
  *dst = __ldg(src);
#endif
}
__device__ __forceinline__ void stage_async(uint4* dst, const uint4* src) {
#if BMF_EMIT_ASYNC
  const unsigned sa = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(src) : "memory");
#else
  *dst = __ldg(src);
#endif
}
__device__ __forceinline__ void stage_wait() {
#if BMF_EMIT_ASYNC
  asm volatile("cp.async.wait_all;\n" ::: "memory");
#endif
}

struct RTile {
  uint4 rec[kTileWords];  // the words' records, the last with the plane's base added
  NbCache nb[kTileWords];
  uint32_t X[kTileWords], Y[kTileWords], Z[kTileWords];
  int x[kTileWords], y[kTileWords], zb[kTileWords], dim[kTileWords], zc[kTileWords];
  int64_t cw[kTileWords], dens[kTileWords], vout[kTileWords], iout[kTileWords];
  float oy[kTileWords], sc[kTileWords];  // the chunk's y origin and scale (2D column fill)
  // per word, the crossing words of the owner lines (x + i, y + j), i, j in
  // {0, 1}: X and Y in blocks zb, zb + 1 ([i][j][b]) and Z in block zb -- what
  // a triangle's three vertex ids are counted from (tile_vertex_id)
  uint32_t ox_[kTileWords][8], oy_[kTileWords][8], oz_[kTileWords][4];
  int voff[kTileWords + 1], toff[kTileWords + 1];  // exclusive vertex / triangle offsets of the tile's words
};

// A crossing end's density: read from the fill's densities, or (2D heightmap
// column fill) computed from the sample's column height with the full fill's
// operations.
__device__ __forceinline__ float end_density(const WordScratch& ws, const float* D, int64_t cw, float oy, float sc,
                                             int dim, int x, int y, int z) {
  if (ws.cols2d) {
    const float py = oy + (float)y * sc;
    const float dy = py * ws.c2d_g;
    return -dy - __ldg(ws.cols2d + cw + (int64_t)x * dim + z) * ws.c2d_height;
  }
  return dens_at(D, dim, x, y, z);
}

// The tile word holding flattened item j: the last t < nt with off[t] <= j.
__device__ __forceinline__ int tile_word(const int* off, int nt, int j) {
  int t = 0;
#pragma unroll
  for (int s = kTileWords / 2; s > 0; s >>= 1)
    if (t + s < nt && off[t + s] <= j) t += s;
  return t;
}

// Chunk-local id of the vertex on the axis-a crossing owned by sample
// (x + i, y + j, zabs), i, j in {0, 1}, zabs in blocks zb, zb + 1 of tile word
// t: nb_vertex_id's count, from the word's staged owner-line crossing words.
__device__ __forceinline__ uint32_t tile_vertex_id(const RTile& R, int t, int i, int j, int zabs, int a) {
  const int b = (zabs >> 5) - R.zb[t], l = zabs & 31;
  const int q = i * 2 + j;
  const uint32_t X = R.ox_[t][q * 2 + b], Y = R.oy_[t][q * 2 + b], lt = lane_lt(l);
  uint32_t id = R.nb[t].vb[i * 4 + j * 2 + b] + __popc(X & lt) + __popc(Y & lt);
  if (l > 0) id += __popc(R.oz_[t][q] & lt);  // then b == 0
  if (a >= 1) id += (X >> l) & 1u;
  if (a >= 2) id += (Y >> l) & 1u;
  return id;
}

__global__ void __launch_bounds__(32 * kEmitWarps, 4) k_emit_words_r(const ChunkDev* __restrict__ chunks,
                                                                 const uint32_t* __restrict__ words,
                                                                 const float* __restrict__ dens, WordScratch ws,
                                                                 MeshOut out) {
  __shared__ uint64_t s_tri[256], s_etris[256];
  __shared__ RTile s_tiles[kEmitWarps];
  const int64_t n = min((int64_t)*ws.ccount, ws.clist_cap);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  RTile& R = s_tiles[warp];
  const int64_t nwarps = (int64_t)gridDim.x * kEmitWarps;
  // A short list (a chunk) is spread over the whole grid, few words per warp:
  // a tile's time is the chain of its phases and rounds, whatever its size
  // (33^3 chunk, ~300 busy words: 16 us as 16-word tiles on 19 warps).  Whole calls
  // without sweeps, us, spread / not: 33^3 48 / 58, 65^3 50 / 62, 129^3 75 / 85, 257^3
  // 158 / 164, Mode Q 129^3 73 / 77; longer lists fill the tiles (32 chunks 188 / 189),
  // and a line at whole instead of half tiles changes nothing (within 0.5 us).
  const bool spread = n <= nwarps * (kTileWords / 2);
  const int64_t tw = spread ? (n + nwarps - 1) / nwarps : kTileWords;
  const int64_t w0 = spread ? (int64_t)warp * gridDim.x + blockIdx.x : (int64_t)blockIdx.x * kEmitWarps + warp;
  if ((spread ? (int64_t)blockIdx.x : (int64_t)blockIdx.x * kEmitWarps) * tw >= n) return;  // no warp has a tile
  for (int i = threadIdx.x; i < 256; i += blockDim.x) {
    s_tri[i] = __ldg(g_tri_cases + i);
    s_etris[i] = g_edge_tris.w[i];
  }
  __syncthreads();
  for (int64_t t0 = w0 * tw; t0 < n; t0 += nwarps * tw) {
    const int nt = (int)min(tw, n - t0);
    // 1. the tile's words
    uint2 pb0 = make_uint2(0u, 0u);  // this lane's word: its plane's bases, the next plane's vertex base
    uint32_t pv1 = 0u;
    if (lane < nt) {
      const uint2 e = ws.clist[t0 + lane];
      const ChunkDev& ch = chunks[e.x];
      const int dim = ch.dim, zc = ch.zc, wi = (int)e.y;
      const int xy = wi / zc;
      R.zb[lane] = wi - xy * zc;
      R.y[lane] = xy % dim;
      R.x[lane] = xy / dim;
      R.dim[lane] = dim;
      R.zc[lane] = zc;
      const uint2* pb = ws.pb + ch.unit0 + R.x[lane];
      pb0 = __ldg(pb);
      if (R.x[lane] + 1 < dim) pv1 = __ldg(&pb[1].x);
      R.cw[lane] = ch.words;
      R.dens[lane] = ch.dens;
      R.vout[lane] = ch.vout;
      R.iout[lane] = ch.iout;
      R.oy[lane] = ch.oy;
      R.sc[lane] = ch.scale;
    }
    __syncwarp();
    // 2. stage the neighbourhoods (zeros outside the chunk): one item per
    // (word, neighbour line) loads the line's blocks zb-1..zb+1; one item per
    // (word, owner line) its vertex bases in blocks zb, zb+1; one per word its
    // index base and count planes -- three loops, so a warp's lanes take the
    // same branch
    // (asynchronous global -> shared copies: a lane issues every copy of its
    // items and waits once, instead of a load-then-store per item)
    for (int k = lane; k < nt * 16; k += 32) {
      const int t = k >> 4, i = (k >> 2) & 3, j = k & 3;
      const int dim = R.dim[t], zc = R.zc[t], zb = R.zb[t];
      const int xx = R.x[t] - 1 + i, yy = R.y[t] - 1 + j;
      uint32_t* dst = R.nb[t].w + (i * 4 + j) * 3;
      if (xx < 0 || yy < 0 || xx >= dim || yy >= dim) {
        dst[0] = dst[1] = dst[2] = 0u;
      } else {
        const uint32_t* L = words + R.cw[t] + (xx * dim + yy) * zc + zb;
        if (zb > 0) stage_async(dst, L - 1); else dst[0] = 0u;
        stage_async(dst + 1, L);
        if (zb + 1 < zc) stage_async(dst + 2, L + 1); else dst[2] = 0u;
      }
    }
    for (int k = lane; k < nt * 4; k += 32) {
      const int t = k >> 2, l = k & 3;
      const int dim = R.dim[t], zc = R.zc[t], zb = R.zb[t];
      const int xx = R.x[t] + (l >> 1), yy = R.y[t] + (l & 1);
      uint32_t* dst = R.nb[t].vb + (l >> 1) * 4 + (l & 1) * 2;
      if (xx < dim && yy < dim) {
        const uint32_t* V = ws.vcnt + R.cw[t] + (xx * dim + yy) * zc + zb;
        stage_async(dst, V);
        if (zb + 1 < zc) stage_async(dst + 1, V + 1); else dst[1] = 0u;
      } else {
        dst[0] = dst[1] = 0u;
      }
    }
    if (lane < nt) {
      const int64_t wi = R.cw[lane] + (R.x[lane] * R.dim[lane] + R.y[lane]) * R.zc[lane] + R.zb[lane];
      stage_async(&R.rec[lane], ws.rec + wi);
    }
    stage_wait();
    __syncwarp();
    // 3. per word: owned crossings, vertex count and triangle count (count
    // planes), scanned over the tile in one word (vertices low, triangles high)
    {
      uint32_t packed = 0u;
      if (lane < nt) {
        NbCache& nb = R.nb[lane];
        // word bases: within the plane + the plane's
        const uint32_t ib = R.rec[lane].w + pb0.y;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          nb.vb[k] += pb0.x;
          nb.vb[4 + k] += pv1;
        }
        R.rec[lane].w = ib;
        if (out.vkey)  // the adjacency build reads the word's primitive base
          ws.rec[R.cw[lane] + (R.x[lane] * R.dim[lane] + R.y[lane]) * R.zc[lane] + R.zb[lane]].w = ib / 3u;
        const int dim = R.dim[lane], x = R.x[lane], y = R.y[lane], zb = R.zb[lane];
        const uint32_t wc = nb.w[(1 * 4 + 1) * 3 + 1];
        const uint32_t X = (x + 1 < dim) ? wc ^ nb.w[(2 * 4 + 1) * 3 + 1] : 0u;
        const uint32_t Y = (y + 1 < dim) ? wc ^ nb.w[(1 * 4 + 2) * 3 + 1] : 0u;
        uint32_t Z = wc ^ ((wc >> 1) | (nb.w[(1 * 4 + 1) * 3 + 2] << 31));
        const int valid = dim - 1 - 32 * zb;
        if (valid < 32) Z &= valid <= 0 ? 0u : ((1u << valid) - 1u);
        R.X[lane] = X;
        R.Y[lane] = Y;
        R.Z[lane] = Z;
        // the owner lines' crossing words, as nb_vertex_id forms them
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int i = q >> 1, j = q & 1;
#pragma unroll
          for (int b = 0; b < 2; ++b) {
            const uint32_t w0 = nb.w[((i + 1) * 4 + (j + 1)) * 3 + b + 1];
            R.ox_[lane][q * 2 + b] = (x + i + 1 < dim) ? w0 ^ nb.w[((i + 2) * 4 + (j + 1)) * 3 + b + 1] : 0u;
            R.oy_[lane][q * 2 + b] = (y + j + 1 < dim) ? w0 ^ nb.w[((i + 1) * 4 + (j + 2)) * 3 + b + 1] : 0u;
          }
          const uint32_t w0 = nb.w[((i + 1) * 4 + (j + 1)) * 3 + 1];
          uint32_t Zq = w0 ^ ((w0 >> 1) | (nb.w[((i + 1) * 4 + (j + 1)) * 3 + 2] << 31));
          if (valid < 32) Zq &= valid <= 0 ? 0u : ((1u << valid) - 1u);
          R.oz_[lane][q] = Zq;
        }
        const uint32_t nv = __popc(X) + __popc(Y) + __popc(Z);
        const uint32_t ntri = __popc(R.rec[lane].x) + 2u * __popc(R.rec[lane].y) + 4u * __popc(R.rec[lane].z);
        packed = nv | (ntri << 16);  // at most 96 and 160 per word
      }
      uint32_t incl = packed;
#pragma unroll
      for (int o = 1; o < kTileWords; o <<= 1) {
        const uint32_t v = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += v;
      }
      if (lane < kTileWords) {
        R.voff[lane + 1] = (int)(incl & 0xFFFFu);
        R.toff[lane + 1] = (int)(incl >> 16);
      }
      if (lane == 0) R.voff[0] = R.toff[0] = 0;
    }
    __syncwarp();
    // 4. one lane per vertex: the k-th vertex of word t is at the cell l whose
    // preceding cells own k or fewer crossings, the (k - that)-th of its axes
    const int nvt = R.voff[nt];
    for (int j = lane; j < nvt; j += 32) {
      const int t = tile_word(R.voff, nt, j);
      const int k = j - R.voff[t];
      const uint32_t X = R.X[t], Y = R.Y[t], Z = R.Z[t];
      int l = 0;
#pragma unroll
      for (int s = 16; s > 0; s >>= 1) {
        const uint32_t m = lane_lt(l + s);
        if ((int)(__popc(X & m) + __popc(Y & m) + __popc(Z & m)) <= k) l += s;
      }
      const uint32_t lt = lane_lt(l);
      const int r = k - (int)(__popc(X & lt) + __popc(Y & lt) + __popc(Z & lt));
      uint32_t own = ((X >> l) & 1u) | (((Y >> l) & 1u) << 1) | (((Z >> l) & 1u) << 2);
      if (r >= 1) own &= own - 1u;
      if (r >= 2) own &= own - 1u;
      const int a = __ffs(own) - 1;
      const NbCache& nb = R.nb[t];
      const int64_t gv = R.vout[t] + (int64_t)nb.vb[0] + k;
      if (gv >= out.vcap) continue;
      const int dim = R.dim[t], x = R.x[t], y = R.y[t], z = 32 * R.zb[t] + l;
      const int x1 = x + (a == 0), y1 = y + (a == 1), z1 = z + (a == 2);
      const float* D = dens + R.dens[t];
      const int64_t cw = R.cw[t];
      const float oy = R.oy[t], sc = R.sc[t];
      const float s0 = end_density(ws, D, cw, oy, sc, dim, x, y, z);
      const float s1 = end_density(ws, D, cw, oy, sc, dim, x1, y1, z1);
      const float mu = (0.0f - s0) / (s1 - s0);
      const float q0[3] = {(float)x, (float)y, (float)z};
      const float dl[3] = {(float)(x1 - x), (float)(y1 - y), (float)(z1 - z)};
      float* P = out.pos + 3 * gv;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const float dv = dl[c] * mu;
        P[c] = dv + q0[c];
      }
      if (out.boundary)
        out.boundary[gv] = (x == 0 || y == 0 || z == 0 || x == dim - 1 || y == dim - 1 || z == dim - 1 ||
                            x1 == dim - 1 || y1 == dim - 1 || z1 == dim - 1);
      if (out.nrm) { out.nrm[3 * gv] = 0.0f; out.nrm[3 * gv + 1] = 0.0f; out.nrm[3 * gv + 2] = 0.0f; }
      if (out.vkey) out.vkey[gv] = vertex_key(x, y, z, a);
      if (out.valence) {
        // inside bits of lines (x-1..x+1, y-1..y+1) at samples z-1..z+1
        uint32_t nbits = 0u;
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int jj = 0; jj < 3; ++jj) {
            const int zr0 = l + 31, b = zr0 >> 5;  // z - 1 relative to block zb - 1
            const uint32_t* w = nb.w + (i * 4 + jj) * 3;
            const uint64_t q = ((uint64_t)w[b + 1] << 32) | w[b];
            nbits |= ((uint32_t)(q >> (zr0 & 31)) & 7u) << (3 * (3 * i + jj));
          }
        // init_valence: the triangles that use this edge in the (up to) four interior
        // cells around it (polygonize skips far-face cells, DMCChunk.cpp:528)
        uint32_t bits = 0u;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const int d1 = c >> 1, d2 = c & 1;
          const int ox = a == 0 ? 0 : -d1, oy = a == 0 ? -d1 : (a == 1 ? 0 : -d2), oz = a == 2 ? 0 : -d2;
          const int e = 4 * a + 2 * d1 + d2;
          const int cx = x + ox, cy = y + oy, cz = z + oz;
          if (cx < 0 || cy < 0 || cz < 0 || cx > dim - 2 || cy > dim - 2 || cz > dim - 2) continue;
          bits |= ((uint32_t)(s_etris[packed_mask(nbits, ox, oy, oz)] >> (5 * e)) & 31u) << (5 * (3 - c));
        }
        out.valence[gv] = (uint8_t)__popc(bits);
        if (out.vadj) out.vadj[gv] = bits;
      }
    }
    // 5. one lane per triangle: the k-th triangle of word t is in the cell l
    // whose preceding cells hold k or fewer (count planes), its (k - that)-th
    const int ntt = R.toff[nt];
    for (int j = lane; j < ntt; j += 32) {
      const int t = tile_word(R.toff, nt, j);
      const int k = j - R.toff[t];
      const uint32_t c0 = R.rec[t].x, c1 = R.rec[t].y, c2 = R.rec[t].z;
      int l = 0;
#pragma unroll
      for (int s = 16; s > 0; s >>= 1) {
        const uint32_t m = lane_lt(l + s);
        if ((int)(__popc(c0 & m) + 2 * __popc(c1 & m) + 4 * __popc(c2 & m)) <= k) l += s;
      }
      const uint32_t lt = lane_lt(l);
      const int r = k - (int)(__popc(c0 & lt) + 2 * __popc(c1 & lt) + 4 * __popc(c2 & lt));
      const NbCache& nb = R.nb[t];
      // the cell's case: corner (dx, dy, dz) is bit 4 dx + 2 dy + dz
      int mask = 0;
#pragma unroll
      for (int d = 0; d < 4; ++d) {
        const uint32_t* w = nb.w + ((1 + (d >> 1)) * 4 + 1 + (d & 1)) * 3;
        const uint64_t q = ((uint64_t)w[2] << 32) | w[1];
        mask |= (int)((q >> l) & 3u) << (2 * d);
      }
      const uint64_t tw = s_tri[mask];
      if (3 * r + 3 > 3 * (int)(tw >> 60)) continue;  // the planes and the case table agree
      const int z = 32 * R.zb[t] + l;
      const int64_t gi = R.iout[t] + (int64_t)R.rec[t].w + 3 * (int64_t)k;
      const int64_t vout = R.vout[t];
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const int e = tri_edge(tw, 3 * r + i);
        // EDGE_V owner of edge e: axis e >> 2, offsets from its two low bits
        const int ea = e >> 2, d1 = (e >> 1) & 1, d2 = e & 1;
        const int ox = ea == 0 ? 0 : d1, oy = ea == 0 ? d1 : (ea == 1 ? 0 : d2), oz = ea == 2 ? 0 : d2;
        const uint32_t vid = tile_vertex_id(R, t, ox, oy, z + oz, ea);
        if (gi + i < out.icap) {
          out.idx[gi + i] = vid;
          if (out.idx_global) out.idx_global[gi + i] = (uint32_t)(vout + vid);
        }
      }
    }
    __syncwarp();  // the next tile overwrites the stage
  }
}

// Mode Q emission over the busy-word list, in the form of k_emit_words_r: a
// warp stages the neighbourhoods of its words (the occupancy words of lines
// (x-1..x+1, y-1..y+1) in blocks zb-1..zb+1, and the vertex base and group-count
// planes of the cell lines (x-1..x, y-1..y) in blocks zb-1, zb), then writes one
// lane per vertex (the k-th vertex group of a word, from its group-count
// planes) and one lane per quad (the k-th interior crossing edge; its four
// cells' masks, groups and vertex ids from the staged lines).  Bound by
// shared-memory wavefronts (0.73 of peak) and issue (0.67): 512 x 65^3 fitting grids
// (3.9 M vertices) 231 us, 512 mixed terrain chunks 132 us; the thread-per-cell form it
// replaces read each quad's four cells from global memory behind bounds checks (512 x
// 65^3 fitting grids: 607 us).
struct QTile {
  uint4 rec[kTileWords][8];        // [2i+j][b]: record of cell line (x-1+i, y-1+j), block zb-1+b
  uint32_t w[kTileWords][27];      // [i][j][b]: line (x-1+i, y-1+j), block zb-1+b
  uint32_t vb[kTileWords][8];      // and its vertex base
  uint32_t ib[kTileWords], X[kTileWords], Y[kTileWords], Z[kTileWords];
  int x[kTileWords], y[kTileWords], zb[kTileWords], dim[kTileWords], zc[kTileWords];
  int64_t cw[kTileWords], dens[kTileWords], vout[kTileWords], iout[kTileWords];
  int voff[kTileWords + 1], qoff[kTileWords + 1];  // exclusive vertex / quad offsets of the tile's words
};

// Corner mask of the cell of line (x-1+i, y-1+j), i, j in {0, 1}, at bit zr in
// [0, 64) of blocks zb-1, zb.
__device__ __forceinline__ int qtile_mask(const uint32_t* w, int i, int j, int zr) {
  int m = 0;
  const int b = zr >> 5, l = zr & 31;
#pragma unroll
  for (int d = 0; d < 4; ++d) {
    const uint32_t* q = w + ((i + (d >> 1)) * 3 + j + (d & 1)) * 3 + b;
    m |= (int)(__funnelshift_r(q[0], q[1], l) & 3u) << (2 * d);
  }
  return m;
}

template <int PLACE>
__global__ void __launch_bounds__(32 * kEmitWarps, 4) k_emit_words_q(const ChunkDev* __restrict__ chunks,
                                                                 const uint32_t* __restrict__ words,
                                                                 const float* __restrict__ dens, WordScratch ws,
                                                                 MeshOut out) {
  __shared__ uint64_t s_grp[256];
  __shared__ QTile s_tiles[kEmitWarps];
  const int64_t n = min((int64_t)*ws.ccount, ws.clist_cap);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  QTile& R = s_tiles[warp];
  const int64_t nwarps = (int64_t)gridDim.x * kEmitWarps;
  const bool spread = n <= nwarps * (kTileWords / 2);  // (as k_emit_words_r)
  const int64_t tw = spread ? (n + nwarps - 1) / nwarps : kTileWords;
  const int64_t w0 = spread ? (int64_t)warp * gridDim.x + blockIdx.x : (int64_t)blockIdx.x * kEmitWarps + warp;
  if ((spread ? (int64_t)blockIdx.x : (int64_t)blockIdx.x * kEmitWarps) * tw >= n) return;  // no warp has a tile
  for (int i = threadIdx.x; i < 256; i += blockDim.x) s_grp[i] = __ldg(g_group_cases + i);
  __syncthreads();
  const bool idx16 = (((uintptr_t)out.idx | (uintptr_t)out.idx_global) & 15) == 0;  // quads as 16-byte stores
  for (int64_t t0 = w0 * tw; t0 < n; t0 += nwarps * tw) {
    const int nt = (int)min(tw, n - t0);
    // 1. the tile's words
    uint2 pb1 = make_uint2(0u, 0u);  // this lane's word: its plane's bases, and the previous plane's vertex base
    uint32_t pv0 = 0u;
    if (lane < nt) {
      const uint2 e = ws.clist[t0 + lane];
      const ChunkDev& ch = chunks[e.x];
      const int dim = ch.dim, zc = ch.zc, wi = (int)e.y;
      const int xy = wi / zc;
      R.zb[lane] = wi - xy * zc;
      R.y[lane] = xy % dim;
      R.x[lane] = xy / dim;
      R.dim[lane] = dim;
      R.zc[lane] = zc;
      const uint2* pb = ws.pb + ch.unit0 + R.x[lane];
      pb1 = __ldg(pb);
      if (R.x[lane] > 0) pv0 = __ldg(&pb[-1].x);
      R.cw[lane] = ch.words;
      R.dens[lane] = ch.dens;
      R.vout[lane] = ch.vout;
      R.iout[lane] = ch.iout;
    }
    __syncwarp();
    // 2. stage the neighbourhoods (zeros outside the chunk)
    for (int k = lane; k < nt * 9; k += 32) {
      const int t = k / 9, l = k - 9 * t, i = l / 3, j = l - 3 * i;
      const int dim = R.dim[t], zc = R.zc[t], zb = R.zb[t];
      const int xx = R.x[t] - 1 + i, yy = R.y[t] - 1 + j;
      uint32_t* dst = R.w[t] + l * 3;
      if (xx < 0 || yy < 0 || xx >= dim || yy >= dim) {
        dst[0] = dst[1] = dst[2] = 0u;
      } else {
        const uint32_t* L = words + R.cw[t] + (xx * dim + yy) * zc + zb;
        if (zb > 0) stage_async(dst, L - 1); else dst[0] = 0u;
        stage_async(dst + 1, L);
        if (zb + 1 < zc) stage_async(dst + 2, L + 1); else dst[2] = 0u;
      }
    }
    for (int k = lane; k < nt * 8; k += 32) {
      const int t = k >> 3, l = k & 7, b = l & 1;
      const int dim = R.dim[t], zc = R.zc[t], zb = R.zb[t] - 1 + b;
      const int xx = R.x[t] - 1 + (l >> 2), yy = R.y[t] - 1 + ((l >> 1) & 1);
      if (xx < 0 || yy < 0 || zb < 0) continue;  // no cell there: never read
      const int64_t wi = R.cw[t] + (xx * dim + yy) * zc + zb;
      stage_async(&R.vb[t][l], ws.vcnt + wi);
      stage_async(&R.rec[t][l], ws.rec + wi);
    }
    stage_wait();
    __syncwarp();
    // 3. per word: its interior crossings (quads), vertex and quad counts,
    // scanned over the tile in one word (vertices low, quads high)
    {
      uint32_t packed = 0u;
      if (lane < nt) {
        const uint32_t* w = R.w[lane];
        const int dim = R.dim[lane], x = R.x[lane], y = R.y[lane], zb = R.zb[lane];
        const uint32_t wc = w[13];  // line (x, y), block zb
        const bool xi = x >= 1 && x <= dim - 2, yi = y >= 1 && y <= dim - 2;
        const uint32_t zu = zbits_upto(dim - 2, zb), zi = zb == 0 ? zu & ~1u : zu;
        const uint32_t X = (yi && x + 1 < dim) ? (wc ^ w[22]) & zi : 0u;
        const uint32_t Y = (xi && y + 1 < dim) ? (wc ^ w[16]) & zi : 0u;
        const uint32_t Z = (xi && yi) ? (wc ^ ((wc >> 1) | (w[14] << 31))) & zu : 0u;
        R.X[lane] = X;
        R.Y[lane] = Y;
        R.Z[lane] = Z;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          R.vb[lane][b] += pv0;
          R.vb[lane][4 + b] += pb1.x;
        }
        const uint4 own = R.rec[lane][7];
        R.ib[lane] = own.w + pb1.y;
        if (ws.quads) ws.quads[R.cw[lane] + (x * dim + R.y[lane]) * R.zc[lane] + zb] = make_uint4(X, Y, Z, R.ib[lane] / 4u);
        const uint32_t nv = __popc(own.x) + 2u * __popc(own.y) + 4u * __popc(own.z);
        packed = nv | ((__popc(X) + __popc(Y) + __popc(Z)) << 16);  // at most 128 and 96 per word
      }
      uint32_t incl = packed;
#pragma unroll
      for (int o = 1; o < kTileWords; o <<= 1) {
        const uint32_t v = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += v;
      }
      if (lane < kTileWords) {
        R.voff[lane + 1] = (int)(incl & 0xFFFFu);
        R.qoff[lane + 1] = (int)(incl >> 16);
      }
      if (lane == 0) R.voff[0] = R.qoff[0] = 0;
    }
    __syncwarp();
    // 4. one lane per vertex: the k-th vertex of word t is in the cell l whose
    // preceding cells hold k or fewer (count planes), its (k - that)-th group
    const int nvt = R.voff[nt];
    for (int jb = 0; jb < nvt; jb += 32) {
      const int j = jb + lane;
      bool in = j < nvt;
      const int t = tile_word(R.voff, nt, in ? j : 0);
      const int k = in ? j - R.voff[t] : 0;
      const uint4 own = R.rec[t][7];
      const uint32_t c0 = own.x, c1 = own.y, c2 = own.z;
      int l = 0;
#pragma unroll
      for (int s = 16; s > 0; s >>= 1) {
        const uint32_t m = lane_lt(l + s);
        if ((int)(__popc(c0 & m) + 2 * __popc(c1 & m) + 4 * __popc(c2 & m)) <= k) l += s;
      }
      const uint32_t lt = lane_lt(l);
      const int g = k - (int)(__popc(c0 & lt) + 2 * __popc(c1 & lt) + 4 * __popc(c2 & lt));
      const int64_t gv = R.vout[t] + (int64_t)R.vb[t][7] + k;
      in = in && gv < out.vcap;
      const int dim = R.dim[t], x = R.x[t], y = R.y[t], z = 32 * R.zb[t] + l;
      const int mask = qtile_mask(R.w[t], 1, 1, 32 + l);
      if (PLACE != 2) {  // (QEF positions come from k_place_qef)
        float P[3];
        q_place<PLACE, true>(dens + R.dens[t], dim, x, y, z, in ? group_edges(mask, g & 3) : 0u, P);
        if (in) {
          out.pos[3 * gv] = P[0];
          out.pos[3 * gv + 1] = P[1];
          out.pos[3 * gv + 2] = P[2];
        }
      }
      if (in) {
        if (out.nrm) { out.nrm[3 * gv] = 0.0f; out.nrm[3 * gv + 1] = 0.0f; out.nrm[3 * gv + 2] = 0.0f; }
        // cells run to dim - 2
        if (out.boundary)
          out.boundary[gv] = (x == 0 || y == 0 || z == 0 || x == dim - 2 || y == dim - 2 || z == dim - 2);
        if (out.vkey) out.vkey[gv] = vertex_key(x, y, z, g);
        if (out.valence) {
          // the group's edges whose four cells exist (q_edge_interior), in quad order
          uint32_t set = group_edges_q(mask, g & 3);
          const auto cut = [&](bool has, uint32_t m) { if (!has) set &= ~m; };
          cut(x > 0, kQuadDx0);
          cut(x + 1 <= dim - 2, kQuadDx1);
          cut(y > 0, kQuadDy0);
          cut(y + 1 <= dim - 2, kQuadDy1);
          cut(z > 0, kQuadDz0);
          cut(z + 1 <= dim - 2, kQuadDz1);
          out.valence[gv] = (uint8_t)__popc(set);
          if (out.vadj) out.vadj[gv] = set;
        }
      }
      __syncwarp();
    }
    // 5. one lane per quad: the k-th interior crossing of word t
    const int nqt = R.qoff[nt];
    for (int j = lane; j < nqt; j += 32) {
      const int t = tile_word(R.qoff, nt, j);
      const int k = j - R.qoff[t];
      const uint32_t X = R.X[t], Y = R.Y[t], Z = R.Z[t];
      int l = 0;
#pragma unroll
      for (int s = 16; s > 0; s >>= 1) {
        const uint32_t m = lane_lt(l + s);
        if ((int)(__popc(X & m) + __popc(Y & m) + __popc(Z & m)) <= k) l += s;
      }
      const uint32_t lt = lane_lt(l);
      const int r = k - (int)(__popc(X & lt) + __popc(Y & lt) + __popc(Z & lt));
      uint32_t ownb = ((X >> l) & 1u) | (((Y >> l) & 1u) << 1) | (((Z >> l) & 1u) << 2);
      if (r >= 1) ownb &= ownb - 1u;
      if (r >= 2) ownb &= ownb - 1u;
      const int a = __ffs(ownb) - 1;
      const uint32_t* w = R.w[t];
      uint32_t q[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        // cell at (b, c) offsets (-1,-1), (0,-1), (0,0), (-1,0) of axes a + 1, a + 2; lb, lc: the edge's place in it
        const int lb = (c == 0 || c == 3) ? 1 : 0, lc = c < 2 ? 1 : 0;
        const int dx = a == 0 ? 0 : (a == 1 ? lc : lb), dy = a == 0 ? lb : (a == 1 ? 0 : lc);
        const int dz = a == 0 ? lc : (a == 1 ? lb : 0);
        const int e = a == 0 ? 2 * dy + dz : (a == 1 ? 4 + 2 * dx + dz : 8 + 2 * dx + dy);
        const int i = 1 - dx, jj = 1 - dy, zr = 32 + l - dz;
        const int m = qtile_mask(w, i, jj, zr);
        const int at = (i * 2 + jj) * 2 + (zr >> 5);
        const uint4 cv = R.rec[t][at];
        const uint32_t ct = lane_lt(zr & 31);
        q[c] = R.vb[t][at] + __popc(cv.x & ct) + 2 * __popc(cv.y & ct) + 4 * __popc(cv.z & ct) +
               (uint32_t)((s_grp[m] >> (4 * e)) & 0xF);
      }
      if (!((w[13] >> l) & 1u)) {  // lower sample outside: reversed
        const uint32_t v = q[1];
        q[1] = q[3];
        q[3] = v;
      }
      const int64_t gi = R.iout[t] + (int64_t)R.ib[t] + 4 * (int64_t)k;
      const uint32_t vo = (uint32_t)R.vout[t];
      if (idx16 && gi + 4 <= out.icap) {
        *reinterpret_cast<uint4*>(out.idx + gi) = make_uint4(q[0], q[1], q[2], q[3]);
        if (out.idx_global)
          *reinterpret_cast<uint4*>(out.idx_global + gi) = make_uint4(q[0] + vo, q[1] + vo, q[2] + vo, q[3] + vo);
      } else {
#pragma unroll
        for (int c = 0; c < 4; ++c)
          if (gi + c < out.icap) {
            out.idx[gi + c] = q[c];
            if (out.idx_global) out.idx_global[gi + c] = q[c] + vo;
          }
      }
    }
    __syncwarp();  // the next tile overwrites the stage
  }
}

// Mode Q QEF placement, one thread per vertex (dense lanes, unlike the
// warp-per-word emit where only surface cells' lanes work): the same
// q_place<2> on the vertex's cell and group, decoded from its key.
template <bool RECORD>
__global__ void __launch_bounds__(128) k_place_qef(const ChunkDev* __restrict__ chunks, int n_chunks,
                                                   const uint32_t* __restrict__ words, const float* __restrict__ dens,
                                                   const uint32_t* __restrict__ vkey,
                                                   const int64_t* __restrict__ d_counts, int64_t vcap,
                                                   float* __restrict__ pos, uint8_t* __restrict__ qflag,
                                                   uint32_t* __restrict__ qlist, uint32_t* __restrict__ qcount,
                                                   float* __restrict__ qseed) {
  const int64_t nv = min(vcap, d_counts[0]);
  for (int64_t v0 = (int64_t)blockIdx.x * blockDim.x; v0 < nv; v0 += (int64_t)gridDim.x * blockDim.x) {
    const bool in = v0 + threadIdx.x < nv;
    const int64_t v = in ? v0 + threadIdx.x : nv - 1;
    const ChunkDev& ch = chunks[find_chunk_by_vertex(chunks, n_chunks, v)];
    const int dim = ch.dim;
    int x, y, z, g;
    vertex_key_decode(vkey[v], x, y, z, g);
    const uint32_t edges = in ? group_edges(cell_mask_at(words + ch.words, dim, ch.zc, x, y, z), g) : 0u;
    float P[3];
    QefSolveInfo info;
    bool used = false;
    q_place<2, true>(dens + ch.dens, dim, x, y, z, edges, P, RECORD ? &info : nullptr, RECORD ? &used : nullptr);
    if (RECORD) {
      // record the branch, and for a QEF-placed vertex its FP32 eigenvectors
      // (the seeds of the wide adjoint), in the list of QEF-placed vertices:
      // one reservation per warp
      __syncwarp();
      const uint32_t take = __ballot_sync(kFull, used);
      uint32_t base = 0u;
      if ((threadIdx.x & 31) == 0 && take) base = atomicAdd(qcount, (uint32_t)__popc(take));
      base = __shfl_sync(kFull, base, 0);
      if (in) qflag[v] = used ? 1 : 0;
      if (used) {
        const uint32_t k = base + __popc(take & lane_lt(threadIdx.x & 31));
        qlist[k] = (uint32_t)v;
#pragma unroll
        for (int r = 0; r < 3; ++r) {
#pragma unroll
          for (int c3 = 0; c3 < 3; ++c3) qseed[9 * (int64_t)k + 3 * r + c3] = info.V[r][c3];
        }
      }
    }
    if (in) {
      pos[3 * v] = P[0];
      pos[3 * v + 1] = P[1];
      pos[3 * v + 2] = P[2];
    }
    __syncwarp();
  }
}

static void launch_place_qef(const ChunkDev* d_chunks, int n_chunks, const uint32_t* words, const float* dens,
                             const MeshOut& out, const int64_t* d_counts, cudaStream_t st) {
  // persistent: as many CTAs as are resident, whatever the arena's capacity
  static std::atomic<int> grid[64] = {};
  const int g = per_device_once(grid, [](int dev) {
    int sms = 0, per_sm = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_place_qef<true>, 128, 0);
    return (sms > 0 ? sms : 1) * (per_sm > 0 ? per_sm : 1);
  });
  const int64_t need = (out.vcap + 127) / 128;
  const int blocks = (int)(need < g ? need : g);
  if (out.qflag) {
    cudaMemsetAsync(out.qcount, 0, sizeof(uint32_t), st);
    k_place_qef<true><<<blocks, 128, 0, st>>>(d_chunks, n_chunks, words, dens, out.vkey, d_counts, out.vcap, out.pos,
                                              out.qflag, out.qlist, out.qcount, out.qseed);
  } else {
    k_place_qef<false><<<blocks, 128, 0, st>>>(d_chunks, n_chunks, words, dens, out.vkey, d_counts, out.vcap, out.pos,
                                               nullptr, nullptr, nullptr, nullptr);
  }
}

int launch_emit(int mode, int placement, const ChunkDev* d_chunks, int n_chunks, const int* d_unit_start,
                int n_units, const uint32_t* words, const float* dens, const uint32_t* flags, WordScratch ws,
                MeshOut out, const int64_t* d_counts, cudaStream_t st) {
  if (mode == 0 && ws.clist) {
    // persistent: one wave of resident CTAs
    static std::atomic<int> grid[64] = {};
    const int g = per_device_once(grid, [](int dev) {
      int sms = 0, per_sm = 0;
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_emit_words_r, 32 * kEmitWarps, 0);
      return (sms > 0 ? sms : 1) * (per_sm > 0 ? per_sm : 1);
    });
    k_emit_words_r<<<g, 32 * kEmitWarps, 0, st>>>(d_chunks, words, dens, ws, out);
  } else if (mode == 0) {
    k_emit<0, 0><<<n_units, 256, 0, st>>>(d_chunks, n_chunks, d_unit_start, words, dens, flags, ws, out);
  } else if (ws.clist) {
    static std::atomic<int> grid[64] = {};  // persistent: one wave of resident CTAs
    const int g = per_device_once(grid, [](int dev) {
      int sms = 0, per_sm = 0;
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_emit_words_q<1>, 32 * kEmitWarps, 0);
      return (sms > 0 ? sms : 1) * (per_sm > 0 ? per_sm : 1);
    });
    if (placement == 0) k_emit_words_q<0><<<g, 32 * kEmitWarps, 0, st>>>(d_chunks, words, dens, ws, out);
    else if (placement == 1) k_emit_words_q<1><<<g, 32 * kEmitWarps, 0, st>>>(d_chunks, words, dens, ws, out);
    else k_emit_words_q<2><<<g, 32 * kEmitWarps, 0, st>>>(d_chunks, words, dens, ws, out);
    if (placement == 2 && out.vcap > 0) {
      launch_place_qef(d_chunks, n_chunks, words, dens, out, d_counts, st);
      return 2;
    }
  } else if (placement == 0) {
    k_emit<1, 0><<<n_units, 256, 0, st>>>(d_chunks, n_chunks, d_unit_start, words, dens, flags, ws, out);
  } else if (placement == 1) {
    k_emit<1, 1><<<n_units, 256, 0, st>>>(d_chunks, n_chunks, d_unit_start, words, dens, flags, ws, out);
  } else {
    k_emit<1, 2><<<n_units, 256, 0, st>>>(d_chunks, n_chunks, d_unit_start, words, dens, flags, ws, out);
  }
  return 1;
}

}  // namespace bmf
