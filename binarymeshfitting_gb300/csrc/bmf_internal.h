// Host-side declarations shared by the library's translation units.
#pragma once

#include "../../include/bmf.h"
#include <atomic>
#include <cstdint>
#include <cuda_runtime.h>

namespace bmf {

// A launch constant worked out once per device (an occupancy-sized grid, a
// shared-memory opt-in done).  Host threads may race on the first call: each
// computes the same value, and the atomic slot makes the publication well
// defined.  compute(dev) must return a non-zero value.
template <class F>
inline int per_device_once(std::atomic<int> (&slot)[64], F compute) {
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return compute(dev);
  int v = slot[dev].load(std::memory_order_acquire);
  if (v == 0) {
    v = compute(dev);
    slot[dev].store(v, std::memory_order_release);
  }
  return v;
}

struct ChunkDev;
struct FieldDev;

// Output arena for one launch of the emit kernels (single chunk or batch).
struct MeshOut {
  float* pos;
  float* nrm;
  uint8_t* boundary;
  uint8_t* valence;
  uint32_t* idx;          // chunk-local vertex ids (one VerticesIndicesBlock per chunk)
  uint32_t* idx_global;   // optional: the same indices offset by the chunk's vertex base
  int64_t vcap, icap;
  // optional: where each vertex came from, (chunk-local linear sample index << 2) | k,
  // k = crossing axis (Mode R) or vertex group (Mode Q); the key the analytic
  // adjacency build starts from.
  uint32_t* vkey = nullptr;
  // optional: per vertex what the adjacency starts from (valence is its number of
  // bits).  Mode R: the triangles that use it in each of the four cells around its
  // edge, 5 bits per cell, ascending; Mode Q: the edges of its group that have a
  // quad, 12 bits in quad order.
  uint32_t* vadj = nullptr;
  // optional (QEF placement with keys): the record the QEF adjoint reads --
  // per vertex whether it took the QEF branch, the list of those vertices
  // (count in *qcount) and their FP32 eigenvectors (9 floats per entry)
  uint8_t* qflag = nullptr;
  uint32_t* qlist = nullptr;
  uint32_t* qcount = nullptr;
  float* qseed = nullptr;
};

// Per-word scratch of the extraction kernels, indexed like the occupancy
// words (chunk.words + (x*dim + y)*zc + zb).
struct WordScratch {
  // The count kernel writes these two for busy words only (words that own a
  // vertex or emit a primitive); nothing reads them for any other word.
  uint32_t* vcnt;  // vertices of the x-plane's words before this one (a word's base is pb[plane].x + vcnt)
  // {3 bit-planes of the per-cell triangle (Mode R) / vertex-group (Mode Q) count,
  // indices of the x-plane's words before this one}; Mode R's emit replaces the
  // last by the word's first primitive (of the chunk), for the adjacency
  uint4* rec;
  // Work list (nullable) of the busy words (those that own a vertex or emit a
  // primitive) as {chunk, word index in the chunk}, in no particular order;
  // *ccount (zeroed before the count kernel) entries, at most clist_cap kept.
  // With room for every word no arena is too small for it: each vertex that the
  // arena holds then gets its key, which the QEF placement, the adjacency and
  // the adjoint take for a cell inside the chunk.
  uint2* clist;
  uint32_t* ccount;
  int64_t clist_cap;
  // Per x-plane (ChunkDev::unit0 + x): its {vertex, index} totals (count
  // kernel), then their exclusive sums over the chunk's planes (k_chunk_scan)
  uint2* pb;
  // Band fill (nullable): its exactness mask, and (Mode R) the list of samples
  // the count kernel finds at an end of a crossing with an inexact density,
  // as {chunk, sample index in the chunk}; *fcount (zeroed before the count
  // kernel) entries, at most fix_cap kept.  A crossing has two ends, so the
  // list holds at most twice the vertex count (2 vcap + 1 suffices).
  const uint32_t* exact = nullptr;
  uint2* fix = nullptr;
  uint32_t* fcount = nullptr;
  int64_t fix_cap = 0;
  // Mode Q's band fill (nullable): per word the samples at an end of a crossing,
  // for launch_fill_need (words layout; only of chunks with a mesh).
  uint32_t* ends = nullptr;
  // Mode Q with sweeps (nullable): per busy word its interior crossings along x, y, z
  // and its first quad (of the chunk), which the emit writes and the adjacency reads.
  uint4* quads = nullptr;
  // The 2D heightmap's column fill (Mode R batches, nullable): no densities
  // are stored; the emit computes a crossing end's density from its (x, z)
  // column height (at chunk.words + x * dim + z) as the full fill does,
  // -(py * g) - n * height with py = chunk.oy + y * scale.
  const float* cols2d = nullptr;
  float c2d_g = 0.0f, c2d_height = 0.0f;
};

// Fill + label.  A terrain field of a single chunk goes through the block or the
// line kernel directly; batches pass their own item queue to
// launch_fill_terrain.
// cols (BMF_FIELD_TERRAIN_2D needs it): the (x, z) column heights from
// launch_columns2d, stored at chunk.words + x * dim + z (a chunk's dim^2
// columns fit its words' span).
void launch_sample_label(const ChunkDev* d_chunks, int n_chunks, const int* d_unit_start, int n_units, int max_dim,
                         const FieldDev& field, const float* dens_in, float* dens_out, uint32_t* words,
                         uint32_t* flags, cudaStream_t st, const float* cols = nullptr);
// The 2D heightmap's column heights of a batch into cols (layout above), over
// items {chunk, first column} of columns2d_item() columns each (null: chunk 0's
// columns in order).
void launch_columns2d(const ChunkDev* d_chunks, const int2* d_items, int n_items, const FieldDev& field, float* cols,
                      cudaStream_t st);
int columns2d_item();
// The 2D heightmap's occupancy words and contains_mesh flags from the column
// heights alone (the column fill: no densities).
void launch_words2d(const ChunkDev* d_chunks, int n_chunks, const int* d_unit_start, int n_units,
                    const FieldDev& field, const float* cols, uint32_t* words, uint32_t* flags, cudaStream_t st);
// Terrain FBM fill over line items {chunk, first line} (kFillLines lines
// each; d_items null = chunk 0's items in order).  d_queue non-null: grid
// persistent CTAs take items from the queue (zeroed by the caller); else one CTA
// per item.
// run = z-samples per step (4, 8, 16 or 32).
// exact (nullable): the band fill's exactness mask (words layout); with it
// the fill may leave decided samples inexact (see k_fill_terrain<RUN, true>)
void launch_fill_terrain(int run, const ChunkDev* d_chunks, const int2* d_items, int n_items, int* d_queue,
                         int grid, const FieldDev& field, float* dens_out, uint32_t* words, uint32_t* flags,
                         uint32_t* exact, cudaStream_t st);
// the band fill applies to fields of the form (py - h) - a * FBM with a > 0,
// and (as the column fill: words and column heights, no densities) to the 2D
// heightmap
bool fill_band_supported(const FieldDev& field);
// The batched-fitting loss (sum over chunks of the mean squared sphere-union
// distance of the chunk's vertices) into *loss and its position gradient into
// grad (vcap * 3, zero past the vertex total); n_partial per-block partial sums.
int launch_fit_loss_spheres(const ChunkDev* d_chunks, int n_chunks, const uint32_t* d_tot, const int64_t* d_totals,
                            int64_t vcap, const float* pos, const float* spheres, int k, float* grad, float* partial,
                            int n_partial, float* loss, cudaStream_t st);
// Adam over n parameters with the step count on the device (advanced after)
int launch_adam(float* p, const float* g, float* m, float* v, int64_t n, int* step, float lr, float b1, float b2,
                float eps, cudaStream_t st);
// exact densities for the samples the count kernel listed in ws.fix (the
// inexact ends of crossings; after launch_count, before launch_emit)
void launch_fill_fixup(const ChunkDev* d_chunks, const uint32_t* words, const WordScratch& ws, const FieldDev& field,
                       float* dens, cudaStream_t st);
// the same for a Mode Q mesh: the ends of all crossings, with grad also their
// neighbours along the axes (what the QEF's central differences read)
void launch_fill_need(bool grad, const ChunkDev* d_chunks, int n_chunks, const int* d_unit_start, int n_units,
                      const uint32_t* flags, const WordScratch& ws, const FieldDev& field, float* dens,
                      cudaStream_t st);
int fill_terrain_items(int dim);          // items of one chunk
int fill_terrain_lines();                 // lines per item
int fill_terrain_resident_ctas(int run, int octaves, bool band);  // persistent grid: SMs x resident CTAs per SM
void launch_cell_masks(int dim, const uint32_t* W, uint8_t* masks, cudaStream_t st);
// The record and unit range of a single chunk, its flags and (nullable) its
// work-list counter zeroed: one small launch instead of two copies and two
// memsets.
void launch_setup_chunk(const ChunkDev& c, ChunkDev* d_c, int* d_units, uint32_t* d_flags, uint32_t* d_ccount,
                        cudaStream_t st);
// Extraction: count -> chunk scan -> emit.  The list counters in ws are zeroed
// by the caller.  flags: the contains_mesh flags the
// fill wrote; flags_out (instead, with flags null): words produced elsewhere,
// whose flags the count kernel adds up here (cleared by the caller).
void launch_count(int mode, const ChunkDev* d_chunks, int n_chunks, const int* d_unit_start, int n_units,
                  const uint32_t* words, const uint32_t* flags, WordScratch ws, cudaStream_t st,
                  uint32_t* flags_out = nullptr);
// Scans each chunk's plane totals in ws.pb, writes chunk totals (vertices,
// indices) to d_tot[2c], and scans those into chunk.vout / chunk.iout, the
// per-chunk info table {voff, vcount, ioff, icount, contains_mesh, status} and
// d_totals {vertices, indices, contains_mesh of chunk 0}.  d_ticket: one int,
// zero before the first call and left zero by each (null for at most 32 chunks).
// sweep (nullable): the work lists of the chunk-by-chunk sweeps.
constexpr int kTotals = 3;
// Work lists of the chunk-by-chunk sweeps: the chunks that have vertices, by
// size (powers of sqrt 2), largest first.  The first n_big are taken by whole
// clusters, the others by single CTAs.
struct SweepLists {
  int* order = nullptr;  // [n_chunks]
  int* head = nullptr;   // {n_big, listed chunks, cluster queue, CTA queue}; launch_sweep_chunks zeroes the queues
  int cluster = 1;       // CTAs per cluster and CTAs in all of the launch that will take the lists
  int ctas = 1;
};
constexpr int kSweepHead = 4;
// The barrier of the whole-mesh sweep kernel's team of CTAs (zeroed once; each
// launch leaves its counters zero) and the CTAs' valence sums.
constexpr int kTeamMax = 256;
struct TeamSync {
  unsigned arrived, left, failed, pad;
  uint32_t seg[kTeamMax];
};
// h_totals (nullable): the same totals in pinned host memory, so that the host
// needs a synchronisation but no copy to read them.
void launch_chunk_scan(ChunkDev* d_chunks, int n_chunks, WordScratch ws, uint32_t* d_tot, const uint32_t* flags,
                       int64_t vcap, int64_t icap, int64_t* d_info, int64_t* d_totals, int64_t* h_totals, int* d_ticket,
                       cudaStream_t st, const SweepLists* sweep = nullptr);
// How the sweeps of n_chunks chunks with `columns` (sum of dim^2) columns in all
// run: one launch per step, one cooperative launch over the whole mesh, or
// chunk by chunk (then cluster and ctas of *s are filled).  equal: all chunks have
// the same dim and about as large meshes.
enum SweepForm { kSweepLaunches, kSweepTeam, kSweepChunks };
SweepForm sweep_form(int mode, int n_chunks, int64_t columns, bool equal, SweepLists* s);
// Returns the kernels launched: Mode Q QEF placement with vertex keys and
// d_counts (total vertices on the device) adds the per-vertex k_place_qef.
int launch_emit(int mode, int placement, const ChunkDev* d_chunks, int n_chunks, const int* d_unit_start,
                int n_units, const uint32_t* words, const float* dens, const uint32_t* flags, WordScratch ws,
                MeshOut out, const int64_t* d_counts, cudaStream_t st);

// One sweep (a dual and a primal step) of MeshProcessor.cpp:130-306.
// normals: 0 none, 1 face normals, 2 sums of vertex normals.  The face normals
// of a sweep only set the vertex normals, which the next face sweep sets
// anew, so with at most three face sweeps they are computed in the last of
// them alone.  A vertex keeps its older normal when its new one has n.y == 0
// (MeshProcessor.cpp:287): the positions before the left-out sweeps are kept,
// x[0] before the first, x[1] before the second, and primal_older_normal takes the normal of such a vertex from them.  Left out: the square roots and divisions of two of three
// sweeps, a float2 gather per list entry and a normal written per vertex.
struct SweepBufs {
  float* x[2] = {nullptr, nullptr};  // positions before the left-out sweeps (null: none left out)
  float* pos = nullptr;                       // positions out
  float* nrm = nullptr;                       // normals out (null: none)
  __host__ __device__ bool keep() const { return x[0] != nullptr; }
};
struct SweepStep {
  int normals, set_colors;
  const float* src;  // positions read, and written (dst may be src)
  float* dst;
  int skipped;  // face sweeps left out before this one (the last face sweep), which sets every vertex's first normal
};
// Face sweeps of iters sweeps (MeshProcessor.cpp:149-163) and those left out.
__host__ __device__ inline int sweep_face_count(int iters) {
  const int mx = iters / 2 - 3 < 10 ? iters / 2 - 3 : 10, f = mx > 3 ? mx : 3;
  return f < iters ? f : iters;
}
__host__ __device__ inline int sweep_skipped(int iters, int sn) {
  const int f = sweep_face_count(iters) - 1;
  return !sn || f < 0 || f > 2 ? 0 : f;
}
__host__ __device__ inline int sweep_colors(int m, int iters) {
  return (m < iters - 1) ? ((m == 3) || (m == 0 && iters <= 3)) : 0;
}
// keep: b.x are there
__host__ __device__ inline SweepStep sweep_step(int m, int iters, int sn, bool keep, const SweepBufs& b) {
  const int last = sweep_face_count(iters) - 1, k = keep ? sweep_skipped(iters, sn) : 0;
  SweepStep s;
  s.normals = !sn ? 0 : (m > last ? 2 : (m < k ? 0 : 1));
  s.set_colors = m < k ? 0 : sweep_colors(m, iters);
  s.src = m >= k ? b.pos : (m == 0 ? b.x[0] : b.x[1]);
  s.dst = m + 1 < k ? b.x[1] : b.pos;
  s.skipped = m == k ? k : 0;
  return s;
}

// MeshProcessor: operates on one flat mesh (vertices [0, nv), prims of N).
struct ProcessScratch {
  uint32_t* off;      // nv + 1 CSR offsets
  uint32_t* cursor;   // nv fill cursors
  uint32_t* adj;      // sum of valences
  float* dual_p;      // 4 * n_prims: dual point, normal x
  float* dual_n;      // 2 * n_prims: normal y, z (unused without normals)
  // positions before the left-out face sweeps (3 * nv each; null: none are left
  // out): x[0] is where the emit put the mesh
  float* x[2] = {nullptr, nullptr};
  uint32_t* tmp;      // scan scratch (block totals)
  int block;          // threads per CTA of the dual / primal sweeps (0 = 256)
};
// nv / n_prims size the grids; when d_counts is given the actual vertex and
// index counts are read from d_counts[0] / d_counts[1] on the device (so the
// sequence can be captured in a CUDA graph before the counts are known).
// Scratch sizes: off nv+1, cursor nv, adj N*n_prims, dual_p 4*n_prims, dual_n
// 2*n_prims, tmp ceil(nv / 4096) + 1.
// Where the vertex->primitive lists come from: a mesh this library extracted
// (grid structure known: built analytically per vertex) or any mesh (atomic
// scatter + per-vertex sort).
struct StructuredAdj {
  int mode;                  // BMF_MODE_R / BMF_MODE_Q; 2: any mesh, as one team (team set, the rest unused)
  const ChunkDev* chunks;    // with vout / iout set
  int n_chunks;
  WordScratch ws;            // scanned counts + per-word records
  const uint32_t* vkey;      // per-vertex keys written by the emit kernel
  const uint32_t* vadj;      // MeshOut::vadj
  // optional (tot and lists.order, or neither): the sweeps run chunk by chunk
  const uint32_t* tot = nullptr;  // per chunk {vertices, indices}
  SweepLists lists;               // filled by launch_chunk_scan
  TeamSync* team = nullptr;       // or (whole mesh, one cooperative launch): the team's barrier, and
  unsigned* team_failed = nullptr;  // where it tells the host of a wait that ran out (pinned)
  int* bwd_queue = nullptr;       // the adjoint sweeps' queue over lists.order (one int, reset by launch_process_bwd)
  // the chunk-by-chunk sweeps keep 16-bit chunk-relative adjacency lists for
  // chunks of at most 65535 primitives unless a later pass reads the
  // adjacency (the fit's adjoint sweeps want 32-bit mesh-wide ids)
  bool wide_adj = false;
};
void launch_adj_build(int mode, const ChunkDev* d_chunks, int n_chunks, WordScratch ws, const uint32_t* vkey,
                      const uint32_t* vadj, const uint32_t* off, const int64_t* d_counts, int64_t vcap,
                      int64_t adj_cap, uint32_t* adj, cudaStream_t st);
// The chunk-by-chunk form of launch_process for StructuredAdj with tot and
// lists set: CSR offsets, adjacency and all sweeps in one launch.
void launch_sweep_chunks(const StructuredAdj& sa, int N, int64_t nv, int64_t n_prims, const int64_t* d_counts,
                         float* pos, float* nrm, const uint8_t* boundary, const uint8_t* valence,
                         const uint32_t* idx, int iters, int process_boundary, int smooth_normals,
                         const ProcessScratch& s, cudaStream_t st);
// Makes the wait of a team's barrier run out, in one CTA that returns after about
// a millisecond: what a failed launch leaves behind.
void launch_team_timeout(TeamSync* sync, unsigned* host_failed, cudaStream_t st);
// Whether any mesh of this size takes the whole-mesh form (StructuredAdj mode 2).
bool sweep_team_mesh(int N, int64_t nv, int64_t n_prims);
// The whole-mesh form of launch_process in one cooperative launch (sa.team set).
void launch_sweep_team(const StructuredAdj& sa, int N, int64_t nv, int64_t n_prims, const int64_t* d_counts,
                       float* pos, float* nrm, const uint8_t* boundary, const uint8_t* valence, const uint32_t* idx,
                       int iters, int process_boundary, int smooth_normals, const ProcessScratch& s, cudaStream_t st);
// Returns the number of kernels launched.
int launch_process(int N, int64_t nv, int64_t n_prims, const int64_t* d_counts, float* pos, float* nrm,
                   const uint8_t* boundary, const uint8_t* valence, const uint32_t* idx, int iters,
                   int process_boundary, int smooth_normals, ProcessScratch s, const StructuredAdj* sa,
                   cudaStream_t st);
// Device-side LOD descriptor generation (bmf_lod.cu).  cap <= kLodMaxLeaves.
constexpr int kLodMaxLeaves = 16384;
size_t lod_scratch_bytes(int cap);
int lod_generate(const bmf_lod_params& p, bmf_chunk_desc* d_descs, int cap, int32_t* d_count, void* scratch,
                 cudaStream_t st);
// GLChunk::format_data: per-vertex p/n/c (unwind 0) or unwound quads with
// one normal each (unwind 1); d_chunks non-null resolves chunk-local indices
// of a batch arena.  Returns the kernels launched.
int launch_format(const ChunkDev* d_chunks, int n_chunks, int64_t nv, int64_t ni, const int64_t* d_counts,
                  const float* pos, const float* nrm, const uint32_t* idx, int unwind, int smooth, float* p, float* n,
                  float* c, int64_t cap, cudaStream_t st);
// Adjoint of a Mode Q mesh's position sweeps (needs launch_process's CSR in s.off /
// s.adj; uses s.dual_p and h, 4 * nv floats, as scratch): dL/d(initial positions)
// into g from dL/d(final positions) of the first n_grad vertices (0 for the
// others); n_prims > 0, iters > 0.  Returns the number of kernels launched.
int launch_process_bwd(int64_t nv, int64_t n_prims, const int64_t* d_counts, const uint8_t* boundary,
                       const uint8_t* valence, const uint32_t* idx, int iters, int process_boundary,
                       const ProcessScratch& s, const float* grad, int64_t n_grad, float* g, float* h,
                       const StructuredAdj* sa, cudaStream_t st);
// Adjoint of Mode Q placement (placement 1 mass point, 2 QEF); accumulates into
// grad_dens (the caller clears it).  wide (QEF): 0 FP32 adjoint, 1 the QEF
// derivative from an FP64 re-solve, 2 from a double-float re-solve; these read
// the forward's record (MeshOut::qflag, qlist, qcount, qseed).  Returns the
// kernels launched.
int launch_place_bwd(int placement, int wide, const ChunkDev* d_chunks, int n_chunks, const uint32_t* words,
                     const float* dens, const uint32_t* vkey, const int64_t* d_counts, int64_t vcap,
                     const float* grad_pos, float* grad_dens, const uint32_t* qlist, const uint32_t* qcount,
                     const float* qseed, const uint8_t* qflag, cudaStream_t st);
// Its wide pass over the list (bmf_adjoint64.cu).
void launch_qef_bwd(int wide, const ChunkDev* d_chunks, int n_chunks, const uint32_t* words, const float* dens,
                    const uint32_t* vkey, int64_t vcap, const float* grad_pos, float* grad_dens, const uint32_t* qlist,
                    const uint32_t* qcount, const float* qseed, cudaStream_t st);
void launch_exclusive_scan_u8_to_u32(const uint8_t* in, uint32_t* out, int64_t n, const int64_t* d_n,
                                     uint32_t* block_tmp, cudaStream_t st);

}  // namespace bmf
