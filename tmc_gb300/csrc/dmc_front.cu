// Dual Marching Cubes front end: per-cell classification, MC polygons, vertex representatives
// and quads, emitted in the reference's order without hash tables.
//
// Order.  The reference CPU path (cpp_dmc/DualMarchingCubes.cpp:16-50, :97-192) appends one
// vertex per contour in cell order, stores quads in a std::map keyed by the dual grid edge
// (3*global_index + axis) and walks the map in key order (DualMarchingCubes.h:663); vertices that
// no complete quad uses are then dropped (DualMarchingCubes.h:685).  A contour's vertex is used
// exactly when one of its edges is an interior grid edge (all four cells around it exist), and a
// quad exists exactly for every crossed interior edge.  So:
//   vertex index = #used contours in earlier cells + rank of the contour among the cell's used ones
//   quad index   = #crossed interior edges owned by earlier grid points + rank of the axis
// Both are exclusive prefix sums over cells; no atomics, no hash table, deterministic output.
//
// Kernels:
//   dmc_classify_kernel  case, contours, per-cell record (counts + edge->vertex rank map) and
//                        per-tile sums for the scan
//   dmc_offsets_kernel   in-tile scan -> per-cell vertex / quad offsets
//   dmc_vertex_point_kernel, dmc_vertex_finish_kernel
//                        vertex representatives (cpp_dmc representative/projection) in float32
//                        and float-float, normals, positions
//   dmc_vertex_search_kernel  the vertices that take the whole 7x7 search, or a coordinate in float64
//   dmc_vertex_kernel    the vertices those leave, with every float64 fallback
//   dmc_vertex_warp_kernel  the reference's 26x26 retry (and short lists whole), one warp per vertex
//   dmc_quad_kernel      each cell emits the quads of its crossed interior edges 0, 3, 8 by
//                        looking up the cells around them
//   dmc_twin_kernel      halfedge twins and vertex degrees of a single volume's quads
#include <cstdio>

#include "common.cuh"
#include "dmc.h"
#include "dmc_cell.cuh"
#include "dmc_repr.cuh"
#include "scan.cuh"

namespace tmc {

__constant__ uint64_t c_case_contour[256] = TMC_CASE_CONTOUR_INIT;

// ------------------------------------------------------------------------------------------
// classification (per-cell helpers in dmc_cell.cuh)
// ------------------------------------------------------------------------------------------
// Records of cells whose edges are all interior (at least one cell away from every border), by case: an
// unambiguous case has one contour, which is then used (rank 0 on every edge); 0 for the ambiguous ones.
struct CaseRecords {
  uint32_t r[256];
};
constexpr CaseRecords make_case_records() {
  constexpr uint64_t contours[256] = TMC_CASE_CONTOUR_INIT;
  CaseRecords t{};
  for (int c = 1; c < 255; c++) {
    if ((contours[c] & 0xF) == 0) continue;  // the contour's size
    int nq = 0;
    const int edge[3][2] = {{0, 1}, {0, 2}, {0, 4}};
    for (int e = 0; e < 3; e++) nq += ((c >> edge[e][0]) ^ (c >> edge[e][1])) & 1;
    t.r[c] = 1u | ((uint32_t)nq << 3);
  }
  return t;
}
__device__ const CaseRecords d_case_records = make_case_records();

// One warp per tile of kScanTile consecutive cells (linear order): the crossed cells in cell order from
// the bit rows (list_tile), then the records of those with an unambiguous case, a cell per lane,
// written densely at their slots with their in-tile offsets and cases, and the tile's packed
// (vertices << 32 | quads) sum.  Ambiguous cells (the asymptotic decider, ~1 % of the cells) go by slot
// to amb_list for dmc_amb_kernel, which runs them densely instead of stalling every warp here on a
// few lanes.
template <int kPerTile>  // warps per tile (block_per_tile)
__global__ void __launch_bounds__(kClassifyThreads) dmc_classify_kernel(CellSpace space, int64_t tile0, int64_t tile1,
                                                                          uint32_t* rec, uint16_t* cellof,
                                                                          uint8_t* ccase, CellMask* mask,
                                                                          unsigned long long* tile_sums,
                                                                          unsigned long long* stats,
                                                                          uint32_t* amb_list, unsigned* amb_n) {
  pdl_begin();
  constexpr unsigned kAll = 0xffffffffu;
  constexpr int kTiles = kClassifyThreads / 32 / kPerTile;  // tiles per block
  __shared__ uint16_t lists[kTiles][kScanTile];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int share = kPerTile == 1 ? 0 : wid;  // the warp's share of its tile
  const int64_t tile = tile0 + (int64_t)blockIdx.x * kTiles + (kPerTile == 1 ? wid : 0);
  if (tile >= tile1) return;  // the whole warp, or the whole block
  uint16_t* list = lists[kPerTile == 1 ? wid : 0];
  const Grid g = space.grid_of_tile(tile);
  const int64_t vbase = tile * kScanTile;  // first cell of the tile in the space
  unsigned long long* tile_sum = nullptr;  // of the tile's warps, when there are several
  int na = 0;
  if (share == 0) na = list_tile(g, space.n, tile, mask, list);
  if (kPerTile > 1) {
    __shared__ int s_na;
    __shared__ unsigned long long s_sum;
    if (threadIdx.x == 0) {
      s_na = na;
      s_sum = 0;
    }
    __syncthreads();
    na = s_na;
    tile_sum = &s_sum;
  }
  unsigned long long local = 0;
  unsigned nact = 0, amb = 0;
  for (int a0 = 32 * share; a0 < na; a0 += 32 * kPerTile) {
    const int a = a0 + lane;
    const uint32_t slot = (uint32_t)(vbase + a);
    bool ambiguous = false;
    uint32_t r = 0;
    if (a < na) {
      const int off = list[a];
      int i, j, k;
      cell_ijk(g, vbase + off - g.vbase, i, j, k);
      const unsigned cs = case_from_bits(g, i, j, k);
      ambiguous = case_ambiguous(cs);
      cellof[slot] = (uint16_t)off;
      ccase[slot] = (uint8_t)cs;
      if (!ambiguous) {
        const bool inner = i >= 1 && j >= 1 && k >= 1 && i <= g.nx - 3 && j <= g.ny - 3 && k <= g.nz - 3;
        r = inner ? __ldg(d_case_records.r + cs)
                  : record_from_contours(g, i, j, k, cs, table_contour(c_case_contour[cs]), false);
        rec[slot] = r;
        local += ((unsigned long long)rec_nv(r) << 32) | (unsigned long long)rec_nq(r);
      }
    }
    nact += __popc(__ballot_sync(kAll, r != 0));
    // ambiguous cells: their ranks to the front of the warp's share (its entries up to here are read)
    const unsigned bal = __ballot_sync(kAll, ambiguous);
    if (bal) {
      __syncwarp();
      if (ambiguous) list[share_entry<kPerTile>(share, amb + __popc(bal & ((1u << lane) - 1u)))] = (uint16_t)a;
      amb += __popc(bal);
    }
  }
  if (amb) {  // one atomic per warp: a single counter takes them all
    unsigned base = 0;
    if (lane == 0) base = atomicAdd(amb_n, amb);
    base = __shfl_sync(kAll, base, 0);
    __syncwarp();
    for (unsigned x = lane; x < amb; x += 32)
      amb_list[base + x] = (uint32_t)(vbase + list[share_entry<kPerTile>(share, x)]);
  }
  for (int o = 16; o; o >>= 1) local += __shfl_down_sync(kAll, local, o);
  if (lane == 0) {
    if (kPerTile == 1) tile_sums[tile] = local;
    else if (local) atomicAdd(tile_sum, local);
    // stats[0]: cells with a record (a used contour, an owned quad or the ambiguous flag); the
    // ambiguous cells' records are never empty, so they count here too
    if (amb) atomicAdd(stats + 1, (unsigned long long)amb);
    if (nact | amb) atomicAdd(stats + 0, (unsigned long long)(nact + amb));
  }
  if (kPerTile > 1) {
    __syncthreads();
    if (threadIdx.x == 0) tile_sums[tile] = *tile_sum;
  }
}

// The ambiguous listed cells: MC polygon with the asymptotic decider (float-float, float64 near the
// isovalue), record, and their counts added to their tile's sum (after the classification wrote it).
__global__ void __launch_bounds__(128) dmc_amb_kernel(CellSpace space, const uint16_t* cellof, uint32_t* rec,
                                                      unsigned long long* tile_sums, const uint32_t* list,
                                                      const unsigned* count) {
  pdl_begin();
  __shared__ uint64_t cc[256];
  for (int c = threadIdx.x; c < 256; c += blockDim.x) cc[c] = c_case_contour[c];
  __syncthreads();
  const unsigned na = *count;
  for (unsigned a = blockIdx.x * blockDim.x + threadIdx.x; a < na; a += gridDim.x * blockDim.x) {
    const uint32_t slot = list[a];
    const int64_t tile = slot >> kTileShift;
    const Grid g = space.grid_of_tile(tile);
    int i, j, k;
    cell_ijk(g, slot_cell(cellof, slot) - g.vbase, i, j, k);
    float u[8];
    load_corners(g, i, j, k, u);
    const uint32_t r = classify_active(g, i, j, k, mc_case(u, g.iso_up), u, cc);
    rec[slot] = r;
    const unsigned long long add = ((unsigned long long)rec_nv(r) << 32) | (unsigned long long)rec_nq(r);
    if (add) atomicAdd(tile_sums + tile, add);
  }
}

// In-tile exclusive scan of the listed cells' records -> per slot the record beside its vertex offset
// (rv, what the quads need of a neighbour in one load) and the quad offset (blocked: 16-byte loads
// and stores over the tile's slots), two entries per vertex (the slot of the cell that generates it
// and its rank there), and the tile's chunks of 32 slots appended to the chunk list (scan.cuh).
// Launched before the host knows the counts, with room for vcap vertices, so that it runs while the host
// wakes, reads them and makes room for the results (70 to 90 us that the GPU waited); with more vertices it
// does nothing and is launched again.
// The entries per vertex, written by the lanes that scan the cells, took half of the pass on dense
// fields (stores to 32 sectors at once); gathered and written in order: 47 M vertices 440 -> 211 us, 16.6 M
// 158 -> 138 us.
__global__ void __launch_bounds__(32 * kOffsetWarps, 4) dmc_offsets_kernel(const CellMask* mask, const uint32_t* rec,
                                                                       const unsigned long long* tile_off,
                                                                       int64_t tiles, uint2* rv, int32_t* qoff,
                                                                       uint32_t* vwork, uint8_t* vrank,
                                                                       uint32_t* chunks, unsigned* nchunks,
                                                                       const unsigned long long* totals, int64_t vcap) {
  pdl_begin();
  if ((int64_t)(*totals >> 32) > vcap) return;  // the whole grid
  __shared__ uint16_t staged[kOffsetWarps][4 * kOffsetStep];
  uint16_t* const vertices = staged[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const int64_t tile = (int64_t)blockIdx.x * kOffsetWarps + (threadIdx.x >> 5);
  const uint32_t listed = tile < tiles ? tile_listed(mask, tile) : 0;
  list_chunks<kOffsetWarps>(tile, listed, chunks, nchunks);
  if (tile >= tiles) return;  // the whole warp
  const int64_t base = tile * kScanTile;
  const int64_t end = base + listed;
  unsigned long long carry = tile_off[tile];
  for (int64_t step = base; step < end; step += kOffsetStep) {  // warp-uniform
    const int64_t first = step + (int64_t)lane * kScanItems;
    uint32_t r[kScanItems];
    load8(rec, first, end, r);
    unsigned long long sum = 0;
#pragma unroll
    for (int s = 0; s < kScanItems; s++) sum += ((unsigned long long)rec_nv(r[s]) << 32) | rec_nq(r[s]);
    const unsigned long long inc = warp_inclusive_scan(sum);
    const unsigned long long before = carry;
    unsigned long long pre = carry + inc - sum;
    carry += __shfl_sync(0xffffffffu, inc, 31);
    uint32_t vo[kScanItems];
    int32_t qo[kScanItems];
#pragma unroll
    for (int s = 0; s < kScanItems; s++) {
      vo[s] = (uint32_t)(pre >> 32);
      qo[s] = (int32_t)(pre & 0xffffffffull);
      pre += ((unsigned long long)rec_nv(r[s]) << 32) | rec_nq(r[s]);
    }
    store8_pairs(rv, first, end, r, vo);
    store8(qoff, first, end, qo);
    // the step's vertices are consecutive: gathered in shared memory (a cell has at most four), written
    // out by the whole warp
    const uint32_t v0 = (uint32_t)(before >> 32), count = (uint32_t)(carry >> 32) - v0;
    __syncwarp();  // the previous step's are written out
#pragma unroll
    for (int s = 0; s < kScanItems; s++)
      for (int q = 0; q < rec_nv(r[s]); q++)  // empty beyond the listed cells
        vertices[vo[s] - v0 + q] = (uint16_t)(((uint32_t)(first - base) + s) | (unsigned)q << kTileShift);
    __syncwarp();
    for (uint32_t e = lane; e < count; e += 32) {
      const unsigned x = vertices[e];
      vwork[v0 + e] = (uint32_t)base + (x & (kScanTile - 1));
      vrank[v0 + e] = (uint8_t)(x >> kTileShift);
    }
  }
}

// ------------------------------------------------------------------------------------------
// vertices (work list from the offsets kernel): the representatives of dmc_repr.cuh, a float32 search with
// certified float-float rounding, bit-identical to the reference's float/double arithmetic.  Its one-step
// form makes the points of nearly all (dmc_vertex_point_kernel, dmc_vertex_search_kernel), the contours it
// leaves take representative_7x7 and the 26x26 retry (dmc_vertex_kernel, dmc_vertex_warp_kernel).
// ------------------------------------------------------------------------------------------
// estimateGradient at a grid point (cpp_dmc/UniformGrid.cpp:512-540): central differences with
// the reference's border indexing ((i<0) ? 0 : (i>=max) ? max-i : i).
__device__ __forceinline__ int grad_index(int i, int max) { return (i < 0) ? 0 : (i >= max) ? max - i : i; }
// a + t*(b - a) in float-float
__device__ __forceinline__ ffx::ff ff_lerp(ffx::ff a, ffx::ff b, float t) {
  return ffx::ff_add(a, ffx::ff_mul_f(ffx::ff_sub(b, a), t));
}

struct Normal64 {
  double n[3];
};
// The reference's float64 normal (UniformGrid::normal on estimateGradient values), for the rare
// vertices whose gradients cancel so much that the float-float result would lose its margin.
__device__ __noinline__ Normal64 normal_f64(const Grid& g, int i, int j, int k, double pu, double pv, double pw,
                                            int flip) {
  const double* inv2d = g.inv2;
  double G[8][3];
  for (int q = 0; q < 8; q++) {
    const int a = i + (q & 1), b = j + ((q >> 1) & 1), c = k + ((q >> 2) & 1);
    const int i0 = grad_index(a - 1, g.nx), i1 = grad_index(a + 1, g.nx);
    const int j0 = grad_index(b - 1, g.ny), j1 = grad_index(b + 1, g.ny);
    const int k0 = grad_index(c - 1, g.nz), k1 = grad_index(c + 1, g.nz);
    G[q][0] = ((double)g.at(i1, b, c) - (double)g.at(i0, b, c)) * inv2d[0];
    G[q][1] = ((double)g.at(a, j1, c) - (double)g.at(a, j0, c)) * inv2d[1];
    G[q][2] = ((double)g.at(a, b, k1) - (double)g.at(a, b, k0)) * inv2d[2];
  }
  const double uu = pu, vv = pv, ww = pw;
  double nv3[3];
  for (int d = 0; d < 3; d++) {
    double gq[8];
    for (int q = 0; q < 8; q++) gq[q] = flip ? G[q][d] * -1. : G[q][d];
    nv3[d] = (1 - ww) * ((1 - vv) * ((1 - uu) * gq[0] + uu * gq[1]) + vv * ((1 - uu) * gq[2] + uu * gq[3])) +
             ww * ((1 - vv) * ((1 - uu) * gq[4] + uu * gq[5]) + vv * ((1 - uu) * gq[6] + uu * gq[7]));
  }
  const double s = sqrt(nv3[0] * nv3[0] + nv3[1] * nv3[1] + nv3[2] * nv3[2]);
  Normal64 r;
  for (int d = 0; d < 3; d++) r.n[d] = nv3[d] / s;
  return r;
}
// The 32 field values behind the central differences at a cell's corners: the corners themselves and,
// along each axis, the four values before and the four after them (one end of every difference is a
// corner).  The reference's border indexing (grad_index): before index 0 comes point 0, after the last
// point comes point 0.
// One axis at a time: the corners stay, the axis's eight outer values are loaded when it is its turn.
struct AxisLines {
  float lo[4], hi[4];  // before and after, the four corner lines in corner order
};
__device__ __forceinline__ void load_axis(const Grid& g, int i, int j, int k, int d, AxisLines& S) {
  const int64_t sy = g.nx, sz = (int64_t)g.nx * g.ny;
  const float* f = g.f + (int64_t)k * sz + (int64_t)j * sy + i;
  const int64_t st = d == 0 ? 1 : (d == 1 ? sy : sz);
  const int at = d == 0 ? i : (d == 1 ? j : k), n = d == 0 ? g.nx : (d == 1 ? g.ny : g.nz);
  const float* lo = at > 0 ? f - st : f;
  const float* hi = at + 2 < n ? f + 2 * st : f - at * st;
  const int64_t sa = d == 0 ? sy : 1, sb = d == 2 ? sy : sz;
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const int64_t o = (q & 1 ? sa : 0) + (q & 2 ? sb : 0);
    S.lo[q] = __ldg(lo + o);
    S.hi[q] = __ldg(hi + o);
  }
}
// the two values of the difference along axis d at corner q
__device__ __forceinline__ void corner_pair(const float c[8], const AxisLines& S, int d, int q, float& hi, float& lo) {
  const int line = d == 0 ? q >> 1 : (d == 1 ? (q & 1) | (q >> 1 & 2) : q & 3);
  const bool up = (q >> d) & 1;
  hi = up ? S.hi[line] : c[q | 1 << d];
  lo = up ? c[q & ~(1 << d)] : S.lo[line];
}

// The normal at local coordinates p from the corner differences, as float pairs normalised; false where float64
// has to decide.  kept: the pairs themselves are kept (within 2^-30 of the reference's float64 normal; false where
// the gradients cancel to below 2^-10 of their size).  Otherwise their float32 roundings are wanted: false where
// these may not be the float64 normal's.  A component errs by 42 2^-48 of its differences' size: 13 2^-48 by each of
// three interpolations (a pair sum 3, a product 2, of the difference of up to twice the size; a sum 3), the scaling.
__device__ __forceinline__ bool normal_ff(const Grid& g, int i, int j, int k, const float c[8], const float p[3],
                                          int flip, bool kept, ffx::ff out[3]) {
  ffx::ff nv3[3];
  float scale = 0;  // largest |difference| * 1/(2 spacing): the size of the interpolation's inputs
#pragma unroll
  for (int d = 0; d < 3; d++) {
    AxisLines S;
    load_axis(g, i, j, k, d, S);
    ffx::ff G[8];
    float md = 0;
#pragma unroll
    for (int q = 0; q < 8; q++) {
      float hi, lo;
      corner_pair(c, S, d, q, hi, lo);
      G[q] = ffx::two_sum(hi, -lo);
      md = fmaxf(md, fabsf(G[q].hi));
    }
    scale = fmaxf(scale, md * g.inv2_hi[d]);
    const ffx::ff a0 = ff_lerp(G[0], G[1], p[0]), a1 = ff_lerp(G[2], G[3], p[0]);
    const ffx::ff a2 = ff_lerp(G[4], G[5], p[0]), a3 = ff_lerp(G[6], G[7], p[0]);
    const ffx::ff b0 = ff_lerp(a0, a1, p[1]), b1 = ff_lerp(a2, a3, p[1]);
    const ffx::ff t = ffx::ff_mul(ff_lerp(b0, b1, p[2]), ffx::ff{g.inv2_hi[d], g.inv2_lo[d]});
    nv3[d] = flip ? ffx::ff_neg(t) : t;
  }
  if (!kept) return unit_certain(nv3, scale * 0x1.5p-43f, out) && pairs_hold(scale, g.inv2_hi);
  float dot, r0;
  unit_ff(nv3, out, dot, r0);
  return dot > 0x1p-80f && dot < 0x1p80f && scale <= 0x1p10f * sqrtf(dot);
}

constexpr int kVertexThreads = 128;

// The current volume's grid and the constants derived from it, cached per thread (a batch mixes
// volumes; consecutive vertices mostly share one).
struct GridCache {
  int vol = -1;
  Grid g{};
  ffx::ff iso_ff{0, 0};
  __device__ __forceinline__ void load(const CellSpace& space, uint32_t vcell) {
    const int v = space.grids ? ld(space.tile_vol + vcell / kScanTile) : 0;
    if (v == vol) return;
    vol = v;
    g = space.grids ? space.grids[v] : space.one;
    iso_ff = ffx::ff_from_double(g.iso);
  }
};

// The contour behind vertex `rank` of a cell: corners, MC polygon, and the edge points and bounding
// boxes of all its contours (slice, cpp_dmc/DualMarchingCubes.cpp:114-136).
struct VertexContour {
  float u[8];
  uint64_t c;
  repr::Boxes bx;
  float pts[36];
  int tsel, tstart;
};
__device__ __forceinline__ bool vertex_contour(const Grid& g, int i, int j, int k, int rank, const uint64_t* cc,
                                               ffx::ff iso_ff, VertexContour& V) {
  load_corners(g, i, j, k, V.u);
  const unsigned cs = mc_case(V.u, g.iso_up);
  V.c = dmc_polygon(cs, V.u, g.iso, cc);
  const int ncnt = cnt_count(V.c);
  int flat = 0, used_seen = 0;
  V.tsel = -1;
  V.tstart = 0;
  for (int t = 0; t < ncnt; t++) {
    V.bx.b[t][0][0] = 1; V.bx.b[t][0][1] = 0;
    V.bx.b[t][1][0] = 1; V.bx.b[t][1][1] = 0;
    V.bx.b[t][2][0] = 1; V.bx.b[t][2][1] = 0;
    const int sz = cnt_size(V.c, t);
    bool used = false;
    for (int q = 0; q < sz; q++) {
      const int e = cnt_edge(V.c, flat + q);
      used = used || edge_interior(g, i, j, k, e);
      bool fb = false;
      const float l = repr::edge_param_fast(e, V.u, g.iso, iso_ff, fb);
      float ui[3];
      repr::local_from_param(e, l, ui);
#pragma unroll
      for (int d = 0; d < 3; d++) {
        V.pts[3 * (flat + q) + d] = ui[d];
        V.bx.b[t][d][0] = V.bx.b[t][d][0] > ui[d] ? ui[d] : V.bx.b[t][d][0];
        V.bx.b[t][d][1] = V.bx.b[t][d][1] < ui[d] ? ui[d] : V.bx.b[t][d][1];
      }
    }
    if (used) {
      if (used_seen == rank) {
        V.tsel = t;
        V.tstart = flat;
      }
      used_seen++;
    }
    flat += sz;
  }
  return V.tsel >= 0;
}

// Position, normal and local coordinates of vertex vidx at local coordinates p of cell (i, j, k).
// p64: the float64 local coordinates when they are not the floats p (the reference's unrounded mean
// point, for contours without any valid projection sample), else null.
// kFF: some volume keeps normals as float pairs (simplification), kAllKept: every one does; the float32 normals
// alone otherwise
// Float64 (1/57 of the float32 rate) is kept to what it must decide: positions that are float64
// outputs, float32 positions and normals whose rounding the float pair does not certify, kept pair
// normals whose gradients cancel to below 2^-10 of their size.  The gradients take 32 field loads (48
// point by point), one axis after another.  16.6 M vertices with float64 positions and pair normals: 1.40
// -> 1.09 ms; 7.6 M with float32 outputs: 0.49 -> 0.30 ms; 47 M of the saddle field, where many
// gradients cancel to below 1/16 (float64 normals before): 15.4 -> 2.49 ms with 72 registers, 10,000
// of them in float64.
template <bool kFF = true, bool kAllKept = false>
__device__ __forceinline__ void vertex_outputs(const Grid& g, int i, int j, int k, int64_t cell,
                                               const float p[3], const double* p64, int64_t vidx,
                                               const DmcVertexOut& out, int flip, repr::Stats& st) {
  const int64_t o = 3 * vidx;
  // a simplified volume: its float32 positions and normals are written after the passes, from the
  // float64 positions and the float-pair normals kept here
  const bool keep64 = kAllKept || (out.n64 && (g.flags & kGridNormal64));
  float2* n2 = reinterpret_cast<float2*>(out.n64);
  // position: UniformGrid::position (cpp_dmc/UniformGrid.h:300-305)
#pragma unroll
  for (int d = 0; d < 3; d++) {
    const int c = d == 0 ? i : (d == 1 ? j : k);
    const double og = d == 0 ? g.ox : (d == 1 ? g.oy : g.oz), sp = d == 0 ? g.dx : (d == 1 ? g.dy : g.dz);
    if (!p64 && !out.v64) {
      const ffx::ff t = ffx::ff_mul(ffx::two_sum((float)c, p[d]), ffx::ff{g.sp_hi[d], g.sp_lo[d]});
      const ffx::ff x = ffx::ff_add_abs(ffx::ff{g.org_hi[d], g.org_lo[d]}, t);
      // below 2^-80 the pairs' low parts run into the end of the float range
      const float mag = fabsf(g.org_hi[d]) + fabsf(t.hi);
      out.v[o + d] = mag > 0x1p-80f && ffx::ff_certain(x, mag * 0x1p-43f) ? x.hi : (float)(og + (c + (double)p[d]) * sp);
    } else {
      const double x = og + (c + (p64 ? p64[d] : (double)p[d])) * sp;
      if (!keep64) out.v[o + d] = (float)x;
      if (out.v64) out.v64[o + d] = x;
    }
  }
  // normal: trilinear interpolation of the 8 corner gradients, normalised (UniformGrid::normal,
  // cpp_dmc/UniformGrid.h:286-298).  When it is kept for the simplification merges it is computed
  // in float-float (relative error ~2^-40, far below the float32 output's 2^-24) on the FP32 pipes.
  ffx::ff nf[3];
  bool pairs = false;  // nf holds the normal
  if (!p64) {
    float c[8];
    load_corners(g, i, j, k, c);
    if (!(kFF && keep64)) {
      float nv3[3];
      const float sgn = flip ? -1.0f : 1.0f;
      float scale = 0;  // largest corner gradient component: the size of the interpolation's inputs
#pragma unroll
      for (int d = 0; d < 3; d++) {
        AxisLines S;
        load_axis(g, i, j, k, d, S);
        float G[8];
#pragma unroll
        for (int q = 0; q < 8; q++) {
          float hi, lo;
          corner_pair(c, S, d, q, hi, lo);
          G[q] = (hi - lo) * g.inv2f[d];
          scale = fmaxf(scale, fabsf(G[q]));
        }
        const float a0 = fmaf(p[0], G[1] - G[0], G[0]), a1 = fmaf(p[0], G[3] - G[2], G[2]);
        const float a2 = fmaf(p[0], G[5] - G[4], G[4]), a3 = fmaf(p[0], G[7] - G[6], G[6]);
        const float b0 = fmaf(p[1], a1 - a0, a0), b1 = fmaf(p[1], a3 - a2, a2);
        nv3[d] = sgn * fmaf(p[2], b1 - b0, b0);
      }
      const float dot = nv3[0] * nv3[0] + nv3[1] * nv3[1] + nv3[2] * nv3[2];
      // The float32 interpolation errs by a few ulps of `scale`; where the gradients cancel to below
      // 1/16 of it (strongly uneven spacing, near critical points) that would exceed ~4e-6 of the
      // unit normal: float pairs instead, as where the squares leave the float range.
      if (dot > 0x1p-100f && dot < 0x1p100f && scale <= 16.0f * sqrtf(dot)) {
        const float rn = rsqrtf(dot);
#pragma unroll
        for (int d = 0; d < 3; d++) nf[d] = ffx::ff_from(nv3[d] * rn);
        pairs = true;
      }
    }
    if (!pairs) pairs = normal_ff(g, i, j, k, c, p, flip, kFF && keep64, nf);
  }
  if (!pairs) {
    const Normal64 n = normal_f64(g, i, j, k, p64 ? p64[0] : (double)p[0], p64 ? p64[1] : (double)p[1],
                                  p64 ? p64[2] : (double)p[2], flip);
#pragma unroll
    for (int d = 0; d < 3; d++) nf[d] = ffx::ff_from_double(n.n[d]);
    st.normal_f64++;
  }
#pragma unroll
  for (int d = 0; d < 3; d++) {
    if (keep64) n2[o + d] = make_float2(nf[d].hi, nf[d].lo);
    else out.n[o + d] = nf[d].hi;
  }
  if (out.vcell) {
    out.vcell[vidx] = cell;
    out.vuvw[o] = p[0];
    out.vuvw[o + 1] = p[1];
    out.vuvw[o + 2] = p[2];
  }
}

__device__ __forceinline__ void flush_stats(const repr::Stats& st, unsigned long long* stats) {
  // representative counters (the reference's failed-projection counts) and float64 fallbacks
  if (st.fail1) atomicAdd(stats + 2, (unsigned long long)st.fail1);
  if (st.fail2) atomicAdd(stats + 3, (unsigned long long)st.fail2);
  if (st.fallback + st.normal_f64) atomicAdd(stats + 7, (unsigned long long)(st.fallback + st.normal_f64));
}

// One-pass vertex kernel over the vertices that dmc_vertex_search_kernel leaves: the 7x7 projection with
// every float64 fallback.  Contours
// without a valid 7x7 sample go on to the tail list (the reference's 26x26 retry, one warp each).
// A list of at most `warp_max` entries is left whole to the warp kernel: one thread's serial
// projection (~0.1 ms) would set the latency of a small call.
__global__ void __launch_bounds__(kVertexThreads) dmc_vertex_kernel(CellSpace space, const uint16_t* cellof, const uint8_t* vrank,
                                                                     const uint32_t* vwork, const uint32_t* list,
                                                                     const unsigned* count, uint32_t* tail_list,
                                                                     unsigned* tail_count, unsigned warp_max,
                                                                     DmcVertexOut out, int flip_all,
                                                                     unsigned long long* stats) {
  pdl_begin();
  __shared__ uint64_t cc[256];
  __shared__ float sample_lb[49 * kVertexThreads];  // per-thread sample bounds, column per thread
  const unsigned n = *count;
  if (n <= warp_max) return;
  for (int c = threadIdx.x; c < 256; c += blockDim.x) cc[c] = c_case_contour[c];
  __syncthreads();
  repr::Stats st;
  GridCache G;
  for (int64_t a = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; a < n; a += (int64_t)gridDim.x * blockDim.x) {
    const int64_t vidx = (int64_t)list[a];
    const uint32_t vcell = slot_cell(cellof, vwork[vidx]);
    const int rank = vrank[vidx];
    G.load(space, vcell);
    const Grid& g = G.g;
    const int64_t cell = vcell - g.vbase;
    int i, j, k;
    cell_ijk(g, cell, i, j, k);
    VertexContour V;
    if (!vertex_contour(g, i, j, k, rank, cc, G.iso_ff, V)) continue;  // cannot happen: counted
    float p[3];
    int prj;
    if (!repr::representative_7x7(V.u, g.iso, V.c, V.tsel, V.pts + 3 * V.tstart, cnt_size(V.c, V.tsel), V.bx, p,
                                  st, sample_lb + threadIdx.x, kVertexThreads, prj)) {
      st.fail1++;
      tail_list[atomicAdd(tail_count, 1u)] = (uint32_t)vidx;
      continue;
    }
    vertex_outputs(g, i, j, k, cell, p, nullptr, vidx, out, flip_all | (g.flags & kGridFlip), st);
  }
  flush_stats(st, stats);
}

// warp-wide winner of the lanes' samples: smallest distance, then smallest loop index
__device__ __forceinline__ repr::LaneBest warp_best(repr::LaneBest b) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    repr::LaneBest x;
    x.d = __shfl_xor_sync(0xffffffffu, b.d, o);
    x.w = __shfl_xor_sync(0xffffffffu, b.w, o);
    x.q = __shfl_xor_sync(0xffffffffu, b.q, o);
    if (repr::lane_better(x, b)) b = x;
  }
  return b;
}

// One warp per vertex: every lane rebuilds the contour and its projection frame (same cell, no
// divergence), the lanes split the samples, and lane 0 writes the outputs.  A listed vertex takes
// ~2 samples per lane for its 7x7 projection and ~22 for the reference's 26x26 retry, instead of up
// to 725 on one thread.  Work: the whole one-pass list when it has at most `warp_max` entries
// (the one-pass kernel then does nothing), otherwise the one-pass kernel's tail list.
__global__ void __launch_bounds__(kVertexThreads) dmc_vertex_warp_kernel(CellSpace space, const uint16_t* cellof, const uint8_t* vrank,
                                                                          const uint32_t* vwork, const uint32_t* list,
                                                                          const unsigned* count,
                                                                          const uint32_t* tail_list,
                                                                          const unsigned* tail_count,
                                                                          unsigned warp_max, DmcVertexOut out,
                                                                          int flip_all, unsigned long long* stats) {
  pdl_begin();
  constexpr int kWarps = kVertexThreads / 32;
  __shared__ uint64_t cc[256];
  __shared__ float coords[kWarps][2][26];  // each warp's sample coordinates
  const bool whole = *count <= warp_max;   // 7x7 projections too, not only retries
  const uint32_t* L = whole ? list : tail_list;
  const int64_t n = whole ? (int64_t)*count : (int64_t)*tail_count;
  if (n == 0) return;
  for (int c = threadIdx.x; c < 256; c += blockDim.x) cc[c] = c_case_contour[c];
  __syncthreads();
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  float* su = coords[wib][0];
  float* sv = coords[wib][1];
  repr::Stats st;
  GridCache G;
  int f64 = 0;
  for (int64_t a = (int64_t)blockIdx.x * kWarps + wib; a < n; a += (int64_t)gridDim.x * kWarps) {
    const int64_t vidx = (int64_t)L[a];
    const uint32_t vcell = slot_cell(cellof, vwork[vidx]);
    const int rank = vrank[vidx];
    G.load(space, vcell);
    const Grid& g = G.g;
    const int64_t cell = vcell - g.vbase;
    int i, j, k;
    cell_ijk(g, cell, i, j, k);
    VertexContour V;
    if (!vertex_contour(g, i, j, k, rank, cc, G.iso_ff, V)) continue;  // cannot happen (warp-uniform)
    const float* pts = V.pts + 3 * V.tstart;
    const int npts = cnt_size(V.c, V.tsel);
    repr::ProjCtx P;
    float us[7], vs[7];
    int f64c = 0;  // float64 sample coordinates: the same on every lane (counted once)
    repr::projection_setup(V.u, g.iso, V.c, V.tsel, pts, npts, V.bx, P, us, vs, f64c);
    if (whole && lane == 0) f64 += f64c;  // a retry's set-up was counted by the one-pass kernel
    repr::LaneBest b = repr::lane_none();
    int ns = 7;
    if (whole) {
      __syncwarp();  // the previous vertex's coordinates are no longer read
      if (lane == 0) {
#pragma unroll
        for (int q = 0; q < 7; q++) {
          su[q] = us[q];
          sv[q] = vs[q];
        }
      }
      __syncwarp();
      b = warp_best(repr::grid_lane(P, su, sv, 7, lane, 32, pts, npts, f64));
      if (b.q == repr::kNoSample && lane == 0) st.fail1++;
    }
    if (b.q == repr::kNoSample) {
      // the reference's retry with 26x26 samples from the same mean point
      __syncwarp();
      if (lane < 26) {
        su[lane] = repr::tail_coord(V.bx.b[V.tsel][P.A][0], V.bx.b[V.tsel][P.A][1], lane + 1);
        sv[lane] = repr::tail_coord(V.bx.b[V.tsel][P.B][0], V.bx.b[V.tsel][P.B][1], lane + 1);
      }
      __syncwarp();
      b = warp_best(repr::grid_lane(P, su, sv, 26, lane, 32, pts, npts, f64));
      ns = 26;
    }
    if (lane == 0) {
      float p[3];
      if (b.q != repr::kNoSample) {
        repr::lane_point(P, su, sv, ns, b, p);
        vertex_outputs(g, i, j, k, cell, p, nullptr, vidx, out, flip_all | (g.flags & kGridFlip), st);
      } else {
        // nothing valid at 26x26 either: the reference keeps its float64 mean point, unrounded
        st.fail2++;
        const repr::Point64 pm = repr::mean_point_exact(pts, npts);
        for (int d = 0; d < 3; d++) p[d] = (float)pm.p[d];
        const bool exact = (double)p[0] == pm.p[0] && (double)p[1] == pm.p[1] && (double)p[2] == pm.p[2];
        vertex_outputs(g, i, j, k, cell, p, exact ? nullptr : pm.p, vidx, out, flip_all | (g.flags & kGridFlip),
                       st);
      }
    }
  }
  st.fallback += f64;
  flush_stats(st, stats);
}

// Crossed edges of every MC case, two bits per edge (dmc_repr.cuh's edge sets)
struct CaseEdges {
  uint32_t m[256];
};
constexpr CaseEdges make_case_edges() {
  CaseEdges t{};
  for (int c = 0; c < 256; c++)
    for (int e = 0; e < 12; e++) {
      const int a = (int)((TMC_PK_EDGE_V0 >> (4 * e)) & 0xF), b = (int)((TMC_PK_EDGE_V1 >> (4 * e)) & 0xF);
      t.m[c] |= (uint32_t)(((c >> a) ^ (c >> b)) & 1) << (2 * e);
    }
  return t;
}
__device__ const CaseEdges d_case_edges = make_case_edges();

// Appends x to a list for the active lanes with `take` set: one atomic per warp.
__device__ __forceinline__ void append(uint32_t* list, unsigned* count, bool take, uint32_t x) {
  const unsigned am = __activemask(), bal = __ballot_sync(am, take);
  if (!bal) return;
  const int lane = threadIdx.x & 31, leader = __ffs(bal) - 1;
  unsigned base = 0;
  if (lane == leader) base = atomicAdd(count, (unsigned)__popc(bal));
  base = __shfl_sync(am, base, leader);
  if (take) list[base + __popc(bal & ((1u << lane) - 1u))] = x;
}

// A warp's entries for a list, gathered in shared memory and appended 32 at a time: one atomic per 32
// entries.  (With one per warp and iteration the list's single counter took a fifth of the point kernel.)
struct WarpList {
  uint32_t* buf;  // 64 entries
  int n = 0;      // the same on every lane
  __device__ __forceinline__ void flush(uint32_t* list, unsigned* count, int k) {
    const int lane = threadIdx.x & 31;
    unsigned base = 0;
    if (lane == 0) base = atomicAdd(count, (unsigned)k);
    base = __shfl_sync(0xffffffffu, base, 0);
    if (lane < k) list[base + lane] = buf[lane];
  }
  // every lane of the warp calls it
  __device__ __forceinline__ void add(uint32_t* list, unsigned* count, bool take, uint32_t x) {
    const unsigned bal = __ballot_sync(0xffffffffu, take);
    if (!bal) return;
    const int lane = threadIdx.x & 31;
    if (take) buf[n + __popc(bal & ((1u << lane) - 1u))] = x;
    n += __popc(bal);
    __syncwarp();
    if (n >= 32) {
      flush(list, count, 32);
      n -= 32;
      const uint32_t rest = buf[32 + lane];
      __syncwarp();
      buf[lane] = rest;
      __syncwarp();
    }
  }
  __device__ __forceinline__ void finish(uint32_t* list, unsigned* count) {
    if (n) flush(list, count, n);
  }
};

// copies a float to shared memory without waiting for it (cp_async_wait)
__device__ __forceinline__ void cp_async4(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// The vertices' projected points, one lane per vertex.  The contour's edge set comes from the cell's
// record and case, so no polygon is walked again; the frame of the search (repr::vertex_frame) sits
// in shared memory, a column per lane, and nothing is written to memory but the point.
// p (local coordinates) goes to vp, or w != 0 marks what is still open: 1 the one-pass kernels' list,
// 4 + plane the missing coordinate of the second list (last_coordinates).
//
// The number of samples a lane still has to bound after its first one varies (none for 70 % of the
// vertices of the noise field, more than ten for 1 %): looping over its own, a lane would keep its
// warp busy until the warp's largest number is reached (6 active lanes per instruction, measured).
// So the warp lists all its lanes' samples and its lanes take them 32 at a time, whosever they are.
// A lane with more than kFewSamples has its samples listed by the whole warp, and a sample's bounds go to
// its lane's words in shared memory: the lanes' own loops over their samples took 43 % of the saddle
// field's time, where a few lanes of most warps have dozens.  The first samples pass through the same code
// (one copy of it: with two the warps waited for instructions a quarter of the time).  The chain vertex ->
// slot -> record and cell -> corners runs one iteration ahead, the corners into shared memory.
// Bound by instruction issue (80 % active, 23 lanes per instruction, 64 registers).  16.6 M vertices
// (512^3 noise): 1.78 -> 1.48 ms; 47 M (1024x1024x64 saddles): 7.66 -> 5.54 ms, with 0.13 ms more for the
// search of what stays open; 2.2 M (256^3 noise): 0.237 -> 0.200 ms.
// The separate set-up and projection kernels before this one (a 144-byte record per vertex written and
// read in between, nine samples bounded per vertex) took 1.15 + 0.85 ms for 5.5 M vertices, one kernel
// with per-lane loops 1.06 ms.
constexpr int kSampleWindow = 256;  // samples listed at a time
constexpr int kFewSamples = 4;
template <bool kBatch>
__global__ void __launch_bounds__(kVertexThreads, 8) dmc_vertex_point_kernel(CellSpace space, const uint16_t* cellof,
                                                                          const uint8_t* ccase, const uint32_t* rec,
                                                                          const uint8_t* vrank, const uint32_t* vwork,
                                                                          int64_t nv, float4* vp, uint32_t* list,
                                                                          uint32_t* wlist, unsigned* count) {
  pdl_begin();
  constexpr int kWarps = kVertexThreads / 32;
  constexpr unsigned kAll = 0xffffffffu;
  __shared__ float frames[repr::kFrameFloats * kVertexThreads];
  __shared__ float corners[8 * kVertexThreads];  // of the next iteration's cells
  __shared__ uint16_t items[kWarps][kSampleWindow];
  __shared__ float lowers[kWarps][kSampleWindow];
  __shared__ unsigned per_lane[kWarps][2][32];
  __shared__ uint32_t lists[kWarps][2][64];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint16_t* item = items[wid];
  float* const lower = lowers[wid];
  unsigned *const smallest = per_lane[wid][0], *const tally = per_lane[wid][1];
  float* const warp_frames = frames + 32 * wid;
  const repr::FrameCol F{warp_frames + lane, kVertexThreads};
  WarpList redo_list{lists[wid][0]}, w_list{lists[wid][1]};
  const int64_t step = (int64_t)gridDim.x * kVertexThreads;
  int64_t first = ((int64_t)blockIdx.x * kWarps + wid) * 32;  // warp-uniform
  auto grid_of = [&](uint32_t vcell) -> const Grid& {
    return kBatch ? space.grids[ld(space.tile_vol + vcell / kScanTile)] : space.one;
  };
  auto fetch_corners = [&](uint32_t vcell) {
    const Grid& g = grid_of(vcell);
    int i, j, k;
    cell_ijk(g, vcell - g.vbase, i, j, k);
    const float* p = g.f + ((int64_t)k * g.ny + j) * g.nx + i;
    const int64_t sy = g.nx, sz = (int64_t)g.nx * g.ny;
    float* c = corners + threadIdx.x;
#pragma unroll
    for (int q = 0; q < 8; q++)
      cp_async4(c + q * kVertexThreads, p + (q & 1) + (q & 2 ? sy : 0) + (q & 4 ? sz : 0));
  };
  // this iteration's record, crossed edges, rank and cell; the next one's slot
  uint32_t r = 0, crossed = 0, vcell = 0, slot_next = 0;
  int rank = 0;
  if (first + lane < nv) {
    const uint32_t slot = vwork[first + lane];
    rank = vrank[first + lane];
    r = rec[slot];
    crossed = d_case_edges.m[ld(ccase + slot)];
    vcell = slot_cell(cellof, slot);
    fetch_corners(vcell);
  }
  if (first + step + lane < nv) slot_next = vwork[first + step + lane];
  for (; first < nv; first += step) {
    const int64_t vidx = first + lane, ahead = vidx + step;
    const bool valid = vidx < nv, more = ahead < nv;
    uint32_t r_next = 0, cs_next = 0, vcell_next = 0, slot_after = 0;
    int rank_next = 0;
    if (more) {
      r_next = rec[slot_next];
      cs_next = ld(ccase + slot_next);
      vcell_next = slot_cell(cellof, slot_next);
      rank_next = vrank[ahead];
      if (ahead + step < nv) slot_after = vwork[ahead + step];
    }
    int prj = -1;
    ffx::ff iso{0, 0};
    cp_async_wait();
    if (valid) {
      const Grid& g = grid_of(vcell);
#pragma unroll
      for (int q = 0; q < 8; q++) F[q] = corners[q * kVertexThreads + threadIdx.x];
      const uint32_t em = repr::edges_of_rank(rec_map(r), rank, crossed);
      const int n = __popc(em);
      // another contour of three edges excludes samples inside its box (one-pass kernels); in a cell
      // with an unused contour some edges have no rank of their own
      bool redo = rec_unused(r);
      if (rec_nv(r) > 1 && n != 3)
        for (int t = 0; t < rec_nv(r); t++)
          redo = redo || (t != rank && __popc(repr::edges_of_rank(rec_map(r), t, crossed)) == 3);
      iso = ffx::ff{g.iso_f, g.iso_lo};
      if (!redo) prj = repr::vertex_frame(F, em, n, g.iso, iso, g.iso_exact);
    }
    uint32_t crossed_next = 0;
    if (more) {
      crossed_next = d_case_edges.m[cs_next];
      fetch_corners(vcell_next);
    }
    // The search: the lane's first sample, then (shared) its neighbours when that one is not surely valid,
    // then the samples whose in-plane distance is within the smallest upper bound.  smallest[lane] is
    // that bound, tally[lane] counts the samples whose lower bound does not exceed it (a later window or
    // round may lower it further: such a count is too large, never too small) and sums their numbers.
    int q0 = 0;
    if (prj >= 0) q0 = repr::seed_sample(F);
    smallest[lane] = __float_as_uint(INFINITY);
    tally[lane] = 0;
    float seed_lb = INFINITY;
    uint64_t need = 0, seen = 1ull << q0;
    bool ring = false;
    for (int round = 0;; round++) {
      const int c = round ? __popcll(need) : 1;
      int upto = c;  // inclusive scan of the lanes' numbers
      if (round) {
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int y = __shfl_up_sync(kAll, upto, o);
          if (lane >= o) upto += y;
        }
      }
      const int from = upto - c, total = round ? __shfl_sync(kAll, upto, 31) : 32;
      for (int w = 0; w < total; w += kSampleWindow) {
        const int end = min(w + kSampleWindow, total);
        if (round) {
          const int hi = min(upto, end);
          __syncwarp();  // the frames are written, the previous window's entries are read
          if (c <= kFewSamples && hi > w) {
            uint64_t m = need;
            for (int k = from; k < hi; k++, m &= m - 1)
              if (k >= w) item[k - w] = (uint16_t)(lane << 6 | (__ffsll((long long)m) - 1));
          }
          for (unsigned x = __ballot_sync(kAll, c > kFewSamples && from < end && upto > w); x; x &= x - 1) {
            const int o = __ffs(x) - 1;  // the owner
            const unsigned m0 = __shfl_sync(kAll, (unsigned)need, o), m1 = __shfl_sync(kAll, (unsigned)(need >> 32), o);
            const unsigned below = (1u << lane) - 1u;
            const int k0 = __shfl_sync(kAll, from, o) - w + __popc(m0 & below);
            const int k1 = __shfl_sync(kAll, from, o) - w + __popc(m0) + __popc(m1 & below);
            if ((m0 >> lane & 1) && (unsigned)k0 < kSampleWindow) item[k0] = (uint16_t)(o << 6 | lane);
            if ((m1 >> lane & 1) && (unsigned)k1 < kSampleWindow) item[k1] = (uint16_t)(o << 6 | 32 | lane);
          }
          __syncwarp();
        }
        for (int k = w + lane; k < end; k += 32) {
          const int x = round ? item[k - w] : lane << 6 | q0;
          const repr::SampleBound b =
              repr::sample_bound(repr::FrameCol{warp_frames + (x >> 6), kVertexThreads}, x & 63);
          if (round) lower[k - w] = b.lb;
          else seed_lb = b.lb;
          if (b.ub < INFINITY) atomicMin(smallest + (x >> 6), __float_as_uint(b.ub));
        }
        if (round) {
          __syncwarp();
          for (int k = w + lane; k < end; k += 32) {
            const int o = item[k - w] >> 6;
            const float lb = lower[k - w];
            if (lb < INFINITY && lb <= __uint_as_float(smallest[o])) atomicAdd(tally + o, 0x10000u + (item[k - w] & 63u));
          }
        }
      }
      __syncwarp();
      if (!__any_sync(kAll, round == 0 || ring)) break;
      const float m = __uint_as_float(smallest[lane]);
      // the seed not surely valid: its neighbours before everything else
      const bool want = prj >= 0 && (round == 0 || ring);
      ring = want && round == 0 && !(m < INFINITY);
      need = 0;
      if (want) need = (ring ? repr::ring_of(q0) : repr::samples_within(F, m)) & ~seen;
      seen |= need;
    }
    const float m = __uint_as_float(smallest[lane]);
    unsigned near = tally[lane];
    if (seed_lb <= m) near += 0x10000u + q0;
    float p[3] = {0, 0, 0};
    int what = repr::kRedo;
    // one sample's lower bound is within the smallest upper bound: it has that bound, is surely valid
    // and the nearest
    if (prj >= 0 && m < INFINITY && near >> 16 == 1) what = repr::sample_point(F, near & 0xffffu, prj, iso, p);
    __syncwarp();  // the frames are read
    if (valid)
      vp[vidx] =
          make_float4(p[0], p[1], p[2], what == repr::kFound ? 0.0f : (what == repr::kRedo ? 1.0f : 4.0f + prj));
    redo_list.add(list, count, valid && what == repr::kRedo, (uint32_t)vidx);
    w_list.add(wlist, count + 2, valid && what == repr::kW64, (uint32_t)vidx);
    r = r_next;
    crossed = crossed_next;
    vcell = vcell_next;
    rank = rank_next;
    slot_next = slot_after;
  }
  redo_list.finish(list, count);
  w_list.finish(wlist, count + 2);
}

// The points whose last coordinate needs float64 (mostly bilinear values exactly on a float midpoint,
// where a box spans the whole cell and the sample coordinates are eighths), listed by
// dmc_vertex_point_kernel: a few per cent of the vertices, so that there nearly every warp would
// wait for the float64 pipe; here every lane has one.  It is the second half of the search kernel's launch:
// the two lists are apart, and short ones are latency, which here runs beside the search's.  Both passes: 64^3
// blobs 20 -> 14 us, 20-volume batch 62 -> 45 us, 131x117x140 35 -> 17 us, 512^3 noise 0.53 -> 0.48 ms.
__device__ __forceinline__ void last_coordinates(const CellSpace& space, const uint16_t* cellof, const uint32_t* vwork,
                                                 const uint32_t* wlist, unsigned n, float4* vp) {
  // from the grid's end: a short search list keeps its first threads
  for (unsigned a = (gridDim.x - 1 - blockIdx.x) * blockDim.x + threadIdx.x; a < n; a += gridDim.x * blockDim.x) {
    const uint32_t vidx = wlist[a];
    const uint32_t vcell = slot_cell(cellof, vwork[vidx]);
    const Grid& g = space.grids ? space.grids[ld(space.tile_vol + vcell / kScanTile)] : space.one;
    int i, j, k;
    cell_ijk(g, vcell - g.vbase, i, j, k);
    float u[8];
    load_corners(g, i, j, k, u);
    const float4 q = vp[vidx];
    float p[3] = {q.x, q.y, q.z};
    const int prj = (int)q.w - 4;
    const float w = repr::vertex_w_f64(u, g.iso, p, prj);
#pragma unroll
    for (int d = 0; d < 3; d++)
      if (d == 2 - prj) p[d] = w;
    vp[vidx] = make_float4(p[0], p[1], p[2], 0.0f);
  }
}

// The reference's float64 mean point of the contour with edge set em (n edges): its edge points summed in
// the polygon's order.  Rare, out of line.
__device__ __noinline__ repr::Point64 contour_mean_f64(const Grid& g, int i, int j, int k, unsigned cs, uint32_t em,
                                                       int n) {
  float u[8];
  load_corners(g, i, j, k, u);
  const uint64_t c = dmc_polygon(cs, u, g.iso, c_case_contour);
  int at = 0;  // where the contour begins in the word
  for (int t = 0; t < cnt_count(c) && !((em >> (2 * cnt_edge(c, at))) & 1); t++) at += cnt_size(c, t);
  repr::Point64 r{{0, 0, 0}};
  for (int q = 0; q < n; q++) {
    float p[3];
    const int e = cnt_edge(c, at + q);
    repr::local_from_param(e, repr::edge_param_exact(e, u, g.iso), p);
    for (int d = 0; d < 3; d++) r.p[d] += p[d];
  }
  for (int d = 0; d < 3; d++) r.p[d] /= n;
  return r;
}

// The edge sets of a cell whose record does not tell its contours apart (some unused): the contour of
// vertex `rank`, and the other contours of three edges
struct ContourSets {
  uint32_t own, others[3];
  int n_others;
};
__device__ __noinline__ ContourSets contour_sets(const Grid& g, int i, int j, int k, unsigned cs, int rank) {
  float u[8];
  load_corners(g, i, j, k, u);
  const uint64_t c = dmc_polygon(cs, u, g.iso, c_case_contour);
  ContourSets S{0, {0, 0, 0}, 0};
  int flat = 0, seen = 0;
  for (int t = 0; t < cnt_count(c); t++) {
    const int sz = cnt_size(c, t);
    uint32_t m = 0;
    bool used = false;
    for (int q = 0; q < sz; q++) {
      const int e = cnt_edge(c, flat + q);
      m |= 1u << (2 * e);
      used = used || edge_interior(g, i, j, k, e);
    }
    if (used && seen++ == rank) S.own = m;
    else if (sz == 3 && S.n_others < 3) S.others[S.n_others++] = m;
    flat += sz;
  }
  return S;
}
__device__ __forceinline__ int vertex_search_frame(const Grid& g, const repr::FrameCol& F, uint32_t r, int rank,
                                                   unsigned cs, int i, int j, int k, ffx::ff mean[3],
                                                   repr::Exclusion& X, uint32_t& em, int& n) {
  float c[8];
  load_corners(g, i, j, k, c);
#pragma unroll
  for (int q = 0; q < 8; q++) F[q] = c[q];
  ContourSets S{0, {0, 0, 0}, 0};
  if (rec_unused(r)) {
    S = contour_sets(g, i, j, k, cs, rank);
  } else {
    const uint32_t crossed = d_case_edges.m[cs];
    S.own = repr::edges_of_rank(rec_map(r), rank, crossed);
    for (int t = 0; t < rec_nv(r); t++) {
      const uint32_t m = repr::edges_of_rank(rec_map(r), t, crossed);
      if (t != rank && __popc(m) == 3 && S.n_others < 3) S.others[S.n_others++] = m;
    }
  }
  em = S.own;
  n = __popc(em);
  const ffx::ff iso{g.iso_f, g.iso_lo};
  // the boxes of the other contours of three edges
  bool ok = true;
  if (n != 3)
    for (; X.n < S.n_others; X.n++)
      ok = repr::contour_box(F, S.others[X.n], g.iso, iso, g.iso_exact, X.lo[X.n], X.hi[X.n]) && ok;
  if (!ok) return -1;
  const uint32_t own = em;
  const int edges = n;
  auto mean64 = [&g, i, j, k, cs, own, edges]() { return contour_mean_f64(g, i, j, k, cs, own, edges); };
  const int prj = repr::vertex_frame<true>(F, em, n, g.iso, iso, g.iso_exact, mean, mean64);
  if (prj > 0)  // the boxes in the frame's axes: (x, z, y) or (y, z, x)
    for (int t = 0; t < X.n; t++) {
      const float l0 = X.lo[t][0], h0 = X.hi[t][0], l1 = X.lo[t][1], h1 = X.hi[t][1];
      X.lo[t][0] = prj == 1 ? l0 : l1;
      X.hi[t][0] = prj == 1 ? h0 : h1;
      X.lo[t][1] = X.lo[t][2];
      X.hi[t][1] = X.hi[t][2];
      X.lo[t][2] = prj == 1 ? l1 : l0;
      X.hi[t][2] = prj == 1 ? h1 : h0;
    }
  return prj;
}
// The listed vertices that take the whole search: several samples as near as one another (exact ties of
// symmetric contours), contours beside one that excludes samples, no sample surely valid.  The edge
// sets, frame and bounds are the point kernel's; samples are evaluated exactly, in float64 where a
// rounding is not certified.  What is left (no valid sample at 7x7, values at the ends of the float
// range) goes to the one-pass kernels' list, which is empty on most fields.
//
// A list of more than `warp_max` entries takes one thread per vertex (bounds first, then the few
// candidates); a shorter one takes a warp per vertex, the lanes splitting the 49 samples, because one
// thread's search of a contour whose samples all tie lasts as long as the rest of a small call (85 us;
// a warp's 14 us; lists of 19,000 take about as long either way).  Before, all of them took the one-pass
// kernels (64^3 blobs 24 us, 512^3 noise 0.67 ms, 1024x1024x64 saddles 3.3 ms); now 14 us, 0.35 and
// 0.96 ms, and the one-pass kernels get what is left (0.05 and 0.14 ms).
__global__ void __launch_bounds__(kVertexThreads) dmc_vertex_search_kernel(CellSpace space, const uint16_t* cellof,
                                                                           const uint8_t* ccase, const uint32_t* rec,
                                                                           const uint8_t* vrank, const uint32_t* vwork,
                                                                           const uint32_t* list, const uint32_t* wlist,
                                                                           unsigned* count,
                                                                           unsigned warp_max, float4* vp, uint32_t* hard,
                                                                           unsigned long long* stats) {
  pdl_begin();
  constexpr unsigned kAll = 0xffffffffu;
  __shared__ float frames[repr::kFrameFloats * kVertexThreads];
  const repr::FrameCol F{frames + threadIdx.x, kVertexThreads};
  const unsigned total = count[0];
  const bool warp = total <= warp_max;  // the lanes of a warp share a vertex
  const int lane = threadIdx.x & 31;
  int f64 = 0;
  const unsigned tid = blockIdx.x * blockDim.x + threadIdx.x, threads = gridDim.x * blockDim.x;
  for (unsigned a = warp ? tid >> 5 : tid; a < total; a += warp ? threads >> 5 : threads) {
    const uint32_t vidx = list[a];
    const uint32_t slot = vwork[vidx];
    const uint32_t r = rec[slot];
    const unsigned cs = ld(ccase + slot);
    const uint32_t vcell = slot_cell(cellof, slot);
    const Grid& g = space.grids ? space.grids[ld(space.tile_vol + vcell / kScanTile)] : space.one;
    int i, j, k;
    cell_ijk(g, vcell - g.vbase, i, j, k);
    ffx::ff mean[3];
    repr::Exclusion X;
    uint32_t em;
    int n;
    const int prj = vertex_search_frame(g, F, r, vrank[vidx], cs, i, j, k, mean, X, em, n);
    const ffx::ff iso{g.iso_f, g.iso_lo};
    auto mean64 = [&]() { return contour_mean_f64(g, i, j, k, cs, em, n); };
    float p[3] = {0, 0, 0};
    int what = repr::kRedo;
    if (warp) {
      // each lane two of the 49 samples; the winner by distance, then loop order
      repr::LaneBest b = repr::lane_none();
      if (prj >= 0) {  // warp-uniform
        repr::ExactSample s[2];
        float u[2], v[2];
        bool open = false;
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int q = lane + 32 * h;
          s[h].state = 0;
          if (q < 49) {
            u[h] = repr::sample_coord_any(F[repr::kUlo], F[repr::kUhi], q / 7 + 1);
            v[h] = repr::sample_coord_any(F[repr::kVlo], F[repr::kVhi], q - 7 * (q / 7) + 1);
            s[h] = repr::exact_sample(F, u[h], v[h], mean, X, g.iso, iso, f64);
            open = open || s[h].state == 2;
          }
        }
        if (__any_sync(kAll, open)) {
          const repr::Point64 pm = mean64();
#pragma unroll
          for (int h = 0; h < 2; h++)
            if (s[h].state == 2) {
              s[h].d = repr::distance_f64(pm, prj, u[h], v[h], s[h].w);
              f64++;
            }
        }
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const repr::LaneBest x{s[h].d, s[h].w, lane + 32 * h};
          if (s[h].state != 0 && repr::lane_better(x, b)) b = x;
        }
        b = warp_best(b);
        if (b.q != repr::kNoSample) {
          what = repr::kFound;
          repr::frame_point(prj, repr::sample_coord_any(F[repr::kUlo], F[repr::kUhi], b.q / 7 + 1),
                            repr::sample_coord_any(F[repr::kVlo], F[repr::kVhi], b.q - 7 * (b.q / 7) + 1), b.w, p);
        }
      }
      if (lane != 0) continue;
    } else if (prj >= 0) {
      what = repr::search_all(F, prj, mean, X, g.iso, iso, mean64, p, f64);
    }
    if (what == repr::kFound) vp[vidx] = make_float4(p[0], p[1], p[2], 0.0f);
    append(hard, count + 3, what != repr::kFound, vidx);
  }
  if (f64) atomicAdd(stats + 7, (unsigned long long)f64);
  const unsigned open = count[2];
  last_coordinates(space, cellof, vwork, wlist, open, vp);
  if (tid == 0 && open) atomicAdd(stats + 7, 3ull * open);
}

// Positions, normals and local coordinates of the projected vertices.  At most 72 registers (seven blocks per
// SM): the gradients' loads are what it waits for, and at the compiler's 109 only four blocks were there to
// cover them (47 M vertices of the saddle field 2.86 -> 2.26 ms, 2.49 since uncertain normals are told apart;
// 16.6 M with pair normals 1.09 -> 0.91 ms; 8 blocks spill more than they cover).
template <bool kBatch, bool kFF>
__global__ void __launch_bounds__(kVertexThreads, 7) dmc_vertex_finish_kernel(CellSpace space, const uint16_t* cellof,
                                                                         const uint32_t* vwork,
                                                                         int64_t nv, const float4* vp,
                                                                         DmcVertexOut out, int flip_all,
                                                                         unsigned long long* stats) {
  pdl_begin();
  repr::Stats st;
  for (int64_t vidx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; vidx < nv;
       vidx += (int64_t)gridDim.x * blockDim.x) {
    const float4 q = vp[vidx];
    if (q.w != 0.0f) continue;  // done by the one-pass kernel
    const uint32_t vcell = slot_cell(cellof, vwork[vidx]);
    const Grid& g = kBatch ? space.grids[ld(space.tile_vol + vcell / kScanTile)] : space.one;
    const int64_t cell = vcell - g.vbase;
    int i, j, k;
    cell_ijk(g, cell, i, j, k);
    const float p[3] = {q.x, q.y, q.z};
    vertex_outputs<kFF, kFF && !kBatch>(g, i, j, k, cell, p, nullptr, vidx, out, flip_all | (g.flags & kGridFlip), st);
  }
  flush_stats(st, stats);
}

// ------------------------------------------------------------------------------------------
// quads: the cell owning a crossed interior edge (its edge 0, 3 or 8) gathers the vertices of the
// four cells around it.  Slot by the side of the edge's first end vertex (get_vertex_pos,
// cpp_dmc/DualMarchingCubes.h:221-224); colour 3*parity(i,j,k) + axis (:177-180).
// ------------------------------------------------------------------------------------------
// Quad corners are vertex indices within the quad's own volume: the space-wide offsets minus the
// volume's first vertex (the scanned tile offset of its first tile; 0 for a single volume).
//
// One warp per chunk of 32 consecutive listed cells of one tile (the chunk list of the offsets pass),
// a cell per lane.  A cell owns the quads of its crossed interior edges 0, 3 and 8; the cells around
// them are six neighbours, each looked up once and independently (a mask word, then record and offset
// in one load).  A crossed edge makes every cell around it listed.  Walking every tile's 64 possible
// chunks, with up to nine dependent look-ups of three loads each, a smooth field took as long as a dense
// one (512^3 periodic: 0.62 ms of a 2.81 ms call; 2.31 ms with the list).
constexpr int kQuadThreads = 256;
// quad around edge axis A from its four cells' vertices, in the order of their cells: the one across
// both axes, then those below the edge along the second and the first, then the owner
template <int E0, int E1, int E2, int E3>
__device__ __forceinline__ int4 quad_corners(const int32_t v[4], int neg) {
  constexpr int kE[4] = {E0, E1, E2, E3};
  int32_t a[4], b[4];
#pragma unroll
  for (int s = 0; s < 4; s++) {
    a[quad_slot(kE[s], 0)] = v[s];
    b[quad_slot(kE[s], 1)] = v[s];
  }
  return neg ? make_int4(b[0], b[1], b[2], b[3]) : make_int4(a[0], a[1], a[2], a[3]);
}
template <bool kBatch>
__global__ void __launch_bounds__(kQuadThreads) dmc_quad_kernel(CellSpace space, const CellMask* mask,
                                                                const uint16_t* cellof, const uint8_t* ccase,
                                                                const uint2* rv, const int32_t* qoff,
                                                                const unsigned long long* tile_off,
                                                                const uint32_t* chunks, const unsigned* nchunks,
                                                                int32_t* quads, uint8_t* colors) {
  pdl_begin();
  constexpr int kWarps = kQuadThreads / 32;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const unsigned n = *nchunks;
  for (unsigned c = blockIdx.x * kWarps + wid; c < n; c += gridDim.x * kWarps) {
    const uint32_t chunk = ld(chunks + c), slot = (chunk & ~31u) + lane;
    if ((uint32_t)lane > (chunk & 31u)) continue;  // the chunk's number of cells minus one
    const uint2 own = ld(rv + slot);
    if (rec_nq(own.x) == 0) continue;
    const unsigned cs = ld(ccase + slot);
    const uint32_t vc = slot_cell(cellof, slot);
    const Grid& g = kBatch ? space.grids[ld(space.tile_vol + vc / kScanTile)] : space.one;
    const int32_t vfirst = kBatch ? (int32_t)(ld(tile_off + g.vbase / kScanTile) >> 32) : 0;
    int i, j, k;
    cell_ijk(g, vc - g.vbase, i, j, k);
    // from the cell's MC case (bit v: corner v at or above the isovalue): corner 0's side, and the
    // crossings of edges 0 (corners 0-1), 3 (0-2) and 8 (0-4); interior: off the lower borders (the
    // edges at the cell's lower corner never lie on the upper ones)
    const int neg = !(cs & 1u);  // first end vertex below the isovalue
    const bool x = (((cs ^ (cs >> 1)) & 1u) != 0) && j > 0 && k > 0;
    const bool y = (((cs ^ (cs >> 2)) & 1u) != 0) && i > 0 && k > 0;
    const bool z = (((cs ^ (cs >> 4)) & 1u) != 0) && i > 0 && j > 0;
    const uint32_t cx = (uint32_t)g.cx(), cxy = cx * (uint32_t)g.cy();
    // neighbours (0,-1,-1), (0,0,-1), (-1,0,-1), (0,-1,0), (-1,0,0), (-1,-1,0)
    const uint32_t off[6] = {cxy + cx, cxy, cxy + 1, cx, 1, cx + 1};
    const bool want[6] = {x, x || y, y, x || z, y || z, z};
    uint32_t ns[6];
#pragma unroll
    for (int s = 0; s < 6; s++) ns[s] = want[s] ? listed_slot(mask, vc - off[s]) : 0u;
    uint2 o[6];
#pragma unroll
    for (int s = 0; s < 6; s++) o[s] = want[s] ? ld(rv + ns[s]) : make_uint2(0, 0);
    auto vertex = [vfirst](uint2 r, int e) { return (int32_t)r.y - vfirst + rec_rank(r.x, e); };
    int64_t q = ld(qoff + slot);
    const int par = (i & 1) | ((j & 1) << 1) | ((k & 1) << 2);
    if (x) {
      const int32_t v[4] = {vertex(o[0], 6), vertex(o[1], 4), vertex(o[3], 2), vertex(own, 0)};
      reinterpret_cast<int4*>(quads)[q] = quad_corners<6, 4, 2, 0>(v, neg);
      if (colors) colors[q] = (uint8_t)(3 * par);
      q++;
    }
    if (y) {
      const int32_t v[4] = {vertex(o[2], 5), vertex(o[1], 7), vertex(o[4], 1), vertex(own, 3)};
      reinterpret_cast<int4*>(quads)[q] = quad_corners<5, 7, 1, 3>(v, neg);
      if (colors) colors[q] = (uint8_t)(3 * par + 1);
      q++;
    }
    if (z) {
      const int32_t v[4] = {vertex(o[5], 10), vertex(o[3], 11), vertex(o[4], 9), vertex(own, 8)};
      reinterpret_cast<int4*>(quads)[q] = quad_corners<10, 11, 9, 8>(v, neg);
      if (colors) colors[q] = (uint8_t)(3 * par + 2);
    }
  }
}

// ------------------------------------------------------------------------------------------
// twins: the halfedges of the quads of one volume, from the cells.
//
// Two quads share a mesh edge across a grid face: the edge joins a vertex of the cell on either side, and
// its halfedges belong to the quads of the face's crossed interior grid edges.  So a cell settles the
// halfedges across its three lower faces.  With two crossed edges on the face (all but the ambiguous
// ones) they are each other's twins, or one is on the border, has no quad, and leaves the other without;
// with four, those with the same vertex on both sides make up one mesh edge, paired by the build's rules
// for edges of up to four halfedges (halfedges.cu).  The quads' numbers come from the cell and its three
// upper neighbours, which own all nine grid edges on the lower faces.  flag is zero on entry; every twin is
// written once.  deg: the quads around each vertex, its contour's interior edges.
//
// 16.6 M quads: 0.355 ms in place of the 1.19 ms that the general build takes (halfedges counted and listed
// by their origin, lists searched for the opposite ones); 2.2 M: 52 us for 157.  A batch's volumes keep
// that build: their chunks are not listed apart.  Bound by instruction issue (68 %) and the scattered
// 4-byte stores; the edges of three and four halfedges out of line (in line, with the ambiguous faces'
// pairs, 0.60 ms).
// ------------------------------------------------------------------------------------------
__host__ __device__ constexpr int cell_edge(int face, int s) {  // the grid edges of lower face x, y, z
  constexpr int e[3][4] = {{3, 8, 7, 11}, {0, 8, 4, 9}, {0, 3, 2, 1}};
  return e[face][s];
}
__host__ __device__ constexpr int across_edge(int face, int s) {  // the same in the cell across it
  constexpr int e[3][4] = {{1, 9, 5, 10}, {2, 11, 6, 10}, {4, 7, 6, 5}};
  return e[face][s];
}
// Mesh edges of three and four halfedges on one face: h, the numbers; from_cell, bit s: halfedge s starts at
// this cell's vertex; same, bits 4 s + t: halfedges s and t have the same vertices on both sides.
__device__ __noinline__ void pair_crowded_face(int4 h4, unsigned from_cell, unsigned same, int32_t* twin, uint8_t* flag) {
  const int h[4] = {h4.x, h4.y, h4.z, h4.w};
  for (int s = 0; s < 4; s++) {
    const unsigned m = same >> (4 * s) & 15u;
    if (__popc(m) < 3) continue;
    int id[4], c = 0;  // the mesh edge's halfedges by number
    bool from[4];
    for (int t = 0; t < 4; t++) {
      if (!(m >> t & 1)) continue;
      int at = c++;
      for (; at > 0 && id[at - 1] > h[t]; at--) {
        id[at] = id[at - 1];
        from[at] = from[at - 1];
      }
      id[at] = h[t];
      from[at] = from_cell >> t & 1;
    }
    int partner[4] = {-1, -1, -1, -1};
    auto pair = [&](int a, int b) {
      partner[a] = id[b];
      partner[b] = id[a];
    };
    if (c == 3) {
      if (from[0] != from[1]) pair(0, 1);
      else if (from[0] != from[2]) pair(0, 2);
      else pair(1, 2);
    } else if (from[0] != from[1]) {
      pair(0, 1);
      pair(2, 3);
    } else {
      pair(0, 2);
      pair(1, 3);
    }
    for (int a = 0; a < c; a++)
      if (id[a] == h[s]) twin[h[s]] = partner[a];
    flag[h[s]] = c == 3 ? 2 : 1;
  }
}
template <int kFace>
__device__ __forceinline__ void face_twins(unsigned cs, uint32_t crossed, uint32_t in, const int q[12], uint32_t own,
                                           const CellMask* mask, const uint2* rv, uint32_t across, int32_t* twin,
                                           uint8_t* flag) {
  uint32_t face = 0;
#pragma unroll
  for (int s = 0; s < 4; s++) face |= 1u << (2 * cell_edge(kFace, s));
  if (!(in & face)) return;
  int h[4];
  unsigned from_cell = 0, there = 0;
#pragma unroll
  for (int s = 0; s < 4; s++) {
    const int e = cell_edge(kFace, s), a = across_edge(kFace, s);
    // quad corners of the two cells' vertices (by the side of the grid edge's first end), adjacent
    const bool neg = !(cs >> edge_v0(e) & 1u);
    const int r0 = quad_slot(e, 0), r1 = quad_slot(e, 1), a0 = quad_slot(a, 0), a1 = quad_slot(a, 1);
    const bool from0 = ((r0 + 1) & 3) == a0, from1 = ((r1 + 1) & 3) == a1;
    h[s] = 4 * q[e] + (neg ? (from1 ? r1 : a1) : (from0 ? r0 : a0));
    from_cell |= (unsigned)(neg ? from1 : from0) << s;
    there |= (in >> (2 * e) & 1u) << s;
  }
  if (__popc(crossed & face) == 4) {
    const uint2 o = ld(rv + listed_slot(mask, across));
    unsigned key[4], same = 0;
#pragma unroll
    for (int s = 0; s < 4; s++)
      key[s] = (unsigned)rec_rank(own, cell_edge(kFace, s)) << 2 | (unsigned)rec_rank(o.x, across_edge(kFace, s));
    bool crowded = false;
#pragma unroll
    for (int s = 0; s < 4; s++) {
      int other = -1, c = 0;
#pragma unroll
      for (int t = 0; t < 4; t++)
        if ((there >> s & there >> t & 1u) && key[s] == key[t]) {
          same |= 1u << (4 * s + t);
          c++;
          if (t != s) other = h[t];
        }
      if (c == 1 || c == 2) twin[h[s]] = other;
      crowded = crowded || c > 2;
    }
    if (crowded) pair_crowded_face(make_int4(h[0], h[1], h[2], h[3]), from_cell, same, twin, flag);
    return;
  }
  int a = -1, b = -1;
#pragma unroll
  for (int s = 0; s < 4; s++)
    if (there >> s & 1) {
      b = a;
      a = h[s];
    }
  twin[a] = b;
  if (b >= 0) twin[b] = a;
}
__global__ void __launch_bounds__(kQuadThreads) dmc_twin_kernel(CellSpace space, const CellMask* mask,
                                                                const uint16_t* cellof, const uint8_t* ccase,
                                                                const uint2* rv, const int32_t* qoff,
                                                                const uint32_t* chunks, const unsigned* nchunks,
                                                                int32_t* twin, uint8_t* flag, int32_t* deg) {
  pdl_begin();
  constexpr int kWarps = kQuadThreads / 32;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const unsigned n = *nchunks;
  const Grid& g = space.one;
  const uint32_t cx = (uint32_t)g.cx(), cxy = cx * (uint32_t)g.cy();
  for (unsigned c = blockIdx.x * kWarps + wid; c < n; c += gridDim.x * kWarps) {
    const uint32_t chunk = ld(chunks + c), slot = (chunk & ~31u) + lane;
    if ((uint32_t)lane > (chunk & 31u)) continue;  // the chunk's number of cells minus one
    const uint2 own = ld(rv + slot);
    const unsigned cs = ld(ccase + slot);
    const uint32_t vc = slot_cell(cellof, slot);
    const int q0 = ld(qoff + slot);
    const uint32_t crossed = d_case_edges.m[cs];
    int i, j, k;
    cell_ijk(g, vc, i, j, k);
    uint32_t in = crossed;  // the crossed edges that have a quad
    if (!(i >= 1 && j >= 1 && k >= 1 && i <= g.nx - 3 && j <= g.ny - 3 && k <= g.nz - 3))
      for (int e = 0; e < 12; e++)
        if (!edge_interior(g, i, j, k, e)) in &= ~(1u << (2 * e));
    auto has = [in](int e) { return (int)(in >> (2 * e) & 1u); };
    for (int t = 0; t < rec_nv(own.x); t++)
      deg[own.y + t] = __popc(repr::edges_of_rank(rec_map(own.x), t, in));
    // the first quads of the upper neighbours and how many they own, where they own one of the edges
    const bool want[3] = {(has(1) | has(9)) != 0, (has(2) | has(11)) != 0, (has(4) | has(7)) != 0};
    const uint32_t off[3] = {1, cx, cxy};
    uint32_t ns[3];
    int first[3], last[3];
#pragma unroll
    for (int s = 0; s < 3; s++) ns[s] = want[s] ? listed_slot(mask, vc + off[s]) : 0u;
#pragma unroll
    for (int s = 0; s < 3; s++) {
      first[s] = want[s] ? ld(qoff + ns[s]) : 0;
      last[s] = first[s] + (want[s] ? rec_nq(ld(rv + ns[s]).x) : 0) - 1;
    }
    // a cell's quads are those of its edges 0 (x), 3 (y), 8 (z), in this order
    int q[12];
    q[0] = q0;
    q[3] = q0 + has(0);
    q[8] = q[3] + has(3);
    q[9] = last[0];
    q[1] = last[0] - has(9);
    q[2] = first[1];
    q[11] = last[1];
    q[4] = first[2];
    q[7] = first[2] + has(4);
    face_twins<0>(cs, crossed, in, q, own.x, mask, rv, vc - 1u, twin, flag);
    face_twins<1>(cs, crossed, in, q, own.x, mask, rv, vc - cx, twin, flag);
    face_twins<2>(cs, crossed, in, q, own.x, mask, rv, vc - cxy, twin, flag);
  }
}

// ------------------------------------------------------------------------------------------
// host-side launches
// ------------------------------------------------------------------------------------------
int dmc_front_count(const CellSpace& space, DmcScratch& s, int sms, cudaStream_t st, Prof* prof,
                    const TileGate* gates, int ngates) {
  const int64_t tiles = ceil_div(space.n, kScanTile);
  int k = 0;
  {
    Stage t(prof, "dmc_classify", st);
    // the ambiguous cells' list lives in qoff until the offsets kernel writes the quad offsets
    auto classify = [&](int64_t t0, int64_t t1, int z0, int z1) {
      k += launch_point_bits(space, z0, z1, sms, st);
      if (t1 <= t0) return;
      uint32_t* amb = reinterpret_cast<uint32_t*>(s.qoff);
      if (block_per_tile(t1 - t0, sms))
        launch(dmc_classify_kernel<8>, (unsigned)(t1 - t0), kClassifyThreads, st, 
            space, t0, t1, s.rec, s.cellof, s.ccase, s.mask, s.tile_sums, s.stats, amb, s.amb_n);
      else
        launch(dmc_classify_kernel<1>, (unsigned)ceil_div(t1 - t0, kClassifyThreads / 32), kClassifyThreads, st, 
            space, t0, t1, s.rec, s.cellof, s.ccase, s.mask, s.tile_sums, s.stats, amb, s.amb_n);
      k++;
    };
    if (ngates == 0) classify(0, tiles, 0, space.one.nz);
    int64_t t0 = 0;
    int z0 = 0;
    for (int q = 0; q < ngates; q++) {
      cudaStreamWaitEvent(st, gates[q].ready, 0);
      const int64_t t1 = (q == ngates - 1) ? tiles : std::min(gates[q].tile_end, tiles);
      classify(t0, t1, z0, gates[q].z_end);
      t0 = std::max(t0, t1);
      z0 = gates[q].z_end;
    }
    // one wave; the list length is only known on the device, so the grid follows the cell count
    static const int r_amb = resident_blocks(dmc_amb_kernel, 128);
    launch(dmc_amb_kernel, (unsigned)wave_grid(r_amb, sms, 16, ceil_div(space.n, 128), 128), 128, st, 
        space, s.cellof, s.rec, s.tile_sums, reinterpret_cast<const uint32_t*>(s.qoff), s.amb_n);
    k++;
  }
  Stage t(prof, "dmc_scan", st);
  scan_tile_sums(s.tile_sums, tiles, s.totals, st);
  return k + 1;
}

int dmc_front_offsets(const CellSpace& space, DmcScratch& s, cudaStream_t st, Prof* prof) {
  Stage t(prof, "dmc_scan", st);
  const int64_t tiles = ceil_div(space.n, kScanTile);
  launch(dmc_offsets_kernel, (unsigned)ceil_div(tiles, kOffsetWarps), 32 * kOffsetWarps, st, s.mask, s.rec, s.tile_sums,
         tiles, s.rv, s.qoff, s.vwork, s.vrank, s.chunks, s.amb_n + 1, s.totals, s.vcap);
  return 1;
}

int dmc_front_emit(const CellSpace& space, DmcScratch& s, DmcVertexOut vo, int64_t nv, int32_t* quads,
                   uint8_t* colors, int flip, const Tuning& tu, cudaStream_t st, Prof* prof) {
  const int sms = tu.sms;
  const int64_t n = space.n;
  // per-vertex grids: whole waves of each kernel's resident blocks
  static const int r_point = resident_blocks(dmc_vertex_point_kernel<false>, kVertexThreads);
  static const int r_point_batch = resident_blocks(dmc_vertex_point_kernel<true>, kVertexThreads);
  static const int r_quad = resident_blocks(dmc_quad_kernel<false>, kQuadThreads);
  static const int r_quad_batch = resident_blocks(dmc_quad_kernel<true>, kQuadThreads);
  auto vgrid = [&](int resident) {
    return (unsigned)wave_grid(resident, sms, tu.vertex_blocks_per_sm, nv, kVertexThreads);
  };
  {
    Stage t(prof, "dmc_vertex_point", st);
    if (space.grids)
      launch(dmc_vertex_point_kernel<true>, vgrid(r_point_batch), kVertexThreads, st, 
          space, s.cellof, s.ccase, s.rec, s.vrank, s.vwork, nv, s.vp, s.fb_list, s.w_list, s.fb_count);
    else
      launch(dmc_vertex_point_kernel<false>, vgrid(r_point), kVertexThreads, st, 
          space, s.cellof, s.ccase, s.rec, s.vrank, s.vwork, nv, s.vp, s.fb_list, s.w_list, s.fb_count);
    // the lists' lengths are only known on the device: one wave, sized for a tenth of the vertices
    // (the search takes a warp per vertex when few are listed, so as many warps as vertices may use)
    static const int r_search = resident_blocks(dmc_vertex_search_kernel, kVertexThreads);
    launch(dmc_vertex_search_kernel, (unsigned)wave_grid(r_search, sms, 1, nv, kVertexThreads), kVertexThreads, st, 
        space, s.cellof, s.ccase, s.rec, s.vrank, s.vwork, s.fb_list, s.w_list, s.fb_count,
        (unsigned)std::min<int64_t>(tu.warp_list_max, 0x7fffffff), s.vp, s.hard_list, s.stats);
  }
  {
    Stage t(prof, "dmc_vertex_finish", st);
#define DMC_FINISH(B, F)                                                                              \
  {                                                                                                   \
    static const int res = resident_blocks(dmc_vertex_finish_kernel<B, F>, kVertexThreads);           \
    launch(dmc_vertex_finish_kernel<B, F>, vgrid(res), kVertexThreads, st, space, s.cellof, s.vwork, nv, s.vp, vo, flip, \
                                                                          s.stats);                   \
  }
    // the pair normals' storing path only when some volume keeps them (simplification)
    if (space.grids) {
      if (vo.n64) DMC_FINISH(true, true) else DMC_FINISH(true, false)
    } else {
      if (vo.n64) DMC_FINISH(false, true) else DMC_FINISH(false, false)
    }
#undef DMC_FINISH
  }
  {
    // the listed vertices: one thread each with every float64 fallback, the 26x26 retries one warp
    // each; a short list (small calls) entirely one warp per vertex
    Stage t(prof, "dmc_vertex", st);
    const unsigned warp_max = (unsigned)std::min<int64_t>(tu.warp_list_max, 0x7fffffff);
    static const int r_vertex = resident_blocks(dmc_vertex_kernel, kVertexThreads);
    const unsigned fb = (unsigned)wave_grid(r_vertex, sms, 8, nv, kVertexThreads);
    launch(dmc_vertex_kernel, fb, kVertexThreads, st, space, s.cellof, s.vrank, s.vwork, s.hard_list, s.fb_count + 3, s.tail_list,
                                                      s.fb_count + 1, warp_max, vo, flip, s.stats);
    launch(dmc_vertex_warp_kernel, (unsigned)std::max(1, sms * 3), kVertexThreads, st, 
        space, s.cellof, s.vrank, s.vwork, s.hard_list, s.fb_count + 3, s.tail_list, s.fb_count + 1, warp_max, vo, flip,
        s.stats);
  }
  Stage t(prof, "dmc_quad", st);
  // one wave: the number of chunks is only known on the device
#define DMC_QUADS(B, R)                                                                                              \
  launch(dmc_quad_kernel<B>, (unsigned)wave_grid(R, sms, tu.quad_blocks_per_sm, ceil_div(n, 32), kQuadThreads / 32),  kQuadThreads, st, space, s.mask, s.cellof, s.ccase, s.rv, s.qoff, s.tile_sums, s.chunks, \
                                              s.amb_n + 1, quads, colors)
  if (space.grids) DMC_QUADS(true, r_quad_batch);
  else DMC_QUADS(false, r_quad);
#undef DMC_QUADS
  return 6;
}

int dmc_front_twins(const CellSpace& space, const DmcScratch& s, int32_t* twin, uint8_t* flag, int32_t* deg, int sms,
                    cudaStream_t st) {
  static const int res = resident_blocks(dmc_twin_kernel, kQuadThreads);
  launch(dmc_twin_kernel, (unsigned)wave_grid(res, sms, 32, ceil_div(space.n, 32), kQuadThreads / 32), kQuadThreads, st,
         space, s.mask, s.cellof, s.ccase, s.rv, s.qoff, s.chunks, s.amb_n + 1, twin, flag, deg);
  return 1;
}

}  // namespace tmc
