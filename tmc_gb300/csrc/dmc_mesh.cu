// DMC mesh post-processing on the GPU: face colouring, vertex valence, P3X3Y simplification
// (colour pass and isolated pass), P3333 simplification, final halfedges and the quad -> triangle
// split.  Follows cpp_dmc/DualMarchingCubes.cpp:488-1460 step by step; every sequential loop of
// the reference is shown to be order-independent (or made so) where it is parallelised:
//
//  * colorFaces (:714-844): faces are reduced class by class (inherited colours 5..23, then the
//    faces whose inherited colour is 4).  Inherited colour = 3*parity(lower grid point) + axis,
//    and two faces sharing an edge come from two grid edges of one grid face, so they never share
//    an inherited colour: inside one class no face reads another face's new colour.  One launch
//    per class, or per group of classes that never meet on a front-end mesh (color_class).
//  * mergeVertices3X3Y (:916-1094): a merge reads valence >= 5 vertices and writes valence-3
//    vertices, so reads never see writes.  Several faces writing the same vertex resolve to the
//    highest face index (the reference's last write), via atomicMax claims.
//  * mark3333 (:1189-1322): marked faces cannot be adjacent and their vertices have valence 3, so
//    no vertex is written twice; the neighbour flags are idempotent.
//  * removals (removeVertices3X3Y / removeQuadrilaterals3X3Y, their 3333 pair): the passes run in
//    place, killing faces and re-targeting corners while every index stays; the halfedges are built
//    once and repaired around the touched vertices after each pass (halfedges.cu,
//    repair_halfedges), and one order-preserving compaction after the last pass gives the
//    reference's numbering, since each of its per-pass compactions keeps the order of what remains.
#include <cmath>

#include "../../include/tmc_gb300.h"
#include "color_groups.h"
#include "dmc_mesh.h"
#include "ffloat.cuh"
#include "halfedges.h"
#include "host_wait.h"
#include "libm_acosf.h"
#include "scan.cuh"

namespace tmc {

namespace {

inline unsigned grid_for(int64_t n, int sms) {
  return (unsigned)std::max<int64_t>(1, std::min<int64_t>(ceil_div(n, 256), (int64_t)sms * 8));
}

// (kernels on grids of grid_for keep to the 32 registers at which its blocks are one wave)
#define FOR_EACH(i, n) for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < (n); i += (int64_t)gridDim.x * blockDim.x)

// Halfedges of a quad mesh: halfedge r of face f is 4f + r; its origin is quad corner r and its
// next 4f + (r+1)%4 (implicit); twins and flags come from the halfedge build.
struct HeView {
  const int32_t* q;
  const int32_t* twin;
  const uint8_t* flag;
};
__device__ __forceinline__ int he_twin(const HeView& he, int64_t h) { return he.twin[h]; }
__device__ __forceinline__ int he_face(const HeView&, int64_t h) { return (int)(h >> 2); }
__device__ __forceinline__ int he_origin(const HeView& he, int64_t h) { return he.q[h]; }
__device__ __forceinline__ int he_flag(const HeView& he, int64_t h) { return he.flag[h]; }
__device__ __forceinline__ int64_t he_next(int64_t h) { return (h & ~(int64_t)3) | ((h + 1) & 3); }

// collectNeighbors (cpp_dmc/DualMarchingCubes.cpp:673-702); halfedge r of face f is 4f + r
__device__ __forceinline__ void neighbors(const HeView& he, int64_t f, int n[4]) {
#pragma unroll
  for (int r = 0; r < 4; r++) {
    const int t = he_twin(he, 4 * f + r);
    n[r] = (t != -1) ? he_face(he, t) : -1;
  }
}

// isNonManifold (:874-885)
__device__ __forceinline__ bool non_manifold(const HeView& he, int64_t f) {
  return he_flag(he, 4 * f) == 1 || he_flag(he, 4 * f + 1) == 1 || he_flag(he, 4 * f + 2) == 1 ||
         he_flag(he, 4 * f + 3) == 1;
}

// ---------------------------------------------------------------------------------------------
// colouring
// ---------------------------------------------------------------------------------------------
// The group a face's inherited colour is reduced in, -1 for colours 0..3.  Of any mesh: a group per colour,
// 5..23 in order, then 4.  Of the front end's own (kFront): inherited colours are those of grid edges, and two
// faces share an edge only when their grid edges lie on one grid face, so most pairs of colours never meet;
// a colour's group is one after the last earlier colour it can meet, which leaves 14 groups, each as
// independent as one colour (tests/test_color_groups_cpu.py derives them).  Small meshes pay per launch:
// 0.4 M faces 57 -> 39 us, 2.2 M 84 -> 65 us; 16.6 M 0.26 ms either way.
constexpr int kColorGroups = 20, kFrontGroups = 14;
template <bool kFront>
__device__ __forceinline__ int color_class(int c) {
  if (!kFront) return c > 4 ? c - 5 : (c == 4 ? 19 : -1);
  // group of colours 4..23, four bits each: 4..19, then 20..23
  constexpr uint64_t lo = TMC_FRONT_GROUPS_LO, hi = TMC_FRONT_GROUPS_HI;
  return c < 4 ? -1 : (int)((c < 20 ? lo >> (4 * (c - 4)) : hi >> (4 * (c - 20))) & 15);
}

// Class histograms and lists are aggregated per block (shared-memory ranks, one global atomic per
// class and block): 20 global counters hit by every face serialise the whole pass otherwise.  The
// order of faces within a class list does not matter (faces of one class never touch).
constexpr int kColorThreads = 256, kColorItems = 8, kColorTile = kColorThreads * kColorItems;

template <bool kFront>
__global__ void __launch_bounds__(kColorThreads) color_count_kernel(const uint8_t* col, int64_t nq, int32_t* cnt) {
  pdl_begin();
  __shared__ int h[20];
  if (threadIdx.x < 20) h[threadIdx.x] = 0;
  __syncthreads();
  const int64_t base = (int64_t)blockIdx.x * kColorTile;
#pragma unroll
  for (int s = 0; s < kColorItems; s++) {
    const int64_t f = base + s * kColorThreads + threadIdx.x;
    if (f < nq) {
      const int k = color_class<kFront>(col[f]);
      if (k >= 0) atomicAdd(&h[k], 1);
    }
  }
  __syncthreads();
  if (threadIdx.x < 20 && h[threadIdx.x]) atomicAdd(cnt + threadIdx.x, h[threadIdx.x]);
}

__global__ void color_offsets_kernel(const int32_t* cnt, int32_t* off, int32_t* cursor) {
  pdl_begin();
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    int s = 0;
    for (int k = 0; k < 20; k++) {
      off[k] = s;
      cursor[k] = s;
      s += cnt[k];
    }
    off[20] = s;
  }
}

template <bool kFront>
__global__ void __launch_bounds__(kColorThreads) color_scatter_kernel(const uint8_t* col, int64_t nq, int32_t* cursor,
                                                                     int32_t* list) {
  pdl_begin();
  __shared__ int h[20], at[20];
  if (threadIdx.x < 20) h[threadIdx.x] = 0;
  __syncthreads();
  const int64_t base = (int64_t)blockIdx.x * kColorTile;
  int ks[kColorItems], rs[kColorItems];
#pragma unroll
  for (int s = 0; s < kColorItems; s++) {
    const int64_t f = base + s * kColorThreads + threadIdx.x;
    ks[s] = (f < nq) ? color_class<kFront>(col[f]) : -1;
    rs[s] = (ks[s] >= 0) ? atomicAdd(&h[ks[s]], 1) : 0;
  }
  __syncthreads();
  if (threadIdx.x < 20 && h[threadIdx.x]) at[threadIdx.x] = atomicAdd(cursor + threadIdx.x, h[threadIdx.x]);
  __syncthreads();
#pragma unroll
  for (int s = 0; s < kColorItems; s++)
    if (ks[s] >= 0) list[at[ks[s]] + rs[s]] = (int32_t)(base + s * kColorThreads + threadIdx.x);
}

__global__ void color_reduce_kernel(HeView he, uint8_t* col, const int32_t* list, const int32_t* off, int k,
                                    int lim) {
  pdl_begin();
  const int64_t b = off[k], e = off[k + 1];
  FOR_EACH(idx, e - b) {
    const int f = list[b + idx];
    int n[4], nc[4];
    neighbors(he, f, n);
#pragma unroll
    for (int r = 0; r < 4; r++) nc[r] = (n[r] != -1) ? (int)col[n[r]] : -1;
    for (int c = 0; c <= lim; c++) {
      if (nc[0] != c && nc[1] != c && nc[2] != c && nc[3] != c) {
        col[f] = (uint8_t)c;
        break;
      }
    }
  }
}

// ---------------------------------------------------------------------------------------------
// valence and patterns
// ---------------------------------------------------------------------------------------------
// vertexValence (:847-871): outgoing halfedges, +1 at the origin of a boundary halfedge's next.
// The outgoing count is the out-degree the halfedge build just counted; only boundary halfedges
// (rare) add with atomics.
// One thread per face (16-byte twin loads; the corners only for a face with a boundary halfedge);
// alive: the live faces (all when NULL).  A caller's quads need not be 16-byte aligned.
__global__ void __launch_bounds__(256, 8) valence_boundary_kernel(HeView he, int64_t nq, int32_t* val, const uint8_t* alive) {
  pdl_begin();
  const bool vec = ((reinterpret_cast<uintptr_t>(he.q) | reinterpret_cast<uintptr_t>(he.twin)) & 15) == 0;
  FOR_EACH(f, nq) {
    if (alive && !alive[f]) continue;
    const int4 t = vec ? reinterpret_cast<const int4*>(he.twin)[f]
                       : make_int4(he.twin[4 * f], he.twin[4 * f + 1], he.twin[4 * f + 2], he.twin[4 * f + 3]);
    if (t.x != -1 && t.y != -1 && t.z != -1 && t.w != -1) continue;
    const int4 q = vec ? reinterpret_cast<const int4*>(he.q)[f]
                       : make_int4(he.q[4 * f], he.q[4 * f + 1], he.q[4 * f + 2], he.q[4 * f + 3]);
    // a boundary halfedge adds one at the origin of its next, the following corner
    if (t.x == -1) atomicAdd(val + q.y, 1);
    if (t.y == -1) atomicAdd(val + q.z, 1);
    if (t.z == -1) atomicAdd(val + q.w, 1);
    if (t.w == -1) atomicAdd(val + q.x, 1);
  }
}

// mark3X3Y (:889-913)
__global__ void __launch_bounds__(256, 8) mark3x3y_kernel(const int4* q, int64_t nq, const int32_t* val, uint8_t* p, const uint8_t* alive) {
  pdl_begin();
  FOR_EACH(f, nq) {
    const int4 v = q[f];
    if (!alive[f]) {
      p[f] = 0;
      continue;
    }
    const int a = val[v.x], b = val[v.y], c = val[v.z], d = val[v.w];
    p[f] = (a == 3 && b >= 5 && c == 3 && d >= 5) || (a >= 5 && b == 3 && c >= 5 && d == 3);
  }
}

// mergeVertices3X3Y, both variants (:916-1094): decide removal, claim written vertices
__global__ void __launch_bounds__(256, 8) merge_claim_kernel(HeView he, int64_t nq, const uint8_t* p, const int32_t* val,
                                   const uint8_t* col, int color_pass, uint8_t* branch, int32_t* own_pos,
                                   int32_t* own_rm) {
  pdl_begin();
  FOR_EACH(f, nq) {
    branch[f] = 0;
    if (!p[f]) continue;
    int n[4];
    neighbors(he, f, n);
    if (color_pass) {
      bool bad = false;
      for (int r = 0; r < 4; r++) {
        if (n[r] >= 0 && non_manifold(he, n[r])) bad = true;
        if (n[r] < 0) bad = true;
      }
      if (bad) continue;
      const int c = col[f];
      bool ok = true;
      for (int r = 0; r < 4; r++)
        if (p[n[r]] && (int)col[n[r]] <= c) ok = false;
      if (!ok) continue;
    } else {
      bool skip = false;
      for (int r = 0; r < 4; r++)
        if (n[r] != -1 && non_manifold(he, n[r])) skip = true;
      for (int r = 0; r < 4; r++)
        if (n[r] != -1 && p[n[r]]) skip = true;
      if (skip) continue;
    }
    const int v0 = he_origin(he, 4 * f), v1 = he_origin(he, 4 * f + 1), v2 = he_origin(he, 4 * f + 2),
              v3 = he_origin(he, 4 * f + 3);
    const int a = val[v0], b = val[v1], c2 = val[v2], d = val[v3];
    if (a == 3 && b >= 5 && c2 == 3 && d >= 5) {
      branch[f] = 1;
      atomicMax(own_pos + v0, (int32_t)f);
      atomicMax(own_rm + v2, (int32_t)f);
    } else if (a >= 5 && b == 3 && c2 >= 5 && d == 3) {
      branch[f] = 2;
      atomicMax(own_pos + v1, (int32_t)f);
      atomicMax(own_rm + v3, (int32_t)f);
    }
  }
}

// The normals kept while simplifying are float pairs (hi, lo) in the 8-byte slots of n64: the front
// end computes them in float-float (within ~2^-40 of the reference's float64 normals), and only their
// float32 roundings leave the library, so they are stored as computed.
__device__ __forceinline__ double pair_to_double(const double* n64, int64_t e) {
  const float2 x = reinterpret_cast<const float2*>(n64)[e];
  return (double)x.x + (double)x.y;
}

// The normal halfway between two, normalised, in float64.  Rare, out of line.
__device__ __noinline__ void middle_normal_f64(double* n64, int dst, int a, int b) {
  double m[3];
  for (int d = 0; d < 3; d++) {
    const double na = pair_to_double(n64, 3 * (int64_t)a + d), nb = pair_to_double(n64, 3 * (int64_t)b + d);
    m[d] = na + 0.5 * (nb - na);
  }
  const double s = sqrt(m[0] * m[0] + m[1] * m[1] + m[2] * m[2]);
  float2* n2 = reinterpret_cast<float2*>(n64);
  for (int d = 0; d < 3; d++) {
    const ffx::ff x = ffx::ff_from_double(m[d] / s);
    n2[3 * (int64_t)dst + d] = make_float2(x.hi, x.lo);
  }
}
// float64 positions and float-pair normals: the float32 outputs are their roundings, written once after the
// last pass.  The positions are the reference's float64 operations; the normals' interpolation and
// normalisation stay in float pairs (within 2^-43, as the front end's are within 2^-40 of the reference's),
// unless the two nearly cancel: a root and three divisions on the float64 pipe, 1/57 of the float32 rate,
// were most of this pass (512^3 noise, both passes: 0.29 -> 0.21 ms; 131x117x140: 49 -> 14 us).
__device__ __forceinline__ void midpoint(double* v64, double* n64, int dst, int a, int b) {
  const float2* n2 = reinterpret_cast<const float2*>(n64);
  ffx::ff m[3];
  double x[3];
#pragma unroll
  for (int d = 0; d < 3; d++) {
    const double pa = v64[3 * (int64_t)a + d], pb = v64[3 * (int64_t)b + d];
    const float2 na = n2[3 * (int64_t)a + d], nb = n2[3 * (int64_t)b + d];
    x[d] = pa + 0.5 * (pb - pa);
    const ffx::ff t = ffx::ff_sub(ffx::ff{nb.x, nb.y}, ffx::ff{na.x, na.y});
    m[d] = ffx::ff_add(ffx::ff{na.x, na.y}, ffx::ff{0.5f * t.hi, 0.5f * t.lo});
  }
#pragma unroll
  for (int d = 0; d < 3; d++) v64[3 * (int64_t)dst + d] = x[d];
  const ffx::ff dot =
      ffx::ff_add(ffx::ff_add(ffx::ff_mul(m[0], m[0]), ffx::ff_mul(m[1], m[1])), ffx::ff_mul(m[2], m[2]));
  if (!(dot.hi > 0x1p-8f && dot.hi < 2.0f)) {  // unit normals: less than 1/8 of one is left
    middle_normal_f64(n64, dst, a, b);
    return;
  }
  // 1 / sqrt(dot): float estimate and one Newton step in float pairs
  const float r0 = rsqrtf(dot.hi);
  const ffx::ff h = ffx::ff_mul_f(ffx::ff_mul_f(dot, r0), r0);
  const ffx::ff r = ffx::ff_mul_f(ffx::ff_sub(ffx::ff_from(1.5f), ffx::ff_mul_f(h, 0.5f)), r0);
  float2* out = reinterpret_cast<float2*>(n64);
#pragma unroll
  for (int d = 0; d < 3; d++) {
    const ffx::ff y = ffx::ff_mul(m[d], r);
    out[3 * (int64_t)dst + d] = make_float2(y.hi, y.lo);
  }
}

// What a pass does to a vertex, in one byte (two arrays cost the next pass two gathers per corner).  Two faces
// may mark one vertex differently, hence the atomic.
constexpr unsigned kTouched = 1, kRemoved = 2;
__device__ __forceinline__ void mark(uint8_t* marks, int v, unsigned m) {
  atomicOr(reinterpret_cast<unsigned*>(marks) + (v >> 2), m << (8 * (v & 3)));
}

// Marks the removed vertices and lists the midpoint merges (destination, two sources); the
// midpoints run densely in midpoint_kernel (a few merging faces per warp would otherwise
// pay the float64 pipe for the whole warp).  Each destination has one owner, and the sources are
// never destinations (valence >= 5 vs valence 3), so the merges are independent.
// marks: the valence-3 corners of the removed faces (merge targets and removed vertices) are touched, the
// vertices the halfedge repair re-pairs around; valive: the removed vertices die.
// The jobs of a block's faces are gathered in shared memory and appended with one global atomic
// per block and iteration (per-warp appends to the one counter serialise on it).
constexpr int kMergeThreads = 256;
__global__ void __launch_bounds__(kMergeThreads) merge_apply_kernel(HeView he, int64_t nq, const uint8_t* branch,
                                                                   const int32_t* own_pos, const int32_t* own_rm,
                                                                   int32_t* vm_second, uint8_t* em, int4* jobs,
                                                                   unsigned* njobs, uint8_t* marks, uint8_t* valive) {
  pdl_begin();
  __shared__ int4 s_jobs[kMergeThreads];
  __shared__ unsigned s_n, s_base;
  // block-uniform loop: every thread reaches the barriers
  for (int64_t f0 = (int64_t)blockIdx.x * kMergeThreads; f0 < nq; f0 += (int64_t)gridDim.x * kMergeThreads) {
    if (threadIdx.x == 0) s_n = 0;
    __syncthreads();
    const int64_t f = f0 + threadIdx.x;
    if (f < nq) {
      const uint8_t br = branch[f];
      em[f] = br != 0;
      if (br) {
        const int v0 = he_origin(he, 4 * f), v1 = he_origin(he, 4 * f + 1), v2 = he_origin(he, 4 * f + 2),
                  v3 = he_origin(he, 4 * f + 3);
        bool job = false;
        int4 jv = make_int4(0, 0, 0, 0);
        if (br == 1) {
          if (own_pos[v0] == f) {
            job = true;
            jv = make_int4(v0, v1, v3, 0);
          }
          mark(marks, v0, kTouched);
          mark(marks, v2, kTouched | kRemoved);
          valive[v2] = 0;
          if (own_rm[v2] == f) vm_second[v2] = v0;
        } else {
          if (own_pos[v1] == f) {
            job = true;
            jv = make_int4(v1, v0, v2, 0);
          }
          mark(marks, v1, kTouched);
          mark(marks, v3, kTouched | kRemoved);
          valive[v3] = 0;
          if (own_rm[v3] == f) vm_second[v3] = v1;
        }
        if (job) s_jobs[atomicAdd(&s_n, 1u)] = jv;
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) s_base = s_n ? atomicAdd(njobs, s_n) : 0u;
    __syncthreads();
    if (threadIdx.x < s_n) jobs[s_base + threadIdx.x] = s_jobs[threadIdx.x];
    __syncthreads();  // s_n and s_jobs are read before the next iteration resets them
  }
}

__global__ void midpoint_kernel(const int4* jobs, const unsigned* njobs, double* v64, double* n64) {
  pdl_begin();
  const int64_t nj = *njobs;
  FOR_EACH(a, nj) {
    const int4 j = jobs[a];
    midpoint(v64, n64, j.x, j.y, j.z);
  }
}

// The float32 positions and normals of the simplified mesh: the roundings of its float64 ones (the
// front end writes float32 values that are the same roundings, so that the passes only carry the
// float64 arrays).
__global__ void float_outputs_kernel(const double* v64, const double* n64, int64_t n, float* v, float* nf) {
  pdl_begin();
  const float2* n2 = reinterpret_cast<const float2*>(n64);
  FOR_EACH(e, n) {
    v[e] = (float)v64[e];
    nf[e] = n2[e].x;  // a normalised pair's high part is its float32 rounding
  }
}

// ---------------------------------------------------------------------------------------------
// compaction helpers
// ---------------------------------------------------------------------------------------------

// removeVertices3X3Y / removeVertices3333 (:1096-1112, :1324-1338): kept vertices move to their
// new index (idx[i] - idx[0]), which becomes their map entry.  One thread per vertex component (x, y or z):
// every load and store is unit-stride across the warp.
// Writes what the result keeps: the float32 positions and normals (roundings of the float64 positions and
// float-pair normals) and, when they are an output (v64o), the float64 positions.  16.6 M vertices, 12 M
// kept: 349 us with the float64 positions and the normals' pairs copied along (nothing reads them), 227 us.
__global__ void __launch_bounds__(256, 8) gather_vertices_kernel(const uint8_t* keep, const int32_t* idx, int64_t nv, const double* v64,
                                       const double* n64, double* v64o, int32_t* map, int64_t cap, unsigned* overflow,
                                       float* vo, float* no) {
  pdl_begin();
  const int first = idx[0];
  FOR_EACH(e, 3 * nv) {
    const uint32_t i = (uint32_t)e / 3u, d = (uint32_t)e - 3u * i;  // 3 nv < 2^32
    // all four loads before the first use: a third of the vertices goes, but a component read in vain
    // costs less than one waited for
    const uint8_t k = keep[i];
    const int64_t o = (int64_t)idx[i] - first;
    const double x = v64[e];
    const float nn = reinterpret_cast<const float2*>(n64)[e].x;
    if (!k) continue;
    if (o < 0 || o >= cap) {
      if (d == 0) atomicAdd(overflow, 1u);
      continue;
    }
    if (v64o) v64o[3 * o + d] = x;
    vo[3 * o + d] = (float)x;
    no[3 * o + d] = nn;
    if (d == 0) map[i] = (int32_t)o;
  }
}

// A killed face's corners that stay clean lose one outgoing halfedge each.
// A live face's corner x, now y, is marked for the halfedge repair: y is dirty when x was touched by the
// pass, and then its out-degree is recounted from zero.
__device__ __forceinline__ void killed_corner(int x, unsigned m, int32_t* deg) {
  if (!(m & kTouched)) atomicSub(deg + x, 1);
}
__device__ __forceinline__ void live_corner(int y, unsigned m, uint8_t* dirty, int32_t* deg) {
  if ((m & kTouched) && y >= 0) {
    dirty[y] = 1;
    deg[y] = 0;
  }
}

// removeVertices3X3Y + removeQuadrilaterals3X3Y (:1096-1137) in place: the merged faces die, the
// corners on removed vertices move to their merge target (which a merge always keeps: the faces
// around a valence-3 vertex are pairwise adjacent and no two adjacent faces merge in one pass).
// Faces and vertices keep their indices; the compaction runs once after the last pass.
// Bound by the latency of the corners' gathers (the four marks are loaded together): 16.6 M faces 216 -> 143 us
// in the first pass, 156 -> 85 us in the second, 178 -> 122 us for apply_3333_kernel, with two bytes per
// corner and the corners one by one before.
__global__ void __launch_bounds__(256, 8) apply_3x3y_kernel(int4* q, int64_t nq, uint8_t* alive, const uint8_t* em, const uint8_t* marks,
                                  const int32_t* vm_second, uint8_t* dirty, int32_t* deg) {
  pdl_begin();
  FOR_EACH(f, nq) {
    const uint8_t a = alive[f], e = em[f];
    const int4 c = q[f];
    if (!a) continue;
    const unsigned m0 = marks[c.x], m1 = marks[c.y], m2 = marks[c.z], m3 = marks[c.w];
    if (e) {
      alive[f] = 0;
      killed_corner(c.x, m0, deg);
      killed_corner(c.y, m1, deg);
      killed_corner(c.z, m2, deg);
      killed_corner(c.w, m3, deg);
      continue;
    }
    if (!((m0 | m1 | m2 | m3) & kTouched)) continue;  // a removed vertex is a touched one
    const int4 y = make_int4(m0 & kRemoved ? vm_second[c.x] : c.x, m1 & kRemoved ? vm_second[c.y] : c.y,
                             m2 & kRemoved ? vm_second[c.z] : c.z, m3 & kRemoved ? vm_second[c.w] : c.w);
    if ((m0 | m1 | m2 | m3) & kRemoved) q[f] = y;
    live_corner(y.x, m0, dirty, deg);
    live_corner(y.y, m1, dirty, deg);
    live_corner(y.z, m2, dirty, deg);
    live_corner(y.w, m3, dirty, deg);
  }
}

// mark3333 (:1189-1322)
__global__ void __launch_bounds__(256, 8) mark3333_kernel(HeView he, int64_t nq, const int32_t* val, uint8_t* p3, uint8_t* rflag,
                                int32_t* vm1, uint8_t* marks, const uint8_t* alive, uint8_t* valive) {
  pdl_begin();
  FOR_EACH(f, nq) {
    if (!alive[f] || non_manifold(he, f)) continue;
    int vq[4], fo[4], vo[4];
    for (int r = 0; r < 4; r++) vq[r] = he_origin(he, 4 * f + r);
    if (val[vq[0]] != 3 || val[vq[1]] != 3 || val[vq[2]] != 3 || val[vq[3]] != 3) continue;
    bool boundary = false;
    for (int r = 0; r < 4; r++) {
      const int twin = he_twin(he, 4 * f + r);
      if (twin == -1) {
        boundary = true;
        break;
      }
      fo[r] = he_face(he, twin);
      const int64_t nx = he_next(he_next(twin));
      vo[r] = he_origin(he, nx);
    }
    if (boundary) continue;
    bool nm = false;
    for (int r = 0; r < 4; r++)
      if (non_manifold(he, fo[r])) nm = true;
    if (nm) continue;
    const int a = val[vo[0]], b = val[vo[1]], c = val[vo[2]], d = val[vo[3]];
    if ((a == 3 && b == 3) || (b == 3 && c == 3) || (c == 3 && d == 3) || (d == 3 && a == 3)) continue;
    if (a == 3 || b == 3 || c == 3 || d == 3) continue;
    if (a == 4 && b == 4 && c == 4 && d == 4) continue;
    for (int r = 0; r < 4; r++) {
      vm1[vq[r]] = vo[r];
      marks[vq[r]] = kTouched;
      marks[vo[r]] = kTouched;
      valive[vq[r]] = 0;
    }
    p3[f] = 1;
    for (int r = 0; r < 4; r++) rflag[fo[r]] = 1;
  }
}

// removeVertices3333 + removeQuadrilaterals3333 (:1324-1382) in place: the four neighbours of a
// marked face die and its corners move to the neighbours' far vertices (kept: their valence is not 3).
__global__ void __launch_bounds__(256, 8) apply_3333_kernel(int4* q, int64_t nq, uint8_t* alive, const uint8_t* rflag, const uint8_t* p3,
                                  const int32_t* vm1, const uint8_t* marks, uint8_t* dirty, int32_t* deg) {
  pdl_begin();
  FOR_EACH(f, nq) {
    const uint8_t a = alive[f], e = rflag[f], moved = p3[f];
    const int4 c = q[f];
    if (!a) continue;
    const unsigned m0 = marks[c.x], m1 = marks[c.y], m2 = marks[c.z], m3 = marks[c.w];
    if (e) {
      alive[f] = 0;
      killed_corner(c.x, m0, deg);
      killed_corner(c.y, m1, deg);
      killed_corner(c.z, m2, deg);
      killed_corner(c.w, m3, deg);
      continue;
    }
    if (!((m0 | m1 | m2 | m3) & kTouched)) continue;  // a moved face's corners are touched
    int4 y = c;
    if (moved) {
      y = make_int4(vm1[c.x], vm1[c.y], vm1[c.z], vm1[c.w]);
      q[f] = y;
    }
    live_corner(y.x, m0, dirty, deg);
    live_corner(y.y, m1, dirty, deg);
    live_corner(y.z, m2, dirty, deg);
    live_corner(y.w, m3, dirty, deg);
  }
}

// The live faces at their compacted indices, corners renumbered (vertex x -> vmap[x]); src[o]: the
// face's index before.  Bound by the latency of the gathers: 16-byte loads and stores (the arrays are
// aligned), everything but the corners' numbers loaded before it is known whether the face is live.
// 16.6 M faces: 164 -> 127 us.
__global__ void gather_live_quads_kernel(const uint8_t* alive, const int32_t* idx, int64_t nq, const int4* q,
                                         const int32_t* vmap, int4* qo, int32_t* src, int64_t cap, unsigned* overflow) {
  pdl_begin();
  FOR_EACH(f, nq) {
    const uint8_t a = alive[f];
    const int64_t o = idx[f];
    const int4 c = q[f];
    if (!a) continue;
    if (o < 0 || o >= cap) {
      atomicAdd(overflow, 1u);
      continue;
    }
    src[o] = (int32_t)f;
    qo[o] = make_int4(vmap[c.x], vmap[c.y], vmap[c.z], vmap[c.w]);
  }
}

// ---------------------------------------------------------------------------------------------
// quad -> triangles (collectTriangles, :1387-1460; minAngle, DualMarchingCubes.h:746-756)
// ---------------------------------------------------------------------------------------------
// minAngle exactly as the reference: three float arc cosines of the host C library (the restated
// kind of libm_acosf.h that the host's acosf is, bit for bit), float minimum in std::min's order.
template <int kAcos>
__device__ __noinline__ float min_angle_all(float ca, float cb, float cc) {
  const float A = libm::acosf_kind(ca, kAcos), B = libm::acosf_kind(cb, kAcos), C = libm::acosf_kind(cc, kAcos);
  const float mAB = (B < A) ? B : A;
  return (C < mAB) ? C : mAB;
}
// Where one cosine is clearly the largest (by 2^-18; all within [-1, 1]) its arc cosine is the minimum:
// acos falls at least as fast as its argument grows, and the library's is within an ulp (2^-22).
template <int kAcos>
__device__ __forceinline__ float min_angle(float a, float b, float c) {
  const float ca = (b * b + c * c - a * a) / (2 * b * c), cb = (a * a + c * c - b * b) / (2 * a * c),
              cc = (b * b + a * a - c * c) / (2 * b * a);
  const float m = fmaxf(ca, fmaxf(cb, cc)), low = fminf(ca, fminf(cb, cc));
  const float mid = fmaxf(fminf(ca, cb), fminf(fmaxf(ca, cb), cc));
  if (ca == ca && cb == cb && cc == cc && m <= 1.0f && low >= -1.0f && mid < m - 0x1p-18f)
    return libm::acosf_kind(m, kAcos);
  return min_angle_all<kAcos>(ca, cb, cc);
}

// the reference's side length: the float of a float64 distance
__device__ __forceinline__ float side_f64(const double* p, const double* q) {
  const double d = (p[0] - q[0]) * (p[0] - q[0]) + (p[1] - q[1]) * (p[1] - q[1]) + (p[2] - q[2]) * (p[2] - q[2]);
  return (float)sqrt(d);
}
// A float64 position as float pairs (2^-47 relative), taken apart with integer operations (a conversion
// would run on the float64 pipe too).
struct PairPoint {
  ffx::ff x[3];
};
__device__ __forceinline__ ffx::ff split_f64(double x) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const int e = (int)(b >> 52) & 0x7ff;
  if (e < 1023 - 60 || e > 1023 + 60) return ffx::ff_from_double(x);  // zero, or far from 1
  const uint32_t sign = (uint32_t)(b >> 63) << 31;
  const float hi = __uint_as_float(sign | (uint32_t)(e - 896) << 23 | ((uint32_t)(b >> 29) & 0x7fffffu));
  const float lo = (float)((uint32_t)b & 0x1fffffffu) * __uint_as_float(sign | (uint32_t)(e - 896 - 52) << 23);
  return ffx::ff{hi, lo};
}
__device__ __forceinline__ PairPoint load_pairs(const double* v) {
  return PairPoint{{split_f64(v[0]), split_f64(v[1]), split_f64(v[2])}};
}
// |p - q|; false when its rounding is not certified.  The differences err by 2^-45.4 of the coordinates'
// magnitudes, so the length by their sum's, and by 2^-43 of itself.
__device__ __forceinline__ bool side_certain(const PairPoint& p, const PairPoint& q, float& out) {
  ffx::ff sum{0, 0};
  float mag = 0;
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const ffx::ff s = ffx::two_sum(p.x[a].hi, -q.x[a].hi);
    const ffx::ff d = ffx::quick_two_sum(s.hi, s.lo + (p.x[a].lo - q.x[a].lo));
    sum = ffx::ff_add_abs(sum, ffx::ff_mul(d, d));
    mag += fabsf(p.x[a].hi) + fabsf(q.x[a].hi);
  }
  if (!(sum.hi > 0x1p-80f && sum.hi < 0x1p80f)) return false;
  // the rounded root and one Newton step
  const float r = sqrtf(sum.hi);
  const ffx::ff sq = ffx::two_prod(r, r);
  const ffx::ff l = ffx::quick_two_sum(r, (((sum.hi - sq.hi) - sq.lo) + sum.lo) * (0.5f * ffx::rcp_est(r)));
  out = l.hi;
  return ffx::ff_certain(l, mag * 0x1p-45f + l.hi * 0x1p-42f);
}

__device__ __forceinline__ void write_split(int32_t* t, int64_t i, int v0, int v1, int v2, int v3, bool first) {
  int32_t* o = t + 6 * i;
  if (first) {
    o[0] = v1; o[1] = v3; o[2] = v0; o[3] = v1; o[4] = v2; o[5] = v3;
  } else {
    o[0] = v0; o[1] = v1; o[2] = v2; o[3] = v0; o[4] = v2; o[5] = v3;
  }
}

// A side from float positions: its length, the reciprocal's estimate and its relative error bound.
struct Side {
  float d, r, e;
};
// Largest cosine of the triangle with sides a, b, c, and the bound of the result's distance to the
// reference's; false when the cosines are not surely inside [-1, 1].
__device__ __forceinline__ bool max_cosine_bounded(const Side& a, const Side& b, const Side& c, float& m, float& em) {
  const float aa = a.d * a.d, bb = b.d * b.d, cc = c.d * c.d;
  const float ab = 0.5f * a.r * b.r, ac = 0.5f * a.r * c.r, bc = 0.5f * b.r * c.r;
  const float cA = (bb + cc - aa) * bc, cB = (aa + cc - bb) * ac, cC = (bb + aa - cc) * ab;
  // first-order propagation of the side errors (doubled), plus the rounding of both evaluations (with
  // the reciprocals' 2^-21)
  const float rel = a.e + b.e + c.e, s = 2.0f * (aa * a.e + bb * b.e + cc * c.e);
  const float eA = 2.0f * (s * bc + fabsf(cA) * rel) + 0x1p-19f;
  const float eB = 2.0f * (s * ac + fabsf(cB) * rel) + 0x1p-19f;
  const float eC = 2.0f * (s * ab + fabsf(cC) * rel) + 0x1p-19f;
  if (!(fabsf(cA) + eA <= 1.f && fabsf(cB) + eB <= 1.f && fabsf(cC) + eC <= 1.f)) return false;
  m = fmaxf(cA, fmaxf(cB, cC));
  em = fmaxf(eA, fmaxf(eB, eC));
  return true;
}

// |p - q| from float positions and a bound of its distance to the reference's float (rounded from
// the float64 length of the float64 difference); each float position is within 2^-24 |x| of its
// float64 value.
struct FloatPoint {
  float x[3];
};
__device__ __forceinline__ FloatPoint load_point(const float* v, int64_t i) {
  return FloatPoint{{v[3 * i], v[3 * i + 1], v[3 * i + 2]}};
}
__device__ __forceinline__ bool side_bounded(const FloatPoint& p, const FloatPoint& q, Side& out) {
  const float dx = p.x[0] - q.x[0], dy = p.x[1] - q.x[1], dz = p.x[2] - q.x[2];
  const float d2 = dx * dx + dy * dy + dz * dz;
  const float mag = fabsf(p.x[0]) + fabsf(q.x[0]) + fabsf(p.x[1]) + fabsf(q.x[1]) + fabsf(p.x[2]) + fabsf(q.x[2]);
  out.r = rsqrtf(d2);  // within two ulps
  out.d = d2 * out.r;
  out.e = mag * 0x1p-23f * out.r + 0x1p-20f;
  return d2 > 0x1p-80f && d2 < 0x1p80f;
}

// The split of quad corners P, where the two candidates' smallest angles are apart by more than the
// error bounds: 1 first (along v1-v3), 0 second, -1 in doubt.
__device__ __forceinline__ int split_bounded(const FloatPoint& P0, const FloatPoint& P1, const FloatPoint& P2,
                                             const FloatPoint& P3) {
  Side d01, d12, d20, d23, d30, d13;
  bool ok = side_bounded(P0, P1, d01);
  ok = side_bounded(P1, P2, d12) && ok;
  ok = side_bounded(P2, P0, d20) && ok;
  ok = side_bounded(P2, P3, d23) && ok;
  ok = side_bounded(P3, P0, d30) && ok;
  ok = side_bounded(P1, P3, d13) && ok;
  float m1, m2, m3, m4, x1, x2, x3, x4;
  if (!(ok && max_cosine_bounded(d01, d12, d20, m1, x1) && max_cosine_bounded(d20, d23, d30, m2, x2) &&
        max_cosine_bounded(d13, d30, d01, m3, x3) && max_cosine_bounded(d12, d23, d13, m4, x4)))
    return -1;
  // smallest angle of a split = acos of its largest cosine (acos decreasing): the first split wins when
  // its largest cosine is smaller.  The bounds place the reference's largest cosines; a further 2^-20
  // between them keeps its angles (acos has slope at least 1 in magnitude, and the library's float
  // acos is within one ulp, at most 2^-22 below pi) strictly ordered the same way.
  const float xb = fmaxf(m1, m2), eb = fmaxf(x1, x2), xc = fmaxf(m3, m4), ec = fmaxf(x3, x4);
  if (xb + eb + 0x1p-20f < xc - ec) return 0;  // b1 > c1
  if (xb - eb > xc + ec + 0x1p-20f) return 1;  // b1 < c1
  return -1;
}
__device__ __forceinline__ void list_quad(uint32_t* list, unsigned* count, bool take, uint32_t x) {
  const int lane = threadIdx.x & 31;
  const unsigned am = __activemask();
  const unsigned bal = __ballot_sync(am, take);
  if (!bal) return;
  const int leader = __ffs(bal) - 1;
  unsigned base = 0;
  if (lane == leader) base = atomicAdd(count, (unsigned)__popc(bal));
  base = __shfl_sync(am, base, leader);
  if (take) list[base + __popc(bal & ((1u << lane) - 1u))] = x;
}

// collectTriangles (:1387-1460), first pass: decides the split from the float positions wherever they
// leave no doubt; the other quads are listed.
__global__ void triangles_fast_kernel(const int32_t* q, int64_t nq, const float* v, int32_t* t, uint32_t* list,
                                      unsigned* count) {
  pdl_begin();
  FOR_EACH(i, nq) {
    const int v0 = q[4 * i], v1 = q[4 * i + 1], v2 = q[4 * i + 2], v3 = q[4 * i + 3];
    const int s = split_bounded(load_point(v, v0), load_point(v, v1), load_point(v, v2), load_point(v, v3));
    if (s >= 0) write_split(t, i, v0, v1, v2, v3, s == 1);
    list_quad(list, count, s < 0, (uint32_t)i);
  }
}

// The reference's decision from the six side lengths: minAngle of the triangles (v0,v1,v2), (v0,v2,v3)
// against (v1,v3,v0), (v1,v2,v3), each from the sides |p0p1|, |p1p2|, |p2p0|; true: the first split.
template <int kAcos>
__device__ __forceinline__ bool split_exact(float d01, float d12, float d20, float d23, float d30, float d13) {
  float m[4];
#pragma unroll 1  // one copy of the arc cosines: the pass is bound by instruction fetch otherwise
  for (int t = 0; t < 4; t++) {
    const float a = t == 0 ? d01 : (t == 1 ? d20 : (t == 2 ? d13 : d12));
    const float b = t == 0 ? d12 : (t == 1 ? d23 : (t == 2 ? d30 : d23));
    const float c = t == 0 ? d20 : (t == 1 ? d30 : (t == 2 ? d01 : d13));
    const float x = min_angle<kAcos>(a, b, c);
    if (t == 0) m[0] = x;
    if (t == 1) m[1] = x;
    if (t == 2) m[2] = x;
    if (t == 3) m[3] = x;
  }
  // (the reference compares the floats as doubles)
  const float b1 = m[1] < m[0] ? m[1] : m[0], b2 = m[0] < m[1] ? m[1] : m[0];
  const float c1 = m[3] < m[2] ? m[3] : m[2], c2 = m[2] < m[3] ? m[3] : m[2];
  return b1 < c1 || (b1 == c1 && b2 <= c2);
}

// collectTriangles (:1387-1460), exact pass over the listed quads: the reference's arithmetic
// step by step.  Six side lengths (float of a float64 distance), minAngle of the four triangles with
// the host library's float acos (libm_acosf.h, kAcos), comparisons of the two splits.
// The float positions are coarse beside a fine grid's cells, so many quads are listed (8 % of the 512^3
// noise field's, 40 % of the 1024x1024x64 saddle field's).  The lengths come from float pairs with
// certified rounding; the quads with one that is not certified (a few per cent) are gathered in shared
// memory and taken in float64 densely, a few lanes of most warps would occupy that pipe otherwise.
// v64 and q64: the float64 positions and the quads that index them; src: the face there of each of q's
// (null when they are the same mesh).
// With twelve arc cosines per quad and every length in float64 the pass took 0.28 ms (noise, 0.38 million
// quads listed) and 4.64 ms (saddle); 0.16 and 2.18 ms so.
constexpr int kSplitThreads = 256;
template <int kAcos>
__global__ void __launch_bounds__(kSplitThreads) triangles_kernel(const int32_t* q, const uint32_t* list,
                                                                  const unsigned* count, const double* v64,
                                                                  const int32_t* q64, const int32_t* src, int32_t* t) {
  pdl_begin();
  __shared__ uint32_t open[2 * kSplitThreads];
  __shared__ unsigned n_open;
  if (threadIdx.x == 0) n_open = 0;
  __syncthreads();
  const int64_t nl = *count;
  const int64_t step = (int64_t)gridDim.x * kSplitThreads;
  for (int64_t base = (int64_t)blockIdx.x * kSplitThreads; base < nl; base += step) {  // block-uniform
    const int64_t a = base + threadIdx.x;
    if (a < nl) {
      const int64_t i = list[a];
      const int v0 = q[4 * i], v1 = q[4 * i + 1], v2 = q[4 * i + 2], v3 = q[4 * i + 3];
      const int32_t* c = q64 + 4 * (src ? (int64_t)src[i] : i);
      const PairPoint p0 = load_pairs(v64 + 3 * (int64_t)c[0]), p1 = load_pairs(v64 + 3 * (int64_t)c[1]),
                      p2 = load_pairs(v64 + 3 * (int64_t)c[2]), p3 = load_pairs(v64 + 3 * (int64_t)c[3]);
      float d01, d12, d20, d23, d30, d13;
      bool ok = side_certain(p0, p1, d01);
      ok = side_certain(p1, p2, d12) && ok;
      ok = side_certain(p2, p0, d20) && ok;
      ok = side_certain(p2, p3, d23) && ok;
      ok = side_certain(p3, p0, d30) && ok;
      ok = side_certain(p1, p3, d13) && ok;
      if (ok) write_split(t, i, v0, v1, v2, v3, split_exact<kAcos>(d01, d12, d20, d23, d30, d13));
      else open[atomicAdd(&n_open, 1u)] = (uint32_t)i;
    }
    __syncthreads();
    const unsigned n = n_open;
    __syncthreads();  // n_open is read before the next round's quads add to it
    if (n >= kSplitThreads || base + step >= nl) {  // block-uniform: a full round, or the last
      for (unsigned x = threadIdx.x; x < n; x += kSplitThreads) {
        const int64_t i = open[x];
        const int v0 = q[4 * i], v1 = q[4 * i + 1], v2 = q[4 * i + 2], v3 = q[4 * i + 3];
        const int32_t* c = q64 + 4 * (src ? (int64_t)src[i] : i);
        const double *P0 = v64 + 3 * (int64_t)c[0], *P1 = v64 + 3 * (int64_t)c[1], *P2 = v64 + 3 * (int64_t)c[2],
                     *P3 = v64 + 3 * (int64_t)c[3];
        write_split(t, i, v0, v1, v2, v3,
                    split_exact<kAcos>(side_f64(P0, P1), side_f64(P1, P2), side_f64(P2, P0), side_f64(P2, P3),
                                       side_f64(P3, P0), side_f64(P1, P3)));
      }
      __syncthreads();
      if (threadIdx.x == 0) n_open = 0;
      __syncthreads();
    }
  }
}

// ---------------------------------------------------------------------------------------------
// driver helpers
// ---------------------------------------------------------------------------------------------
// Scratch of one call: arrays cut from one reserved block (256-byte aligned), on their own when it is
// used up.
struct Pool {
  cudaStream_t st;
  std::vector<void*> temp;
  cudaError_t err = cudaSuccess;
  char* at = nullptr;
  size_t left = 0;
  explicit Pool(cudaStream_t s) : st(s) {}
  void reserve(size_t bytes) {
    void* p = nullptr;
    if (err != cudaSuccess) return;
    err = cudaMallocAsync(&p, bytes, st);
    if (err != cudaSuccess) return;
    temp.push_back(p);
    at = (char*)p;
    left = bytes;
  }
  template <typename T>
  T* get(int64_t n) {
    const size_t bytes = ((size_t)std::max<int64_t>(n, 4) * sizeof(T) + 255) & ~(size_t)255;
    if (err != cudaSuccess) return nullptr;
    if (bytes <= left) {
      void* p = at;
      at += bytes;
      left -= bytes;
      return (T*)p;
    }
    void* p = nullptr;
    err = cudaMallocAsync(&p, bytes, st);
    if (err == cudaSuccess) temp.push_back(p);
    return (T*)p;
  }
  ~Pool() {
    for (void* p : temp) cudaFreeAsync(p, st);
  }
};

struct HeBufs {
  int32_t* twin = nullptr;
  uint8_t* flag = nullptr;
  int32_t* hv = nullptr;
  HeWork w{};
  // counters, zeroed together: non-manifold edges, overflow, merge jobs of the passes, handle counts,
  // quads of the exact triangle split, colour classes
  unsigned long long* zero = nullptr;
  unsigned long long* nm = nullptr;
  unsigned* ovf = nullptr;
  // repairs after the simplification passes: what a pass did to the vertices (marks) and the dirty ones
  // (dnew); the compacted faces' indices before (src); handle counters
  uint8_t* marks = nullptr;
  uint8_t* dnew = nullptr;
  int32_t* src = nullptr;
  HeUpdateWork u{};
  unsigned long long* hcount = nullptr;
};

// colorFaces (:714-844) on a mesh whose halfedges are built: the inherited colours in `col` become
// the reduced ones, group by group (colours 5..23 to the lowest of 0..4 free among the neighbours,
// then colour 4, the last group, to the lowest of 0..3).  Returns the number of kernels launched.
// cnt: 24 zeroed words; front: the mesh is as the front end made it.
int color_faces(const HeView& he, uint8_t* col, int64_t nq, int32_t* cnt, bool front, Pool& pool, int sms,
                cudaStream_t st) {
  int32_t* off = pool.get<int32_t>(24);
  int32_t* cursor = pool.get<int32_t>(24);
  int32_t* list = pool.get<int32_t>(std::max<int64_t>(nq, 1));
  if (pool.err) return 0;
  const unsigned gc = (unsigned)std::max<int64_t>(1, ceil_div(nq, kColorTile));
  if (front) launch(color_count_kernel<true>, gc, kColorThreads, st, col, nq, cnt);
  else launch(color_count_kernel<false>, gc, kColorThreads, st, col, nq, cnt);
  launch(color_offsets_kernel, 1, 32, st, cnt, off, cursor);
  if (front) launch(color_scatter_kernel<true>, gc, kColorThreads, st, col, nq, cursor, list);
  else launch(color_scatter_kernel<false>, gc, kColorThreads, st, col, nq, cursor, list);
  const unsigned gq = grid_for(std::max<int64_t>(nq, 1), sms);
  const int groups = front ? kFrontGroups : kColorGroups;
  for (int k = 0; k < groups; k++) launch(color_reduce_kernel, gq, 256, st, he, col, list, off, k, k + 1 < groups ? 4 : 3);
  return groups + 3;
}

// Fills and one copy in one launch (16 bytes at a time; the arrays' pool blocks are whole multiples, so a
// last partial one stays inside).  As fills and copies of the stream's own they cost 5 to 6 us each between
// short kernels, three or four per pass: 131x117x140 with all outputs 648 -> 595 us with one launch each.
struct Fill {
  uint4* p;
  int64_t n;  // of 16 bytes
  uint32_t v;
};
Fill fill(void* p, size_t bytes, uint32_t v) {
  return Fill{reinterpret_cast<uint4*>(p), (int64_t)((bytes + 15) / 16), v};
}
struct Fills {
  Fill f[4];
};
__global__ void __launch_bounds__(256) fill_and_copy_kernel(Fills fills, const uint4* from, uint4* to, int64_t n) {
  pdl_begin();
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const uint32_t v = fills.f[q].v;
    FOR_EACH(i, fills.f[q].n) fills.f[q].p[i] = make_uint4(v, v, v, v);
  }
  FOR_EACH(i, n) to[i] = from[i];
}
int fill_and_copy(const std::vector<Fill>& fills, const void* from, void* to, size_t bytes, int sms, cudaStream_t st) {
  Fills f{};
  int64_t most = (int64_t)((bytes + 15) / 16);
  for (size_t q = 0; q < fills.size(); q++) {  // at most four
    f.f[q] = fills[q];
    most = std::max(most, fills[q].n);
  }
  launch(fill_and_copy_kernel, grid_for(std::max<int64_t>(most, 1), sms), 256, st, f,
         reinterpret_cast<const uint4*>(from), reinterpret_cast<uint4*>(to), (int64_t)((bytes + 15) / 16));
  return 1;
}

// vertexValence (:847-871): the out-degrees of the halfedge build plus the boundary corrections
// (alive: the live faces, all when NULL)
int vertex_valence(const HeView& he, const int32_t* deg, int64_t nv, int64_t nq, int32_t* val, int sms,
                   cudaStream_t st, const uint8_t* alive = nullptr) {
  cudaMemcpyAsync(val, deg, nv * sizeof(int32_t), cudaMemcpyDeviceToDevice, st);
  launch(valence_boundary_kernel, grid_for(std::max<int64_t>(nq, 1), sms), 256, st, he, nq, val, alive);
  return 1;
}

constexpr int kZeroWords = 32;  // [0,1] non-manifold, [2] overflow, [3..6] handles, [7] jobs, [8] split, [16..27] colours
constexpr int kZeroJobs = 7, kZeroSplit = 8, kZeroColors = 16;

HeBufs halfedge_buffers(Pool& pool, int64_t NV, int64_t NQ) {
  HeBufs hw;
  hw.twin = pool.get<int32_t>(4 * NQ);
  hw.flag = pool.get<uint8_t>(4 * NQ);
  hw.hv = pool.get<int32_t>(NV);
  hw.w.deg = pool.get<int32_t>(NV);
  hw.w.off = pool.get<int32_t>(NV);
  hw.w.rank = pool.get<int32_t>(4 * NQ);
  hw.w.list = pool.get<int2>(4 * NQ);
  hw.w.hv_key = pool.get<unsigned long long>(NV);
  hw.w.tiles = pool.get<unsigned long long>(scan_tiles(NV) + 2);
  hw.w.total = pool.get<unsigned long long>(2);
  hw.zero = pool.get<unsigned long long>(kZeroWords);
  hw.nm = hw.zero;
  hw.w.non_manifold = hw.nm;
  hw.ovf = reinterpret_cast<unsigned*>(hw.zero + 2);
  hw.hcount = hw.zero + 3;
  return hw;
}

// Buffers of the simplification passes, their halfedge repairs and the final compaction.  What a pass
// resets lies together: `fresh` (bucket sizes, marks and dirty vertices) is zeroed and `owner` (claims and
// merge targets) set to -1.
struct PassBufs {
  int32_t* val;
  uint8_t *p, *em, *branch;   // p and em adjacent (both zero for P3333)
  size_t face_stride;         // from p to em
  uint8_t* fresh;
  size_t fresh_bytes;
  int32_t* owner;
  int32_t *own_pos, *own_rm, *vm_second;
  int4* jobs;
  uint8_t *alive, *valive;    // faces, then vertices: one scan numbers both
  int32_t *idx_q, *idx;       // likewise; vertex x becomes idx[x] - idx[0], and idx[0] faces are kept
};
PassBufs pass_buffers(Pool& pool, HeBufs& hw, int64_t NV, int64_t NQ) {
  PassBufs b;
  const int64_t nv16 = (NV + 15) / 16 * 16, nq16 = (NQ + 15) / 16 * 16;
  hw.src = pool.get<int32_t>(NQ);
  hw.u.drank = pool.get<int32_t>(4 * NQ);
  hw.u.dmask = pool.get<uint8_t>(NQ);
  hw.u.boff = hw.w.off;    // the build's scratch is idle after the one build
  hw.u.blist = hw.w.list;
  hw.u.bkey = pool.get<int32_t>(4 * NQ);
  hw.u.tiles = hw.w.tiles;
  hw.u.total = hw.w.total;
  b.val = pool.get<int32_t>(NV);
  b.face_stride = (size_t)nq16;
  b.p = pool.get<uint8_t>(2 * nq16);
  b.em = b.p + nq16;
  b.branch = pool.get<uint8_t>(NQ);
  b.fresh_bytes = (size_t)(6 * nv16);
  b.fresh = pool.get<uint8_t>(6 * nv16);
  hw.u.bcnt = reinterpret_cast<int32_t*>(b.fresh);
  hw.marks = b.fresh + 4 * nv16;
  hw.dnew = b.fresh + 5 * nv16;
  b.owner = pool.get<int32_t>(3 * NV);
  b.own_pos = b.owner;
  b.own_rm = b.owner + NV;
  b.vm_second = b.owner + 2 * NV;
  b.jobs = pool.get<int4>(NQ);
  b.alive = pool.get<uint8_t>(NQ + NV);
  b.valive = b.alive + NQ;
  b.idx_q = pool.get<int32_t>(NQ + NV);
  b.idx = b.idx_q + NQ;
  return b;
}

}  // namespace

DmcPostStatus dmc_color_valence(const int32_t* quads, int64_t nq, int64_t nv, uint8_t* colors, int32_t* valence,
                                int sms, cudaStream_t st) {
  DmcPostStatus s;
  if (nq == 0) {
    if (nv > 0) s.err = cudaMemsetAsync(valence, 0, nv * sizeof(int32_t), st);
    return s;
  }
  Pool pool(st);
  pool.reserve(72 * (size_t)nq + 20 * (size_t)std::max<int64_t>(nv, 1) + 32 * 256);
  HeBufs hw = halfedge_buffers(pool, std::max<int64_t>(nv, 1), nq);
  if ((s.err = pool.err) != cudaSuccess) return s;
  cudaMemsetAsync(hw.zero, 0, kZeroWords * sizeof(unsigned long long), st);
  HeOut ho{hw.twin, hw.flag, hw.hv};
  s.launches += build_halfedges(quads, 4, nq, nv, ho, hw.w, sms, st, false);
  const HeView he{quads, hw.twin, hw.flag};
  s.launches += color_faces(he, colors, nq, reinterpret_cast<int32_t*>(hw.zero + kZeroColors), false, pool, sms, st);
  if ((s.err = pool.err) != cudaSuccess) return s;
  s.launches += vertex_valence(he, hw.w.deg, nv, nq, valence, sms, st);
  s.err = cudaGetLastError();
  return s;
}

// what its buffers add up to, per face and per vertex
size_t dmc_postprocess_bytes(uint32_t flags, int64_t nv, int64_t nq) {
  const bool passes = (flags & (TMC_DMC_P3X3Y_COLOR | TMC_DMC_P3X3Y_ISOLATED | TMC_DMC_P3333)) && nq > 0;
  return (passes ? 144 : 74) * (size_t)std::max<int64_t>(nq, 1) + (passes ? 56 : 24) * (size_t)std::max<int64_t>(nv, 1) + 64 * 256;
}

DmcPostStatus dmc_postprocess(const DmcMesh& in, uint32_t flags, int sms, cudaStream_t st, DmcPostOut* out,
                              unsigned long long* h_cnt, Prof* prof, bool borrowed, const ReadyFn* ready,
                              const TwinsFn* twins) {
  DmcPostStatus s;
  out->mesh = in;
  const bool c3x3y = flags & TMC_DMC_P3X3Y_COLOR, i3x3y = flags & TMC_DMC_P3X3Y_ISOLATED,
             p3333 = flags & TMC_DMC_P3333, want_t = flags & TMC_OUT_TRIANGLES, want_he = flags & TMC_OUT_HALFEDGES;
  if (!(c3x3y || i3x3y || p3333 || want_t || want_he)) return s;
  // the repairs and handles read quads and flags 4 at a time: front-end meshes are 16-byte aligned
  if (reinterpret_cast<uintptr_t>(in.quads) & 15) {
    s.err = cudaErrorInvalidValue;
    return s;
  }
  Pool pool(st);
  const int64_t NV = std::max<int64_t>(in.nv, 1), NQ = std::max<int64_t>(in.nq, 1);
  pool.reserve(dmc_postprocess_bytes(flags, in.nv, in.nq));

  DmcMesh cur = in;
  HeBufs hw = halfedge_buffers(pool, NV, NQ);
  unsigned long long* tiles = pool.get<unsigned long long>(scan_tiles(NV + NQ) + 2);
  unsigned long long* total = pool.get<unsigned long long>(2);
  if (pool.err) {
    s.err = pool.err;
    return s;
  }
  const unsigned gq = grid_for(NQ, sms);
  const bool simplify = (c3x3y || i3x3y || p3333) && in.nq > 0;
  // the counters and what else a call starts from
  auto start = [&](std::vector<Fill> fills) {
    fills.push_back(fill(hw.zero, kZeroWords * sizeof(unsigned long long), 0u));
    if (twins && cur.nq > 0) fills.push_back(fill(hw.flag, 4 * (size_t)NQ, 0u));
    s.launches += fill_and_copy(fills, nullptr, nullptr, 0, sms, st);
  };
  auto build_he = [&](bool handles) {
    Stage tm(prof, "dmc_halfedges", st);
    HeOut ho{hw.twin, hw.flag, hw.hv};
    if (!twins || cur.nq == 0) {
      s.launches += build_halfedges(cur.quads, 4, cur.nq, cur.nv, ho, hw.w, sms, st, handles);
      return;
    }
    s.launches += (*twins)(hw.twin, hw.flag, hw.w.deg);
    if (handles)
      s.launches +=
          halfedge_handles(cur.quads, 4, cur.nq, cur.nv, nullptr, hw.twin, hw.flag, hw.hv, hw.w, hw.hcount, sms, st);
  };
  auto retire = [&](void* ptr) {
    if (!ptr) return;
    bool mine = false;
    for (auto& q : out->owned)
      if (q == ptr) {
        q = nullptr;
        mine = true;
      }
    if (!mine) out->freed.push_back(ptr);
    if (mine || !borrowed) cudaFreeAsync(ptr, st);
  };
  auto adopt = [&](void* ptr) { out->owned.push_back(ptr); };

  // ---- simplification (simplify3X3Y :1139-1182, simplify3333 :1362-1385) ----
  // In place: faces and vertices keep their indices through the passes (alive / valive flags), the
  // halfedges are built once and repaired after each pass, and one order-preserving compaction after
  // the last pass gives the reference's numbering (each of its per-pass compactions keeps the order
  // of what remains, and every rule that compares indices compares them in the same order).
  bool compacted = false;
  uint8_t *alive = nullptr, *valive = nullptr;
  int32_t *idx = nullptr, *idx_q = nullptr, *map = nullptr;
  int64_t nv0 = cur.nv, nq0 = cur.nq;  // the uncompacted mesh
  int64_t nv2 = nv0, nq2 = nq0;        // and what is left of it
  int32_t* q0 = cur.quads;
  if (simplify) {
    const PassBufs b = pass_buffers(pool, hw, NV, NQ);
    int32_t *val = b.val, *own_pos = b.own_pos, *own_rm = b.own_rm, *vm_second = b.vm_second;
    uint8_t *p = b.p, *em = b.em, *branch = b.branch;
    alive = b.alive;
    valive = b.valive;
    idx = b.idx;
    idx_q = b.idx_q;
    map = b.vm_second;
    if ((s.err = pool.err) != cudaSuccess) return s;
    start({fill(alive, (size_t)(NQ + NV), 0x01010101u)});
    build_he(false);
    const HeView he{q0, hw.twin, hw.flag};
    // what is left after the last pass, counted before its repair and the handles: they run while the host
    // takes the counts and makes room for the result
    cudaEvent_t counted = nullptr;
    auto count_live = [&]() {
      Stage tm(prof, "dmc_compact", st);
      s.launches += scan_flags(alive, nq0 + nv0, idx_q, tiles, total, st);
      cudaMemcpyAsync(h_cnt, total, sizeof(unsigned long long), cudaMemcpyDeviceToHost, st);
      cudaMemcpyAsync(h_cnt + 1, idx, sizeof(int32_t), cudaMemcpyDeviceToHost, st);
      counted = host_mark(st);
    };
    // what a pass starts from: its marks and the vertices' valences (vertexValence :847-871)
    auto begin_pass = [&](const std::vector<Fill>& fills) {
      s.launches += fill_and_copy(fills, hw.w.deg, val, (size_t)nv0 * sizeof(int32_t), sms, st);
      launch(valence_boundary_kernel, gq, 256, st, he, nq0, val, alive);
      s.launches += 2;
    };
    auto repair = [&]() {
      Stage tm(prof, "dmc_halfedges", st);
      HeOut ho{hw.twin, hw.flag, nullptr};
      s.launches += repair_halfedges(q0, nq0, nv0, alive, hw.dnew, ho, hw.w.deg, hw.u, sms, st);
    };
    // P3X3Y: colour pass, then isolated pass
    for (int pass = 0; pass < 2; pass++) {
      if ((pass == 0 && !c3x3y) || (pass == 1 && !i3x3y)) continue;
      if (pass == 0) {
        Stage tm(prof, "dmc_color", st);
        s.launches += color_faces(he, cur.colors, nq0, reinterpret_cast<int32_t*>(hw.zero + kZeroColors), true, pool, sms,
                                  st);
        if ((s.err = pool.err) != cudaSuccess) return s;
      }
      {
        Stage tm(prof, "dmc_p3x3y", st);
        begin_pass({fill(b.owner, 3 * (size_t)NV * sizeof(int32_t), 0xffffffffu), fill(b.fresh, b.fresh_bytes, 0u)});
        launch(mark3x3y_kernel, gq, 256, st, reinterpret_cast<const int4*>(q0), nq0, val, p, alive);
        launch(merge_claim_kernel, gq, 256, st, he, nq0, p, val, cur.colors, pass == 0, branch, own_pos, own_rm);
        unsigned* njobs = reinterpret_cast<unsigned*>(hw.zero + kZeroJobs) + pass;
        launch(merge_apply_kernel, gq, kMergeThreads, st, he, nq0, branch, own_pos, own_rm, vm_second, em, b.jobs, njobs,
               hw.marks, valive);
        static const int r_mid = resident_blocks(midpoint_kernel, 256);  // one wave over the merge list
        launch(midpoint_kernel, (unsigned)wave_grid(r_mid, sms, 1, nq0, 256), 256, st, b.jobs, njobs, cur.v64, cur.n64);
        launch(apply_3x3y_kernel, gq, 256, st, reinterpret_cast<int4*>(q0), nq0, alive, em, hw.marks, vm_second, hw.dnew,
               hw.w.deg);
        s.launches += 5;
      }
      if (!p3333 && (pass == 1 || !i3x3y)) count_live();
      repair();
    }
    // P3333
    if (p3333) {
      {
        Stage tm(prof, "dmc_p3333", st);
        uint8_t* p3 = p;
        uint8_t* rflag = em;
        int32_t* vm1 = own_pos;
        begin_pass({fill(p3, 2 * b.face_stride, 0u) /* and rflag behind it */, fill(b.fresh, b.fresh_bytes, 0u),
                    fill(vm1, (size_t)NV * sizeof(int32_t), 0xffffffffu)});
        launch(mark3333_kernel, gq, 256, st, he, nq0, val, p3, rflag, vm1, hw.marks, alive, valive);
        launch(apply_3333_kernel, gq, 256, st, reinterpret_cast<int4*>(q0), nq0, alive, rflag, p3, vm1, hw.marks, hw.dnew,
               hw.w.deg);
        s.launches += 2;
      }
      count_live();
      repair();
    }
    // the output's vertex handles and edge counts, on the uncompacted mesh (before it is released)
    if (want_he) {
      Stage tm(prof, "dmc_halfedges", st);
      s.launches += halfedge_handles(q0, 4, nq0, nv0, alive, hw.twin, hw.flag, hw.hv, hw.w, hw.hcount, sms, st);
    }
    // ---- the one compaction: live vertices and faces, in order ----
    if ((s.err = host_wait_mark(counted, st)) != cudaSuccess) return s;
    nq2 = (int64_t) * reinterpret_cast<const int32_t*>(h_cnt + 1);
    nv2 = (int64_t)h_cnt[0] - nq2;
    // nothing died: no pass changed the mesh, and it stays as it is (with its halfedges)
    compacted = nv2 != nv0 || nq2 != nq0;
    if (compacted) {  // made anew below
      retire(cur.v);
      retire(cur.n);
      cur.v = cur.n = nullptr;
    }
  }
  // The result's arrays in one allocation: made one by one behind the frees of what they replace, the pool
  // mapped memory anew for them (1.4 ms of a 512^3 call's 12.4, the GPU waiting).
  struct Part {
    void** p;
    size_t bytes;
  };
  std::vector<Part> parts;
  auto part = [&](auto** p, int64_t count) {
    parts.push_back(Part{reinterpret_cast<void**>(p), ((size_t)std::max<int64_t>(count, 1) * sizeof(**p) + 255) & ~(size_t)255});
  };
  DmcMesh nx = cur;
  nx.nv = nv2;
  nx.nq = nq2;
  const bool new_floats = !cur.v;  // compacted, or left to be made here
  if (new_floats) {
    part(&nx.v, 3 * nv2);
    part(&nx.n, 3 * nv2);
  }
  if (compacted) {
    nx.v64 = nx.n64 = nullptr;
    if (flags & TMC_OUT_POS_F64) part(&nx.v64, 3 * nv2);
    part(&nx.quads, 4 * nq2);
  }
  int32_t *he4 = nullptr, *hv = nullptr, *hf = nullptr, *tr = nullptr;
  if (want_he) {
    part(&he4, 16 * nq2);
    part(&hv, nv2);
    part(&hf, nq2);
  }
  if (want_t) part(&tr, 6 * nq2);
  if (!parts.empty()) {
    size_t bytes = 0;
    for (const Part& x : parts) bytes += x.bytes;
    void* block = nullptr;
    if ((s.err = cudaMallocAsync(&block, bytes, st)) != cudaSuccess) return s;
    adopt(block);
    char* at = (char*)block;
    for (const Part& x : parts) {
      *x.p = at;
      at += x.bytes;
    }
  }
  const DmcMesh old = cur;  // the uncompacted mesh
  cur = nx;
  if (compacted) {
    Stage tm(prof, "dmc_compact", st);
    // vertex map into vm_second (free after the passes)
    launch(gather_vertices_kernel, grid_for(3 * nv0, sms), 256, st, valive, idx, nv0, old.v64, old.n64, cur.v64, map, nv2,
                                                                   hw.ovf, cur.v, cur.n);
    launch(gather_live_quads_kernel, gq, 256, st, alive, idx_q, nq0, reinterpret_cast<const int4*>(q0), map,
                                                 reinterpret_cast<int4*>(cur.quads), hw.src, nq2, hw.ovf);
    s.launches += 2;
    // the inherited colours are only read by the colour pass; they are not carried along
    retire(old.n64);
  } else if ((simplify || new_floats) && cur.nv > 0) {
    // the float32 outputs of a mesh no pass changed
    launch(float_outputs_kernel, grid_for(3 * cur.nv, sms), 256, st, cur.v64, cur.n64, 3 * cur.nv, cur.v, cur.n);
    s.launches += 1;
  }
  // ---- final halfedges and triangles ----
  if (s.err == cudaSuccess && ready) {
    (*ready)(cur.v, (size_t)cur.nv * 3 * sizeof(float));
    (*ready)(cur.n, (size_t)cur.nv * 3 * sizeof(float));
    if (flags & TMC_OUT_POS_F64) (*ready)(cur.v64, (size_t)cur.nv * 3 * sizeof(double));
    (*ready)(cur.quads, (size_t)cur.nq * 4 * sizeof(int32_t));
  }
  if (!simplify) start({});
  if (want_he) {
    if (!simplify) build_he(true);  // the front-end mesh as it is: one build with the handles
    Stage tm(prof, "dmc_halfedges", st);
    if (compacted) {
      s.launches += pack_compacted_halfedges(cur.quads, cur.nq, hw.src, idx_q, hw.twin, he4, hf, valive, idx, nv0, hw.hv,
                                             hv, sms, st);
    } else {
      s.launches += pack_halfedges4(cur.quads, 4, hw.twin, 4 * cur.nq, he4, hf, sms, st);
      cudaMemcpyAsync(hv, hw.hv, cur.nv * sizeof(int32_t), cudaMemcpyDeviceToDevice, st);
    }
    if (ready) {
      (*ready)(he4, (size_t)cur.nq * 16 * sizeof(int32_t));
      (*ready)(hv, (size_t)cur.nv * sizeof(int32_t));
      (*ready)(hf, (size_t)cur.nq * sizeof(int32_t));
    }
    // read by the caller when the stream is done (the compaction's counts in h_cnt are read by now)
    cudaMemcpyAsync(h_cnt + 2, hw.nm, sizeof(unsigned long long), cudaMemcpyDeviceToHost, st);
    out->non_manifold = h_cnt + 2;
    out->nhe = 4 * cur.nq;
    out->he = he4;
    out->he_v = hv;
    out->he_f = hf;
  }
  if (want_t) {
    Stage tm(prof, "dmc_triangles", st);
    uint32_t* tlist = pool.get<uint32_t>(std::max<int64_t>(cur.nq, 1));
    unsigned* tcount = reinterpret_cast<unsigned*>(hw.zero + kZeroSplit);
    if ((s.err = pool.err) == cudaSuccess) {
      static const int r_fast = resident_blocks(triangles_fast_kernel, 256);
      launch(triangles_fast_kernel, (unsigned)wave_grid(r_fast, sms, 8, cur.nq, 256), 256, st, cur.quads, cur.nq, cur.v, tr,
             tlist, tcount);
      const unsigned gt = grid_for(cur.nq, sms);
      const int kind = libm::host_acosf_kind();
      // positions from the uncompacted mesh, by its quads
#define TRIANGLES(K)                                                                                               \
  launch(triangles_kernel<K>, gt, kSplitThreads, st, cur.quads, tlist, tcount, old.v64, q0, compacted ? hw.src : nullptr, tr)
      if (kind == libm::kAcosfFused) TRIANGLES(libm::kAcosfFused);
      else if (kind == libm::kAcosfSeparate) TRIANGLES(libm::kAcosfSeparate);
      else TRIANGLES(libm::kAcosfCorrect);
#undef TRIANGLES
      s.launches += 2;
      if (ready) (*ready)(tr, (size_t)cur.nq * 6 * sizeof(int32_t));
    }
    out->nt = 2 * cur.nq;
    out->tris = tr;
  }
  if (compacted) {
    retire(old.v64);
    retire(old.quads);
  }
  {
    std::vector<void*> keepv;
    for (void* q : out->owned)
      if (q) keepv.push_back(q);
    out->owned.swap(keepv);
  }
  if (s.err == cudaSuccess) s.err = cudaGetLastError();
  out->mesh = cur;
  return s;
}

}  // namespace tmc
