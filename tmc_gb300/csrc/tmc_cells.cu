// Topologically correct Marching Cubes (TMC) on the GPU, emitted in the reference's order.
//
// Order.  The reference CPU path t_mc (mc/MarchingCubes.cpp:151-317) walks cells in grid order
// and creates a vertex for a crossed edge the first time a cell touches it (std::map keyed by the
// global edge), in edge order 0..11, followed by the cell's inner vertices (p_slice,
// :323-1299); triangles are appended cell by cell.  The first cell touching an edge is the
// lowest-index cell around it, so each cell "owns" a fixed subset of its edges (those whose lower
// neighbours across the edge do not exist).  Hence
//   vertex index   = #vertices of earlier cells + rank among the cell's owned edges (or inner)
//   triangle index = #triangles of earlier cells + rank in the cell
// both exclusive prefix sums over cells; a triangle corner on an edge owned by a neighbour reads
// that neighbour's record.  No hash table, no atomics, deterministic output.
//
// Kernels:
//   tmc_classify_kernel  per-cell record: owned crossed edges, table triangle counts; ambiguous
//                        cells listed
//   tmc_amb_key/cursor/sort_kernel  the ambiguous list sorted by MC case
//   tmc_amb_decide_kernel, tmc_amb_count_kernel
//                        the ambiguous cells' p_slice once (float pairs; float64 for those left in
//                        doubt): counts into the cell records,
//                        triangles (local codes) and inner-vertex parameters into AmbRec records
//   tmc_offsets_kernel   in-tile scan -> per-cell vertex / triangle offsets
//   tmc_emit_kernel      edge vertices and table triangles
//   tmc_ambiguous_kernel the ambiguous cells' triangles and inner vertices from their records
//   tmc_inner_again_kernel, tmc_ambiguous_again_kernel
//                        the inner vertices and cells that need p_slice a second time
#include "ffloat.cuh"
#include "listing.cuh"
#include "scan.cuh"
#include "tmc_cells.h"

namespace tmc {

__constant__ uint64_t c_tmc_tris[256] = TMC_TRIANGLES_INIT;

// per-cell record
//   bits 0-11  owned crossed edges
//   bits 12-14 inner vertices (0, 1 or 6)
//   bits 15-20 triangles
//   bit 21     ambiguous case
//   bit 22     a singular face the reference cannot triangulate (cell emits no triangle)
__device__ __forceinline__ uint32_t trec_owned(uint32_t r) { return r & 0xFFF; }
__device__ __forceinline__ int trec_inner(uint32_t r) { return (r >> 12) & 7; }
__device__ __forceinline__ int trec_ntri(uint32_t r) { return (r >> 15) & 63; }
__device__ __forceinline__ int trec_nv(uint32_t r) { return __popc(trec_owned(r)) + trec_inner(r); }

// cell counts stay below 2^32 (checked by the runtime), so 32-bit division suffices
__device__ __forceinline__ void tcell_ijk(const Grid& g, int64_t c, int& i, int& j, int& k) {
  const uint32_t cx = (uint32_t)(g.nx - 1), cy = (uint32_t)(g.ny - 1);
  const uint32_t cc = (uint32_t)c;  // cell indices of a volume stay below 2^32
  const uint32_t r = g.div_cx.div(cc);
  i = (int)(cc - r * cx);
  const uint32_t kk = g.div_cy.div(r);
  j = (int)(r - kk * cy);
  k = (int)kk;
}

__device__ __forceinline__ void tload_corners(const Grid& g, int i, int j, int k, float u[8]) {
  const float* p = g.f + ((int64_t)k * g.ny + j) * g.nx + i;
  const int64_t sy = g.nx, sz = (int64_t)g.nx * g.ny;
  u[0] = __ldg(p);
  u[1] = __ldg(p + 1);
  u[2] = __ldg(p + sy);
  u[3] = __ldg(p + sy + 1);
  u[4] = __ldg(p + sz);
  u[5] = __ldg(p + sz + 1);
  u[6] = __ldg(p + sz + sy);
  u[7] = __ldg(p + sz + sy + 1);
}

// Edges a cell creates first: across the edge, along each other axis, the cell either sits on the
// far side of the edge (offset 1) or no lower neighbour exists (index 0).
__device__ __forceinline__ uint32_t owned_edges(int i, int j, int k) {
  uint32_t m = 0;
#pragma unroll
  for (int e = 0; e < 12; e++) {
    const int off = edge_off(e), ax = edge_axis(e);
    bool own = true;
    if (ax != 0) own = own && (((off >> 0) & 1) || i == 0);
    if (ax != 1) own = own && (((off >> 1) & 1) || j == 0);
    if (ax != 2) own = own && (((off >> 2) & 1) || k == 0);
    m |= (uint32_t)own << e;
  }
  return m;
}

// Owner cell of local edge e of cell (i,j,k) and the edge's local index there.
__device__ __forceinline__ void edge_owner(int i, int j, int k, int e, int& oi, int& oj, int& ok, int& oe) {
  const int off = edge_off(e), ax = edge_axis(e);
  const int gi = i + (off & 1), gj = j + ((off >> 1) & 1), gk = k + ((off >> 2) & 1);
  oi = (ax == 0) ? gi : (gi > 0 ? gi - 1 : 0);
  oj = (ax == 1) ? gj : (gj > 0 ? gj - 1 : 0);
  ok = (ax == 2) ? gk : (gk > 0 ? gk - 1 : 0);
  const int o = (gi - oi) | ((gj - oj) << 1) | ((gk - ok) << 2);  // offset of the edge in the owner
  // local edge with that offset and axis
#pragma unroll
  for (int q = 0; q < 12; q++)
    if (edge_axis(q) == ax && edge_off(q) == o) oe = q;
}

// ------------------------------------------------------------------------------------------
// cell geometry in float64 for the ambiguous path
// ------------------------------------------------------------------------------------------
// UGrid::gradient (mc/MarchingCubes.cpp:1451-1509): one-sided differences on the border
__device__ __forceinline__ void tmc_point_gradient(const Grid& g, int i, int j, int k, double out[3]) {
  if (i == 0) out[0] = ((double)g.at(i + 1, j, k) - (double)g.at(i, j, k)) / g.dx;
  else if (i == g.nx - 1) out[0] = ((double)g.at(i, j, k) - (double)g.at(i - 1, j, k)) / g.dx;
  else out[0] = ((double)g.at(i + 1, j, k) - (double)g.at(i - 1, j, k)) / (2 * g.dx);
  if (j == 0) out[1] = ((double)g.at(i, j + 1, k) - (double)g.at(i, j, k)) / g.dy;
  else if (j == g.ny - 1) out[1] = ((double)g.at(i, j, k) - (double)g.at(i, j - 1, k)) / g.dy;
  else out[1] = ((double)g.at(i, j + 1, k) - (double)g.at(i, j - 1, k)) / (2 * g.dy);
  if (k == 0) out[2] = ((double)g.at(i, j, k + 1) - (double)g.at(i, j, k)) / g.dz;
  else if (k == g.nz - 1) out[2] = ((double)g.at(i, j, k) - (double)g.at(i, j, k - 1)) / g.dz;
  else out[2] = ((double)g.at(i, j, k + 1) - (double)g.at(i, j, k - 1)) / (2 * g.dz);
}

__device__ __forceinline__ void cell_trilinear3(const double q[8][3], double u, double v, double w, double out[3]) {
#pragma unroll
  for (int d = 0; d < 3; d++)
    out[d] = (1 - w) * ((1 - v) * (q[0][d] + u * (q[1][d] - q[0][d])) + v * (q[2][d] + u * (q[3][d] - q[2][d]))) +
             w * ((1 - v) * (q[4][d] + u * (q[5][d] - q[4][d])) + v * (q[6][d] + u * (q[7][d] - q[6][d])));
}

// The isovalue's parameter on crossed edge e (t_mc's edge coordinates, mc/MarchingCubes.cpp:241-254),
// float64.  p_slice reads them only on a singular face and in the tunnel / hexagon branch, so they
// are computed there, not for every ambiguous cell.
__device__ __forceinline__ double edge_coord(const double F[8], double iso, int e) {
  const int v0 = edge_v0(e), v1 = edge_v1(e);
  return (iso - F[v0]) / (F[v1] - F[v0]);
}

// e_vert (mc/MarchingCubes.cpp:902-911): local coordinate d of the point on edge e
__device__ __forceinline__ double e_vert(const double ecoord[12], int e, int d) {
  return (edge_axis(e) == d) ? ecoord[e] : (double)((edge_off(e) >> d) & 1);
}

// Triangles of p_slice: written out (3 vertex indices each), or, in the counting pass, kept as local
// vertex codes (0..11 the crossed edges, 12..17 the inner vertices; 5 bits each) in the cell's
// ambiguous-cell record, the first kAmbRecTris of them.  n counts them all.
constexpr int kAmbRecTris = 36;
struct TriSink {
  int32_t* out;     // 3 per triangle, or NULL
  uint16_t* codes;  // packed codes, or NULL
  int n;
  __device__ __forceinline__ void put(int a, int b, int c) {
    if (out) {
      out[3 * n] = a;
      out[3 * n + 1] = b;
      out[3 * n + 2] = c;
    } else if (codes && n < kAmbRecTris) {
      codes[n] = (uint16_t)(a | b << 5 | c << 10);
    }
    n++;
  }
};

// The record the counting pass keeps of an ambiguous cell, so that the emission pass does not run
// p_slice again (32 words, 16-byte aligned):
//   w[0]     slot of the cell
//   w[1]     bits 0-7 MC case, 8-13 triangles, 14-16 inner vertices, 17 triangles beyond the record
//            (emission runs p_slice again), 18 a singular face the reference cannot triangulate,
//            19 the parameters are float pairs (hi, lo) in the first three float64 slots, the bound of
//            their errors the first float of the fourth
//   w[2..13] six float64 parameters of the inner vertices: (u, v, w) of the single inner vertex, or
//            (u0, u1, v0, v1, w0, w1) of the six hexagon corners
//   w[14..31] kAmbRecTris triangles as packed local codes (TriSink)
constexpr int kAmbRecWords = 32;
struct __align__(16) AmbRec {
  uint32_t slot, info;
  double prm[6];
  uint16_t tri[kAmbRecTris];
};
static_assert(sizeof(AmbRec) == 4 * kAmbRecWords && kAmbRecWords == kTmcAmbRecWords, "ambiguous-cell record size");

struct AmbResult {
  int inner;     // inner vertices created
  bool error;    // singular face without a valid triangulation
};

// p_slice after the edge vertices (mc/MarchingCubes.cpp:418-1296), float64 throughout.
// vid[e]: global index of the vertex on crossed edge e; ibase: index of the first inner vertex.
// When `geo` is set, inner vertices are written there (positions/normals); when `prm` is set, the
// parameters they are made from (AmbRec::prm).
struct InnerOut {
  float* v;
  float* n;
  double* v64;
};

// Corners (u, v, w) of the inner hexagon (:831-840) from the quadratic's two roots per axis
__device__ __forceinline__ void hex_corners(const double ui[2], const double vi[2], const double wi[2],
                                            double hvt[6][3]) {
  const double c[6][3] = {{ui[0], vi[0], wi[0]}, {ui[0], vi[0], wi[1]}, {ui[1], vi[0], wi[1]},
                          {ui[1], vi[1], wi[1]}, {ui[1], vi[1], wi[0]}, {ui[0], vi[1], wi[0]}};
#pragma unroll
  for (int s = 0; s < 6; s++)
#pragma unroll
    for (int d = 0; d < 3; d++) hvt[s][d] = c[s][d];
}

// One inner vertex at local parameters (u, v, w): trilinear position and normal of the cell's corners,
// the normal normalised (the reference's arithmetic, :1073-1083 and :1283-1293).
__device__ __forceinline__ void inner_vertex(const double (*P)[3], const double (*N)[3], double u, double v, double w,
                                             const InnerOut& geo, int64_t index) {
  double ip[3], in[3];
  cell_trilinear3(P, u, v, w, ip);
  cell_trilinear3(N, u, v, w, in);
  const double factor = sqrt(in[0] * in[0] + in[1] * in[1] + in[2] * in[2]);
  const int64_t o = 3 * index;
  for (int q = 0; q < 3; q++) {
    geo.v[o + q] = (float)ip[q];
    geo.n[o + q] = (float)(in[q] / factor);
    if (geo.v64) geo.v64[o + q] = ip[q];
  }
}

// The triangles of contours without an inner vertex (:1128-1176).  vid(e): the vertex on edge e.
template <typename Vid>
__device__ __forceinline__ void slice_contours(uint64_t c, int cnt, const Vid& vid, TriSink& tri) {
  int flat = 0;
  for (int t = 0; t < cnt; t++) {
    const int sz = cnt_size(c, t);
    int e[6];
    for (int q = 0; q < 6; q++) e[q] = (q < sz) ? vid[cnt_edge(c, flat + q)] : -1;
    switch (sz) {
      case 3: tri.put(e[0], e[1], e[2]); break;
      case 4: tri.put(e[0], e[1], e[2]); tri.put(e[0], e[2], e[3]); break;
      case 5: tri.put(e[0], e[1], e[2]); tri.put(e[0], e[2], e[3]); tri.put(e[0], e[3], e[4]); break;
      case 6:
        tri.put(e[0], e[1], e[3]); tri.put(e[1], e[2], e[3]); tri.put(e[0], e[3], e[4]); tri.put(e[0], e[4], e[5]);
        break;
      default: break;
    }
    flat += sz;
  }
}
// The triangles around one inner vertex (:1262-1281): contours of three edges stay triangles, the
// others fan around it; returns whether any does.
template <typename Vid>
__device__ __forceinline__ bool slice_fans(uint64_t c, int cnt, const Vid& vid, int32_t inner, TriSink& tri) {
  bool used = false;
  int flat = 0;
  for (int t = 0; t < cnt; t++) {
    const int sz = cnt_size(c, t);
    if (sz == 3) {
      tri.put(vid[cnt_edge(c, flat)], vid[cnt_edge(c, flat + 1)], vid[cnt_edge(c, flat + 2)]);
    } else {
      used = true;
      for (int r = 0; r < sz; r++) tri.put(vid[cnt_edge(c, flat + r)], vid[cnt_edge(c, flat + (r + 1) % sz)], inner);
    }
    flat += sz;
  }
  return used;
}

__device__ AmbResult p_slice_dev(unsigned ic, const double F[8], double iso, const int32_t vid[12], int32_t ibase,
                                 TriSink& tri, const double (*P)[3], const double (*N)[3], const InnerOut* geo,
                                 double* prm) {
  AmbResult res{0, false};
  uint64_t to = ~0ull;
  int f_flag = 0;
#pragma unroll 1
  for (int f = 0; f < 6; f++) {
    const uint32_t fv = face_v_pack(f), fe = face_e_pack(f);
    const double f0 = F[nib(fv, 0)], f1 = F[nib(fv, 1)], f2 = F[nib(fv, 2)], f3 = F[nib(fv, 3)];
    int fc = 0;
    if (f0 >= iso) fc |= 1;
    if (f1 >= iso) fc |= 2;
    if (f2 >= iso) fc |= 4;
    if (f3 >= iso) fc |= 8;
    int sep = 0;
    if (fc == 6 || fc == 9) {
      const double val = decider(f0, f1, f2, f3);
      if (val > iso) sep = 1;
      else if (val < iso) sep = 0;
      else {
        f_flag |= 1 << f;
        const unsigned e_flag = 0x218;
        // an ambiguous face: its four edges are crossed
        double ec0 = edge_coord(F, iso, nib(fe, 0)), ec1 = edge_coord(F, iso, nib(fe, 1)),
               ec2 = edge_coord(F, iso, nib(fe, 2)), ec3 = edge_coord(F, iso, nib(fe, 3));
        if ((e_flag >> (f * 2)) & 1) { ec0 = 1 - ec0; ec2 = 1 - ec2; }
        if ((e_flag >> (f * 2)) & 2) { ec1 = 1 - ec1; ec3 = 1 - ec3; }
        const bool c1 = (ec1 < ec3 && ec0 > ec2), c2 = (ec1 > ec3 && ec0 < ec2);
        if (!c1 && !c2) {
          res.error = true;
          return res;
        }
        sep = (fc == 6) ? (c1 ? 0 : 1) : (c1 ? 1 : 0);
      }
    }
    face_segments(fc, sep, fe, to);
  }
  const uint64_t c = connect_contours(to, case_edge_mask(ic));
  const int cnt = cnt_count(c);

  // inner-ambiguity quadratic (:715-795)
  double ui[2] = {0, 0}, vi[2] = {0, 0}, wi[2] = {0, 0};
  unsigned q_sol = 0;
  const double a = (F[0] - F[1]) * (-F[6] + F[7] + F[4] - F[5]) - (F[4] - F[5]) * (-F[2] + F[3] + F[0] - F[1]);
  const double b = (iso - F[0]) * (-F[6] + F[7] + F[4] - F[5]) + (F[0] - F[1]) * (F[6] - F[4]) -
                   (iso - F[4]) * (-F[2] + F[3] + F[0] - F[1]) - (F[4] - F[5]) * (F[2] - F[0]);
  const double cc = (iso - F[0]) * (F[6] - F[4]) - (iso - F[4]) * (F[2] - F[0]);
  double d = b * b - 4 * a * cc;
  if (d > 0) {
    d = sqrt(d);
    ui[0] = (-b - d) / (2 * a);
    ui[1] = (-b + d) / (2 * a);
    double g1 = F[0] * (1 - ui[0]) + F[1] * ui[0];
    double g2 = F[2] * (1 - ui[0]) + F[3] * ui[0];
    vi[0] = (iso - g1) / (g2 - g1);
    if (isnan(vi[0]) || isinf(vi[0])) vi[0] = -1.f;
    g1 = F[0] * (1 - ui[1]) + F[1] * ui[1];
    g2 = F[2] * (1 - ui[1]) + F[3] * ui[1];
    vi[1] = (iso - g1) / (g2 - g1);
    if (isnan(vi[1]) || isinf(vi[1])) vi[1] = -1.f;
    g1 = F[0] * (1 - ui[0]) + F[1] * ui[0];
    g2 = F[4] * (1 - ui[0]) + F[5] * ui[0];
    wi[0] = (iso - g1) / (g2 - g1);
    if (isnan(wi[0]) || isinf(wi[0])) wi[0] = -1.f;
    g1 = F[0] * (1 - ui[1]) + F[1] * ui[1];
    g2 = F[4] * (1 - ui[1]) + F[5] * ui[1];
    wi[1] = (iso - g1) / (g2 - g1);
    if (isnan(wi[1]) || isinf(wi[1])) wi[1] = -1.f;
    if (f_flag & 1) { if (wi[0] < wi[1]) wi[0] = 0; else wi[1] = 0; }
    if (f_flag & 2) { if (wi[0] > wi[1]) wi[1] = 1; else wi[1] = 1; }
    if (f_flag & 4) { if (vi[0] < vi[1]) vi[0] = 0; else vi[1] = 0; }
    if (f_flag & 8) { if (vi[0] > vi[1]) vi[0] = 1; else vi[1] = 1; }
    if (f_flag & 16) { if (ui[0] < ui[1]) ui[0] = 0; else ui[1] = 0; }
    if (f_flag & 32) { if (ui[0] > ui[1]) ui[0] = 1; else ui[1] = 1; }
    if (0 < ui[0] && ui[0] < 1) q_sol |= 1;
    if (0 < ui[1] && ui[1] < 1) q_sol |= 2;
    if (0 < vi[0] && vi[0] < 1) q_sol |= 4;
    if (0 < vi[1] && vi[1] < 1) q_sol |= 8;
    if (0 < wi[0] && wi[0] < 1) q_sol |= 16;
    if (0 < wi[1] && wi[1] < 1) q_sol |= 32;
  }

  if (__popc(q_sol) == 6) {
    // tunnel or 12-vertex contour: inner hexagon (:831-1083)
    double ecoord[12];
    const uint32_t emask = case_edge_mask(ic);
    for (int e = 0; e < 12; e++) ecoord[e] = (emask >> e) & 1 ? edge_coord(F, iso, e) : 0.0;
    double hvt[6][3];
    hex_corners(ui, vi, wi, hvt);
    int not_tunnel = 0xF;
    if (cnt == 3) {
      const double uc_min = (ui[0] < ui[1]) ? ui[0] : ui[1];
      const double uc_max = (ui[0] < ui[1]) ? ui[1] : ui[0];
      int flat = 0;
      for (int t = 0; t < cnt; t++) {
        const int sz = cnt_size(c, t);
        if (sz == 3) {
          double umin = 2, umax = -2;
          const int e0 = cnt_edge(c, flat), e1 = cnt_edge(c, flat + 1), e2 = cnt_edge(c, flat + 2);
          const double u_e0 = e_vert(ecoord, e0, 0), u_e1 = e_vert(ecoord, e1, 0), u_e2 = e_vert(ecoord, e2, 0);
          umin = (u_e0 < umin) ? u_e0 : umin;
          umin = (u_e1 < umin) ? u_e1 : umin;
          umin = (u_e2 < umin) ? u_e2 : umin;
          umax = (u_e0 > umax) ? u_e0 : umax;
          umax = (u_e1 > umax) ? u_e1 : umax;
          umax = (u_e2 > umax) ? u_e1 : umax;  // the reference keeps u_e1 here
          if (uc_min > umax || uc_max < umin) {
            not_tunnel = t;
            tri.put(vid[e0], vid[e1], vid[e2]);
          }
        }
        flat += sz;
      }
    }
    if (geo)
      for (int s = 0; s < 6; s++) inner_vertex(P, N, hvt[s][0], hvt[s][1], hvt[s][2], *geo, (int64_t)ibase + s);
    if (prm) {
      prm[0] = ui[0]; prm[1] = ui[1]; prm[2] = vi[0]; prm[3] = vi[1]; prm[4] = wi[0]; prm[5] = wi[1];
    }
    res.inner = 6;
    unsigned char tcon[12];
    int flat = 0;
    for (int t = 0; t < cnt; t++) {
      const int sz = cnt_size(c, t);
      if (not_tunnel != t) {
        for (int r = 0; r < sz; r++) {
          unsigned idx = (unsigned)-1;
          double dist = 1000.;
          const int ci = cnt_edge(c, flat + r);
          const double ue = e_vert(ecoord, ci, 0), ve = e_vert(ecoord, ci, 1), we = e_vert(ecoord, ci, 2);
          for (int s = 0; s < 6; s++) {
            const double uval = ue - hvt[s][0], vval = ve - hvt[s][1], wval = we - hvt[s][2];
            const double val = uval * uval + vval * vval + wval * wval;
            if (dist > val) {
              idx = (unsigned)s;
              dist = val;
            }
          }
          tcon[ci] = (unsigned char)idx;
        }
        for (int r = 0; r < sz; r++) {
          const int tid1 = cnt_edge(c, flat + r), tid2 = cnt_edge(c, flat + (r + 1) % sz);
          const int cid1 = tcon[tid1], cid2 = tcon[tid2];
          const int rr = (cid1 - cid2) < 0 ? cid2 - cid1 : cid1 - cid2;
          const int dst = rr > 2 ? 6 - rr : rr;
          if (dst == 0) {
            tri.put(vid[tid1], vid[tid2], ibase + cid1);
          } else if (dst == 1) {
            double l1 = 0, l2 = 0;
            {
              const double a0 = e_vert(ecoord, tid1, 0) - hvt[cid2][0], a1 = e_vert(ecoord, tid1, 1) - hvt[cid2][1],
                           a2 = e_vert(ecoord, tid1, 2) - hvt[cid2][2];
              l1 = a0 * a0 + a1 * a1 + a2 * a2;
              const double b0 = e_vert(ecoord, tid2, 0) - hvt[cid1][0], b1 = e_vert(ecoord, tid2, 1) - hvt[cid1][1],
                           b2 = e_vert(ecoord, tid2, 2) - hvt[cid1][2];
              l2 = b0 * b0 + b1 * b1 + b2 * b2;
            }
            if (l1 < l2) {
              tri.put(vid[tid1], vid[tid2], ibase + cid2);
              tri.put(vid[tid1], ibase + cid2, ibase + cid1);
            } else {
              tri.put(vid[tid1], vid[tid2], ibase + cid1);
              tri.put(vid[tid2], ibase + cid2, ibase + cid1);
            }
          } else if (dst == 2) {
            const int dmax = (cid1 > cid2) ? cid1 : cid2, dmin = (cid1 < cid2) ? cid1 : cid2;
            const int cidm = ((dmax + 2) % 6 == dmin) ? (dmax + 1) % 6 : (dmax + dmin) / 2;
            tri.put(vid[tid1], vid[tid2], ibase + cidm);
            tri.put(vid[tid1], ibase + cidm, ibase + cid1);
            tri.put(vid[tid2], ibase + cid2, ibase + cidm);
          }
        }
      }
      flat += sz;
    }
    if (cnt == 1) {
      const bool s_ = decider(F[0], F[1], F[2], F[3]) <= iso;
      const bool of_ = (wi[1] < wi[0]) ? s_ : !s_;
      const int t0 = ibase, t1 = ibase + 1, t2 = ibase + 2, t3 = ibase + 3, t4 = ibase + 4, t5 = ibase + 5;
      if (!of_) {
        tri.put(t0, t2, t1); tri.put(t2, t4, t3); tri.put(t0, t5, t4); tri.put(t0, t4, t2);
      } else {
        tri.put(t0, t1, t2); tri.put(t2, t3, t4); tri.put(t0, t4, t5); tri.put(t0, t2, t4);
      }
    }
    return res;
  }
  // no tunnel
  const unsigned nr_u = ((q_sol & 0x5) == 0x5) + ((q_sol & 0xA) == 0xA);
  const unsigned nr_v = ((q_sol & 0x11) == 0x11) + ((q_sol & 0x22) == 0x22);
  const unsigned nr_w = ((q_sol & 0x18) == 0x18) + ((q_sol & 0x24) == 0x24);
  const unsigned nr_t = nr_u + nr_v + nr_w;
  if (nr_t == nr_u || nr_t == nr_v || nr_t == nr_w) {
    slice_contours(c, cnt, vid, tri);
    return res;
  }
  // saddle points: one inner vertex (:1178-1296)
  const unsigned fs00 = q_sol & 1, fs01 = (q_sol >> 1) & 1, fs10 = (q_sol >> 2) & 1, fs11 = (q_sol >> 3) & 1,
                 fs20 = (q_sol >> 4) & 1, fs21 = (q_sol >> 5) & 1;
  const unsigned fc1 = fs00 * fs10 + fs01 * fs11;
  const unsigned fc2 = fs00 * fs20 + fs01 * fs21;
  const unsigned fc3 = fs10 * fs21 + fs11 * fs20;
  const unsigned c_faces = fc1 + fc2 + fc3;
  double uc = 0, vc = 0, wc = 0;
  if (c_faces == 2) {
    if (fc1 == 0) {
      uc = fs00 * ui[0] + fs01 * ui[1]; vc = fs10 * vi[0] + fs11 * vi[1]; wc = fs10 * wi[1] + fs11 * wi[0];
    } else if (fc2 == 0) {
      uc = fs00 * ui[0] + fs01 * ui[1]; vc = fs00 * vi[0] + fs01 * vi[1]; wc = fs00 * wi[1] + fs01 * wi[0];
    } else if (fc3 == 0) {
      uc = fs10 * ui[0] + fs11 * ui[1]; vc = fs10 * vi[0] + fs11 * vi[1]; wc = fs10 * wi[0] + fs11 * wi[1];
    }
  } else if (c_faces == 3) {
    uc = (fs00 * ui[0] + fs01 * ui[1]) / (int)(fs00 + fs01);
    vc = (fs10 * vi[0] + fs11 * vi[1]) / (int)(fs10 + fs11);
    wc = (fs20 * wi[0] + fs21 * wi[1]) / (int)(fs20 + fs21);
  } else if (c_faces == 4) {
    const unsigned nu = fs00 + fs01, nv = fs10 + fs11, nw = fs20 + fs21;
    if (nw == 1) {
      uc = fs20 * ui[0] + fs21 * ui[1]; vc = fs21 * vi[0] + fs20 * vi[1]; wc = fs20 * wi[0] + fs21 * wi[1];
    } else if (nv == 1) {
      uc = fs10 * ui[0] + fs11 * ui[1]; vc = fs10 * vi[0] + fs11 * vi[1]; wc = fs11 * wi[0] + fs10 * wi[1];
    } else if (nu == 1) {
      uc = fs00 * ui[0] + fs01 * ui[1]; vc = fs00 * vi[0] + fs01 * vi[1]; wc = fs00 * wi[0] + fs01 * wi[1];
    }
  }
  const bool pt_used = slice_fans(c, cnt, vid, ibase, tri);
  if (pt_used) {
    res.inner = 1;
    if (geo) inner_vertex(P, N, uc, vc, wc, *geo, ibase);
    if (prm) {
      prm[0] = uc; prm[1] = vc; prm[2] = wc;
    }
  }
  return res;
}

// corner data of an ambiguous cell in float64: values, positions, normals
struct AmbCell {
  double F[8];
  double P[8][3];
  double N[8][3];
};

// corner positions and gradients (the inner vertices' trilinear sources)
__device__ __forceinline__ void amb_geometry(const Grid& g, int i, int j, int k, double P[8][3], double N[8][3]) {
  for (int q = 0; q < 8; q++) {
    const int ii = i + (q & 1), jj = j + ((q >> 1) & 1), kk = k + ((q >> 2) & 1);
    P[q][0] = g.ox + ii * g.dx;
    P[q][1] = g.oy + jj * g.dy;
    P[q][2] = g.oz + kk * g.dz;
    tmc_point_gradient(g, ii, jj, kk, N[q]);
  }
}

// One inner vertex of the emission: local parameters (u, v, w) of cell (i, j, k), written at index
// `at` of the outputs.
// The field difference along axis d at grid point p as the two values and whether it is one-sided
// (UGrid::gradient, mc/MarchingCubes.cpp:1451-1509).
__device__ __forceinline__ bool axis_pair(const Grid& g, const int p[3], int d, float& hi, float& lo) {
  const int n = d == 0 ? g.nx : (d == 1 ? g.ny : g.nz);
  int a[3] = {p[0], p[1], p[2]}, b[3] = {p[0], p[1], p[2]};
  const bool low = p[d] == 0, high = p[d] == n - 1;
  if (!high) a[d] += 1;
  if (!low) b[d] -= 1;
  hi = g.at(a[0], a[1], a[2]);
  lo = g.at(b[0], b[1], b[2]);
  return low || high;
}

// The reference's float64 arithmetic (:1073-1083 and :1283-1293), one axis after another.
__device__ __noinline__ void inner_vertex_f64(const Grid& g, int i, int j, int k, double u, double v, double w,
                                              const TmcVertexOut out, int64_t at) {
  double ip[3], in[3];
#pragma unroll
  for (int d = 0; d < 3; d++) {
    const double o = d == 0 ? g.ox : (d == 1 ? g.oy : g.oz), h = d == 0 ? g.dx : (d == 1 ? g.dy : g.dz);
    const int c0 = d == 0 ? i : (d == 1 ? j : k);
    double P[8], N[8];
#pragma unroll
    for (int q = 0; q < 8; q++) {
      const int p[3] = {i + (q & 1), j + ((q >> 1) & 1), k + ((q >> 2) & 1)};
      P[q] = o + (c0 + ((q >> d) & 1)) * h;
      float hi, lo;
      const bool one = axis_pair(g, p, d, hi, lo);
      N[q] = ((double)hi - (double)lo) / (one ? h : 2 * h);
    }
    ip[d] = (1 - w) * ((1 - v) * (P[0] + u * (P[1] - P[0])) + v * (P[2] + u * (P[3] - P[2]))) +
            w * ((1 - v) * (P[4] + u * (P[5] - P[4])) + v * (P[6] + u * (P[7] - P[6])));
    in[d] = (1 - w) * ((1 - v) * (N[0] + u * (N[1] - N[0])) + v * (N[2] + u * (N[3] - N[2]))) +
            w * ((1 - v) * (N[4] + u * (N[5] - N[4])) + v * (N[6] + u * (N[7] - N[6])));
  }
  const double factor = sqrt(in[0] * in[0] + in[1] * in[1] + in[2] * in[2]);
#pragma unroll
  for (int d = 0; d < 3; d++) {
    out.v[3 * at + d] = (float)ip[d];
    out.n[3 * at + d] = (float)(in[d] / factor);
    if (out.v64) out.v64[3 * at + d] = ip[d];
  }
}

// A coordinate of an inner vertex, o + (c + t) h, in float pairs; false where its float32 rounding may not be the
// float64 position's.  e: bound of t's error.  The pairs err by 2^-43 of the sum's terms; below 2^-80 their low
// parts leave the float range.
__device__ __forceinline__ bool inner_position_ff(const Grid& g, int d, int c, ffx::ff t, float e, float& out) {
  const ffx::ff h{g.sp_hi[d], g.sp_lo[d]}, o{g.org_hi[d], g.org_lo[d]};
  const ffx::ff y = ffx::ff_mul(ffx::ff_add(ffx::ff_from((float)c), t), h), x = ffx::ff_add(o, y);
  const float mag = fabsf(o.hi) + fabsf(y.hi);
  out = x.hi;
  return mag > 0x1p-80f && ffx::ff_certain(x, mag * 0x1p-43f + e * h.hi);
}

// The same for float32 outputs in float-float: positions as float64 rounds them, normals within 2^-30 of the
// float64 ones.  Writes nothing where float64 has to decide: kArithmetic, a position's rounding is left open or the
// gradients cancel to below 2^-10 of their size.  e: bound of the parameters' errors (0: none to speak of).  Each moves a gradient component by at
// most twice its inputs' size, so the normal by 10.4 e times their ratio to the gradient; kParameters where that may
// be more than 2^-20 (some 2^-30 in fact; steep fields, whose parameters have to come from float64).  At 2^-24 a
// quarter of the saddle field's are made again, 3.3 -> 4.3 ms instead of 3.45.
enum { kDone = 0, kArithmetic = 1, kParameters = 2 };
__device__ __noinline__ int inner_vertex_ff(const Grid& g, int i, int j, int k, ffx::ff U, ffx::ff V, ffx::ff W, float e,
                                             const TmcVertexOut out, int64_t at) {
  auto lerp = [](ffx::ff a, ffx::ff b, ffx::ff t) {
    return ffx::ff_add_abs(a, ffx::ff_mul(ffx::ff_add_abs(b, ffx::ff_neg(a)), t));
  };
  ffx::ff in[3];
  float scale = 0;
#pragma unroll
  for (int d = 0; d < 3; d++) {
    ffx::ff N[8];  // in units of 1 / (2 spacing)
#pragma unroll
    for (int q = 0; q < 8; q++) {
      const int p[3] = {i + (q & 1), j + ((q >> 1) & 1), k + ((q >> 2) & 1)};
      float hi, lo;
      const float m = axis_pair(g, p, d, hi, lo) ? 2.0f : 1.0f;
      const ffx::ff x = ffx::two_sum(hi, -lo);
      N[q] = ffx::ff{x.hi * m, x.lo * m};
      scale = fmaxf(scale, fabsf(N[q].hi) * g.inv2_hi[d]);
    }
    const ffx::ff t = lerp(lerp(lerp(N[0], N[1], U), lerp(N[2], N[3], U), V),
                           lerp(lerp(N[4], N[5], U), lerp(N[6], N[7], U), V), W);
    in[d] = ffx::ff_mul(t, ffx::ff{g.inv2_hi[d], g.inv2_lo[d]});
  }
  ffx::ff n[3];
  float dot, r0, x[3];
  unit_ff(in, n, dot, r0);
  if (e > 0.0f && !(10.5f * e * scale * r0 <= 0x1p-20f)) return kParameters;
  bool ok = dot > 0x1p-80f && dot < 0x1p80f && scale <= 0x1p10f * sqrtf(dot);
#pragma unroll
  for (int d = 0; d < 3; d++)
    ok = inner_position_ff(g, d, d == 0 ? i : (d == 1 ? j : k), d == 0 ? U : (d == 1 ? V : W), 0.0f, x[d]) && ok;
  if (!ok) return kArithmetic;
#pragma unroll
  for (int d = 0; d < 3; d++) {
    out.v[3 * at + d] = x[d];
    out.n[3 * at + d] = n[d].hi;
  }
  return kDone;
}

__device__ void load_amb_cell(const Grid& g, int i, int j, int k, const float u[8], AmbCell& a, bool geometry) {
#pragma unroll
  for (int q = 0; q < 8; q++) a.F[q] = u[q];
  if (geometry) amb_geometry(g, i, j, k, a.P, a.N);
}

// ------------------------------------------------------------------------------------------
// kernels
// ------------------------------------------------------------------------------------------
// What the classification knows of a cell from its case alone, as the bits of its record: the crossed
// edges among those it owns away from the lower borders, the table's triangles or the ambiguous flag.
__device__ __forceinline__ uint32_t case_record(unsigned cs, uint32_t owned) {
  return (case_edge_mask(cs) & owned) | (case_ambiguous(cs) ? (1u << 21) : (uint32_t)(c_tmc_tris[cs] & 0xF) << 15);
}
// One warp per tile of kScanTile consecutive cells: the crossed cells in cell order from the bit rows
// (list_tile), then their records at their slots, a cell per lane; ambiguous cells are listed by slot
// (amb_list) for the counting pass, which adds to this tile's sums.
template <int kPerTile>  // warps per tile (block_per_tile)
__global__ void __launch_bounds__(kClassifyThreads) tmc_classify_kernel(CellSpace space, int64_t tile0, int64_t tile1,
                                                                          uint32_t* rec, uint16_t* cellof,
                                                                          uint8_t* ccase, CellMask* mask,
                                                                          unsigned long long* tile_sums,
                                                                          unsigned long long* stats,
                                                                          uint32_t* amb_list, unsigned* amb_n) {
  pdl_begin();
  constexpr unsigned kAll = 0xffffffffu;
  constexpr int kTiles = kClassifyThreads / 32 / kPerTile;  // tiles per block
  __shared__ uint16_t lists[kTiles][kScanTile];
  __shared__ uint32_t inner_rec[256];  // records of cells off the lower borders
  for (int c = threadIdx.x; c < 256; c += blockDim.x) inner_rec[c] = case_record(c, owned_edges(1, 1, 1));
  __syncthreads();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int share = kPerTile == 1 ? 0 : wid;  // the warp's share of its tile
  const int64_t tile = tile0 + (int64_t)blockIdx.x * kTiles + (kPerTile == 1 ? wid : 0);
  if (tile >= tile1) return;  // the whole warp, or the whole block
  uint16_t* list = lists[kPerTile == 1 ? wid : 0];
  const Grid g = space.grid_of_tile(tile);
  const int64_t vbase = tile * kScanTile;
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
  unsigned amb = 0;
  for (int a0 = 32 * share; a0 < na; a0 += 32 * kPerTile) {
    const int a = a0 + lane;
    const uint32_t slot = (uint32_t)(vbase + a);
    bool listed = false;
    if (a < na) {
      const int off = list[a];
      int i, j, k;
      tcell_ijk(g, vbase + off - g.vbase, i, j, k);
      const unsigned cs = case_from_bits(g, i, j, k);
      const uint32_t r = (i > 0 && j > 0 && k > 0) ? inner_rec[cs] : case_record(cs, owned_edges(i, j, k));
      listed = (r >> 21) & 1;
      rec[slot] = r;
      cellof[slot] = (uint16_t)off;
      ccase[slot] = (uint8_t)cs;
      local += ((unsigned long long)trec_nv(r) << 32) | (unsigned long long)trec_ntri(r);
    }
    // ambiguous cells: their ranks to the front of the warp's share (its entries up to here are read)
    const unsigned bal = __ballot_sync(kAll, listed);
    if (bal) {
      __syncwarp();
      if (listed) list[share_entry<kPerTile>(share, amb + __popc(bal & ((1u << lane) - 1u)))] = (uint16_t)a;
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
    if (amb) atomicAdd(stats + 1, (unsigned long long)amb);
    if (share == 0 && na) atomicAdd(stats + 0, (unsigned long long)na);
    if (kPerTile == 1) tile_sums[tile] = local;
    else if (local) atomicAdd(tile_sum, local);
  }
  if (kPerTile > 1) {
    __syncthreads();
    if (threadIdx.x == 0) tile_sums[tile] = *tile_sum;
  }
}

// The classification lists the ambiguous cells in no useful order; p_slice's branches follow the MC
// case, so the list is sorted by case (counting sort over the 256 cases) before the float64 passes:
// the lanes of a warp then mostly take the same branches (the float64 pipe issues for the whole warp
// whatever its active lanes).  Key pass: each cell's case and the per-case counts.
//
// The passes over the list are launched before the host knows how many cells it has, with records for `cap`
// of them; a longer list (amb_cells) makes them do nothing, and the host launches them again with more.
// Waiting for the number first cost 30 us (small calls) to 85 us.
__device__ __forceinline__ unsigned amb_cells(const unsigned* n, unsigned cap) { return *n > cap ? 0u : *n; }
__global__ void __launch_bounds__(256) tmc_amb_key_kernel(const uint8_t* ccase, const uint32_t* list, const unsigned* count,
                                                          unsigned cap, uint8_t* key, unsigned* hist) {
  pdl_begin();
  __shared__ unsigned h[256];
  const unsigned n = amb_cells(count, cap);
  h[threadIdx.x] = 0;
  __syncthreads();
  for (unsigned a = blockIdx.x * blockDim.x + threadIdx.x; a < n; a += gridDim.x * blockDim.x) {
    const unsigned cs = ccase[list[a]];
    key[a] = (uint8_t)cs;
    atomicAdd(&h[cs], 1u);
  }
  __syncthreads();
  if (h[threadIdx.x]) atomicAdd(hist + threadIdx.x, h[threadIdx.x]);
}

// exclusive scan of the 256 counts into the scatter cursors (one block of 256 threads)
__global__ void tmc_amb_cursor_kernel(const unsigned* hist, unsigned* cursor) {
  pdl_begin();
  __shared__ unsigned x[256];
  x[threadIdx.x] = hist[threadIdx.x];
  __syncthreads();
  for (int o = 1; o < 256; o <<= 1) {
    const unsigned y = threadIdx.x >= (unsigned)o ? x[threadIdx.x - o] : 0u;
    __syncthreads();
    x[threadIdx.x] += y;
    __syncthreads();
  }
  cursor[threadIdx.x] = x[threadIdx.x] - hist[threadIdx.x];
}

// A block ranks its cells per case in shared memory and takes each case's range with one atomic: the
// per-case cursors are few and hot (one atomic per cell: 1.58 ms for the 11 M ambiguous cells of the
// 1024x1024x64 saddle field, 0.31 ms for the 1.3 M of the 512^3 noise field; 0.08 and 0.02 ms so).
constexpr int kSortItems = 8, kSortTile = 256 * kSortItems;
__global__ void __launch_bounds__(256) tmc_amb_sort_kernel(const uint32_t* list, const uint8_t* key,
                                                           const unsigned* count, unsigned cap, unsigned* cursor,
                                                           uint32_t* sorted) {
  pdl_begin();
  __shared__ unsigned h[256];
  const int64_t n = amb_cells(count, cap);
  for (int64_t base = (int64_t)blockIdx.x * kSortTile; base < n; base += (int64_t)gridDim.x * kSortTile) {
    h[threadIdx.x] = 0;
    __syncthreads();
    unsigned k[kSortItems], rank[kSortItems];
#pragma unroll
    for (int s = 0; s < kSortItems; s++) {
      const int64_t a = base + s * 256 + threadIdx.x;
      k[s] = a < n ? key[a] : 0u;
      rank[s] = a < n ? atomicAdd(&h[k[s]], 1u) : 0u;
    }
    __syncthreads();
    const unsigned c = h[threadIdx.x];
    __syncthreads();
    if (c) h[threadIdx.x] = atomicAdd(cursor + threadIdx.x, c);
    __syncthreads();
#pragma unroll
    for (int s = 0; s < kSortItems; s++) {
      const int64_t a = base + s * 256 + threadIdx.x;
      if (a < n) sorted[h[k[s]] + rank[s]] = list[a];
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------------------------------------
// p_slice's decisions on the FP32 pipes: float pairs with error bounds
// ------------------------------------------------------------------------------------------
// The float64 pipe runs at 1/57 of the float32 rate, and p_slice needs some 250 float64 operations
// per cell for a handful of decisions: which side of the isovalue each saddle face's decider lies on,
// and which roots of the inner quadratic lie in (0, 1).  Here each is computed in float pairs with a
// bound of its distance to the reference's float64 value (whose own roundings are some 2^-7 of it),
// and taken when the bound leaves no doubt.  A cell with any doubt, a singular face, an inner hexagon,
// or an inner vertex whose float64 position is an output, is left to the float64 kernel: 0.3 % of the
// ambiguous cells of the 512^3 noise field, 21 % of the 1024x1024x64 field of near-singular saddles.
// Both passes: 0.17 + 0.07 ms and 1.35 + 2.0 ms; 0.64 and 5.94 ms with every cell in float64.
//
// The corner values and the isovalue are scaled by the power of two that brings the largest into
// [1, 2) (the parameters do not change), away from both ends of the float range.
struct Root {
  ffx::ff x;
  float e;  // bound
};
// 1: x surely in (0, 1), 0: surely not, -1: in doubt
__device__ __forceinline__ int in_unit(const Root& r) {
  const float e = r.e * 1.01f, y = (1.0f - r.x.hi) - r.x.lo;
  if (r.x.hi > e && y > e) return 1;
  if (r.x.hi < -e || y < -e) return 0;
  return -1;
}
// (iso - g1) / (g2 - g1) with g1 = f0 + u (f1 - f0), g2 = f2 + u (f3 - f2)
__device__ __forceinline__ Root cross_root(float f0, float f1, float f2, float f3, ffx::ff iso, const Root& u) {
  using namespace ffx;
  const ff d0 = two_sum(f1, -f0), d1 = two_sum(f3, -f2);
  const ff g1 = ff_add_abs(ff_from(f0), ff_mul(u.x, d0)), g2 = ff_add_abs(ff_from(f2), ff_mul(u.x, d1));
  const ff num = ff_add_abs(iso, ff_neg(g1)), den = ff_add_abs(g2, ff_neg(g1));
  const float step = (1.0f + 2.0f * fabsf(u.x.hi)) * 0x1p-42f;  // of each pair operation here
  const float e1 = fabsf(d0.hi) * u.e + step, e2 = fabsf(d1.hi) * u.e + step;
  const float en = e1 + step, ed = e1 + e2 + 2 * step, ad = fabsf(den.hi);
  Root v;
  if (!(ad > 4 * ed && ad > 0x1p-60f)) return Root{ff_from(0.0f), INFINITY};
  v.x = ff_quot(num, den, rcp_est(den.hi));
  v.e = ((en + fabsf(v.x.hi) * ed) * rcp_est(ad - ed) + fabsf(v.x.hi) * 0x1p-42f) * 1.01f;
  return v;
}

// Contours and roots of one ambiguous cell with scaled corners f; false when in doubt.  The roots are
// those of mc/MarchingCubes.cpp:715-795, q_sol its bit set (0 without real roots).
__device__ __forceinline__ bool slice_decide(const float f[8], ffx::ff iso, unsigned cs, uint64_t& contours,
                                             Root u[2], Root v[2], Root w[2], unsigned& q_sol) {
  using namespace ffx;
  uint64_t to = ~0ull;
  bool ok = true;
#pragma unroll
  for (int q = 0; q < 6; q++) {
    const uint32_t fv = face_v_pack(q);
    const int fc = face_case(cs, fv);
    int sep = 0;
    if (fc == 6 || fc == 9) {
      const float a = f[nib(fv, 0)], b = f[nib(fv, 1)], c = f[nib(fv, 2)], d = f[nib(fv, 3)];
      const ff num = ff_add_abs(two_prod(a, d), ff_neg(two_prod(b, c)));
      const ff den = ff_add_abs(two_sum(a, -b), two_sum(d, -c));
      // decider > isovalue  <=>  num - iso den has den's sign; magnitudes 8 and 16
      const ff t = ff_add_abs(num, ff_neg(ff_mul(iso, den)));
      ok = ok && fabsf(t.hi) > 0x1p-38f && fabsf(den.hi) > 0x1p-24f;
      sep = (t.hi > 0.0f) == (den.hi > 0.0f);
    }
    face_segments(fc, sep, face_e_pack(q), to);
  }
  if (!ok) return false;
  contours = connect_contours(to, case_edge_mask(cs));
  // a = d01 t1 - d45 t2, b = i0 t1 + d01 d64 - i4 t2 - d45 d20, c = i0 d64 - i4 d20, t1 = d76 + d45,
  // t2 = d32 + d01, i = iso - f.  The d are exact; with T1, T2, I0, I4 the sums of the magnitudes that
  // t1, t2, i0, i4 add up, each product errs by at most 2^-43.8 of the product of those (the pair sums
  // by 2^-46, the pair product by 2^-45), their sums by 2^-45 more.
  const ff d01 = two_sum(f[0], -f[1]), d45 = two_sum(f[4], -f[5]), d64 = two_sum(f[6], -f[4]), d20 = two_sum(f[2], -f[0]);
  const ff d76 = two_sum(f[7], -f[6]), d32 = two_sum(f[3], -f[2]);
  const ff t1 = ff_add_abs(d76, d45), t2 = ff_add_abs(d32, d01);
  const ff i0 = ff_add_abs(iso, ff_from(-f[0])), i4 = ff_add_abs(iso, ff_from(-f[4]));
  const ff a = ff_add_abs(ff_mul(d01, t1), ff_neg(ff_mul(d45, t2)));
  const ff b = ff_add_abs(ff_add_abs(ff_mul(i0, t1), ff_mul(d01, d64)),
                          ff_neg(ff_add_abs(ff_mul(i4, t2), ff_mul(d45, d20))));
  const ff c = ff_add_abs(ff_mul(i0, d64), ff_neg(ff_mul(i4, d20)));
  const float m01 = fabsf(d01.hi), m45 = fabsf(d45.hi), m64 = fabsf(d64.hi), m20 = fabsf(d20.hi);
  const float T1 = fabsf(d76.hi) + m45, T2 = fabsf(d32.hi) + m01;
  const float I0 = fabsf(iso.hi) + fabsf(f[0]), I4 = fabsf(iso.hi) + fabsf(f[4]);
  const float Ea = (m01 * T1 + m45 * T2) * 0x1p-43f + 0x1p-80f;
  const float Eb = (I0 * T1 + m01 * m64 + I4 * T2 + m45 * m20) * 0x1p-43f + 0x1p-80f;
  const float Ec = (I0 * m64 + I4 * m20) * 0x1p-43f + 0x1p-80f;
  const float aa = fabsf(a.hi), ab = fabsf(b.hi), ac = fabsf(c.hi);
  const ff b2 = ff_mul(b, b), ac4 = ff_mul(ff{4 * a.hi, 4 * a.lo}, c);
  const ff d = ff_add_abs(b2, ff_neg(ac4));
  const float Ed = (2 * ab * Eb + 4 * (aa * Ec + ac * Ea) + (b2.hi + fabsf(ac4.hi)) * 0x1p-43f + 0x1p-70f) * 1.01f;
  q_sol = 0;
  if (d.hi < -Ed) return true;  // no real roots
  if (!(d.hi > 2 * Ed && aa > 4 * Ea)) return false;
  // s = sqrt(d): the rounded root and one Newton step
  const float s0 = sqrtf(d.hi), rs = rcp_est(s0);
  const ff p = two_prod(s0, s0);
  const ff s = quick_two_sum(s0, (((d.hi - p.hi) - p.lo) + d.lo) * (0.5f * rs));
  const float Es = Ed * rs + s0 * 0x1p-43f;
  const ff a2{2 * a.hi, 2 * a.lo};
  const float ra = rcp_est(a2.hi);
#pragma unroll
  for (int r = 0; r < 2; r++) {
    const ff n = ff_add_abs(ff_neg(b), r == 0 ? ff_neg(s) : s);
    u[r].x = ff_quot(n, a2, ra);
    const float au = fabsf(u[r].x.hi);
    u[r].e = ((Eb + Es + (ab + s0) * 0x1p-45f + au * (2 * Ea)) * rcp_est(2 * (aa - Ea)) + au * 0x1p-42f) * 1.01f;
    v[r] = cross_root(f[0], f[1], f[2], f[3], iso, u[r]);
    w[r] = cross_root(f[0], f[1], f[4], f[5], iso, u[r]);
    const int x = in_unit(u[r]), y = in_unit(v[r]), z = in_unit(w[r]);
    if (x < 0 || y < 0 || z < 0) return false;
    q_sol |= (unsigned)x << r | (unsigned)y << (2 + r) | (unsigned)z << (4 + r);
  }
  return true;
}

struct IdentityVid {  // local codes: edges 0..11
  __device__ __forceinline__ int operator[](int e) const { return e; }
};

// The inner vertex of a cell with saddle points (mc/MarchingCubes.cpp:1178-1261), from the certain
// roots, and the bound e of its parameters' errors (the values themselves are some 2^-10 of that off); false when
// the bound is above 2^-28.
__device__ __forceinline__ bool slice_center(unsigned q_sol, const Root u[2], const Root v[2], const Root w[2],
                                             ffx::ff out[3], float& e) {
  using namespace ffx;
  const unsigned f00 = q_sol & 1, f01 = (q_sol >> 1) & 1, f10 = (q_sol >> 2) & 1, f11 = (q_sol >> 3) & 1,
                 f20 = (q_sol >> 4) & 1, f21 = (q_sol >> 5) & 1;
  const unsigned fc1 = f00 * f10 + f01 * f11, fc2 = f00 * f20 + f01 * f21, fc3 = f10 * f21 + f11 * f20;
  const unsigned faces = fc1 + fc2 + fc3;
  e = 0;
  // s0 x0 + s1 x1
  auto pick = [&e](unsigned s0, const Root& x0, unsigned s1, const Root& x1) {
    e = fmaxf(e, (s0 ? x0.e : 0.0f) + (s1 ? x1.e : 0.0f));
    return ff_add_abs(s0 ? x0.x : ff_from(0.0f), s1 ? x1.x : ff_from(0.0f));
  };
  auto half = [](ff x, unsigned n) { return n == 2 ? ff{0.5f * x.hi, 0.5f * x.lo} : x; };
  out[0] = out[1] = out[2] = ff_from(0.0f);
  if (faces == 2) {
    if (fc1 == 0) {
      out[0] = pick(f00, u[0], f01, u[1]); out[1] = pick(f10, v[0], f11, v[1]); out[2] = pick(f10, w[1], f11, w[0]);
    } else if (fc2 == 0) {
      out[0] = pick(f00, u[0], f01, u[1]); out[1] = pick(f00, v[0], f01, v[1]); out[2] = pick(f00, w[1], f01, w[0]);
    } else if (fc3 == 0) {
      out[0] = pick(f10, u[0], f11, u[1]); out[1] = pick(f10, v[0], f11, v[1]); out[2] = pick(f10, w[0], f11, w[1]);
    }
  } else if (faces == 3) {
    if (!(f00 + f01) || !(f10 + f11) || !(f20 + f21)) return false;
    out[0] = half(pick(f00, u[0], f01, u[1]), f00 + f01);
    out[1] = half(pick(f10, v[0], f11, v[1]), f10 + f11);
    out[2] = half(pick(f20, w[0], f21, w[1]), f20 + f21);
  } else if (faces == 4) {
    if (f20 + f21 == 1) {
      out[0] = pick(f20, u[0], f21, u[1]); out[1] = pick(f21, v[0], f20, v[1]); out[2] = pick(f20, w[0], f21, w[1]);
    } else if (f10 + f11 == 1) {
      out[0] = pick(f10, u[0], f11, u[1]); out[1] = pick(f10, v[0], f11, v[1]); out[2] = pick(f11, w[0], f10, w[1]);
    } else if (f00 + f01 == 1) {
      out[0] = pick(f00, u[0], f01, u[1]); out[1] = pick(f00, v[0], f01, v[1]); out[2] = pick(f00, w[0], f01, w[1]);
    }
  }
  return e <= 0x1p-28f;
}

// Ambiguous cells from the case-sorted list, on the FP32 pipes: what tmc_amb_count_kernel writes for
// them, or their place in the list appended to `doubt` for that kernel.
__global__ void __launch_bounds__(128) tmc_amb_decide_kernel(CellSpace space, const uint16_t* cellof, uint32_t* rec,
                                                             unsigned long long* tile_sums, const uint32_t* list,
                                                             const unsigned* count, unsigned cap, AmbRec* recs,
                                                             uint32_t* doubt, unsigned* ndoubt) {
  pdl_begin();
  const unsigned na = amb_cells(count, cap);
  for (unsigned a = blockIdx.x * blockDim.x + threadIdx.x; a < na; a += gridDim.x * blockDim.x) {
    const uint32_t slot = list[a];
    const int64_t vcell = slot_cell(cellof, slot);
    const Grid& g = space.grids ? space.grids[ld(space.tile_vol + vcell / kScanTile)] : space.one;
    int i, j, k;
    tcell_ijk(g, vcell - g.vbase, i, j, k);
    float f[8];
    tload_corners(g, i, j, k, f);
    unsigned cs = 0;
    float m = fabsf(g.iso_f);
#pragma unroll
    for (int v = 0; v < 8; v++) {
      cs |= (unsigned)(f[v] >= g.iso_up) << v;
      m = fmaxf(m, fabsf(f[v]));
    }
    const bool pos64 = (g.flags & kGridPos64) != 0;
    // scale by 2^-e, e the exponent of the largest value (in two exact steps: e may be near the ends)
    const int ex = (int)(ffx::fbits(m) >> 23) - 127;
    bool ok = m > 0x1p-100f && m < 0x1p100f;
    const float sc = ffx::bitsf((uint32_t)(127 - (ok ? ex : 0)) << 23);
#pragma unroll
    for (int v = 0; v < 8; v++) f[v] *= sc;
    const ffx::ff iso{g.iso_f * sc, g.iso_lo * sc};
    uint64_t c = 0;
    Root u[2], v[2], w[2];
    unsigned q_sol = 0;
    ok = ok && slice_decide(f, iso, cs, c, u, v, w, q_sol) && __popc(q_sol) != 6;
    if (ok) {
      AmbRec& R = recs[a];
      TriSink ts{nullptr, R.tri, 0};
      const int cnt = cnt_count(c);
      const unsigned nr_u = ((q_sol & 0x5) == 0x5) + ((q_sol & 0xA) == 0xA);
      const unsigned nr_v = ((q_sol & 0x11) == 0x11) + ((q_sol & 0x22) == 0x22);
      const unsigned nr_w = ((q_sol & 0x18) == 0x18) + ((q_sol & 0x24) == 0x24);
      const unsigned nr_t = nr_u + nr_v + nr_w;
      int inner = 0;
      if (nr_t == nr_u || nr_t == nr_v || nr_t == nr_w) {
        slice_contours(c, cnt, IdentityVid{}, ts);
      } else {
        ffx::ff x[3];
        float e = 0, at;
        ok = !pos64 && slice_center(q_sol, u, v, w, x, e);
        // the emission's float32 position, from these parameters, has to be the float64 one's rounding
#pragma unroll
        for (int d = 0; d < 3; d++) ok = ok && inner_position_ff(g, d, d == 0 ? i : (d == 1 ? j : k), x[d], e, at);
        if (ok && slice_fans(c, cnt, IdentityVid{}, 12, ts)) {
          inner = 1;
          float2* prm = reinterpret_cast<float2*>(R.prm);
#pragma unroll
          for (int d = 0; d < 3; d++) prm[d] = make_float2(x[d].hi, x[d].lo);
          prm[3] = make_float2(e, 0.0f);
        }
      }
      if (ok) {
        R.slot = slot;
        R.info = cs | (uint32_t)ts.n << 8 | (uint32_t)inner << 14 | (1u << 19);
        rec[slot] |= (uint32_t)inner << 12 | (uint32_t)ts.n << 15;
        const unsigned long long add = ((unsigned long long)inner << 32) | (unsigned long long)ts.n;
        if (add) atomicAdd(tile_sums + (slot >> kTileShift), add);
      }
    }
    if (!ok) doubt[atomicAdd(ndoubt, 1u)] = a;
  }
}

// Ambiguous cells in doubt (places in the case-sorted list): p_slice in counting mode (float64); the counts go
// into the cell record and, atomically, into the cell's tile sum (one thread per listed cell, no
// tile barrier to wait on).  The triangles (as local codes) and the inner vertices' parameters go
// into the cell's ambiguous-cell record, which the emission pass reads instead of running p_slice.
__global__ void __launch_bounds__(128) tmc_amb_count_kernel(CellSpace space, const uint16_t* cellof, uint32_t* rec,
                                                            unsigned long long* tile_sums,
                                                            unsigned long long* stats, const uint32_t* list,
                                                            const uint32_t* doubt, const unsigned* count,
                                                            AmbRec* recs, unsigned* overflow) {
  pdl_begin();
  const unsigned na = *count;
  unsigned long long sing = 0;
  for (unsigned x = blockIdx.x * blockDim.x + threadIdx.x; x < na; x += gridDim.x * blockDim.x) {
    const unsigned a = doubt[x];
    const uint32_t slot = list[a];
    const int64_t vcell = slot_cell(cellof, slot);
    const Grid g = space.grid_of_tile(vcell / kScanTile);
    const int64_t cell = vcell - g.vbase;
    int i, j, k;
    tcell_ijk(g, cell, i, j, k);
    float u[8];
    tload_corners(g, i, j, k, u);
    unsigned cs = 0;
#pragma unroll
    for (int v = 0; v < 8; v++) cs |= (unsigned)(u[v] >= g.iso_up) << v;
    AmbCell amb;
    load_amb_cell(g, i, j, k, u, amb, false);
    int32_t vid[12];
    for (int e = 0; e < 12; e++) vid[e] = e;  // local codes: edges 0..11, inner vertices from 12
    AmbRec& R = recs[a];
    TriSink ts{nullptr, R.tri, 0};
    const AmbResult ar = p_slice_dev(cs, amb.F, g.iso, vid, 12, ts, amb.P, amb.N, nullptr, R.prm);
    R.slot = slot;
    R.info = cs | (uint32_t)ts.n << 8 | (uint32_t)ar.inner << 14 | (ts.n > kAmbRecTris ? (1u << 17) : 0u) |
             (ar.error ? (1u << 18) : 0u);
    rec[slot] |= (uint32_t)ar.inner << 12 | (uint32_t)ts.n << 15 | (ar.error ? (1u << 22) : 0u);
    const unsigned long long add = ((unsigned long long)ar.inner << 32) | (unsigned long long)ts.n;
    if (add) atomicAdd(tile_sums + (slot >> kTileShift), add);
    if (ts.n > kAmbRecTris) atomicAdd(overflow, 1u);
    sing += ar.error;
  }
  if (sing) atomicAdd(stats + 5, sing);
}

// In-tile exclusive scan of the listed cells' records -> per slot the record beside its vertex offset
// (rv, what the emission needs of a neighbour in one load) and the triangle offset, and the tile's
// chunks of 32 slots appended to the chunk list (common.cuh, list_chunks).
__global__ void __launch_bounds__(32 * kOffsetWarps) tmc_offsets_kernel(const CellMask* mask, const uint32_t* rec,
                                                                       const unsigned long long* tile_off,
                                                                       int64_t tiles, uint2* rv, int32_t* toff,
                                                                       uint32_t* chunks, unsigned* nchunks,
                                                                       const unsigned* gate, unsigned cap) {
  pdl_begin();
  if (*gate > cap) return;  // the whole grid: the counts are not complete
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
    for (int s = 0; s < kScanItems; s++) sum += ((unsigned long long)trec_nv(r[s]) << 32) | trec_ntri(r[s]);
    const unsigned long long inc = warp_inclusive_scan(sum);
    unsigned long long pre = carry + inc - sum;
    carry += __shfl_sync(0xffffffffu, inc, 31);
    uint32_t vo[kScanItems];
    int32_t to[kScanItems];
#pragma unroll
    for (int s = 0; s < kScanItems; s++) {
      vo[s] = (uint32_t)(pre >> 32);
      to[s] = (int32_t)(pre & 0xffffffffull);
      pre += ((unsigned long long)trec_nv(r[s]) << 32) | trec_ntri(r[s]);
    }
    store8_pairs(rv, first, end, r, vo);
    store8(toff, first, end, to);
  }
}

// An edge vertex's two field values and the two ends' field differences along each axis, as pairs of
// points: for the edge's own axis the ends share their values.  Borders: one-sided differences over
// one spacing (UGrid::gradient, mc/MarchingCubes.cpp:1451-1509), bit d of `one` for the first end and
// bit 4 + d for the second.
struct EdgeStencil {
  float f0, f1;
  float hi[2][3], lo[2][3];  // end, axis
  int one;
};
__device__ __forceinline__ void load_stencil(const Grid& g, const int p0[3], int ax, EdgeStencil& S) {
  const int64_t sy = g.nx, sz = (int64_t)g.nx * g.ny;
  const float* f = g.f + (int64_t)p0[2] * sz + (int64_t)p0[1] * sy + p0[0];
  const int64_t sa = ax == 0 ? 1 : (ax == 1 ? sy : sz);
  S.f0 = __ldg(f);
  S.f1 = __ldg(f + sa);
  S.one = 0;
#pragma unroll
  for (int d = 0; d < 3; d++) {
    const int64_t sd = d == 0 ? 1 : (d == 1 ? sy : sz);
    const int n = d == 0 ? g.nx : (d == 1 ? g.ny : g.nz);
    const bool own = d == ax;
    // first end: its neighbour before (after, on the edge's axis, is the second end)
    const bool low = p0[d] == 0, high = p0[d] == n - 1;  // the upper border is never on the edge's axis
    const float* l0 = low ? f : f - sd;
    const float* h0 = own ? f + sd : (high ? f : f + sd);
    S.lo[0][d] = __ldg(l0);
    S.hi[0][d] = __ldg(h0);
    S.one |= (int)(low || (!own && high)) << d;
    // second end
    const float* e = f + sa;
    const bool last = own ? p0[d] + 1 == n - 1 : high;
    S.lo[1][d] = __ldg(own ? f : (low ? e : e - sd));
    S.hi[1][d] = __ldg(last ? e : e + sd);
    S.one |= (int)(last || (!own && low)) << (4 + d);
  }
}

// The float32 normal from the gradient at edge parameter l in float pairs; false where its rounding may not be the
// float64 normal's.  el: bound of l's error.  A component errs by less than 32 2^-48 of its inputs' size (two pair
// sums of 3 2^-48, a product of 4, the difference up to twice the size; the scaling) and by their difference times el.
__device__ __forceinline__ bool edge_normal_ff(const Grid& g, const EdgeStencil& S, ffx::ff l, float el, float out[3]) {
  ffx::ff in[3], n[3];
  float scale = 0;
#pragma unroll
  for (int d = 0; d < 3; d++) {
    const ffx::ff s{g.inv2_hi[d], g.inv2_lo[d]};
    const float m0 = (S.one >> d) & 1 ? 2.0f : 1.0f, m1 = (S.one >> (4 + d)) & 1 ? 2.0f : 1.0f;
    // differences in units of 1 / (2 spacing); doubling is exact
    const ffx::ff a = ffx::two_sum(S.hi[0][d], -S.lo[0][d]), b = ffx::two_sum(S.hi[1][d], -S.lo[1][d]);
    const ffx::ff a2{a.hi * m0, a.lo * m0}, b2{b.hi * m1, b.lo * m1};
    in[d] = ffx::ff_mul(ffx::ff_add(a2, ffx::ff_mul(l, ffx::ff_sub(b2, a2))), s);
    scale = fmaxf(scale, fmaxf(fabsf(a2.hi), fabsf(b2.hi)) * s.hi);
  }
  const bool ok = unit_certain(in, scale * (0x1p-43f + 2 * el), n) && pairs_hold(scale, g.inv2_hi);
#pragma unroll
  for (int d = 0; d < 3; d++) out[d] = n[d].hi;
  return ok;
}

struct Float3 {
  float x[3];
};
// the reference's float64 normal, for the few edge vertices the float pairs do not serve
__device__ __noinline__ Float3 edge_normal_f64(const Grid& g, const EdgeStencil S) {
  const double f0 = S.f0, f1 = S.f1, l = (g.iso - f0) / (f1 - f0);
  const double sp[3] = {g.dx, g.dy, g.dz};
  double in[3];
  for (int d = 0; d < 3; d++) {
    const double n0 = ((double)S.hi[0][d] - (double)S.lo[0][d]) / ((S.one >> d) & 1 ? sp[d] : 2 * sp[d]);
    const double n1 = ((double)S.hi[1][d] - (double)S.lo[1][d]) / ((S.one >> (4 + d)) & 1 ? sp[d] : 2 * sp[d]);
    in[d] = (1 - l) * n0 + l * n1;
  }
  const double nl = sqrt(in[0] * in[0] + in[1] * in[1] + in[2] * in[2]);
  Float3 r;
  for (int d = 0; d < 3; d++) r.x[d] = (float)(in[d] / nl);
  return r;
}
// the same from float pairs where they decide its rounding
__device__ __noinline__ Float3 edge_normal_precise(const Grid& g, const EdgeStencil S) {
  const ffx::ff num = ffx::ff_sub(ffx::ff{g.iso_f, g.iso_lo}, ffx::ff_from(S.f0)), den = ffx::two_sum(S.f1, -S.f0);
  const ffx::ff l = ffx::ff_div(num, den);
  // the quotient's own error, and the isovalue's as a pair (2^-48 of it)
  const float el = 0x1p-43f + fabsf(g.iso_f) * 0x1p-47f * fabsf(ffx::rcp_est(den.hi));
  Float3 r;
  if (fabsf(den.hi) > 0x1p-90f && edge_normal_ff(g, S, l, el, r.x)) return r;
  return edge_normal_f64(g, S);
}

// The vertex on local edge e of cell (i, j, k), written at index idx.
// kF64: positions as t_mc (mc/MarchingCubes.cpp:241-254) in float64.  Otherwise the edge parameter l is a
// float32 quotient (within 2^-22) and the position within an ulp of what it gives (the grid coordinate
// i + l formed exactly as a float pair), and normals in float32, whose
// interpolation errs by a few ulps of its inputs' size: where the gradients cancel to below 1/16 of
// that it would exceed ~4e-6 of the unit normal, and the float pairs take over.
template <bool kF64>
__device__ __forceinline__ void edge_vertex(const Grid& g, int i, int j, int k, int e, const TmcVertexOut& out,
                                            int64_t idx) {
  const int v0 = edge_v0(e), ax = edge_axis(e);
  const int p0[3] = {i + (v0 & 1), j + ((v0 >> 1) & 1), k + ((v0 >> 2) & 1)};
  EdgeStencil S;
  load_stencil(g, p0, ax, S);
  const int64_t base = 3 * idx;
  if (kF64) {
    const double F0 = S.f0, F1 = S.f1;
    const double l = (g.iso - F0) / (F1 - F0);
#pragma unroll
    for (int d = 0; d < 3; d++) {
      const double o = d == 0 ? g.ox : (d == 1 ? g.oy : g.oz), h = d == 0 ? g.dx : (d == 1 ? g.dy : g.dz);
      const double a = o + p0[d] * h, b = d == ax ? o + (p0[d] + 1) * h : a;
      const double x = (1 - l) * a + l * b;
      out.v[base + d] = (float)x;
      out.v64[base + d] = x;
    }
    const Float3 n = edge_normal_precise(g, S);
#pragma unroll
    for (int d = 0; d < 3; d++) out.n[base + d] = n.x[d];
    return;
  }
  // the isovalue with its remainder: near 1000 a float is 3e-5 off, a good part of a small difference
  const float l = ((g.iso_f - S.f0) + g.iso_lo) / (S.f1 - S.f0);
#pragma unroll
  for (int d = 0; d < 3; d++) {
    // origin + (index + l) * spacing, with index + l exact as a float pair
    const ffx::ff t = (d == ax) ? ffx::two_sum((float)p0[d], l) : ffx::ff_from((float)p0[d]);
    const ffx::ff x = ffx::ff_add(ffx::ff{g.org_hi[d], g.org_lo[d]}, ffx::ff_mul(t, ffx::ff{g.sp_hi[d], g.sp_lo[d]}));
    out.v[base + d] = x.hi + x.lo;
  }
  float in[3], scale = 0;
#pragma unroll
  for (int d = 0; d < 3; d++) {
    const float s = g.inv2f[d];  // the border's 1/spacing is its double, exactly
    const float n0 = (S.hi[0][d] - S.lo[0][d]) * ((S.one >> d) & 1 ? 2 * s : s);
    const float n1 = (S.hi[1][d] - S.lo[1][d]) * ((S.one >> (4 + d)) & 1 ? 2 * s : s);
    in[d] = fmaf(l, n1 - n0, n0);
    scale = fmaxf(scale, fmaxf(fabsf(n0), fabsf(n1)));
  }
  const float dot = in[0] * in[0] + in[1] * in[1] + in[2] * in[2];
  if (dot > 0x1p-100f && dot < 0x1p100f && scale <= 16.0f * sqrtf(dot)) {
    const float rn = rsqrtf(dot);
#pragma unroll
    for (int d = 0; d < 3; d++) out.n[base + d] = in[d] * rn;
    return;
  }
  const Float3 n = edge_normal_precise(g, S);
#pragma unroll
  for (int d = 0; d < 3; d++) out.n[base + d] = n.x[d];
}

// Vertex index of crossed edge e of a cell, within the cell's volume, wherever its owner is (vfirst:
// the volume's first vertex in the space-wide numbering; first: the cell's first vertex, space-wide).
__device__ __forceinline__ int32_t border_vertex_id(const Grid& g, int i, int j, int k, int e, uint32_t own,
                                                    int32_t first, int32_t vfirst, const CellMask* mask,
                                                    const uint2* rv) {
  if (own & (1u << e)) return first - vfirst + __popc(own & ((1u << e) - 1u));
  int oi, oj, ok, oe = 0;
  edge_owner(i, j, k, e, oi, oj, ok, oe);
  const uint2 o = ld(rv + listed_slot(mask, (uint32_t)g.vcell(oi, oj, ok)));  // crossed edge: listed owner
  return (int32_t)o.y - vfirst + __popc(trec_owned(o.x) & ((1u << oe) - 1u));
}
// The same for all crossed edges (em) of a cell.
__device__ __forceinline__ void tmc_vertex_ids(const Grid& g, int i, int j, int k, uint32_t em, uint32_t own,
                                               int32_t first, int32_t vfirst, const CellMask* mask, const uint2* rv,
                                               int32_t vid[12]) {
#pragma unroll
  for (int e = 0; e < 12; e++) vid[e] = -1;
  // crossed edges as a mask, lowest first: the lanes of a warp resolve their k-th edges together
  for (uint32_t m = em; m; m &= m - 1) {
    const int e = __ffs(m) - 1;
    vid[e] = border_vertex_id(g, i, j, k, e, own, first, vfirst, mask, rv);
  }
}

// The vertex indices on the crossed edges of an interior cell (no index 0), into its column of vid.
// Nine of the edges belong to six neighbours; every neighbour that owns a crossed one is looked up
// once, and the six look-ups (a mask word, then the record and offset in one load) are independent.
__device__ __forceinline__ void interior_vertex_ids(int64_t vcell, int cx, int64_t cxy, uint32_t em, uint32_t own,
                                                    int32_t first, int32_t vfirst, const CellMask* mask,
                                                    const uint2* rv, int32_t* vid) {
  // neighbour (0,-1,-1): its edge 6 is edge 0 here; (0,0,-1): 5, 6 are 1, 2; (-1,0,-1): 5 is 3;
  // (0,-1,0): 6, 10 are 4, 9; (-1,0,0): 5, 10 are 7, 11; (-1,-1,0): 10 is 8
  const int64_t off[6] = {-cxy - cx, -cxy, -cxy - 1, -(int64_t)cx, -1, -(int64_t)cx - 1};
  constexpr int kEdge[6][2] = {{0, -1}, {1, 2}, {3, -1}, {4, 9}, {7, 11}, {8, -1}};
  constexpr int kOwner[6][2] = {{6, -1}, {5, 6}, {5, -1}, {6, 10}, {5, 10}, {10, -1}};
  uint32_t slot[6];
#pragma unroll
  for (int q = 0; q < 6; q++) {
    const uint32_t want = (1u << kEdge[q][0]) | (kEdge[q][1] >= 0 ? 1u << (kEdge[q][1] & 15) : 0u);
    slot[q] = (em & want) ? listed_slot(mask, (uint32_t)(vcell + off[q])) : 0xffffffffu;
  }
  uint2 o[6];
#pragma unroll
  for (int q = 0; q < 6; q++) o[q] = slot[q] != 0xffffffffu ? ld(rv + slot[q]) : make_uint2(0, 0);
#pragma unroll
  for (int q = 0; q < 6; q++)
#pragma unroll
    for (int t = 0; t < 2; t++)
      if (kEdge[q][t] >= 0)  // columns of edges that are not crossed are never read
        vid[32 * (kEdge[q][t] & 15)] =
            (int32_t)o[q].y - vfirst + __popc(trec_owned(o[q].x) & ((1u << (kOwner[q][t] & 15)) - 1u));
#pragma unroll
  for (int e = 5; e <= 10; e = e == 6 ? 10 : e + 1) vid[32 * e] = first - vfirst + __popc(own & ((1u << e) - 1u));
}

// Ambiguous cells from the counting pass's records, 32 to a warp: the recorded triangles with the
// cells' vertex indices, and the inner vertices from the recorded parameters, both taken one per lane
// (a cell has 1 to 36 triangles and 0, 1 or 6 inner vertices; the lane's cell is found by a binary
// search in the running counts).  Cells whose triangles overflow their records are left out
// (tmc_ambiguous_again_kernel).  Float32 outputs take positions and normals from float pairs, one
// axis after another (96 registers; 254 with float64 positions and all 24 gradients of a cell held
// at once).  512^3 noise: 0.81 -> 0.41 ms; 1024x1024x64 saddles, 11 M ambiguous cells: 10.3 -> 3.3 ms (3.2
// before the positions' roundings were looked at).
constexpr int kAmbThreads = 128;
__device__ __forceinline__ int owner_of(const int32_t* upto, int t) {  // first cell with upto[cell] > t
  int o = 0;
#pragma unroll
  for (int s = 16; s > 0; s >>= 1)
    if (upto[o + s - 1] <= t) o += s;
  return o;
}
__global__ void __launch_bounds__(kAmbThreads) tmc_ambiguous_kernel(CellSpace space, const CellMask* mask,
                                                                    const uint16_t* cellof, const uint2* rv,
                                                                    const int32_t* toff,
                                                                    const unsigned long long* tile_off,
                                                                    TmcVertexOut out, int32_t* tris,
                                                                    const AmbRec* recs, const unsigned* count,
                                                                    uint32_t* open, unsigned* nopen) {
  pdl_begin();
  constexpr int kWarps = kAmbThreads / 32;
  constexpr unsigned kAll = 0xffffffffu;
  __shared__ int32_t vids[kWarps][18 * 32];     // local code (edge, then inner vertex), cell
  __shared__ int32_t tupto[kWarps][32], iupto[kWarps][32], tbase[kWarps][32];
  __shared__ int4 cells[kWarps][32];            // i, j, k, volume
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int32_t* vid = vids[wid];
  const unsigned na = *count, step = gridDim.x * kAmbThreads;
  for (unsigned a0 = (blockIdx.x * kWarps + wid) * 32; a0 < na; a0 += step) {
    const unsigned a = a0 + lane;
    const uint32_t info = a < na ? recs[a].info : 0u;
    // a singular face: the reference emits nothing for the cell
    const bool on = a < na && !((info >> 17) & 3);
    int nt = 0, ni = 0, vol = 0;
    int32_t vfirst = 0;
    if (on) {
      nt = (int)((info >> 8) & 63);
      ni = (int)((info >> 14) & 7);
      const uint32_t slot = recs[a].slot;
      const int64_t vcell = slot_cell(cellof, slot);
      const uint2 r = ld(rv + slot);
      vol = space.grids ? ld(space.tile_vol + vcell / kScanTile) : 0;
      const Grid& g = space.grids ? space.grids[vol] : space.one;
      vfirst = (int32_t)(ld(tile_off + g.vbase / kScanTile) >> 32);
      int i, j, k;
      tcell_ijk(g, vcell - g.vbase, i, j, k);
      const uint32_t em = case_edge_mask(info & 0xFF), own = trec_owned(r.x);
      if (i > 0 && j > 0 && k > 0) {
        interior_vertex_ids(vcell, g.cx(), (int64_t)g.cx() * g.cy(), em, own, (int32_t)r.y, vfirst, mask, rv, vid + lane);
      } else {
        for (uint32_t m = em; m; m &= m - 1) {
          const int e = __ffs(m) - 1;
          vid[32 * e + lane] = border_vertex_id(g, i, j, k, e, own, (int32_t)r.y, vfirst, mask, rv);
        }
      }
      const int32_t ibase = (int32_t)r.y - vfirst + __popc(own);
      for (int q = 0; q < ni; q++) vid[32 * (12 + q) + lane] = ibase + q;
      cells[wid][lane] = make_int4(i, j, k, vol);
    }
    int tu = nt, iu = ni;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(kAll, tu, o), y = __shfl_up_sync(kAll, iu, o);
      if (lane >= o) {
        tu += x;
        iu += y;
      }
    }
    tupto[wid][lane] = tu;
    iupto[wid][lane] = iu;
    tbase[wid][lane] = nt ? ld(toff + recs[a].slot) - (tu - nt) : 0;
    const int ttotal = __shfl_sync(kAll, tu, 31), itotal = __shfl_sync(kAll, iu, 31);
    __syncwarp();
    for (int t = lane; t < ttotal; t += 32) {
      const int o = owner_of(tupto[wid], t);
      const int q = t - (o ? tupto[wid][o - 1] : 0);
      const unsigned code = recs[a0 + o].tri[q];
      int32_t* w = tris + 3 * ((int64_t)tbase[wid][o] + t);
      w[0] = vid[32 * (code & 31) + o];
      w[1] = vid[32 * ((code >> 5) & 31) + o];
      w[2] = vid[32 * ((code >> 10) & 31) + o];
    }
    for (int t = lane; t < itotal; t += 32) {
      const int o = owner_of(iupto[wid], t);
      const int from = o ? iupto[wid][o - 1] : 0, q = t - from;
      const int4 c = cells[wid][o];
      const Grid& g = space.grids ? space.grids[c.w] : space.one;
      const double* prm = recs[a0 + o].prm;
      if ((recs[a0 + o].info >> 19) & 1) {  // float pairs: one inner vertex, float32 outputs
        const float2* x = reinterpret_cast<const float2*>(prm);
        const ffx::ff U{x[0].x, x[0].y}, V{x[1].x, x[1].y}, W{x[2].x, x[2].y};
        const int64_t at = (int64_t)vid[32 * 12 + o] + (int32_t)(ld(tile_off + g.vbase / kScanTile) >> 32);
        const int what = inner_vertex_ff(g, c.x, c.y, c.z, U, V, W, x[3].x, out, at);
        if (what == kArithmetic)
          inner_vertex_f64(g, c.x, c.y, c.z, ffx::ff_to_double(U), ffx::ff_to_double(V), ffx::ff_to_double(W), out, at);
        const bool again = what == kParameters;
        const unsigned am = __activemask(), bal = __ballot_sync(am, again);
        if (bal) {  // for tmc_inner_again_kernel
          const int leader = __ffs(bal) - 1;
          unsigned base = 0;
          if (lane == leader) base = atomicAdd(nopen, (unsigned)__popc(bal));
          base = __shfl_sync(am, base, leader);
          if (again) open[base + __popc(bal & ((1u << lane) - 1u))] = a0 + o;
        }
        continue;
      }
      double u = prm[0], v = prm[1], w = prm[2];
      if (iupto[wid][o] - from > 1) {  // corner q of the inner hexagon (hex_corners)
        u = prm[(0x1C >> q) & 1];
        v = prm[2 + ((0x38 >> q) & 1)];
        w = prm[4 + ((0x0E >> q) & 1)];
      }
      // vertices are numbered within the volume; the outputs start at its first one
      const int64_t at = (int64_t)vid[32 * (12 + q) + o] + (int32_t)(ld(tile_off + g.vbase / kScanTile) >> 32);
      // float64 outputs requested for this volume: the reference's float64 arithmetic
      if ((g.flags & kGridPos64) || inner_vertex_ff(g, c.x, c.y, c.z, ffx::ff_from_double(u), ffx::ff_from_double(v),
                                                    ffx::ff_from_double(w), 0.0f, out, at) != kDone)
        inner_vertex_f64(g, c.x, c.y, c.z, u, v, w, out, at);
    }
    __syncwarp();  // the columns are read
  }
}

// The inner vertices whose normals need the reference's float64 parameters (listed by tmc_ambiguous_kernel): p_slice
// again for them, one thread per vertex.
__global__ void __launch_bounds__(128) tmc_inner_again_kernel(CellSpace space, const uint16_t* cellof, const uint2* rv,
                                                              TmcVertexOut out, const AmbRec* recs,
                                                              const uint32_t* open, const unsigned* nopen) {
  pdl_begin();
  const unsigned n = *nopen;
  for (unsigned x = blockIdx.x * blockDim.x + threadIdx.x; x < n; x += gridDim.x * blockDim.x) {
    const AmbRec& R = recs[open[x]];
    const uint32_t slot = R.slot;
    const int64_t vcell = slot_cell(cellof, slot);
    const uint2 r = rv[slot];
    const Grid& g = space.grids ? space.grids[ld(space.tile_vol + vcell / kScanTile)] : space.one;
    int i, j, k;
    tcell_ijk(g, vcell - g.vbase, i, j, k);
    float u[8];
    tload_corners(g, i, j, k, u);
    AmbCell amb;
    load_amb_cell(g, i, j, k, u, amb, false);
    int32_t vid[12];
    for (int e = 0; e < 12; e++) vid[e] = e;
    double prm[6] = {0, 0, 0, 0, 0, 0};
    TriSink ts{nullptr, nullptr, 0};
    p_slice_dev(R.info & 0xFF, amb.F, g.iso, vid, 12, ts, amb.P, amb.N, nullptr, prm);
    inner_vertex_f64(g, i, j, k, prm[0], prm[1], prm[2], out, (int64_t)(int32_t)r.y + __popc(trec_owned(r.x)));
  }
}

// The cells with more triangles than their records hold: p_slice again, one thread per record.  Launched
// only when the counting pass found one.
__global__ void __launch_bounds__(128) tmc_ambiguous_again_kernel(CellSpace space, const CellMask* mask,
                                                            const uint16_t* cellof, const uint2* rv,
                                                            const int32_t* toff,
                                                            const unsigned long long* tile_off, TmcVertexOut out,
                                                            int32_t* tris, const AmbRec* recs, const unsigned* count) {
  pdl_begin();
  const unsigned na = *count;
  for (unsigned a = blockIdx.x * blockDim.x + threadIdx.x; a < na; a += gridDim.x * blockDim.x) {
    const AmbRec& R = recs[a];
    const uint32_t info = R.info;
    if (((info >> 17) & 3) != 1) continue;
    const uint32_t slot = R.slot;
    const int64_t vcell = slot_cell(cellof, slot);
    const uint2 r = rv[slot];
    const Grid g = space.grid_of_tile(vcell / kScanTile);
    const int32_t vfirst = (int32_t)(tile_off[g.vbase / kScanTile] >> 32);
    int i, j, k;
    tcell_ijk(g, vcell - g.vbase, i, j, k);
    const unsigned cs = info & 0xFF;
    const uint32_t em = case_edge_mask(cs);
    const uint32_t own = trec_owned(r.x);
    int32_t vid[12];
    tmc_vertex_ids(g, i, j, k, em, own, (int32_t)r.y, vfirst, mask, rv, vid);
    const int32_t ibase = (int32_t)r.y - vfirst + __popc(own);
    // inner vertices are numbered within the volume: shift the outputs to its first vertex
    InnerOut io{out.v + 3 * (int64_t)vfirst, out.n + 3 * (int64_t)vfirst, out.v64 ? out.v64 + 3 * (int64_t)vfirst : nullptr};
    const int ni = (int)((info >> 14) & 7);
    int32_t* t = tris + 3 * (int64_t)toff[slot];
    float u[8];
    tload_corners(g, i, j, k, u);
    AmbCell amb;
    load_amb_cell(g, i, j, k, u, amb, ni > 0);
    TriSink ts{t, nullptr, 0};
    p_slice_dev(cs, amb.F, g.iso, vid, ibase, ts, amb.P, amb.N, &io, nullptr);
  }
}

// One warp per chunk of 32 consecutive listed cells of one tile (the chunk list of the offsets pass).
// A cell owns 0 to 12 vertices (1.06 on average on the 512^3 noise field, at most 3 away from the
// lower borders) and 0 to 5 triangles: with a cell per lane the lanes of a warp run as long as the
// largest, so the warp lists its vertices and then its triangles and takes them one per lane.
// Outputs are contiguous across the lanes.  Each cell's vertex indices (interior_vertex_ids) go to
// shared memory, a column per cell, where the triangle lanes pick them by edge.  Ambiguous cells'
// triangles come from their records (tmc_ambiguous_kernel).
// Bound by the latency of the field and neighbour loads (long_scoreboard, 58 % issue active, 24 lanes
// per instruction); 64 registers for four blocks per SM (80 registers and three blocks: 4 % slower).
// 512^3 noise field, 17.0 M vertices and 33.7 M triangles: 0.81 ms, 2.30 ms with a cell per lane;
// float64 positions (190x151x171 blobs): 20 us, 116 us with every normal in float64.
constexpr int kEmitThreads = 256;
__device__ const uint64_t d_tmc_tris[256] = TMC_TRIANGLES_INIT;
// kPos64: some volume of the launch wants float64 positions (the float64 edge-vertex path is
// compiled only into that instantiation)
template <bool kBatch, bool kPos64>
__global__ void __launch_bounds__(kEmitThreads, 4) tmc_emit_kernel(CellSpace space, const CellMask* mask,
                                                                const uint16_t* cellof, const uint8_t* ccase,
                                                                const uint2* rv, const int32_t* toff,
                                                                const unsigned long long* tile_off,
                                                                const uint32_t* chunks, const unsigned* nchunks,
                                                                TmcVertexOut out, int32_t* tris) {
  pdl_begin();
  constexpr int kWarps = kEmitThreads / 32;
  constexpr unsigned kAll = 0xffffffffu;
  __shared__ int32_t vids[kWarps][12 * 32];    // edge, cell
  __shared__ uint16_t items[kWarps][12 * 32];  // cell << 4 | edge, or cell << 4 | triangle
  __shared__ int4 cells[kWarps][32];           // i, j, k, first vertex minus its place in the list
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int32_t* vid = vids[wid];
  uint16_t* item = items[wid];
  int4* cell = cells[wid];
  const unsigned n = *nchunks;
  for (unsigned q = blockIdx.x * kWarps + wid; q < n; q += gridDim.x * kWarps) {
    const uint32_t chunk = chunks[q], slot0 = chunk & ~31u, slot = slot0 + lane;
    const bool in = (uint32_t)lane <= (chunk & 31u);  // the chunk's number of cells minus one
    const int64_t tile = slot0 >> kTileShift;
    const Grid& g = kBatch ? space.grids[ld(space.tile_vol + tile)] : space.one;
    const int32_t vfirst = kBatch ? (int32_t)(ld(tile_off + g.vbase / kScanTile) >> 32) : 0;
    uint2 r = make_uint2(0, 0);
    unsigned cs = 0;
    int64_t vcell = 0;
    int i = 0, j = 0, k = 0;
    if (in) {
      r = ld(rv + slot);
      cs = ld(ccase + slot);
      vcell = slot_cell(cellof, slot);
      tcell_ijk(g, vcell - g.vbase, i, j, k);
    }
    const uint32_t own = trec_owned(r.x);
    const bool amb = (r.x >> 21) & 1;
    const int nt = amb ? 0 : trec_ntri(r.x);  // of the table, for an unambiguous case
    // the vertices
    int upto = __popc(own);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(kAll, upto, o);
      if (lane >= o) upto += y;
    }
    int from = upto - __popc(own);
    int total = __shfl_sync(kAll, upto, 31);
    cell[lane] = make_int4(i, j, k, (int32_t)r.y - from);
    for (uint32_t m = own; m; m &= m - 1) item[from++] = (uint16_t)(lane << 4 | (__ffs(m) - 1));
    __syncwarp();
    for (int t = lane; t < total; t += 32) {
      const int x = item[t];
      const int4 c = cell[x >> 4];
      if (kPos64 && (!kBatch || (g.flags & kGridPos64))) edge_vertex<true>(g, c.x, c.y, c.z, x & 15, out, c.w + t);
      else edge_vertex<false>(g, c.x, c.y, c.z, x & 15, out, c.w + t);
    }
    // the vertex indices of the cells with triangles
    if (nt) {
      const uint32_t em = case_edge_mask(cs);
      if (i > 0 && j > 0 && k > 0) {
        interior_vertex_ids(vcell, g.cx(), (int64_t)g.cx() * g.cy(), em, own, (int32_t)r.y, vfirst, mask, rv, vid + lane);
      } else {
        for (uint32_t m = em; m; m &= m - 1) {
          const int e = __ffs(m) - 1;
          vid[32 * e + lane] = border_vertex_id(g, i, j, k, e, own, (int32_t)r.y, vfirst, mask, rv);
        }
      }
    }
    __syncwarp();  // the vertex list is read
    // the triangles
    upto = nt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(kAll, upto, o);
      if (lane >= o) upto += y;
    }
    from = upto - nt;
    total = __shfl_sync(kAll, upto, 31);
    const int32_t to = nt ? ld(toff + slot) - from : 0;
    for (int t = 0; t < nt; t++) item[from + t] = (uint16_t)(lane << 4 | t);
    __syncwarp();
    for (int t0 = 0; t0 < total; t0 += 32) {  // warp-uniform: the shuffles need every lane
      const int t = t0 + lane, x = t < total ? item[t] : 0, o = x >> 4;
      const unsigned ocs = __shfl_sync(kAll, cs, o);
      const int32_t oto = __shfl_sync(kAll, to, o);
      if (t < total) {
        // reversed winding (t_mc, mc/MarchingCubes.cpp:276-294)
        const unsigned tw = (unsigned)(__ldg(d_tmc_tris + ocs) >> (4 + 12 * (x & 15)));
        int32_t* w = tris + 3 * ((int64_t)oto + t);
        w[0] = vid[32 * ((tw >> 8) & 0xF) + o];
        w[1] = vid[32 * ((tw >> 4) & 0xF) + o];
        w[2] = vid[32 * (tw & 0xF) + o];
      }
    }
    __syncwarp();  // vid, item and cell are read
  }
}

// ------------------------------------------------------------------------------------------
// host-side launches
// ------------------------------------------------------------------------------------------
int64_t tmc_tiles(const CellSpace& space) { return ceil_div(space.n, kScanTile); }

int tmc_classify(const CellSpace& space, TmcScratch& s, int sms, cudaStream_t st, Prof* prof, const TileGate* gates,
                 int ngates) {
  const int64_t tiles = tmc_tiles(space);
  // the ambiguous-cell list lives in toff until the offsets kernel overwrites it
  uint32_t* amb_cells = reinterpret_cast<uint32_t*>(s.toff);
  int k = 0;
  {
    Stage t(prof, "tmc_classify", st);
    auto classify = [&](int64_t t0, int64_t t1, int z0, int z1) {
      k += launch_point_bits(space, z0, z1, sms, st);
      if (t1 <= t0) return;
      if (block_per_tile(t1 - t0, sms))
        launch(tmc_classify_kernel<8>, (unsigned)(t1 - t0), kClassifyThreads, st, 
            space, t0, t1, s.rec, s.cellof, s.ccase, s.mask, s.tile_sums, s.stats, amb_cells, s.amb_n);
      else
        launch(tmc_classify_kernel<1>, (unsigned)ceil_div(t1 - t0, kClassifyThreads / 32), kClassifyThreads, st, 
            space, t0, t1, s.rec, s.cellof, s.ccase, s.mask, s.tile_sums, s.stats, amb_cells, s.amb_n);
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
  }
  return k;
}

int tmc_count(const CellSpace& space, TmcScratch& s, int sms, cudaStream_t st, Prof* prof) {
  const int64_t tiles = tmc_tiles(space);
  const uint32_t* amb_list = reinterpret_cast<const uint32_t*>(s.toff);
  const int64_t cap = s.amb_cap;
  const unsigned cap32 = (unsigned)cap;
  {
    Stage ta(prof, "tmc_amb_count", st);
    // the list sorted by MC case (the records follow its order, so the emission pass is sorted too)
    auto blocks = [&](int64_t per) {
      return (unsigned)std::max<int64_t>(1, std::min<int64_t>(ceil_div(cap, per), (int64_t)sms * 8));
    };
    launch(tmc_amb_key_kernel, blocks(256), 256, st, s.ccase, amb_list, s.amb_n, cap32, s.amb_key, s.amb_hist);
    launch(tmc_amb_cursor_kernel, 1, 256, st, s.amb_hist, s.amb_hist + 256);
    launch(tmc_amb_sort_kernel, blocks(kSortTile), 256, st, amb_list, s.amb_key, s.amb_n, cap32, s.amb_hist + 256,
           s.amb_sorted);
    static const int r_decide = resident_blocks(tmc_amb_decide_kernel, 128);
    launch(tmc_amb_decide_kernel, (unsigned)wave_grid(r_decide, sms, 16, cap, 128), 128, st, space, s.cellof, s.rec,
           s.tile_sums, s.amb_sorted, s.amb_n, cap32, reinterpret_cast<AmbRec*>(s.amb_rec), s.amb_doubt,
           s.amb_hist + 512);
    static const int r_amb = resident_blocks(tmc_amb_count_kernel, 128);
    launch(tmc_amb_count_kernel, (unsigned)wave_grid(r_amb, sms, 4, cap, 128), 128, st, space, s.cellof, s.rec,
           s.tile_sums, s.stats, s.amb_sorted, s.amb_doubt, s.amb_hist + 512, reinterpret_cast<AmbRec*>(s.amb_rec),
           reinterpret_cast<unsigned*>(s.totals + 1));
  }
  Stage t(prof, "tmc_scan", st);
  scan_tile_sums(s.tile_sums, tiles, s.totals, st, s.amb_n, cap32);
  return 6;
}

int tmc_offsets(const CellSpace& space, TmcScratch& s, cudaStream_t st, Prof* prof) {
  Stage t(prof, "tmc_scan", st);
  const int64_t tiles = tmc_tiles(space);
  launch(tmc_offsets_kernel, (unsigned)ceil_div(tiles, kOffsetWarps), 32 * kOffsetWarps, st, s.mask, s.rec, s.tile_sums,
         tiles, s.rv, s.toff, s.chunks, s.amb_n + 1, s.amb_n, (unsigned)s.amb_cap);
  return 1;
}

int tmc_emit(const CellSpace& space, TmcScratch& s, int64_t n_amb, int64_t n_overflow, TmcVertexOut vo, int32_t* tris,
             const Tuning& tu, cudaStream_t st, Prof* prof) {
  const int sms = tu.sms;
  {
    Stage t(prof, "tmc_emit", st);
    // whole waves; the number of chunks is only known on the device
#define TMC_EMIT(B, P)                                                                                          \
  {                                                                                                             \
    static const int res = resident_blocks(tmc_emit_kernel<B, P>, kEmitThreads);                                \
    const int64_t blocks = wave_grid(res, sms, tu.emit_blocks_per_sm, ceil_div(space.n, 32), kEmitThreads / 32); \
    launch(tmc_emit_kernel<B, P>, (unsigned)blocks, kEmitThreads, st, space, s.mask, s.cellof, s.ccase, s.rv, s.toff, \
                                                                     s.tile_sums, s.chunks, s.amb_n + 1, vo, tris);  \
  }
    const bool pos64 = vo.v64 != nullptr;
    if (space.grids) {
      if (pos64) TMC_EMIT(true, true) else TMC_EMIT(true, false)
    } else {
      if (pos64) TMC_EMIT(false, true) else TMC_EMIT(false, false)
    }
#undef TMC_EMIT
  }
  if (n_amb == 0) return 1;
  Stage t2(prof, "tmc_ambiguous", st);
  static const int r_amb = resident_blocks(tmc_ambiguous_kernel, kAmbThreads);
  launch(tmc_ambiguous_kernel, (unsigned)wave_grid(r_amb, sms, 8, n_amb, kAmbThreads), kAmbThreads, st, 
      space, s.mask, s.cellof, s.rv, s.toff, s.tile_sums, vo, tris, reinterpret_cast<const AmbRec*>(s.amb_rec),
      s.amb_n, s.amb_doubt, s.amb_hist + 513);
  int launched = 2;
  if (space.grids || !vo.v64) {  // float64 outputs take no parameters as pairs
    static const int r_again = resident_blocks(tmc_inner_again_kernel, 128);
    launch(tmc_inner_again_kernel, (unsigned)wave_grid(r_again, sms, 4, n_amb, 128), 128, st, space, s.cellof, s.rv, vo,
           reinterpret_cast<const AmbRec*>(s.amb_rec), s.amb_doubt, s.amb_hist + 513);
    launched++;
  }
  if (n_overflow == 0) return launched;
  launch(tmc_ambiguous_again_kernel, (unsigned)std::max<int64_t>(1, std::min<int64_t>(ceil_div(n_amb, 128), (int64_t)sms * 2)), 128, st, space, s.mask, s.cellof, s.rv, s.toff, s.tile_sums, vo, tris,
                                             reinterpret_cast<const AmbRec*>(s.amb_rec), s.amb_n);
  return launched + 1;
}

}  // namespace tmc
