// Internal interface between the runtime (C ABI) and the DMC kernels.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "common.cuh"
#include "profiler.h"

namespace tmc {

struct DmcVertexOut {
  float* v;        // 3 per vertex
  float* n;        // 3 per vertex
  double* v64;     // optional
  double* n64;     // optional: normals kept while the mesh is simplified, as float pairs (hi, lo) per 8-byte slot
  int64_t* vcell;  // optional (with vuvw)
  float* vuvw;
};

struct DmcScratch {
  uint32_t* rec;                  // per listed cell (slot)
  uint2* rv;                      // per listed cell (slot): record and vertex offset
  int32_t* qoff;                  // per listed cell (slot)
  uint32_t* vwork;                // per vertex: slot of the generating cell
  unsigned long long* tile_sums;  // per scan tile
  unsigned long long* totals;     // [0] = (vertices << 32) | quads
  unsigned long long* stats;      // 8 counters
  // per vertex: the projected points, those that take the whole search, those that lack a coordinate,
  // those left to the one-pass kernels
  float4* vp;
  uint32_t* fb_list;
  uint32_t* w_list;
  uint32_t* hard_list;
  unsigned* fb_count;             // entries of [0] fb_list, [1] tail_list, [2] w_list, [3] hard_list
  uint32_t* tail_list;            // vertices without a valid 7x7 sample (26x26 retry)
  // listed cells (common.cuh): rec, rv and qoff hold one entry per listed cell at its slot
  CellMask* mask;                 // per 32 cells of the space
  uint16_t* cellof;               // per slot: in-tile offset of the listed cell
  uint8_t* ccase;                 // per slot: the listed cell's MC case
  uint8_t* vrank;                 // per vertex: rank among its cell's vertices (vwork: the cell's slot)
  unsigned* amb_n;                // [0] listed cells with an ambiguous case (their slots wait in qoff), [1] chunks
  uint32_t* chunks;               // kScanTile / 32 per tile: the chunk list (scan.cuh)
  int64_t vcap;                   // vertices that vwork and vrank have room for
};

// Each launcher returns the number of kernels it launched.  The counters (stats, totals, amb_n,
// fb_count) are zero when a call starts.
// Per-cell scratch is indexed in the cell space (space.n cells, padding included).
// gates: classify the tiles of each gate once its event has completed (a host field arriving in
// slabs); none: the whole field is on the device
int dmc_front_count(const CellSpace& space, DmcScratch& s, int sms, cudaStream_t st, Prof* prof = nullptr,
                    const TileGate* gates = nullptr, int ngates = 0);
// Offsets of the listed cells and the vertices' cells (vwork, vrank), after dmc_front_count; nothing when there
// are more than vcap vertices.
int dmc_front_offsets(const CellSpace& space, DmcScratch& s, cudaStream_t st, Prof* prof = nullptr);
// Quads hold vertex indices within their own volume; vertices and quads of the volumes follow one
// another in the output arrays.
int dmc_front_emit(const CellSpace& space, DmcScratch& s, DmcVertexOut vo, int64_t nv, int32_t* quads,
                   uint8_t* colors, int flip, const Tuning& tu, cudaStream_t st, Prof* prof = nullptr);

// Twins and flags (zero on entry) of the halfedges of a single volume's quads, as build_halfedges makes them,
// and the number of quads around each vertex, after dmc_front_emit.
int dmc_front_twins(const CellSpace& space, const DmcScratch& s, int32_t* twin, uint8_t* flag, int32_t* deg, int sms,
                    cudaStream_t st);

}  // namespace tmc
