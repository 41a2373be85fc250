// Internal interface: topologically correct Marching Cubes kernels.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "common.cuh"
#include "profiler.h"

namespace tmc {

struct TmcVertexOut {
  float* v;
  float* n;
  double* v64;  // optional
};

constexpr int kTmcAmbRecWords = 32;

struct TmcScratch {
  uint32_t* rec;
  uint2* rv;            // record and vertex offset
  int32_t* toff;
  unsigned long long* tile_sums;
  unsigned long long* totals;
  unsigned long long* stats;
  unsigned* amb_n;      // [0] ambiguous cells listed by the classification, [1] chunks
  uint32_t* amb_rec;    // kTmcAmbRecWords words per ambiguous cell: what the counting pass keeps of
                        // its p_slice for the emission pass (tmc_cells.cu, AmbRec)
  uint32_t* amb_sorted; // the ambiguous cells' slots sorted by MC case (one per ambiguous cell)
  uint8_t* amb_key;     // their cases, in list order (one per ambiguous cell)
  uint32_t* amb_doubt;  // places in amb_sorted that float pairs could not decide, then records whose inner vertex needs
                        // float64 parameters (one per ambiguous cell)
  unsigned* amb_hist;   // 514: per-case counts, scatter cursors, cells in doubt, inner vertices to be made again
  // listed cells (common.cuh): rec, rv and toff hold one entry per listed cell at its slot, the
  // ambiguous-cell list holds slots
  CellMask* mask;       // per 32 cells of the space
  uint16_t* cellof;     // per slot: in-tile offset of the listed cell
  uint8_t* ccase;       // per slot: its MC case
  uint32_t* chunks;     // kScanTile / 32 per tile: the chunk list (scan.cuh)
  int64_t amb_cap;      // ambiguous cells that amb_rec, amb_sorted, amb_key and amb_doubt have room for
};

// The counters (stats, totals, amb_n, amb_hist) are zero when a call starts.
// Per-cell scratch is indexed in the cell space; triangles hold vertex indices within their own
// volume, and the volumes' vertices and triangles follow one another in the outputs.
int64_t tmc_tiles(const CellSpace& space);
// Classification: records of the crossed cells and the list of the ambiguous ones, whose number it
// leaves in *s.amb_n.  gates: as dmc_front_count's (classification of a host field arriving in slabs).
int tmc_classify(const CellSpace& space, TmcScratch& s, int sms, cudaStream_t st, Prof* prof = nullptr,
                 const TileGate* gates = nullptr, int ngates = 0);
// The ambiguous cells' counts (p_slice) into their records and s.amb_rec, then the totals: totals[0] =
// (vertices << 32) | triangles, totals[1] = cells with more triangles than their records hold (tmc_emit's
// n_overflow).  With more than s.amb_cap ambiguous cells it does nothing, and neither does tmc_offsets.
int tmc_count(const CellSpace& space, TmcScratch& s, int sms, cudaStream_t st, Prof* prof = nullptr);
// Vertex and triangle offsets of the listed cells, after tmc_count.  The host reads the totals and makes room
// for the results while it runs.
int tmc_offsets(const CellSpace& space, TmcScratch& s, cudaStream_t st, Prof* prof = nullptr);
int tmc_emit(const CellSpace& space, TmcScratch& s, int64_t n_amb, int64_t n_overflow, TmcVertexOut vo, int32_t* tris,
             const Tuning& tu, cudaStream_t st, Prof* prof = nullptr);

}  // namespace tmc
