// Listing the cells of a scan tile that the isosurface crosses (the classification front end shared
// by DMC and TMC): the points' sides as bit rows, the crossed cells from them by word operations, and
// their slots in cell order (CellMask, common.cuh).
#pragma once
#include "common.cuh"
#include "generators.cuh"
#include "scan.cuh"

namespace tmc {

static_assert(kScanTile == 1 << kTileShift, "listed-cell slots assume 2048-cell scan tiles");

// The points' sides: bit x of row (j, k) of Grid::bits is f(x, j, k) >= isovalue, row after row of
// Grid::wpr words.  One pass over the field, one ballot per 32 points: every later question of the
// classification is about these 1/32 of the field's bytes (16.8 MB of a 512^3 field, which the L2
// keeps).  Asking the field itself, each point compared for the four rows of cells around it and each
// cell's case put together from ballots, took 160-210 warp instructions per 32 cells and 0.66 ms at
// 512^3, bound by instruction issue; this pass is bound by the field's read (0.10 ms at 512^3, 5.2 TB/s)
// and the listing after it by its records (0.13 ms on the noise field; with one append per 32 cells to
// the ambiguous list's counter instead of one per tile: 0.28 ms).
// kGen: the field is generated (Grid::gen): every point is evaluated once and written to
// Grid::gen_out for the passes that follow.
// One launch covers planes z0 .. z1 of a single volume, or volumes of a batch (blockIdx.y).
constexpr int kBitThreads = 256;
constexpr int kMaxGridRows = 65535;  // largest gridDim.y
template <bool kGen>
__global__ void __launch_bounds__(kBitThreads) point_bits_kernel(Grid one, const Grid* grids, int z0, int z1) {
  pdl_begin();
  const Grid& g = grids ? grids[blockIdx.y] : one;
  const int lane = threadIdx.x & 31;
  const uint32_t wpr = (uint32_t)g.wpr;
  const uint32_t first = grids ? 0u : (uint32_t)z0 * (uint32_t)g.ny * wpr;
  const uint32_t words = (uint32_t)(grids ? g.nz : z1) * (uint32_t)g.ny * wpr;
  const float iso = g.iso_up;
  const int nx = g.nx;
  const uint32_t warps = gridDim.x * (kBitThreads / 32);
  // 32 words to a warp: word t's points across the lanes, then its ballot kept by lane t
  const uint32_t w0 = (first >> 5) + blockIdx.x * (kBitThreads / 32) + (threadIdx.x >> 5);
  for (uint64_t base = (uint64_t)w0 * 32; base < words; base += (uint64_t)warps * 32) {
    uint32_t row = g.div_wpr.div((uint32_t)base), w = (uint32_t)base - row * wpr, mine = 0;
    const int n = (int)(words - base < 32 ? words - base : 32);
    const float* p = g.f + (int64_t)row * nx;
    if (kGen) {
      const GenParams& P = *g.gen;
      const float2* tx = (const float2*)__ldg((const unsigned long long*)&P.tab[0]);
      const float2* ty = (const float2*)__ldg((const unsigned long long*)&P.tab[1]);
      const float2* tz = (const float2*)__ldg((const unsigned long long*)&P.tab[2]);
      const int surf = __ldg(&P.surface);
      int k = (int)(row / (uint32_t)g.ny), j = (int)(row - (uint32_t)k * (uint32_t)g.ny);
      for (int t = 0; t < n; t++) {
        const int x = (int)w * 32 + lane;
        float v = 0;
        if (x < nx) {
          v = tx ? combine_terms(surf, __ldg(tx + x), __ldg(ty + j), __ldg(tz + k)) : generated_at(P, g.gd, x, j, k);
          g.gen_out[(int64_t)row * nx + x] = v;
        }
        const unsigned b = __ballot_sync(0xffffffffu, x < nx && v >= iso);
        if (lane == t) mine = b;
        if (++w == wpr) {
          w = 0;
          row++;
          if (++j == g.ny) {
            j = 0;
            k++;
          }
        }
      }
    } else {
#pragma unroll 1
      for (int t = 0; t < n; t += 8) {
        float v[8];
#pragma unroll
        for (int s = 0; s < 8; s++) {  // eight words' loads in flight
          const int x = (int)w * 32 + lane;
          v[s] = (t + s < n && x < nx) ? __ldg(p + x) : -INFINITY;
          if (++w == wpr) {
            w = 0;
            p += nx;
          }
        }
#pragma unroll
        for (int s = 0; s < 8; s++) {
          const unsigned b = __ballot_sync(0xffffffffu, v[s] >= iso);
          if (lane == t + s) mine = b;
        }
      }
    }
    if (lane < n && base + lane >= first) g.bits[base + lane] = mine;
  }
}

// Launches the pass over planes z0 .. z1 of a single volume, or over all planes of a batch's volumes: a grid row
// per volume, as many volumes to a launch as a grid has rows.
inline int launch_point_bits(const CellSpace& space, int z0, int z1, int sms, cudaStream_t st) {
  static const int res = resident_blocks(point_bits_kernel<false>, kBitThreads);
  const bool batch = space.grids != nullptr;
  const int64_t words = batch ? space.max_bit_words : (int64_t)(z1 - z0) * space.one.ny * space.one.wpr;
  const int64_t need = ceil_div(ceil_div(words, 32) + 1, kBitThreads / 32);
  // two waves; a batch shares them among its volumes (at least a block each)
  const int64_t cap = std::max<int64_t>(1, (int64_t)res * sms * 2 / space.n_volumes);
  const unsigned blocks = (unsigned)std::min(need, cap);
  if (!batch) {
    if (space.one.gen) point_bits_kernel<true><<<blocks, kBitThreads, 0, st>>>(space.one, nullptr, z0, z1);
    else point_bits_kernel<false><<<blocks, kBitThreads, 0, st>>>(space.one, nullptr, z0, z1);
    return 1;
  }
  int k = 0;
  for (int v = 0; v < space.n_volumes; v += kMaxGridRows, k++) {
    const dim3 grid(blocks, (unsigned)std::min(kMaxGridRows, space.n_volumes - v));
    point_bits_kernel<false><<<grid, kBitThreads, 0, st>>>(space.one, space.grids + v, z0, z1);
  }
  return k;
}

// Bits x .. x + 31 of a row (lo) and x + 1 .. x + 32 (hi); x within the row.  Reads the word after
// x's, which may belong to the next row (its bits are not used then) or be the padding at the end.
__device__ __forceinline__ void row_bits(const uint32_t* row, int x, uint32_t& lo, uint32_t& hi) {
  const uint32_t a = ld(row + (x >> 5)), b = ld(row + (x >> 5) + 1);
  const int s = x & 31;
  lo = __funnelshift_r(a, b, s);
  hi = (lo >> 1) | ((b >> s) << 31);
}

// MC case of cell (i, j, k) from the bit rows
__device__ __forceinline__ unsigned case_from_bits(const Grid& g, int i, int j, int k) {
  const int64_t py = g.wpr, pz = (int64_t)g.ny * g.wpr;
  const uint32_t* r = g.bits + k * pz + j * py + (i >> 5);
  const int s = i & 31;
  unsigned c = 0;
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const uint32_t* p = r + (q & 1 ? py : 0) + (q & 2 ? pz : 0);
    c |= (__funnelshift_r(ld(p), ld(p + 1), s) & 3u) << (2 * q);
  }
  return c;
}

// The crossed cells (case neither 0 nor 255) among the 32 cells from local cell c0 on, in linear order:
// per piece of a row, the words of its four rows of points, each with its neighbour bit beside it.
__device__ __forceinline__ uint32_t crossed_word(const Grid& g, int64_t c0, int n) {
  if (n <= 0) return 0;
  const uint32_t cc = (uint32_t)c0, r = g.div_cx.div(cc);
  int i = (int)(cc - r * (uint32_t)g.cx());
  int k = (int)g.div_cy.div(r);
  int j = (int)(r - (uint32_t)k * (uint32_t)g.cy());
  const int64_t py = g.wpr, pz = (int64_t)g.ny * g.wpr;
  uint32_t out = 0;
  for (int at = 0; at < n;) {
    const int len = min(n - at, g.cx() - i);
    const uint32_t* row = g.bits + k * pz + j * py;
    uint32_t any = 0, all = 0xffffffffu;
#pragma unroll
    for (int q = 0; q < 4; q++) {
      uint32_t lo, hi;
      row_bits(row + (q & 1 ? py : 0) + (q & 2 ? pz : 0), i, lo, hi);
      any |= lo | hi;
      all &= lo & hi;
    }
    const uint32_t bits = any & ~all & (len == 32 ? 0xffffffffu : (1u << len) - 1u);
    out |= bits << at;
    at += len;
    i = 0;
    if (++j == g.cy()) {
      j = 0;
      k++;
    }
  }
  return out;
}

// How the classification kernels share tiles: one warp per tile (eight tiles per block), or, for spaces
// of few tiles, all eight warps of a block on one (the first lists it): a warp that walks a dense
// tile's 2048 cells alone sets the latency of a small call (57x48x71: 11.1 us, 5.7 us so).
constexpr int kClassifyThreads = 256;
inline bool block_per_tile(int64_t tiles, int sms) { return tiles <= (int64_t)sms * 8; }
// entry p of a warp's share of a tile's list: the warps take chunks of 32 entries in turn
template <int kPerTile>
__device__ __forceinline__ int share_entry(int wid, int p) {
  return kPerTile == 1 ? p : 32 * wid + 32 * kPerTile * (p >> 5) + (p & 31);
}

// One warp lists a tile: its 64 mask words (two per lane) with their in-tile prefixes go to `mask`
// (CellMask per 32 cells), the listed cells' in-tile offsets to `list` in cell order.  Returns their
// number; every lane of the warp calls it.
__device__ __forceinline__ int list_tile(const Grid& g, int64_t space_n, int64_t tile, CellMask* mask, uint16_t* list) {
  constexpr unsigned kAll = 0xffffffffu;
  constexpr int kWords = kScanTile / 32;  // 64
  const int lane = threadIdx.x & 31;
  const int64_t c0 = tile * kScanTile - g.vbase + 64 * lane;  // the lane's first cell in its volume
  const int64_t lim = min(space_n - g.vbase, g.ncells()) - c0;
  const uint32_t a = crossed_word(g, c0, (int)min(lim, (int64_t)32));
  const uint32_t b = crossed_word(g, c0 + 32, (int)min(lim - 32, (int64_t)32));
  const int ca = __popc(a), cb = __popc(b);
  int x = ca + cb;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(kAll, x, o);
    if (lane >= o) x += y;
  }
  int at = x - ca - cb;
  reinterpret_cast<uint4*>(mask + tile * kWords)[lane] = make_uint4(a, (uint32_t)at, b, (uint32_t)(at + ca));
  for (uint32_t m = a; m; m &= m - 1) list[at++] = (uint16_t)(64 * lane + __ffs(m) - 1);
  for (uint32_t m = b; m; m &= m - 1) list[at++] = (uint16_t)(64 * lane + 32 + __ffs(m) - 1);
  __syncwarp();
  return __shfl_sync(kAll, x, 31);
}

}  // namespace tmc
