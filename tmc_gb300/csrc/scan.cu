#include <cooperative_groups.h>

#include "scan.cuh"

namespace tmc {

// Scans all tile sums in place: a block of 1024 threads, or a cluster of kScanCluster of them.  Each warp owns
// a contiguous segment of 32 * rounds sums: its lanes add up their sums of all rounds (independent loads,
// eight in flight), the warps' totals are scanned in shared memory and the blocks' exchanged through it,
// and each warp walks its rounds again, eight at a time, and writes its exclusive prefixes.
// The pass is the latency and bandwidth of one SM, and little else runs beside it: a round at a time in both
// walks, each waiting for its load and its warp scan, one block took 37 us for the 65,152 tiles of 512^3
// cells, 29 us as it is now, and a cluster of eight 7 us.  Up to kScanAlone tiles, eight rounds, a block
// takes 2 to 5 us by itself and need not wait for others.
constexpr int kScanCluster = 8;
constexpr int64_t kScanAlone = 8192;
constexpr int kRoundsAhead = 8;
template <int kBlocks>
__device__ __forceinline__ void scan_sums(unsigned long long* sums, int64_t ntiles, unsigned long long* totals) {
  constexpr int T = 1024, W = T / 32;
  __shared__ unsigned long long wsum[W];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t rounds = (ntiles + kBlocks * T - 1) / (kBlocks * T);
  const int64_t seg = ((int64_t)(kBlocks > 1 ? blockIdx.x : 0) * W + w) * 32 * rounds + lane;
  unsigned long long run = 0;
  for (int64_t r = 0; r < rounds; r += kRoundsAhead) {
    unsigned long long v[kRoundsAhead];
#pragma unroll
    for (int q = 0; q < kRoundsAhead; q++) {
      const int64_t i = seg + 32 * (r + q);
      v[q] = r + q < rounds && i < ntiles ? sums[i] : 0ull;
    }
#pragma unroll
    for (int q = 0; q < kRoundsAhead; q++) run += v[q];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) run += __shfl_xor_sync(0xffffffffu, run, o);
  if (lane == 0) wsum[w] = run;
  __syncthreads();
  if (w == 0) wsum[lane] = warp_inclusive_scan(wsum[lane]);
  __syncthreads();
  unsigned long long pre = w ? wsum[w - 1] : 0ull, before = 0;  // sums of the blocks before this one
  if (kBlocks > 1) {
    const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    cluster.sync();  // every block's total is in its shared memory
    for (int b = 0; b < (int)blockIdx.x; b++) before += *cluster.map_shared_rank(wsum + W - 1, b);
    pre += before;
    cluster.sync();  // and has been read
  }
  for (int64_t r = 0; r < rounds; r += kRoundsAhead) {
    unsigned long long v[kRoundsAhead], x[kRoundsAhead];
#pragma unroll
    for (int q = 0; q < kRoundsAhead; q++) {
      const int64_t i = seg + 32 * (r + q);
      v[q] = r + q < rounds && i < ntiles ? sums[i] : 0ull;
    }
#pragma unroll
    for (int q = 0; q < kRoundsAhead; q++) x[q] = warp_inclusive_scan(v[q]);
#pragma unroll
    for (int q = 0; q < kRoundsAhead; q++) {
      const int64_t i = seg + 32 * (r + q);
      if (r + q < rounds && i < ntiles) sums[i] = pre + x[q] - v[q];
      pre += __shfl_sync(0xffffffffu, x[q], 31);
    }
  }
  if (threadIdx.x == T - 1 && (kBlocks == 1 || blockIdx.x == kBlocks - 1)) totals[0] = before + wsum[W - 1];
}
__global__ void __launch_bounds__(1024) scan_tile_sums_kernel(unsigned long long* sums, int64_t ntiles,
                                                              unsigned long long* totals, const unsigned* gate,
                                                              unsigned cap) {
  pdl_begin();
  if (gate && *gate > cap) return;  // the whole grid
  scan_sums<1>(sums, ntiles, totals);
}
__global__ void __cluster_dims__(kScanCluster) __launch_bounds__(1024)
    scan_tile_sums_cluster_kernel(unsigned long long* sums, int64_t ntiles, unsigned long long* totals,
                                  const unsigned* gate, unsigned cap) {
  pdl_begin();
  if (gate && *gate > cap) return;  // the whole grid
  scan_sums<kScanCluster>(sums, ntiles, totals);
}
void scan_tile_sums(unsigned long long* sums, int64_t ntiles, unsigned long long* totals, cudaStream_t st,
                    const unsigned* gate, unsigned cap) {
  if (ntiles <= kScanAlone) launch(scan_tile_sums_kernel, 1, 1024, st, sums, ntiles, totals, gate, cap);
  else launch(scan_tile_sums_cluster_kernel, kScanCluster, 1024, st, sums, ntiles, totals, gate, cap);
}
}  // namespace tmc

namespace tmc {

// Generic compaction scan of 0/1 flags (one byte each): out[i] = number of set flags before i.
__global__ void __launch_bounds__(kScanThreads) flag_tile_sum_kernel(const uint8_t* flags, int64_t n,
                                                                    unsigned long long* tile_sums) {
  pdl_begin();
  uint32_t f[kScanItems];
  load8(flags, (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanItems, n, f);
  unsigned long long s = 0;
#pragma unroll
  for (int q = 0; q < kScanItems; q++) s += f[q] != 0;
  unsigned long long tot;
  block_exclusive_scan<unsigned long long>(s, &tot);
  if (threadIdx.x == 0) tile_sums[blockIdx.x] = tot;
}

__global__ void __launch_bounds__(kScanThreads) flag_offsets_kernel(const uint8_t* flags, int64_t n,
                                                                   const unsigned long long* tile_off, int32_t* out) {
  pdl_begin();
  const int64_t first = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanItems;
  uint32_t f[kScanItems];
  load8(flags, first, n, f);
  int32_t sum = 0;
#pragma unroll
  for (int s = 0; s < kScanItems; s++) sum += f[s] != 0;
  int32_t tot;
  int32_t pre = (int32_t)tile_off[blockIdx.x] + block_exclusive_scan(sum, &tot);
  int32_t o[kScanItems];
#pragma unroll
  for (int s = 0; s < kScanItems; s++) {
    o[s] = pre;
    pre += f[s] != 0;
  }
  store8(out, first, n, o);
}
int64_t scan_tiles(int64_t n) { return (n + kScanTile - 1) / kScanTile; }

int scan_flags(const uint8_t* flags, int64_t n, int32_t* out, unsigned long long* tile_sums,
               unsigned long long* total, cudaStream_t st) {
  const int64_t tiles = scan_tiles(n);
  if (tiles == 0) {
    cudaMemsetAsync(total, 0, sizeof(unsigned long long), st);
    return 0;
  }
  launch(flag_tile_sum_kernel, (unsigned)tiles, kScanThreads, st, flags, n, tile_sums);
  scan_tile_sums(tile_sums, tiles, total, st);
  launch(flag_offsets_kernel, (unsigned)tiles, kScanThreads, st, flags, n, tile_sums, out);
  return 3;
}

}  // namespace tmc

namespace tmc {

// Exclusive scan of non-negative int32 values: out[i] = sum of in[0..i).
__global__ void __launch_bounds__(kScanThreads) i32_tile_sum_kernel(const int32_t* in, int64_t n,
                                                                   unsigned long long* tile_sums) {
  pdl_begin();
  uint32_t x[kScanItems];
  load8(reinterpret_cast<const uint32_t*>(in), (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanItems, n,
        x);
  unsigned long long s = 0;
#pragma unroll
  for (int q = 0; q < kScanItems; q++) s += x[q];
  unsigned long long tot;
  block_exclusive_scan<unsigned long long>(s, &tot);
  if (threadIdx.x == 0) tile_sums[blockIdx.x] = tot;
}

__global__ void __launch_bounds__(kScanThreads) i32_offsets_kernel(const int32_t* in, int64_t n,
                                                                  const unsigned long long* tile_off, int32_t* out) {
  pdl_begin();
  const int64_t first = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanItems;
  uint32_t x[kScanItems];
  load8(reinterpret_cast<const uint32_t*>(in), first, n, x);
  unsigned long long sum = 0;
#pragma unroll
  for (int s = 0; s < kScanItems; s++) sum += x[s];
  unsigned long long tot;
  unsigned long long pre = tile_off[blockIdx.x] + block_exclusive_scan(sum, &tot);
  int32_t o[kScanItems];
#pragma unroll
  for (int s = 0; s < kScanItems; s++) {
    o[s] = (int32_t)pre;
    pre += x[s];
  }
  store8(out, first, n, o);
}

int scan_i32(const int32_t* in, int64_t n, int32_t* out, unsigned long long* tile_sums, unsigned long long* total,
             cudaStream_t st) {
  const int64_t tiles = scan_tiles(n);
  if (tiles == 0) {
    cudaMemsetAsync(total, 0, sizeof(unsigned long long), st);
    return 0;
  }
  launch(i32_tile_sum_kernel, (unsigned)tiles, kScanThreads, st, in, n, tile_sums);
  scan_tile_sums(tile_sums, tiles, total, st);
  launch(i32_offsets_kernel, (unsigned)tiles, kScanThreads, st, in, n, tile_sums, out);
  return 3;
}

}  // namespace tmc
