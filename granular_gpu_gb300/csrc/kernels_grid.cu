// kernels_grid.cu — uniform-grid neighbour structure.
//
// Replaces neighbor_search_{granular,boundary,upsampled}
// (GranularSystem.cu:65-395) and the primitives of CUDAFunctions.cuh:54-107:
//   cell key per particle  -> stable LSD radix sort of (key, index)
//   -> one gather of every SoA field -> cell_start from the sorted keys.
// The sort is stable, as thrust::sort_by_key on int keys is, so the sorted
// order is identical; it sorts only ceil(log2(C+1)) key bits.
#include <algorithm>
#include <mutex>
#include <utility>

#include "common.cuh"

namespace gg {

constexpr int kSortThreads = 256;
constexpr int kSortItems = 16;
constexpr int kSortTile = kSortThreads * kSortItems;  // 4096
constexpr int kScanThreads = 256;
constexpr int kScanItems = 16;
constexpr int kScanTile = kScanThreads * kScanItems;   // 4096
constexpr int kScanTopThreads = 1024;
constexpr int kScanTopItems = 16;
constexpr int64_t kScanMaxBlocks = (int64_t)kScanTopThreads * kScanTopItems;

int key_bits(int C) {
  int b = 1;
  while (b < 31 && ((int64_t)1 << b) <= (int64_t)C) ++b;
  return b;  // keys take values 0..C
}

// ------------------------------------------------------------------ hash

// mapParticles2Cells_CUDA (CUDAFunctions.cuh:91-107) with the sort's value
// array (thrust::sequence, GranularSystem.cu:71-73) produced in one pass.
// One block per sort tile: the block also counts the tile's first radix
// digits (bits 0-7), hist0 digit-major [256][tiles], so the sort's first
// pass does not read the keys again for its histogram.
__global__ void __launch_bounds__(kSortThreads) k_hash(Grid g, const float4* __restrict__ pos, int n,
                                                       uint32_t* __restrict__ keys, uint32_t* __restrict__ vals,
                                                       uint32_t* __restrict__ keys_copy, int tiles,
                                                       uint32_t* __restrict__ hist0) {
  __shared__ uint32_t h[256];
  h[threadIdx.x] = 0;
  __syncthreads();
  const int base = blockIdx.x * kSortTile;
  const unsigned lt = lanemask_lt();
#pragma unroll 4
  for (int r = 0; r < kSortItems; ++r) {
    const int i = base + r * kSortThreads + threadIdx.x;
    uint32_t d = 0u;
    if (i < n) {
      const float4 p = pos[i];
      const int3 c = floor_cell(g, make_float3(p.x, p.y, p.z));
      const uint32_t k = (uint32_t)cell_key(g, c.x, c.y, c.z);
      keys[i] = k;
      vals[i] = (uint32_t)i;
      if (keys_copy) keys_copy[i] = k;
      d = k & 255u;
    }
    // one shared-memory atomic per distinct digit of the warp (sorted or
    // nearly sorted keys share their digit across the warp)
    const unsigned peers = __match_any_sync(0xffffffffu, i < n ? d : 256u);
    if (i < n && (peers & lt) == 0) atomicAdd(&h[d], (uint32_t)__popc(peers));
  }
  __syncthreads();
  hist0[threadIdx.x * tiles + blockIdx.x] = h[threadIdx.x];
}

// ------------------------------------------------------------ block scan

// Exclusive scan of one int per thread across a block of kThreads threads;
// returns the block total in *total.
template <int kThreads>
__device__ __forceinline__ int block_exclusive_scan(int v, int* total) {
  __shared__ int warp_tot[kThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_tot[warp] = x;
  __syncthreads();
  if (warp == 0) {
    int w = lane < kThreads / 32 ? warp_tot[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    if (lane < kThreads / 32) warp_tot[lane] = w;
  }
  __syncthreads();
  const int warp_prefix = warp ? warp_tot[warp - 1] : 0;
  *total = warp_tot[kThreads / 32 - 1];
  __syncthreads();
  return warp_prefix + x - v;
}

// -------------------------------------------------------- exclusive scan
//
// The scans and the long sort's kernels are launched chained: the render
// points' grid of 2.5 M 0.108 to 0.091 ms a substep, of 1 M 0.106 to 0.077,
// the sort of 655,000 particles 0.087 to 0.064 and of 8.4 M 0.212 to 0.193,
// the compaction of 51,000 0.040 to 0.029.

__global__ void k_scan_reduce(const int32_t* in, int64_t n, int32_t* bsum) {
  const int t = (int)pdl_wait(threadIdx.x);
  const int64_t base = (int64_t)blockIdx.x * kScanTile + (int64_t)t * kScanItems;
  int s = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    const int64_t i = base + k;
    if (i < n) s += in[i];
  }
  int tot;
  block_exclusive_scan<kScanThreads>(s, &tot);
  if (t == 0) bsum[blockIdx.x] = tot;
}

__global__ void k_scan_top(int32_t* bsum, int nb, int32_t* total_out) {
  const int t = (int)pdl_wait(threadIdx.x);
  const int base = t * kScanTopItems;
  int v[kScanTopItems];
  int s = 0;
#pragma unroll
  for (int k = 0; k < kScanTopItems; ++k) {
    v[k] = (base + k < nb) ? bsum[base + k] : 0;
    s += v[k];
  }
  int tot;
  int run = block_exclusive_scan<kScanTopThreads>(s, &tot);
#pragma unroll
  for (int k = 0; k < kScanTopItems; ++k) {
    if (base + k < nb) bsum[base + k] = run;
    run += v[k];
  }
  if (t == 0 && total_out) *total_out = tot;
}

__global__ void k_scan_down(const int32_t* in, int32_t* out, int64_t n, const int32_t* bsum) {
  const int t = (int)pdl_wait(threadIdx.x);
  const int64_t base = (int64_t)blockIdx.x * kScanTile + (int64_t)t * kScanItems;
  int v[kScanItems];
  int s = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    const int64_t i = base + k;
    v[k] = i < n ? in[i] : 0;
    s += v[k];
  }
  int tot;
  int run = block_exclusive_scan<kScanThreads>(s, &tot) + bsum[blockIdx.x];
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    const int64_t i = base + k;
    if (i < n) out[i] = run;
    run += v[k];
  }
}

gg_status exclusive_scan(const int32_t* in, int32_t* out, int64_t n, SortScratch& s, cudaStream_t st,
                         int32_t* total_out_dev) {
  if (n <= 0) {
    if (total_out_dev) GG_CUDA(cudaMemsetAsync(total_out_dev, 0, sizeof(int32_t), st));
    return GG_OK;
  }
  const int64_t nb = (n + kScanTile - 1) / kScanTile;
  if (nb > kScanMaxBlocks || nb > s.scan_block_entries) {
    set_error("exclusive_scan: input larger than the scan scratch");
    return GG_ERR_INVALID_ARGUMENT;
  }
  GG_CUDA(launch_chained(k_scan_reduce, (int)nb, kScanThreads, st, in, n, s.scan_blocks));
  GG_CUDA(launch_chained(k_scan_top, 1, kScanTopThreads, st, s.scan_blocks, (int)nb, total_out_dev));
  GG_CUDA(launch_chained(k_scan_down, (int)nb, kScanThreads, st, in, out, n, s.scan_blocks));
  if (s.counter) *s.counter += 3;
  GG_CUDA(cudaGetLastError());
  return GG_OK;
}

// ------------------------------------------------------------ radix sort

// Per-tile histogram of one 8-bit digit; hist is digit-major [256][tiles].
// The thread's 16 keys are loaded before any is counted, so that their
// loads are in flight together; counts are aggregated over the lanes of a
// warp holding the same digit (one shared-memory atomic per digit).
__global__ void __launch_bounds__(kSortThreads) k_radix_hist(const uint32_t* keys, int n, int shift,
                                                             int tiles, uint32_t* hist) {
  __shared__ uint32_t h[256];
  const int t = (int)pdl_wait(threadIdx.x);
  h[t] = 0;
  const int base = blockIdx.x * kSortTile;
  uint32_t k[kSortItems];
#pragma unroll
  for (int r = 0; r < kSortItems; ++r) {
    const int i = base + r * kSortThreads + t;
    k[r] = i < n ? keys[i] : 0u;
  }
  __syncthreads();
  const unsigned lt = lanemask_lt();
#pragma unroll
  for (int r = 0; r < kSortItems; ++r) {
    const bool valid = base + r * kSortThreads + t < n;
    const uint32_t d = (k[r] >> shift) & 255u;
    const unsigned peers = __match_any_sync(0xffffffffu, valid ? d : 256u);
    if (valid && (peers & lt) == 0) atomicAdd(&h[d], (uint32_t)__popc(peers));
  }
  __syncthreads();
  hist[t * tiles + blockIdx.x] = h[t];
}

// Stable scatter of one digit: items are ranked in index order within the
// tile (rounds of 256 consecutive items; within a round by warp, then by
// lane).  offs holds the exclusive scan of the digit-major [256][tiles]
// histogram.  The thread's 16 keys and values are loaded before the first
// round, so that the rounds wait on no global load.  In a round, the first
// lane of each group of equal digits in a warp posts the group's size in
// wcnt; after the writes it adds the size to the digit's running base and
// clears its entry, so that wcnt is all zero between rounds.
__global__ void __launch_bounds__(kSortThreads) k_radix_scatter(const uint32_t* kin,
                                                                const uint32_t* vin,
                                                                uint32_t* kout,
                                                                uint32_t* vout, int n, int shift,
                                                                int tiles, const uint32_t* offs) {
  constexpr int W = kSortThreads / 32;
  __shared__ uint32_t base_d[256];
  __shared__ uint32_t wcnt[W][256];
  const int t = (int)pdl_wait(threadIdx.x), warp = t >> 5;
  const int base = blockIdx.x * kSortTile;
  uint32_t k[kSortItems], v[kSortItems];
#pragma unroll
  for (int r = 0; r < kSortItems; ++r) {
    const int i = base + r * kSortThreads + t;
    k[r] = i < n ? kin[i] : 0u;
    v[r] = i < n ? vin[i] : 0u;
  }
#pragma unroll
  for (int w = 0; w < W; ++w) wcnt[w][t] = 0;
  base_d[t] = offs[t * tiles + blockIdx.x];
  __syncthreads();
  const unsigned lt = lanemask_lt();
#pragma unroll
  for (int r = 0; r < kSortItems; ++r) {
    const bool valid = base + r * kSortThreads + t < n;
    const uint32_t d = (k[r] >> shift) & 255u;
    const unsigned peers = __match_any_sync(0xffffffffu, valid ? d : 256u);
    const bool leader = valid && (peers & lt) == 0;
    const uint32_t cnt = (uint32_t)__popc(peers);
    if (leader) wcnt[warp][d] = cnt;
    __syncthreads();
    if (valid) {
      uint32_t dst = base_d[d] + (uint32_t)__popc(peers & lt);
      for (int w = 0; w < warp; ++w) dst += wcnt[w][d];
      kout[dst] = k[r];
      vout[dst] = v[r];
    }
    __syncthreads();
    if (leader) {
      atomicAdd(&base_d[d], cnt);
      wcnt[warp][d] = 0;
    }
    __syncwarp();
  }
}

// ------------------------------------------------------------ short sort
//
// The same sort for inputs of at most kShortTiles tiles, in one launch for
// the keys and one a digit (against four a digit): the launches and the gaps
// between them were most of its time there.  A scatter block adds up the
// tile histograms itself (256 threads, one a digit, at most 128 rows) where
// the long sort scans them in three launches, and counts the next digit of
// each item at the tile it lands in.  The counts rotate through three
// tables: a pass reads one, adds to the next, and clears its row of the one
// after that.  Measured on a GB300, hash and sort against the long sort:
// 1,000 particles 18 and 50 us, 51,000 28 and 70 us, 125,000 50 and 95 us
// (two digits, two and three); 200,000 on caller memory with the cell table
// 51 and 97 us.  The rows that every block adds up set the limit.
constexpr int kShortTiles = 128;
constexpr int64_t short_max(int items) { return (int64_t)kShortTiles * kSortThreads * items; }
constexpr int64_t kShortMax = short_max(16);  // 524,288; with 16 items a thread, fewer where fewer make as many tiles

// A tile's keys and their first digits' counts.  kPacked: positions are
// float[3], else float4.
template <int kItems, bool kPacked>
__global__ void __launch_bounds__(kSortThreads) k_hash_short(Grid g, const float* pos, int n,
                                                             uint32_t* keys,
                                                             uint32_t* keys_copy, int tiles,
                                                             uint32_t* hist) {
  __shared__ uint32_t h[256];
  const int t = (int)pdl_wait(threadIdx.x);
  h[t] = 0;
  __syncthreads();
  const int base = blockIdx.x * kSortThreads * kItems;
  const unsigned lt = lanemask_lt();
#pragma unroll
  for (int r = 0; r < kItems; ++r) {
    const int i = base + r * kSortThreads + t;
    uint32_t d = 256u;
    if (i < n) {
      float3 p;
      if (kPacked) p = make_float3(pos[3 * (int64_t)i], pos[3 * (int64_t)i + 1], pos[3 * (int64_t)i + 2]);
      else p = f3(reinterpret_cast<const float4*>(pos)[i]);
      const int3 c = floor_cell(g, p);
      const uint32_t k = (uint32_t)cell_key(g, c.x, c.y, c.z);
      keys[i] = k;
      if (keys_copy) keys_copy[i] = k;
      d = k & 255u;
    }
    const unsigned peers = __match_any_sync(0xffffffffu, d);
    if (i < n && (peers & lt) == 0) atomicAdd(&h[d], (uint32_t)__popc(peers));
  }
  __syncthreads();
  const int row = blockIdx.x * 256 + t;
  hist[row] = h[t];
  hist[tiles * 256 + row] = 0;
}

// One digit: k_radix_scatter with the offsets worked out in the block.  vin
// null: the values are the indices.
template <int kItems>
__global__ void __launch_bounds__(kSortThreads) k_scatter_short(const uint32_t* kin,
                                                                const uint32_t* vin,
                                                                uint32_t* kout,
                                                                uint32_t* vout, int n, int pass,
                                                                int tiles, uint32_t* hist, int last) {
  constexpr int W = kSortThreads / 32, kTile = kSortThreads * kItems;
  __shared__ uint32_t base_d[256];
  __shared__ uint32_t wcnt[W][256];
  const int t = (int)pdl_wait(threadIdx.x), warp = t >> 5, shift = 8 * pass;
  const int base = blockIdx.x * kTile;
  const int64_t table = (int64_t)tiles * 256;
  const uint32_t* cur = hist + (pass % 3) * table;
  uint32_t* next = hist + ((pass + 1) % 3) * table;
  uint32_t k[kItems], v[kItems];
#pragma unroll
  for (int r = 0; r < kItems; ++r) {
    const int i = base + r * kSortThreads + t;
    k[r] = i < n ? kin[i] : 0u;
    v[r] = vin ? (i < n ? vin[i] : 0u) : (uint32_t)i;
  }
#pragma unroll
  for (int w = 0; w < W; ++w) wcnt[w][t] = 0;
  hist[((pass + 2) % 3) * table + blockIdx.x * 256 + t] = 0;
  uint32_t before = 0, total = 0;
#pragma unroll 16
  for (int b = 0; b < tiles; ++b) {
    const uint32_t c = cur[b * 256 + t];
    if (b < (int)blockIdx.x) before += c;
    total += c;
  }
  int all;
  base_d[t] = before + (uint32_t)block_exclusive_scan<kSortThreads>((int)total, &all);
  __syncthreads();
  const unsigned lt = lanemask_lt();
#pragma unroll
  for (int r = 0; r < kItems; ++r) {
    const bool valid = base + r * kSortThreads + t < n;
    const uint32_t d = (k[r] >> shift) & 255u;
    const unsigned peers = __match_any_sync(0xffffffffu, valid ? d : 256u);
    const bool leader = valid && (peers & lt) == 0;
    const uint32_t cnt = (uint32_t)__popc(peers);
    if (leader) wcnt[warp][d] = cnt;
    __syncthreads();
    if (valid) {
      uint32_t dst = base_d[d] + (uint32_t)__popc(peers & lt);
      for (int w = 0; w < warp; ++w) dst += wcnt[w][d];
      kout[dst] = k[r];
      vout[dst] = v[r];
      if (!last) atomicAdd(&next[dst / kTile * 256 + ((k[r] >> (shift + 8)) & 255u)], 1u);
    }
    __syncthreads();
    if (leader) {
      atomicAdd(&base_d[d], cnt);
      wcnt[warp][d] = 0;
    }
    __syncwarp();
  }
}

template <int kItems, bool kPacked>
static gg_status short_sort_items(const Grid& g, const float* pos, int n, SortScratch& s, uint32_t* keys_out,
                                  uint32_t* perm_out, uint32_t* keys_unsorted_out, cudaStream_t st, gg_system* prof) {
  const int tiles = (n + kSortThreads * kItems - 1) / (kSortThreads * kItems);
  const int passes = (key_bits(g.C) + 7) / 8;
  if (prof) prof_begin(prof, PC_HASH, st);
  GG_CUDA(launch_chained(k_hash_short<kItems, kPacked>, tiles, kSortThreads, st, g, pos, n, s.k[0], keys_unsorted_out,
                         tiles, s.hist));
  if (prof) prof_end(prof, PC_HASH, n, st);
  if (prof) prof_begin(prof, PC_SORT, st);
  for (int p = 0; p < passes; ++p) {
    const bool last = p == passes - 1;
    GG_CUDA(launch_chained(k_scatter_short<kItems>, tiles, kSortThreads, st, s.k[p & 1], p ? s.v[p & 1] : nullptr,
                           last ? keys_out : s.k[(p & 1) ^ 1], last ? perm_out : s.v[(p & 1) ^ 1], n, p, tiles, s.hist,
                           last ? 1 : 0));
  }
  if (prof) prof_end(prof, PC_SORT, n, st);
  if (s.counter) *s.counter += 1 + passes;
  GG_CUDA(cudaGetLastError());
  return GG_OK;
}

template <bool kPacked>
static gg_status short_sort(const Grid& g, const float* pos, int64_t n, SortScratch& s, uint32_t* keys_out,
                            uint32_t* perm_out, uint32_t* keys_unsorted_out, cudaStream_t st, gg_system* prof) {
  auto sort = n <= short_max(4)   ? short_sort_items<4, kPacked>
              : n <= short_max(8) ? short_sort_items<8, kPacked>
                                  : short_sort_items<16, kPacked>;
  return sort(g, pos, (int)n, s, keys_out, perm_out, keys_unsorted_out, st, prof);
}

gg_status sort_scratch_alloc(SortScratch& s, int64_t capacity) {
  if (capacity < 1) capacity = 1;
  s.capacity = capacity;
  const int64_t tiles = (capacity + kSortTile - 1) / kSortTile;
  s.hist_entries = std::max<int64_t>(tiles, 3 * kShortTiles) * 256;
  // scan blocks must cover the largest scanned array: hist, cell table, particles
  s.scan_block_entries = kScanMaxBlocks;
  for (int i = 0; i < 2; ++i) {
    GG_CUDA(cudaMalloc(&s.k[i], sizeof(uint32_t) * capacity));
    GG_CUDA(cudaMalloc(&s.v[i], sizeof(uint32_t) * capacity));
  }
  GG_CUDA(cudaMalloc(&s.hist, sizeof(uint32_t) * s.hist_entries));
  GG_CUDA(cudaMalloc(&s.scan_blocks, sizeof(int32_t) * s.scan_block_entries));
  return GG_OK;
}

void sort_scratch_free(SortScratch& s) {
  for (int i = 0; i < 2; ++i) {
    cudaFree(s.k[i]);
    cudaFree(s.v[i]);
    s.k[i] = s.v[i] = nullptr;
  }
  cudaFree(s.hist);
  cudaFree(s.scan_blocks);
  s.hist = nullptr;
  s.scan_blocks = nullptr;
}

// Stable LSD sort of the (key, value) pairs held in s.k[0], s.v[0]; the
// last pass writes keys_out / perm_out.  s.hist already holds the first
// digit's tile histogram (counted by the hash kernel).
static gg_status radix_sort_pairs(const Grid& g, int64_t n, SortScratch& s, uint32_t* keys_out, uint32_t* perm_out,
                                  cudaStream_t st) {
  const int nn = (int)n;
  const int bits = key_bits(g.C);
  const int passes = (bits + 7) / 8;
  const int tiles = (int)((n + kSortTile - 1) / kSortTile);
  int src = 0;
  for (int p = 0; p < passes; ++p) {
    const int shift = 8 * p;
    const bool last = p == passes - 1;
    uint32_t* ko = last ? keys_out : s.k[src ^ 1];
    uint32_t* vo = last ? perm_out : s.v[src ^ 1];
    if (p > 0) {
      GG_CUDA(launch_chained(k_radix_hist, tiles, kSortThreads, st, s.k[src], nn, shift, tiles, s.hist));
      if (s.counter) *s.counter += 1;
    }
    gg_status rc = exclusive_scan((const int32_t*)s.hist, (int32_t*)s.hist, (int64_t)tiles * 256, s, st, nullptr);
    if (rc != GG_OK) return rc;
    GG_CUDA(launch_chained(k_radix_scatter, tiles, kSortThreads, st, s.k[src], s.v[src], ko, vo, nn, shift, tiles,
                           s.hist));
    if (s.counter) *s.counter += 1;
    src ^= 1;
  }
  GG_CUDA(cudaGetLastError());
  return GG_OK;
}

gg_status grid_sort(const Grid& g, const float4* pos, int64_t n, SortScratch& s, uint32_t* keys_out,
                    uint32_t* perm_out, uint32_t* keys_unsorted_out, cudaStream_t st, gg_system* prof) {
  if (n <= 0) return GG_OK;
  if (n > s.capacity) {
    set_error("grid_sort: more elements than the sort scratch holds");
    return GG_ERR_INVALID_ARGUMENT;
  }
  if (n <= kShortMax)
    return short_sort<false>(g, reinterpret_cast<const float*>(pos), n, s, keys_out, perm_out, keys_unsorted_out, st,
                             prof);
  const int nn = (int)n;
  if (prof) prof_begin(prof, PC_HASH, st);
  const int tiles = (int)((n + kSortTile - 1) / kSortTile);
  k_hash<<<tiles, kSortThreads, 0, st>>>(g, pos, nn, s.k[0], s.v[0], keys_unsorted_out, tiles, s.hist);
  if (s.counter) *s.counter += 1;
  if (prof) prof_end(prof, PC_HASH, n, st);
  if (prof) prof_begin(prof, PC_SORT, st);
  gg_status rc = radix_sort_pairs(g, n, s, keys_out, perm_out, st);
  if (prof) prof_end(prof, PC_SORT, n, st);
  return rc;
}

// ------------------------------------------------------------ cell start

// countingInCell_CUDA (CUDAFunctions.cuh:54-61) and its scan, from the
// sorted keys in one launch.  The cells 0 .. C and the sorted keys form one
// merged order, a cell before the keys that are its own or later; cell c's
// start is the number of keys before it.  Key k has k keys and keys[k] + 1
// cells before it, so its place is k + keys[k] + 1, and a warp finds the
// kCellWindow consecutive places that are its own by searching the keys:
// however the particles crowd, a warp has no more than that many.  It notes
// the first particle of each cell that has one, and fills the others from
// the right with the next cell's first.  (Clearing, counting with atomics
// and scanning took five launches: 24 us for 1,000 particles in 15,000 cells
// against 10 us here, 24 and 16 us for 125,000 in 247,000, 54 and 28 us for
// 655,000 and 77 and 71 us for 8.4 M in 3.8 M.  The same by windows of 256
// cells took 919 us on the last one, whose out-of-grid cell is crowded.)
constexpr int kCellWindow = 512, kCellWarps = 8;

// The number of keys whose place is before `place`, by all lanes of a warp:
// 32 probes a step.
__device__ __forceinline__ int keys_before(const uint32_t* keys, int n, int64_t place, int lane) {
  int lo = 0, len = n;
  while (len > 32) {
    const int step = (len + 31) >> 5;
    const int at = lane * step + step - 1;  // the last of this lane's part
    const unsigned less = __ballot_sync(0xffffffffu, at < len && (int64_t)(lo + at) + keys[lo + at] + 1 < place);
    const int skip = __popc(less) * step;   // (parts wholly before, which come first)
    lo += skip;
    len = min(step, len - skip);
  }
  return lo + __popc(__ballot_sync(0xffffffffu, lane < len && (int64_t)(lo + lane) + keys[lo + lane] + 1 < place));
}

__global__ void __launch_bounds__(32 * kCellWarps) k_cell_start(const uint32_t* keys, int n, int entries,
                                                                int32_t* cell_start) {
  __shared__ int s_first[kCellWarps][kCellWindow];
  __shared__ int s_key[kCellWarps + 1];
  const int t = (int)pdl_wait(threadIdx.x), lane = t & 31, w = t >> 5;
  const int64_t place = ((int64_t)blockIdx.x * kCellWarps + w) * kCellWindow;
  const int mine = keys_before(keys, n, place, lane);
  const int end = w == kCellWarps - 1 ? keys_before(keys, n, place + kCellWindow, lane) : 0;
  if (lane == 0) {
    s_key[w] = mine;
    if (w == kCellWarps - 1) s_key[kCellWarps] = end;
  }
  __syncthreads();
  const int k0 = s_key[w], k1 = s_key[w + 1];
  const int64_t c0 = place - k0;  // the cells c0 .. c0 + own - 1 are this warp's
  const int own = (int)min(place + kCellWindow - k1, (int64_t)entries) - (int)min(c0, (int64_t)entries);
  if (own <= 0) return;
  int* first = s_first[w];
#pragma unroll
  for (int k = lane; k < kCellWindow; k += 32) first[k] = k1;
  __syncwarp();
#pragma unroll 4
  for (int p = k0 + lane; p < k1; p += 32) {
    const int64_t c = (int64_t)keys[p] - c0;
    if (c >= 0 && c < own && (p == k0 || keys[p - 1] != keys[p])) first[c] = p;
  }
  __syncwarp();
  // a lane's consecutive cells from the right, then the lanes' firsts
  constexpr int kOwn = kCellWindow / 32;
  int v[kOwn];
#pragma unroll
  for (int k = 0; k < kOwn; ++k) v[k] = first[lane * kOwn + k];
#pragma unroll
  for (int k = kOwn - 2; k >= 0; --k) v[k] = min(v[k], v[k + 1]);
  int rest = v[0];
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_down_sync(0xffffffffu, rest, o);
    if (lane + o < 32) rest = min(rest, y);
  }
  int right = __shfl_down_sync(0xffffffffu, rest, 1);
  if (lane == 31) right = k1;
  __syncwarp();
#pragma unroll
  for (int k = 0; k < kOwn; ++k) first[lane * kOwn + k] = min(v[k], right);
  __syncwarp();
  for (int k = lane; k < own; k += 32) cell_start[c0 + k] = first[k];
}

gg_status cell_start_build(const Grid& g, const uint32_t* sorted_keys, int64_t n, int32_t* cell_start,
                           SortScratch& s, cudaStream_t st, gg_system* prof) {
  if (prof) prof_begin(prof, PC_CELLSTART, st);
  const int entries = g.C + 1;
  if (n > 0) {
    GG_CUDA(launch_chained(k_cell_start, blocks_for(n + entries, kCellWindow * kCellWarps), 32 * kCellWarps, st,
                           sorted_keys, (int)n, entries, cell_start));
    if (s.counter) *s.counter += 1;
  } else {
    GG_CUDA(cudaMemsetAsync(cell_start, 0, sizeof(int32_t) * (size_t)entries, st));
  }
  if (prof) prof_end(prof, PC_CELLSTART, entries, st);
  GG_CUDA(cudaGetLastError());
  return GG_OK;
}

// --------------------------------------------------------------- reorder

// The gathers of GranularSystem.cu:97-135 for every permuted field in one
// pass.  adaptive_last_step and merge_velocity are not permuted, as in the
// reference.
__global__ void k_reorder_granular(int n, const uint32_t* perm,
                                   const float4* pos_in, float4* pos_out,
                                   const float4* vel_in, float4* vel_out,
                                   const float* mass_in, float* mass_out,
                                   const float* rs_in, float* rs_out,
                                   const int32_t* units_in, int32_t* units_out,
                                   const float* merge_in, float* merge_out,
                                   const int32_t* mu_in, int32_t* mu_out,
                                   const int32_t* mc_in, int32_t* mc_out,
                                   const int32_t* rm_in, int32_t* rm_out,
                                   const int32_t* als_in, int32_t* als_out) {
  const int p = blockIdx.x * blockDim.x + (int)pdl_wait(threadIdx.x);
  if (p >= n) return;
  // every load first: without __restrict__ (pdl_wait) a load does not move
  // ahead of a store, and each would wait for the one before it.  8.4 M
  // particles 0.169 ms with a plain launch, 0.222 field by field, 0.164 this way.
  const int32_t als = als_in[p];  // stays where it is
  const uint32_t s = perm[p];
  const float4 pos = pos_in[s], vel = vel_in[s];
  const float mass = mass_in[s], rs = rs_in[s], merge = merge_in[s];
  const int32_t units = units_in[s], mu = mu_in[s], mc = mc_in[s], rm = rm_in[s];
  als_out[p] = als;
  pos_out[p] = pos;
  vel_out[p] = vel;
  mass_out[p] = mass;
  rs_out[p] = rs;
  units_out[p] = units;
  merge_out[p] = merge;
  mu_out[p] = mu;
  mc_out[p] = mc;
  rm_out[p] = rm;
}

gg_status reorder_granular(gg_system* S, cudaStream_t st) {
  if (S->n <= 0) return GG_OK;
  Granular& G = S->g;
  const int a = G.cur, b = G.cur ^ 1;
  prof_begin(S, PC_REORDER, st);
  GG_CUDA(launch_chained(
      k_reorder_granular, blocks_for(S->n, 256), 256, st, (int)S->n, G.perm, G.pos[a], G.pos[b], G.vel[a], G.vel[b], G.mass[a], G.mass[b], G.rs[a], G.rs[b],
      G.units[a], G.units[b], G.merge[a], G.merge[b], G.merge_units[a], G.merge_units[b],
      G.merge_count[a], G.merge_count[b], G.remove[a], G.remove[b], G.als[a], G.als[b]));
  count_launches(S, 1);
  prof_end(S, PC_REORDER, S->n, st);
  G.cur = b;
  GG_CUDA(cudaGetLastError());
  return GG_OK;
}

__global__ void k_gather2(int n, const uint32_t* perm, const float4* a_in,
                          float4* a_out, const float4* b_in,
                          float4* b_out) {
  const int p = blockIdx.x * blockDim.x + (int)pdl_wait(threadIdx.x);
  if (p >= n) return;
  const uint32_t s = perm[p];
  const float4 a = a_in[s];  // (both loads first, as in k_reorder_granular)
  float4 b = make_float4(0.f, 0.f, 0.f, 0.f);
  if (b_in) b = b_in[s];
  a_out[p] = a;
  if (b_in) b_out[p] = b;
}

__global__ void k_gather_boundary(int n, const uint32_t* __restrict__ perm, const float4* __restrict__ p_in,
                                  float4* __restrict__ p_out, const int32_t* __restrict__ a_in,
                                  int32_t* __restrict__ a_out) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const uint32_t s = perm[p];
  p_out[p] = p_in[s];
  a_out[p] = a_in[s];
}

gg_status reorder_boundary(gg_system* S, const uint32_t* perm, cudaStream_t st) {
  if (S->nb <= 0) return GG_OK;
  k_gather_boundary<<<blocks_for(S->nb, 256), 256, 0, st>>>((int)S->nb, perm, S->b.pos, S->b.pos_alt,
                                                            S->b.animated, S->b.animated_alt);
  count_launches(S, 1);
  std::swap(S->b.pos, S->b.pos_alt);
  std::swap(S->b.animated, S->b.animated_alt);
  GG_CUDA(cudaGetLastError());
  return GG_OK;
}

gg_status reorder_upsampled(gg_system* S, const uint32_t* perm, cudaStream_t st) {
  if (S->nu <= 0) return GG_OK;
  const int a = S->u.cur, b = a ^ 1;
  GG_CUDA(launch_chained(k_gather2, blocks_for(S->nu, 256), 256, st, (int)S->nu, perm, S->u.pos[a], S->u.pos[b],
                         S->u.vel[a], S->u.vel[b]));
  count_launches(S, 1);
  S->u.cur = b;
  GG_CUDA(cudaGetLastError());
  return GG_OK;
}


// ------------------------------------------------------------ grid build without allocation
//
// gg_grid_build_noalloc: the grid build above (cell keys, stable radix sort,
// cell start table) for callers that cannot allocate device memory, such as
// code hosted inside an engine or framework that owns every device
// allocation, or a loop that must not allocate once it is running.  The
// caller passes device buffers for the positions and for every output; the
// sort's scratch (two key/value ping-pong buffers and three tables of the
// per-tile digit counts) lives in the file-scope array below, sized for at
// most kNoAllocMaxParticles particles.  Every GPU that loads this library
// holds that array (about 4.4 MiB) until the process exits.

constexpr int64_t kNoAllocMaxParticles = 1 << 18;
constexpr int64_t kNoAllocMaxCells = 1 << 24;
static_assert(kNoAllocMaxParticles <= kShortMax, "the short sort reaches the limit");
constexpr size_t kNoAllocPairWords = 4 * (size_t)kNoAllocMaxParticles;   // k0, k1, v0, v1
constexpr size_t kNoAllocHistWords = 3 * 256 * (size_t)kShortTiles;
constexpr size_t kNoAllocWords = kNoAllocPairWords + kNoAllocHistWords;

static __device__ __align__(256) uint32_t g_noalloc_scratch[kNoAllocWords];

namespace {
// Saves the calling thread's current device and restores it on scope exit.
struct DeviceGuard {
  int saved = 0;
  cudaError_t status;
  DeviceGuard() { status = cudaGetDevice(&saved); }
  ~DeviceGuard() {
    if (status == cudaSuccess) cudaSetDevice(saved);
  }
};

constexpr int kNoAllocMaxDevices = 64;
std::mutex g_noalloc_mu;
uint32_t* g_noalloc_dev[kNoAllocMaxDevices] = {};

// The array's name is a host-side stand-in, not a device address: the
// address is looked up once per device, with that device current.
gg_status noalloc_scratch(int device, uint32_t** out) {
  if (device < 0 || device >= kNoAllocMaxDevices) {
    set_error("gg_grid_build_noalloc: device ordinal out of range");
    return GG_ERR_INVALID_ARGUMENT;
  }
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  if (!g_noalloc_dev[device]) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) return cuda_status(e, "gg_grid_build_noalloc: cudaGetSymbolAddress");
    g_noalloc_dev[device] = (uint32_t*)p;
  }
  *out = g_noalloc_dev[device];
  return GG_OK;
}
}  // namespace

}  // namespace gg

extern "C" gg_status gg_grid_build_noalloc(int32_t device, const float* d_pos, int64_t n,
                                           const int32_t cell_size[3], float cell_length,
                                           uint32_t* d_sorted_keys, uint32_t* d_perm, int32_t* d_cell_start,
                                           void* stream) {
  using namespace gg;
  try {
    if (!cell_size || !(cell_length > 0.0f) || n < 0 || (n > 0 && (!d_pos || !d_sorted_keys || !d_perm)) ||
        !d_cell_start) {
      set_error("gg_grid_build_noalloc: null buffer or invalid size");
      return GG_ERR_INVALID_ARGUMENT;
    }
    if (cell_size[0] <= 0 || cell_size[1] <= 0 || cell_size[2] <= 0) {
      set_error("gg_grid_build_noalloc: cell_size must be positive");
      return GG_ERR_INVALID_ARGUMENT;
    }
    const int64_t C = (int64_t)cell_size[0] * cell_size[1] * cell_size[2];
    if (n > kNoAllocMaxParticles || C > kNoAllocMaxCells) {
      set_error("gg_grid_build_noalloc: at most 262144 particles and 16777216 cells (static scratch limit); "
                "use gg_grid_create/gg_grid_build for larger inputs");
      return GG_ERR_CAPACITY;
    }
    // the caller's current device is put back on every return path
    DeviceGuard guard;
    if (guard.status != cudaSuccess) return cuda_status(guard.status, "gg_grid_build_noalloc: cudaGetDevice");
    GG_CUDA(cudaSetDevice(device));
    uint32_t* base = nullptr;
    gg_status rc = noalloc_scratch(device, &base);
    if (rc != GG_OK) return rc;
    SortScratch s;
    s.k[0] = base;
    s.k[1] = base + kNoAllocMaxParticles;
    s.v[0] = base + 2 * kNoAllocMaxParticles;
    s.v[1] = base + 3 * kNoAllocMaxParticles;
    s.hist = base + kNoAllocPairWords;
    s.capacity = kNoAllocMaxParticles;
    s.hist_entries = (int64_t)kNoAllocHistWords;
    Grid g;
    g.L = cell_length;
    g.nx = cell_size[0];
    g.ny = cell_size[1];
    g.nz = cell_size[2];
    g.C = (int)C;
    cudaStream_t st = (cudaStream_t)stream;
    if (n > 0) {
      rc = short_sort<true>(g, d_pos, n, s, d_sorted_keys, d_perm, nullptr, st, nullptr);
      if (rc != GG_OK) return rc;
    }
    // (the sort's tables are written before they are read, so what the last
    // call left there needs no clearing)
    return cell_start_build(g, d_sorted_keys, n, d_cell_start, s, st, nullptr);
  } catch (...) {
    set_error("gg_grid_build_noalloc: internal error");
    return GG_ERR_INVALID_ARGUMENT;
  }
}
