// CSR -> CSC of a matrix whose rows have ascending columns (as the build
// emits them), for sm_100a.
//
// The columns are cut into bins of 1024, and the rows, in the order in which
// they are taken, into blocks.  A row's entries in a bin are one run of it, so the
// partition by bins is a copy and nothing has to be ranked; only the partition
// inside the bins is a radix pass:
//   1. split: where each row's columns enter every bin (one sweep of the columns,
//      which also checks that they ascend and are in the matrix; the caller looks
//      at the outcome before it allocates the staging);
//   2. sizes of the (bin, block) pieces and their exclusive sums;
//   3. copy: a warp per (bin, block) lays its rows' runs end to end (low ten bits
//      of the column, place k of the row, value), 32 entries at a time;
//   4. per bin, tiles of entries: histogram of the low bits, scan over (bin, digit,
//      tile), which holds the column pointers, and a stable scatter.
// Within a column the entries come out in the order of k, whatever the
// scheduling.  145M entries of 200,000 rows, 70^3 columns: 2.54 ms (split 0.5,
// copy 0.8, scatter 1.05) against 4.53 for the radix sort of rows in any order
// (kernels_transpose.cu), whose first pass ranks a tile's entries by nine bits and
// whose staging is 12 bytes per entry instead of 10.  What bounds it: the
// instructions of the split's sweep (73% of issue), the copy's loads of runs of two or three
// entries, the scatter's rank counters, one shared-memory round trip after another.
#include <algorithm>
#include <cstdint>

#include "internal.h"

namespace raptr {

namespace {

constexpr int kShift = 10, kRange = 1 << kShift;  // columns of a bin
constexpr int kMaxBins = 1024;
constexpr int kSplitThreads = 256;
// rows whose splits are written together, and where m is small: one per warp
constexpr int kSplitRows = 64, kSplitFew = kSplitThreads / 32;
constexpr int kPiece = 16384;       // entries of a piece that a warp copies alone
constexpr int kCopyWarps = 4;
constexpr int kBatch = 4;           // windows of 32 entries loaded together
constexpr int kTile = 65536;        // entries of a tile of step 4
constexpr int kScatterWarps = 16, kItems = 8, kScatterBlocks = 2;
constexpr int kScatterThreads = kScatterWarps * 32;
constexpr int kChunk = kScatterThreads * kItems;  // entries ranked together

// Step 1.  split[q * m + k] = the first entry (from the row's start) of the
// k-th row in bin q or later, q in [0, bins]; begin[k] = the row's start.
// flags: 1 = a column or an order entry out of range, 2 = columns that do not
// ascend (or a row of more than 65535 entries).
template <int ROWS>
__global__ void __launch_bounds__(kSplitThreads) sorted_split_kernel(int64_t m, int64_t n, int bins,
                                                                     const int64_t* __restrict__ rp,
                                                                     const int32_t* __restrict__ col,
                                                                     const int32_t* __restrict__ order,
                                                                     uint16_t* __restrict__ split,
                                                                     int64_t* __restrict__ begin,
                                                                     int32_t* __restrict__ flags) {
  extern __shared__ uint16_t sh_split[];  // [row][bin], rows of an odd number of words
  const int pitch = ((bins + 2) | 2) & ~1 | 2;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int bad = 0;
  for (int64_t kb = int64_t(blockIdx.x) * ROWS; kb < m; kb += int64_t(gridDim.x) * ROWS) {
    // some block has seen that it is not this matrix's way
    if (__syncthreads_or(threadIdx.x == 0 && *(volatile int32_t*)flags != 0)) break;
    for (int i = w; i < ROWS && kb + i < m; i += kSplitThreads / 32) {
      const int64_t k = kb + i;
      uint16_t* first = sh_split + i * pitch;
      const int64_t r = order ? int64_t(__ldg(order + k)) : k;
      int64_t b = 0, e = 0;
      if (r >= 0 && r < m) {
        b = rp[r];
        e = rp[r + 1];
      } else {
        bad |= 1;
      }
      if (lane == 0) begin[k] = b;
      const int len = int(max(min(e - b, int64_t(65535)), int64_t(0)));
      if (e - b != len) bad |= 2;
      const int32_t* p = col + b;
      int last = -1;  // the column before the chunk
      for (int i0 = lane; i0 - lane < len; i0 += 128) {
        int c[4];
#pragma unroll
        for (int u = 0; u < 4; u++) c[u] = i0 + 32 * u < len ? __ldg(p + i0 + 32 * u) : INT32_MAX;
#pragma unroll
        for (int u = 0; u < 4; u++) {
          int before = __shfl_up_sync(0xffffffffu, c[u], 1);
          before = lane == 0 ? last : before;
          last = __shfl_sync(0xffffffffu, c[u], 31);
          if (i0 + 32 * u < len) {
            const int q = c[u] >> kShift, qb = max(before, -1) >> kShift;  // -1 before the row
            if (unsigned(c[u]) >= unsigned(n)) {
              bad |= 1;
            } else if (c[u] <= before) {
              bad |= 2;
            } else if (q != qb) {
              for (int t = qb + 1; t <= q; t++) first[t] = uint16_t(i0 + 32 * u);
            }
          }
        }
      }
      if (__any_sync(0xffffffffu, bad)) break;
      // bins after the row's last entry
      const int lastc = len > 0 ? __ldg(p + len - 1) : -1;
      const int q1 = lastc < 0 ? 0 : min((lastc >> kShift) + 1, bins);
      for (int t = q1 + lane; t <= bins; t += 32) first[t] = uint16_t(len);
    }
    __syncthreads();
    const int rows = int(min(int64_t(ROWS), m - kb));
    for (int t = w; t <= bins; t += kSplitThreads / 32)
      for (int i = lane; i < rows; i += 32) split[int64_t(t) * m + kb + i] = sh_split[i * pitch + t];
    __syncthreads();
  }
  if (bad) atomicOr(flags, bad);
}

// The k-th lowest set bit of `bits` (k below their number).
__device__ __forceinline__ int nth_bit(unsigned bits, int k) {
  int at = 0;
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) {
    const int c = __popc((bits >> at) & ((1u << s) - 1u));
    if (c <= k) {
      k -= c;
      at += s;
    }
  }
  return at;
}

// Step 2.  size[q * blocks + b] = entries of the b-th block of rows in bin q;
// flags[1] = the most of any piece, where that is above kPiece.
__global__ void __launch_bounds__(kCopyWarps * 32)
    sorted_sizes_kernel(int64_t m, int bins, int blocks, int rows_per_block, const uint16_t* __restrict__ split,
                        int32_t* __restrict__ flags, int64_t* __restrict__ size) {
  const int lane = threadIdx.x & 31;
  const int64_t id = int64_t(blockIdx.x) * kCopyWarps + (threadIdx.x >> 5);
  if (id >= int64_t(bins) * blocks) return;
  const int64_t q = id / blocks, b = id - q * blocks;
  if (*flags != 0) return;
  const int64_t k1 = min((b + 1) * rows_per_block, m);
  const uint16_t* s0 = split + q * m;
  int sum = 0;
  for (int64_t k = b * rows_per_block + lane; k < k1; k += 32) sum += int(s0[m + k]) - int(s0[k]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if (lane == 0) {
    size[id] = sum;
    if (sum > kPiece) atomicMax(flags + 1, sum);
  }
}

// tile_first[q] = the tiles of the bins before q (each has at least one).  Sets
// flag 4 where the rows taken do not hold nnz entries in all (an order that
// repeats rows): from here on every kernel does nothing unless *flags is 0, which
// makes the pieces' sums, and with them all places below, those of the matrix.
__global__ void __launch_bounds__(kMaxBins) sorted_tiles_kernel(int bins, int blocks, int64_t nnz,
                                                                const int64_t* __restrict__ off,
                                                                int32_t* __restrict__ flags,
                                                                int32_t* __restrict__ tile_first) {
  __shared__ int sums[32];
  const int q = threadIdx.x, lane = q & 31, w = q >> 5;
  const bool stop = *flags != 0 || off[int64_t(bins) * blocks] != nnz;
  if (__syncthreads_or(stop)) {
    if (q == 0) *flags |= 4;
    return;
  }
  int v = 0;
  if (q < bins) {
    const int64_t entries = off[int64_t(q + 1) * blocks] - off[int64_t(q) * blocks];
    v = int(max((entries + kTile - 1) / kTile, int64_t(1)));
  }
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) sums[w] = x;
  __syncthreads();
  int before = x - v;
  for (int i = 0; i < w; i++) before += sums[i];
  if (q < bins) tile_first[q] = before;
  if (q == bins - 1) tile_first[bins] = before + v;
}

// Step 3, one warp per (bin, block); the bins of one block of rows run next to
// each other, so that the sectors that hold the ends of runs are read once.  Where
// pieces are long (rows whose columns are neighbours, or all the same), `parts`
// warps share a piece, each a run of part_rows rows of it whose place follows from the
// splits: 3,000 rows of the same 1100 of 2^20 columns, 65,536 entries a piece, 2.0 ms
// with a warp for each, 0.93 by the radix sort, 0.57 so.
template <bool SHARED>
__global__ void __launch_bounds__(kCopyWarps * 32)
    sorted_copy_kernel(int64_t m, int bins, int blocks, int rows_per_block, int parts, int part_rows,
                       const int32_t* __restrict__ col, const float* __restrict__ val,
                       const uint16_t* __restrict__ split, const int64_t* __restrict__ begin,
                       const int64_t* __restrict__ off, const int32_t* __restrict__ flags,
                       uint16_t* __restrict__ st_low, int32_t* __restrict__ st_k, float* __restrict__ st_v) {
  const int lane = threadIdx.x & 31;
  const int64_t id = int64_t(blockIdx.x) * kCopyWarps + (threadIdx.x >> 5);
  const int64_t task = SHARED ? id / parts : id;
  if (task >= int64_t(bins) * blocks) return;
  if (*flags != 0) return;
  const int64_t b = task / bins, q = task - b * bins;
  const int32_t c0 = int32_t(q << kShift);
  int64_t out = off[q * blocks + b];
  int64_t kb = b * rows_per_block, k1 = min(kb + rows_per_block, m);
  const uint16_t* s0 = split + q * m;
  if (SHARED) {
    const int64_t first = kb;
    kb = min(kb + (id - task * parts) * part_rows, k1);
    int sum = 0;
    for (int64_t k = first + lane; k < kb; k += 32) sum += int(s0[m + k]) - int(s0[k]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    out += sum;
    k1 = min(kb + part_rows, k1);
  }
  for (int64_t k = kb; k < k1; k += 32) {
    // the rows with entries in the bin, moved to the low lanes
    uint32_t lo = 0, hi = 0;
    if (k + lane < k1) {
      lo = s0[k + lane];
      hi = s0[m + k + lane];
    }
    const unsigned some = __ballot_sync(0xffffffffu, hi > lo);
    if (!some) continue;
    const int rows = __popc(some);
    const int src = lane < rows ? nth_bit(some, lane) : 0;
    lo = __shfl_sync(0xffffffffu, lo, src);
    hi = __shfl_sync(0xffffffffu, hi, src);
    const int64_t b0 = lane < rows ? begin[k + src] : 0;
    const int len = lane < rows ? int(hi - lo) : 0;
    int incl = len;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += x;
    }
    const int total = __shfl_sync(0xffffffffu, incl, 31), excl = incl - len;
    // the entry at place f of the runs end to end is at from[row] + f
    const int64_t from = lane < rows ? b0 + lo - excl : 0;
    int done = 0;  // rows that begin before the window
    for (int f0 = 0; f0 < total; f0 += 32 * kBatch) {
      int c[kBatch], id[kBatch];
      float v[kBatch];
#pragma unroll
      for (int u = 0; u < kBatch; u++) {
        const int f = f0 + 32 * u + lane;
        const unsigned at = unsigned(excl - (f0 + 32 * u));
        const unsigned starts = __reduce_or_sync(0xffffffffu, lane < rows && at < 32u ? 1u << at : 0u);
        const int r = done + __popc(starts & (0xffffffffu >> (31 - lane))) - 1;
        done += __popc(starts);
        const int64_t g = __shfl_sync(0xffffffffu, from, r) + f;
        id[u] = int(k) + __shfl_sync(0xffffffffu, src, r);
        const bool in = f < total;
        c[u] = in ? __ldg(col + g) - c0 : 0;
        v[u] = in ? __ldg(val + g) : 0.f;
      }
#pragma unroll
      for (int u = 0; u < kBatch; u++) {
        const int f = f0 + 32 * u + lane;
        if (f < total) {
          st_low[out + f] = uint16_t(c[u]);
          st_k[out + f] = id[u];
          st_v[out + f] = v[u];
        }
      }
    }
    out += total;
  }
}

// Tile t: its bin, its place among the bin's tiles, and its entries [e0, e0 + n).
struct Tile {
  int bin, at, of, n;
  int64_t e0;
};
__device__ __forceinline__ Tile find_tile(int t, int bins, int blocks, const int32_t* __restrict__ tile_first,
                                          const int64_t* __restrict__ off) {
  int lo = 0, hi = bins;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (tile_first[mid] <= t) lo = mid;
    else hi = mid;
  }
  Tile r;
  r.bin = lo;
  r.at = t - tile_first[lo];
  r.of = tile_first[lo + 1] - tile_first[lo];
  r.e0 = off[int64_t(lo) * blocks] + int64_t(r.at) * kTile;
  r.n = int(max(min(off[int64_t(lo + 1) * blocks] - r.e0, int64_t(kTile)), int64_t(0)));
  return r;
}
// Where the count of digit d of a tile stands: (bin, digit, tile) order, the order
// of the CSC, so that the exclusive sums are the places.
__device__ __forceinline__ int64_t hist_at(const Tile& t, const int32_t* __restrict__ tile_first, int d) {
  return int64_t(kRange) * tile_first[t.bin] + int64_t(d) * t.of + t.at;
}

__global__ void __launch_bounds__(512) sorted_hist_kernel(int bins, int blocks, const int32_t* __restrict__ tile_first,
                                                          const int64_t* __restrict__ off,
                                                          const uint16_t* __restrict__ st_low,
                                                          const int32_t* __restrict__ flags,
                                                          int64_t* __restrict__ hist) {
  __shared__ int cnt[kRange];
  const int t = blockIdx.x;
  if (*flags != 0) return;
  const bool used = t < tile_first[bins];
  for (int d = threadIdx.x; d < kRange; d += 512) cnt[d] = 0;
  __syncthreads();
  Tile tile{};
  if (used) {
    tile = find_tile(t, bins, blocks, tile_first, off);
    constexpr int U = 8;
    for (int i0 = threadIdx.x; i0 < tile.n; i0 += 512 * U) {
      int d[U];
#pragma unroll
      for (int u = 0; u < U; u++) d[u] = i0 + 512 * u < tile.n ? __ldg(st_low + tile.e0 + i0 + 512 * u) : -1;
#pragma unroll
      for (int u = 0; u < U; u++)
        if (d[u] >= 0) atomicAdd(cnt + (d[u] & (kRange - 1)), 1);
    }
    __syncthreads();
  }
  // the places beyond the last tile's are unused, and zero
  for (int d = threadIdx.x; d < kRange; d += 512)
    hist[used ? hist_at(tile, tile_first, d) : int64_t(kRange) * t + d] = cnt[d];
}

__global__ void sorted_cp_kernel(int64_t n, int64_t nnz, const int32_t* __restrict__ tile_first,
                                 const int64_t* __restrict__ place, const int32_t* __restrict__ flags,
                                 int64_t* __restrict__ cp) {
  const int64_t c = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (c > n || *flags != 0) return;
  const int q = int(c >> kShift), d = int(c & (kRange - 1));
  cp[c] = c == n ? nnz : place[int64_t(kRange) * tile_first[q] + int64_t(d) * (tile_first[q + 1] - tile_first[q])];
}

// Shared memory of a scatter block.
struct ScatterShared {
  int64_t to[kRange];                        // next place of each digit, less its start in the chunk
  int start[kRange];                         // of each digit in the chunk's order
  int sums[kScatterWarps];
  unsigned short wcnt[kScatterWarps][kRange];  // per warp: entries of the digit, then those of the warps before
  int k[kChunk];                             // the chunk in the order of its digits
  float v[kChunk];
  unsigned short d[kChunk];
};

// Stable partition of a tile by the low bits, kChunk entries at a time, put in
// order in shared memory first: the four or so entries of a digit then leave as one
// run.  Written from where they are read, each 4-byte store is a sector of its own:
// 1.54 ms for the 290M of them in 145M entries, against 1.06.  Two blocks of 16 warps and
// 4096 entries per SM: 2.85 ms for the whole transpose, one block of 8192 entries 3.20,
// two of 8 warps 2.89.
__global__ void __launch_bounds__(kScatterThreads, kScatterBlocks)
    sorted_scatter_kernel(int bins, int blocks, const int32_t* __restrict__ tile_first,
                          const int64_t* __restrict__ off, const int64_t* __restrict__ place,
                          const int32_t* __restrict__ flags, const uint16_t* __restrict__ st_low,
                          const int32_t* __restrict__ st_k, const float* __restrict__ st_v,
                          int32_t* __restrict__ trow, float* __restrict__ tval) {
  extern __shared__ __align__(16) unsigned char sh_scatter[];
  ScatterShared& sh = *reinterpret_cast<ScatterShared*>(sh_scatter);
  constexpr int kDigits = kRange / kScatterThreads;  // digits of a thread, neighbours
  const int t = blockIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5, d0 = threadIdx.x * kDigits;
  if (*flags != 0 || t >= tile_first[bins]) return;
  const Tile tile = find_tile(t, bins, blocks, tile_first, off);
  int64_t at[kDigits];  // next place of the thread's digits
#pragma unroll
  for (int j = 0; j < kDigits; j++) at[j] = place[hist_at(tile, tile_first, d0 + j)];
  for (int c0 = 0; c0 < tile.n; c0 += kChunk) {
    for (int i = threadIdx.x; i < kScatterWarps * kRange / 8; i += kScatterThreads)
      reinterpret_cast<uint4*>(&sh.wcnt[0][0])[i] = make_uint4(0, 0, 0, 0);
    int dig[kItems], rnk[kItems], kk[kItems];
    float vv[kItems];
#pragma unroll
    for (int it = 0; it < kItems; it++) {
      const int i = c0 + w * (kItems * 32) + it * 32 + lane;
      const bool in = i < tile.n;
      dig[it] = in ? int(__ldcs(st_low + tile.e0 + i)) & (kRange - 1) : -1;
      kk[it] = in ? __ldcs(st_k + tile.e0 + i) : 0;
      vv[it] = in ? __ldcs(st_v + tile.e0 + i) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int it = 0; it < kItems; it++) {
      const int d = dig[it];
      const unsigned peers = __match_any_sync(0xffffffffu, d);
      const int r = __popc(peers & ((1u << lane) - 1u));
      int base = 0;
      if (d >= 0) base = sh.wcnt[w][d];
      __syncwarp();
      if (d >= 0 && r == 0) sh.wcnt[w][d] = (unsigned short)(base + __popc(peers));
      __syncwarp();
      rnk[it] = base + r;
    }
    __syncthreads();
    // per digit: the entries of the warps before each warp; over digits: the starts
    int tot[kDigits], mine = 0;
#pragma unroll
    for (int j = 0; j < kDigits; j++) {
      int sum = 0;
#pragma unroll
      for (int x = 0; x < kScatterWarps; x++) {
        const int c = sh.wcnt[x][d0 + j];
        sh.wcnt[x][d0 + j] = (unsigned short)sum;
        sum += c;
      }
      tot[j] = sum;
      mine += sum;
    }
    int x = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) sh.sums[w] = x;
    __syncthreads();
    int first = x - mine;
    for (int i = 0; i < w; i++) first += sh.sums[i];
#pragma unroll
    for (int j = 0; j < kDigits; j++) {
      sh.start[d0 + j] = first;
      sh.to[d0 + j] = at[j] - first;
      first += tot[j];
      at[j] += tot[j];
    }
    __syncthreads();
#pragma unroll
    for (int it = 0; it < kItems; it++) {
      const int d = dig[it];
      if (d >= 0) {
        const int pos = sh.start[d] + sh.wcnt[w][d] + rnk[it];
        sh.k[pos] = kk[it];
        sh.v[pos] = vv[it];
        sh.d[pos] = (unsigned short)d;
      }
    }
    __syncthreads();
    const int cn = min(tile.n - c0, kChunk);
#pragma unroll 4
    for (int i = threadIdx.x; i < cn; i += kScatterThreads) {
      const int64_t pos = sh.to[sh.d[i]] + i;
      trow[pos] = sh.k[i];
      tval[pos] = sh.v[i];
    }
    __syncthreads();
  }
}

size_t split_smem(int bins, int rows) { return size_t(rows) * size_t((((bins + 2) | 2) & ~1) | 2) * 2; }

}  // namespace

bool transpose_sorted_plan(int64_t m, int64_t n, int64_t nnz, SortedPlan* p) {
  if (m <= 0 || n <= 0 || nnz <= 0 || m > INT32_MAX) return false;
  const int64_t bins = (n + kRange - 1) >> kShift;
  // 32 rows' runs in a bin should fill a window of 32 or so.  At one entry per row
  // and bin (200,000 rows, 343,000 columns) 2.43 ms against 3.87 for the radix sort,
  // at two 4.0 against 8.3; with fewer the splits outweigh the entries.
  if (bins < 2 || bins > kMaxBins || nnz < m * bins) return false;
  p->bins = int(bins);
  // Blocks of 256 rows, and of fewer where that leaves warps idle.  At 145M entries
  // in 335 bins: 2.54 ms for all; blocks of 1024 rows 2.81 (the pieces of the
  // middle bins are the longest, and last), 512 2.63, 128 2.55.
  p->rows_per_block = 256;
  while (p->rows_per_block > 64 && bins * ((m + p->rows_per_block - 1) / p->rows_per_block) < 148 * 64)
    p->rows_per_block /= 2;
  p->blocks = int((m + p->rows_per_block - 1) / p->rows_per_block);
  p->max_tiles = nnz / kTile + bins;
  return p->max_tiles < INT32_MAX / 2;
}

int64_t sorted_hist_elems(const SortedPlan& p) { return int64_t(kRange) * p.max_tiles; }

cudaError_t launch_sorted_split(const SortedPlan& p, int64_t m, int64_t n, int64_t nnz, const int64_t* rp,
                                const int32_t* col, const int32_t* order, const SortedScratch& w, cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(w.flags, 0, 2 * sizeof(int32_t), s);
  if (e != cudaSuccess) return e;
  // a block's rows share its writes of the splits, but fewer rows than SMs want are
  // better spread (64 rows of 60,000 entries: 2.9 ms for the whole transpose, 0.67 so)
  const bool few = m < int64_t(kSplitRows) * 148 * 2;
  const int rows = few ? kSplitFew : kSplitRows;
  const unsigned gs = unsigned(std::min<int64_t>((m + rows - 1) / rows, 148 * 32));
  const int64_t tasks = int64_t(p.bins) * p.blocks;
  const unsigned gt = unsigned((tasks + kCopyWarps - 1) / kCopyWarps);
  auto split = few ? sorted_split_kernel<kSplitFew> : sorted_split_kernel<kSplitRows>;
  e = cudaFuncSetAttribute(split, cudaFuncAttributeMaxDynamicSharedMemorySize, int(split_smem(kMaxBins, rows)));
  if (e != cudaSuccess) return e;
  split<<<gs, kSplitThreads, split_smem(p.bins, rows), s>>>(m, n, p.bins, rp, col, order, w.split, w.begin, w.flags);
  sorted_sizes_kernel<<<gt, kCopyWarps * 32, 0, s>>>(m, p.bins, p.blocks, p.rows_per_block, w.split, w.flags, w.size);
  note_launches(2);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  if ((e = launch_scan_i64(w.size, tasks, w.off, w.scan_tmp, s)) != cudaSuccess) return e;
  sorted_tiles_kernel<<<1, kMaxBins, 0, s>>>(p.bins, p.blocks, nnz, w.off, w.flags, w.tile_first);
  note_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_sorted_move(const SortedPlan& p, int64_t m, int64_t n, int64_t nnz, int most, const int32_t* col,
                               const float* val, const SortedScratch& w, int64_t* cp, int32_t* trow, float* tval,
                               cudaStream_t s) {
  cudaError_t e = cudaFuncSetAttribute(sorted_scatter_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       int(sizeof(ScatterShared)));
  if (e != cudaSuccess) return e;
  int parts = 1;
  while (most / parts > kPiece && p.rows_per_block / parts > 8) parts *= 2;
  const int64_t tasks = int64_t(p.bins) * p.blocks * parts;
  const unsigned gt = unsigned((tasks + kCopyWarps - 1) / kCopyWarps);
  auto copy = parts > 1 ? sorted_copy_kernel<true> : sorted_copy_kernel<false>;
  copy<<<gt, kCopyWarps * 32, 0, s>>>(m, p.bins, p.blocks, p.rows_per_block, parts, p.rows_per_block / parts, col, val,
                                      w.split, w.begin, w.off, w.flags, w.st_low, w.st_k, w.st_v);
  sorted_hist_kernel<<<unsigned(p.max_tiles), 512, 0, s>>>(p.bins, p.blocks, w.tile_first, w.off, w.st_low, w.flags,
                                                           w.hist);
  note_launches(2);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  if ((e = launch_scan_i64(w.hist, sorted_hist_elems(p), w.place, w.scan_tmp, s)) != cudaSuccess) return e;
  sorted_cp_kernel<<<unsigned((n + 256) / 256), 256, 0, s>>>(n, nnz, w.tile_first, w.place, w.flags, cp);
  sorted_scatter_kernel<<<unsigned(p.max_tiles), kScatterThreads, sizeof(ScatterShared), s>>>(
      p.bins, p.blocks, w.tile_first, w.off, w.place, w.flags, w.st_low, w.st_k, w.st_v, trow, tval);
  note_launches(2);
  return cudaGetLastError();
}

}  // namespace raptr
