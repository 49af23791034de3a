// Batched MLEM for sm_100a: K frames that share one system matrix run as
// one multi-right-hand-side pass per half-iteration (SpMM), so every matrix
// entry is read once per frame tile instead of once per frame.
//
// Layout: images X (n x K) and measurements Y (m x K) are frame-minor
// (X[j*K + f]); the ratios E sit at the rows' positions in the transpose's
// order, like the single-frame e, in one block per tile: the tile of KT
// frames from f0 holds E[f0*m + k*KT + (f - f0)], so that the back pass
// over a tile gathers from m*KT floats (82 MB for 4 frames at 5.14M rows,
// inside L2) instead of 16 bytes out of each row of an m x K array, whose
// sectors for a 4-frame tile spread over 164 MB and missed L2 (33 ms per
// 4-frame back pass, against 3.9 ms for one frame).  A pass handles a tile
// of KT consecutive frames.  Within a warp, lanes split into EPW entry slots of
// LPE lanes, each lane owning VEC frames (LPE*VEC = KT, EPW*LPE = 32): per
// step a warp reads EPW matrix entries and gathers EPW rows of KT frames,
// coalesced.  The value type is binary16 (with the per-row scale folded
// into E, as in the FP16 single-frame form) or float.  Grids are sized to
// the GPU and every warp loops over rows / columns (persistent CTAs).  The
// back pass can take the columns in a given order: voxels in compact
// (y, z) tubes along x keep the ratio rows that concurrent warps gather
// (the channels crossing those voxels) within L2.
#include <algorithm>
#include <cstdint>
#include <vector>

#include <cuda_fp16.h>

#include "internal.h"

namespace raptr {

namespace {

constexpr int kThreads = 256;

// Blocks of a pass: one warp per item up to 64 blocks per SM, so that
// blocks are short enough for the scheduler to interleave the kernels of
// other streams (batches of other geometries served at the same time).
unsigned grid_warps(int64_t items) {
  int64_t b = (items * 32 + kThreads - 1) / kThreads;
  if (b < 1) b = 1;
  if (b > 148 * 64) b = 148 * 64;
  return unsigned(b);
}

constexpr int kColsPerWarp = 48;  // back pass: columns a warp takes before its block ends
// CTAs per SM the passes are compiled for: 5 forward (48 registers), 4 back (57,122
// rows of 70^3, 64 frames in tiles of 64 / 16 / 4, back pass with 3, 4, 5, 6: 767,
// 802, 1059, 827 / 1008, 1037, 1249, 1897 / 1686, 1582, 2139, 2589 us; forward with
// 3, 4, 5: 643, 601, 606 / 980, 879, 922 / 2005, 1763, 1672, and 5 is 2-4 % faster
// on 5.14M rows).
constexpr int kForwardBlocks = 5, kBackBlocks = 4;
constexpr double kBackGroupBytes = 48.0 * (1 << 20);  // ratios of a back-pass row-block group

__device__ __forceinline__ float to_f(float v) { return v; }
__device__ __forceinline__ float to_f(__half v) { return __half2float(v); }

// Four frames per lane (one 16-byte gather), KT/4 lanes per entry slot.
template <int KT>
struct Split {
  static constexpr int VEC = 4;
  static constexpr int LPE = KT / VEC;
  static constexpr int EPW = 32 / LPE;
};

__device__ __forceinline__ float4 ld4(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }

__device__ __forceinline__ void fma4(float (&a)[4], float w, float4 x) {
  a[0] += w * x.x;
  a[1] += w * x.y;
  a[2] += w * x.z;
  a[3] += w * x.w;
}

// acc += the entries [b, e) of a row or column times the frames at `at` + index *
// stride: the lane's slot's entries, its four frames, two entries per slot in
// flight.  A 64-frame tile has two slots, which keep sums of their own for the two
// (as many roundings in a row as at 32 frames, four slots).  (Reading 32 entries'
// indices and values at once and handing them to the slots by shuffles is 10-40 %
// slower: the slots' loads are broadcasts, and the gathers wait for the shuffles.)
template <int KT, typename VT>
__device__ __forceinline__ void gather_entries(const int32_t* __restrict__ idx, const VT* __restrict__ val, int64_t b,
                                               int64_t e, const float* __restrict__ at, int64_t stride, int lane,
                                               float (&acc)[4]) {
  using S = Split<KT>;
  int64_t k = b + lane / S::LPE;
  float odd[4] = {0.f, 0.f, 0.f, 0.f};
  for (; k + S::EPW < e; k += 2 * S::EPW) {
    const int c0 = __ldg(idx + k), c1 = __ldg(idx + k + S::EPW);
    const float w0 = to_f(val[k]), w1 = to_f(val[k + S::EPW]);
    const float4 x0 = ld4(at + int64_t(c0) * stride);
    const float4 x1 = ld4(at + int64_t(c1) * stride);
    fma4(acc, w0, x0);
    fma4(S::EPW > 2 ? acc : odd, w1, x1);
  }
  if (k < e) fma4(acc, to_f(val[k]), ld4(at + int64_t(__ldg(idx + k)) * stride));
  if (S::EPW <= 2) {
#pragma unroll
    for (int v = 0; v < 4; v++) acc[v] += odd[v];
  }
}

// Forward: Et[rank_i*KT + f - f0] = sc_i * Y[i*K + f] / (sc_i * sum_j v_ij
// X[j*K + f]) for the frames f of the tile (0 where Y == 0), Et = E + f0*m
// the tile's block of ratios; sc = rscale (FP16) or 1.  The images are gathered from Xg with row stride xs:
// X + f0 and K, or a compact copy of the tile's frames and KT (a 4-frame
// tile then gathers from n*16 bytes instead of 16 bytes of each 256-byte
// row of a 64-frame X).
template <int KT, typename VT>
__global__ void __launch_bounds__(kThreads, kForwardBlocks) batch_forward_kernel(int64_t m, int K, int f0,
                                                                 const int64_t* __restrict__ rp,
                                                                 const int32_t* __restrict__ col,
                                                                 const VT* __restrict__ val,
                                                                 const float* __restrict__ rscale,
                                                                 const float* __restrict__ Y,
                                                                 const float* __restrict__ Xg, int xs,
                                                                 const int32_t* __restrict__ rank,
                                                                 float* __restrict__ Et) {
  using S = Split<KT>;
  const int lane = threadIdx.x & 31;
  const int es = lane / S::LPE, fg = lane % S::LPE;
  const int fbase = f0 + fg * S::VEC;
  const float* __restrict__ X = Xg + fg * S::VEC;  // the lane's four frames
  const int64_t nw = (int64_t(gridDim.x) * blockDim.x) >> 5;
  for (int64_t r = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; r < m; r += nw) {
    float acc[S::VEC];
#pragma unroll
    for (int v = 0; v < S::VEC; v++) acc[v] = 0.f;
    const int64_t b = rp[r], e = rp[r + 1];
    if constexpr (KT == 8) {
      // (as gather_entries, whose loop is compiled differently here: 5.14M rows of 70^3,
      // FP16, 11.2 ms, so 10.2; every other width is as fast or faster with it)
      int64_t k = b + es;
      for (; k + S::EPW < e; k += 2 * S::EPW) {
        const int c0 = __ldg(col + k), c1 = __ldg(col + k + S::EPW);
        const float w0 = to_f(val[k]), w1 = to_f(val[k + S::EPW]);
        const float4 x0 = ld4(X + int64_t(c0) * xs);
        const float4 x1 = ld4(X + int64_t(c1) * xs);
        fma4(acc, w0, x0);
        fma4(acc, w1, x1);
      }
      if (k < e) fma4(acc, to_f(val[k]), ld4(X + int64_t(__ldg(col + k)) * xs));
    } else {
      gather_entries<KT>(col, val, b, e, X, xs, lane, acc);
    }
#pragma unroll
    for (int o = S::LPE; o < 32; o <<= 1)
#pragma unroll
      for (int v = 0; v < S::VEC; v++) acc[v] += __shfl_xor_sync(0xffffffffu, acc[v], o);
    if (es == 0) {
      const float sc = rscale ? __ldg(rscale + r) : 1.f;
      const int64_t dst = rank ? int64_t(__ldg(rank + r)) : r;
#pragma unroll
      for (int v = 0; v < S::VEC; v++) {
        const float yi = __ldg(Y + r * K + fbase + v);
        Et[dst * KT + fg * S::VEC + v] = yi == 0.f ? 0.f : sc * __fdiv_rn(yi, sc * acc[v]);
      }
    }
  }
}

// Back projection and update for the frames of the tile:
// c = sum_k v_kj Eb[k*KT + f - f0] (Eb = E + f0*m, the tile's block of
// ratios; FP32, the FP16 values dominate its error),
// XX = X*c/(S+(S==0)), acc[f] += sum_j XX (FP64).  Warps take the columns that
// have entries (the first *n_full of cols) from the counter *next (zero at
// launch).  The others (where few views are measured two thirds of them) have c =
// 0, so XX = X*0/(S+(S==0)), which is 0 unless X is not finite; the threads of the last
// group's pass share them afterwards.
//
// With a row-block group (seg non-null), only the column's entries whose
// rows lie in blocks [b0, b1) of the transpose's row order are summed
// (entries seg[j*segw + b0] .. seg[j*segw + b1] of column j): the ratios of
// those rows then stay in L2 while every column reads them.  The partial
// sums of all but the last group go to P (n x KT, tile-local frames); the
// last group adds them and finishes as above.  mode: 0 = the whole column
// at once, 1 = first group, 2 = a middle group, 3 = the last group.
template <int KT, typename VT>
__global__ void __launch_bounds__(kThreads, kBackBlocks) batch_back_kernel(int64_t n, int K, int f0, unsigned long long* next,
                                                              const int64_t* __restrict__ cp,
                                                              const int32_t* __restrict__ trow,
                                                              const VT* __restrict__ tval,
                                                              const float* __restrict__ Eb,
                                                              const float* __restrict__ X,
                                                              const float* __restrict__ sens,
                                                              const int32_t* __restrict__ cols,
                                                              const int64_t* __restrict__ n_full,
                                                              float* __restrict__ XX, double* __restrict__ acc,
                                                              const int32_t* __restrict__ seg, int segw, int b0,
                                                              int b1, int mode, float* __restrict__ P) {
  using S = Split<KT>;
  const int lane = threadIdx.x & 31;
  const int es = lane / S::LPE, fg = lane % S::LPE;
  const int fbase = f0 + fg * S::VEC;
  // the lane's four frames of this tile's block of ratios
  const float* __restrict__ Et = Eb + fg * S::VEC;
  double fsum[S::VEC];
#pragma unroll
  for (int v = 0; v < S::VEC; v++) fsum[v] = 0.0;
  __shared__ double red[KT];  // the block's image sums per frame of the tile
  for (int i = threadIdx.x; i < KT; i += blockDim.x) red[i] = 0.0;
  __syncthreads();
  const unsigned long long count = (unsigned long long)*n_full;
  for (int taken = 0; taken < kColsPerWarp; taken++) {
    // columns are handed out one at a time (their lengths vary ~20-fold)
    unsigned long long q = 0;
    if (lane == 0) q = atomicAdd(next, 1ull);
    q = __shfl_sync(0xffffffffu, q, 0);
    if (q >= count) break;
    const int64_t j = __ldg(cols + q);
    float s[S::VEC];
#pragma unroll
    for (int v = 0; v < S::VEC; v++) s[v] = 0.f;
    int64_t b = cp[j], e = cp[j + 1];
    if (seg) {
      const int64_t c0 = b;
      b = c0 + __ldg(seg + j * segw + b0);
      e = c0 + __ldg(seg + j * segw + b1);
    }
    gather_entries<KT>(trow, tval, b, e, Et, KT, lane, s);
#pragma unroll
    for (int o = S::LPE; o < 32; o <<= 1)
#pragma unroll
      for (int v = 0; v < S::VEC; v++) s[v] += __shfl_xor_sync(0xffffffffu, s[v], o);
    if (es == 0 && mode != 0) {
      float4* pp = reinterpret_cast<float4*>(P + j * KT + (fbase - f0));
      if (mode == 2 || mode == 3) {
        const float4 q4 = *pp;
        s[0] += q4.x;
        s[1] += q4.y;
        s[2] += q4.z;
        s[3] += q4.w;
      }
      if (mode != 3) {
        *pp = make_float4(s[0], s[1], s[2], s[3]);
        continue;
      }
    }
    if (es == 0) {
      float dvs = __ldg(sens + j);
      dvs += float(dvs == 0.f);
#pragma unroll
      for (int v = 0; v < S::VEC; v++) {
        const float xx = __fdiv_rn(__fmul_rn(X[j * K + fbase + v], s[v]), dvs);
        XX[j * K + fbase + v] = xx;
        fsum[v] += double(xx);
      }
    }
  }
  if (es == 0)
#pragma unroll
    for (int v = 0; v < S::VEC; v++)
      if (fsum[v] != 0.0) atomicAdd(red + (fbase - f0) + v, fsum[v]);
  __syncthreads();
  for (int i = threadIdx.x; i < KT; i += blockDim.x)
    if (red[i] != 0.0) atomicAdd(acc + f0 + i, red[i]);
  if (mode == 0 || mode == 3) {
    const int64_t empty = (n - int64_t(count)) * S::LPE;
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < empty; i += int64_t(gridDim.x) * blockDim.x) {
      const int64_t j = __ldg(cols + int64_t(count) + i / S::LPE);
      const int f = f0 + int(i % S::LPE) * S::VEC;
      float dvs = __ldg(sens + j);
      dvs += float(dvs == 0.f);
#pragma unroll
      for (int v = 0; v < S::VEC; v++) {
        const float xx = __fdiv_rn(__fmul_rn(X[j * K + f + v], 0.f), dvs);
        XX[j * K + f + v] = xx;
        if (xx != 0.f) atomicAdd(acc + f + v, double(xx));
      }
    }
  }
}

// flag[q] = 1 where the q-th column of the order has entries; then, with pos its
// exclusive sums, cols = those columns in order, followed by the others.
__global__ void batch_flag_kernel(int64_t n, const int64_t* __restrict__ cp, const int32_t* __restrict__ order,
                                  int64_t* __restrict__ flag) {
  const int64_t q = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (q >= n) return;
  const int64_t j = order ? int64_t(order[q]) : q;
  flag[q] = cp[j + 1] > cp[j] ? 1 : 0;
}
__global__ void batch_columns_kernel(int64_t n, const int64_t* __restrict__ cp, const int32_t* __restrict__ order,
                                     const int64_t* __restrict__ pos, int32_t* __restrict__ cols) {
  const int64_t q = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (q >= n) return;
  const int64_t j = order ? int64_t(order[q]) : q;
  cols[cp[j + 1] > cp[j] ? pos[q] : pos[n] + q - pos[q]] = int32_t(j);
}

// Xt[j*t + f'] = X[j*K + f0 + f'], the tile's frames of every image row
// (t a multiple of 4: one 16-byte copy per thread and step).
__global__ void batch_tile_images_kernel(int64_t n, int K, int f0, int t, const float* __restrict__ X,
                                         float* __restrict__ Xt) {
  const int q = t / 4;
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n * q; i += int64_t(gridDim.x) * blockDim.x) {
    const int64_t j = i / q;
    const int v = int(i - j * q) * 4;
    *reinterpret_cast<float4*>(Xt + j * t + v) = *reinterpret_cast<const float4*>(X + j * K + f0 + v);
  }
}

// X = XX * (1 / acc[f]) for all frames.  A thread's four frames stay the same (the
// grid's threads are a multiple of K / 4), so their scales are taken once.
__global__ void batch_normalise_kernel(int64_t n, int K, int64_t threads, float* __restrict__ X,
                                       const float* __restrict__ XX, const double* __restrict__ acc) {
  const int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t >= threads) return;
  const int f = int(t % (K / 4)) * 4;
  float sc[4];
#pragma unroll
  for (int v = 0; v < 4; v++) sc[v] = float(1.0 / acc[f + v]);
  const int64_t total = n * (K / 4);
  for (int64_t i = t; i < total; i += threads) {
    const float4 x = reinterpret_cast<const float4*>(XX)[i];
    reinterpret_cast<float4*>(X)[i] = make_float4(x.x * sc[0], x.y * sc[1], x.z * sc[2], x.w * sc[3]);
  }
}

// A back pass over row blocks [b0, b1) of the transpose (mode as in
// batch_back_kernel; mode 0 = every row at once, without seg).
struct BackGroup {
  int b0 = 0, b1 = 0, mode = 0;
};

template <int KT, typename VT>
cudaError_t launch_tile(const BatchArgs& a, bool forward, int f0, double* acc, unsigned long long* next,
                        const BackGroup& grp, cudaStream_t s) {
  if (forward) {
    const bool compact = a.Xt && KT < a.K;
    if (compact) {
      int64_t blocks = (a.n * (KT / 4) + kThreads - 1) / kThreads;
      if (blocks > 148 * 8) blocks = 148 * 8;
      batch_tile_images_kernel<<<unsigned(std::max<int64_t>(blocks, 1)), kThreads, 0, s>>>(a.n, a.K, f0, KT, a.X,
                                                                                         a.Xt);
      note_launches(1);
    }
    batch_forward_kernel<KT, VT><<<grid_warps(a.m), kThreads, 0, s>>>(
        a.m, a.K, f0, a.rp, a.col, static_cast<const VT*>(a.val), a.half ? a.rscale : nullptr, a.Y,
        compact ? a.Xt : a.X + f0, compact ? KT : a.K, a.rank, a.E + int64_t(f0) * a.m);
  } else {
    // blocks for all columns at kColsPerWarp columns a warp (a warp takes no more),
    // and enough to fill the GPU
    const int64_t per = kColsPerWarp * (kThreads / 32);
    const int64_t blocks = std::max<int64_t>((a.n + per - 1) / per, std::min<int64_t>(148 * 10, grid_warps(a.n)));
    batch_back_kernel<KT, VT><<<unsigned(blocks), kThreads, 0, s>>>(a.n, a.K, f0, next, a.cp, a.trow, static_cast<const VT*>(a.tval),
                                                  a.E + int64_t(f0) * a.m,
                                                  a.X, a.S, a.cols, a.n_full, a.XX, acc, grp.mode ? a.seg : nullptr,
                                                  a.seg_blocks + 1, grp.b0, grp.b1, grp.mode, a.P);
  }
  note_launches(1);
  return cudaGetLastError();
}

template <typename VT>
cudaError_t launch_tile_kt(int kt, const BatchArgs& a, bool forward, int f0, double* acc, unsigned long long* next,
                           const BackGroup& grp, cudaStream_t s) {
  switch (kt) {
    case 4: return launch_tile<4, VT>(a, forward, f0, acc, next, grp, s);
    case 8: return launch_tile<8, VT>(a, forward, f0, acc, next, grp, s);
    case 16: return launch_tile<16, VT>(a, forward, f0, acc, next, grp, s);
    case 32: return launch_tile<32, VT>(a, forward, f0, acc, next, grp, s);
    case 64: return launch_tile<64, VT>(a, forward, f0, acc, next, grp, s);
    default: return cudaErrorInvalidValue;
  }
}

// seg[j*(B+1) + b] = the offset in column j of its first entry whose row
// (position in the transpose's order) is at least b*m/B: lane b of the
// column's warp searches boundary b (entries ascend within a column).
__global__ void block_seg_kernel(int64_t n, int64_t m, int B, const int64_t* __restrict__ cp,
                                 const int32_t* __restrict__ trow, int32_t* __restrict__ seg) {
  const int lane = threadIdx.x & 31;
  const int64_t nw = (int64_t(gridDim.x) * blockDim.x) >> 5;
  for (int64_t j = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; j < n; j += nw) {
    const int64_t c0 = cp[j], c1 = cp[j + 1];
    for (int b = lane; b <= B; b += 32) {
      const int64_t kb = m * b / B;
      int64_t lo = c0, hi = c1;  // first entry with trow >= kb
      while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        if (int64_t(__ldg(trow + mid)) < kb) lo = mid + 1;
        else hi = mid;
      }
      seg[j * (B + 1) + b] = int32_t(lo - c0);
    }
  }
}

}  // namespace

cudaError_t launch_block_seg(int64_t n, int64_t m, int B, const int64_t* cp, const int32_t* trow, int32_t* seg,
                             cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  block_seg_kernel<<<grid_warps(n), kThreads, 0, s>>>(n, m, B, cp, trow, seg);
  note_launches(1);
  return cudaGetLastError();
}

bool batch_tile_supported(int K, int kt) {
  return (kt == 4 || kt == 8 || kt == 16 || kt == 32 || kt == 64) && K > 0 && K % 4 == 0;
}

int batch_tile_at(int K, int kt, int f0) {
  int t = kt;
  while (t > K - f0) t >>= 1;
  return t;
}

cudaError_t launch_batch_columns(int64_t n, const int64_t* cp, const int32_t* order, int64_t* flag, int64_t* pos,
                                 int64_t* scan_tmp, int32_t* cols, cudaStream_t s) {
  const unsigned blocks = unsigned((n + kThreads - 1) / kThreads);
  batch_flag_kernel<<<blocks, kThreads, 0, s>>>(n, cp, order, flag);
  note_launches(1);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = launch_scan_i64(flag, n, pos, scan_tmp, s);
  if (e != cudaSuccess) return e;
  batch_columns_kernel<<<blocks, kThreads, 0, s>>>(n, cp, order, pos, cols);
  note_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_batch_iteration(const BatchArgs& a, int kt, double* acc, unsigned long long* next, cudaStream_t s,
                                   cudaEvent_t ev_mid) {
  // Tiles of kt frames while that many remain, then the largest power of
  // two (>= 4, since K is a multiple of 4) that fits: 40 frames at kt = 32
  // run as 32 + 8, so no frame slot is computed for nothing.
  // Back-pass row-block groups of a tile: the tile's ratios of one group
  // (rows of g blocks of the transpose's order) should fit in about half of
  // L2, so that the column gathers of the group find them there.
  auto groups = [&](int t) {
    std::vector<BackGroup> out;
    if (!a.seg || !a.P || a.seg_blocks < 2) {
      out.push_back(BackGroup{});
      return out;
    }
    const double block_bytes = double(a.m) / a.seg_blocks * t * sizeof(float);
    const int g = std::max(1, int(kBackGroupBytes / std::max(block_bytes, 1.0)));
    if (g >= a.seg_blocks) {
      out.push_back(BackGroup{});
      return out;
    }
    for (int b = 0; b < a.seg_blocks; b += g) {
      BackGroup q;
      q.b0 = b;
      q.b1 = std::min(a.seg_blocks, b + g);
      q.mode = b == 0 ? 1 : (q.b1 == a.seg_blocks ? 3 : 2);
      out.push_back(q);
    }
    return out;
  };
  cudaError_t e = cudaMemsetAsync(acc, 0, size_t(a.K) * sizeof(double), s);
  if (e == cudaSuccess)
    e = cudaMemsetAsync(next, 0, size_t(a.K / 4) * size_t(std::max(a.seg_blocks, 1)) * sizeof(unsigned long long), s);
  const BackGroup whole;
  for (int f0 = 0; f0 < a.K && e == cudaSuccess; f0 += batch_tile_at(a.K, kt, f0)) {
    const int t = batch_tile_at(a.K, kt, f0);
    e = a.half ? launch_tile_kt<__half>(t, a, true, f0, acc, nullptr, whole, s)
               : launch_tile_kt<float>(t, a, true, f0, acc, nullptr, whole, s);
  }
  if (e == cudaSuccess && ev_mid) e = cudaEventRecord(ev_mid, s);
  for (int f0 = 0; f0 < a.K && e == cudaSuccess; f0 += batch_tile_at(a.K, kt, f0)) {
    const int t = batch_tile_at(a.K, kt, f0);
    for (const BackGroup& q : groups(t)) {
      if (e != cudaSuccess) break;
      e = a.half ? launch_tile_kt<__half>(t, a, false, f0, acc, next, q, s)
                 : launch_tile_kt<float>(t, a, false, f0, acc, next, q, s);
      next++;
    }
  }
  if (e == cudaSuccess) {
    const int64_t q = a.K / 4;
    const int64_t threads = std::min<int64_t>(a.n * q, std::max<int64_t>(int64_t(148) * 8 * kThreads / q, 1) * q);
    batch_normalise_kernel<<<unsigned((threads + kThreads - 1) / kThreads), kThreads, 0, s>>>(a.n, a.K, threads, a.X,
                                                                                             a.XX, acc);
    note_launches(1);
    e = cudaGetLastError();
  }
  return e;
}

}  // namespace raptr
