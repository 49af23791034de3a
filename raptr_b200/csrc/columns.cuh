// The column loop of the single-frame back projections (FP32 and FP16), which
// differ in how a column's dot product is taken.
#pragma once

#include <cstdint>
#include <type_traits>

#include "common.cuh"

namespace raptr {

constexpr int kShortColumn = 64;    // entries of a column that four are taken of together

constexpr int kColumnCost = 64;     // entries that the looking at a column counts for

// Columns up to which the back pass has a warp for each (EACH below).  In units, few
// columns fall to few warps, and the draws are as many as without units: FP32 back
// projection of 300 columns of 5,000 entries 41 us in units, 23 so; 50 of 40 20 and 11;
// 18,000 of 1,000 77 and 75.
constexpr int64_t kEachColumn = 148 * 16 * 8;

// Count of a unit of columns, of `total` in all: 32 units to a warp that is
// resident, but no less than a draw takes to serve (2048 entries).
__device__ __forceinline__ int64_t column_unit(int64_t total) {
  const int64_t u = total / (int64_t(kDrawWarps) * 32);
  return u < 2048 ? 2048 : u;
}

// Neumaier compensated addition: (s, c) += v.
__device__ __forceinline__ void two_sum_add(float& s, float& c, float v) {
  const float t = s + v;
  if (fabsf(s) >= fabsf(v))
    c += (s - t) + v;
  else
    c += (v - t) + s;
  s = t;
}

// An FP32 sum with its compensation.
struct CompensatedSum {
  float s = 0.f, c = 0.f;
  __device__ __forceinline__ void add_lane_xor(const CompensatedSum& o, int x) {
    const float so = __shfl_xor_sync(0xffffffffu, o.s, x), co = __shfl_xor_sync(0xffffffffu, o.c, x);
    two_sum_add(s, c, so);
    c += co;
  }
};

// Sums of four values over the warp: lane l gets that of value l / 8.
__device__ __forceinline__ float warp_sum4(const float (&s)[4], int lane) {
  const bool h = (lane & 16) != 0, q = (lane & 8) != 0;
  float a = (h ? s[2] : s[0]) + __shfl_xor_sync(0xffffffffu, h ? s[0] : s[2], 16);
  float b = (h ? s[3] : s[1]) + __shfl_xor_sync(0xffffffffu, h ? s[1] : s[3], 16);
  a = (q ? b : a) + __shfl_xor_sync(0xffffffffu, q ? a : b, 8);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
  return a;
}
__device__ __forceinline__ float warp_sum4(const CompensatedSum (&s)[4], int lane) {
  const bool h = (lane & 16) != 0, q = (lane & 8) != 0;
  CompensatedSum a = h ? s[2] : s[0], b = h ? s[3] : s[1];
  a.add_lane_xor(h ? s[0] : s[2], 16);
  b.add_lane_xor(h ? s[1] : s[3], 16);
  CompensatedSum t = q ? b : a;
  t.add_lane_xor(q ? a : b, 8);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) t.add_lane_xor(t, o);
  return t.s + t.c;
}

// Dot products of four columns of at most kShortColumn entries with e, in sums
// of type Sum (float, or CompensatedSum: the FP16 form); lane l gets that of column
// l / 8.  All loads of the four are in flight together.
template <class Sum, class VT, class F>
__device__ __forceinline__ float short_columns(const int32_t* __restrict__ trow, const VT* __restrict__ tval,
                                               const int64_t (&b)[4], const int (&len)[4],
                                               const float* __restrict__ e, int lane, F to_float) {
  Sum s[4];
  int r[4][2];
  VT w[4][2];
#pragma unroll
  for (int k = 0; k < 4; k++)
#pragma unroll
    for (int u = 0; u < 2; u++) {
      const bool in = lane + 32 * u < len[k];
      r[k][u] = in ? __ldcs(trow + b[k] + lane + 32 * u) : -1;
      w[k][u] = in ? __ldcs(tval + b[k] + lane + 32 * u) : VT(0);
    }
#pragma unroll
  for (int k = 0; k < 4; k++) {
    if constexpr (std::is_same_v<Sum, float>) {
      s[k] = 0.f;
#pragma unroll
      for (int u = 0; u < 2; u++)
        if (r[k][u] >= 0) s[k] += to_float(w[k][u]) * __ldg(e + r[k][u]);
    } else {
#pragma unroll
      for (int u = 0; u < 2; u++)
        if (r[k][u] >= 0) two_sum_add(s[k].s, s[k].c, to_float(w[k][u]) * __ldg(e + r[k][u]));
    }
  }
  return warp_sum4(s, lane);
}

// c_j = <column j, e> for every column, by `dot(b, e)` (one column of any
// length) and `dot4(b[4], len[4])` (four short ones).  With UPDATE the MLEM
// update follows: out_j = x_j*c_j/(s_j + (s_j==0)), and the sum of the lane's
// out_j is returned; without it c_j is stored.
//
// Columns run from none to 10^4 entries and more, so the work is cut into
// units by entries, a column counting kColumnCost entries more than it has:
// unit k takes the columns that begin in [k*E, (k+1)*E) of that count.  Warps
// draw units from the counter at `next` (zero at launch), or take them by a
// grid stride without one.  A unit's columns are looked at 32 at a time, so
// that their pointers, x and sensitivities are read and their results written
// together and an empty column (two thirds of them, where few views are
// measured) costs next to nothing.
//
// One column per draw, as before, was bound by the draws (0.5 ms for 343,000
// columns whatever they hold); several columns per draw by the warp that drew
// the longest.  Back pass of 70^3 voxels, FP32 / FP16: 1,000 rows 242 / 240 ->
// 31 / 31 us, 20,000 rows 252 / 248 -> 54 / 52, 200,000 rows 528 / 460 -> 224 /
// 193, 5.14M rows (100 rays) 4.3 / 3.4 -> 4.1 / 3.5 ms; units of 1024 or 4096
// entries and 8 or 16 units to a warp are 2-10 % slower on some of these.
//
// With EACH, for few columns, there are no units: every warp takes a column, and
// neighbours (which may be long together) go to different blocks.
template <bool UPDATE, bool EACH, class Dot, class Dot4>
__device__ __forceinline__ double back_columns(int64_t n, const int64_t* __restrict__ cp,
                                               const float* __restrict__ x, const float* __restrict__ sens,
                                               float* __restrict__ out, unsigned long long* next, Dot dot,
                                               Dot4 dot4) {
  const int lane = threadIdx.x & 31;
  const int64_t total = EACH ? n : cp[n] + kColumnCost * n, unit = EACH ? 1 : column_unit(total);
  if (EACH) next = nullptr;
  double sum = 0.0;
  int64_t k = EACH   ? int64_t(threadIdx.x >> 5) * gridDim.x + blockIdx.x
              : next ? warp_next(next, lane)
                     : (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  while (k * unit < total) {
    const int64_t p0 = k * unit, p1 = p0 + unit;
    // the first column at p0 or later, 32 probes at a time
    int64_t j0 = EACH ? k : 0, hi = EACH ? k : n;
    while (j0 < hi) {
      const int64_t step = (hi - j0 + 31) >> 5, j = j0 + lane * step;
      const bool before = j < hi && cp[j] + kColumnCost * j < p0;
      const int c = __popc(__ballot_sync(0xffffffffu, before));
      if (c == 0) break;
      hi = min(hi, j0 + c * step);
      j0 += (c - 1) * step + 1;
    }
    bool more = true;
    for (; more && j0 < n; j0 += 32) {
      const int64_t j = j0 + lane;
      int64_t b = 0, e = 0;
      bool own = false;
      if (j < n) {
        b = cp[j];
        e = cp[j + 1];
        own = EACH ? j == k : b + kColumnCost * j < p1;
      }
      more = __all_sync(0xffffffffu, own);
      const int len = own ? int(min(e - b, int64_t(kShortColumn + 1))) : 0;
      float c = 0.f;
      unsigned shorts = __ballot_sync(0xffffffffu, len > 0 && len <= kShortColumn);
      unsigned longs = __ballot_sync(0xffffffffu, len > kShortColumn);
      while (longs) {
        const int i = __ffs(longs) - 1;
        longs &= longs - 1;
        const float v = dot(__shfl_sync(0xffffffffu, b, i), __shfl_sync(0xffffffffu, e, i));
        if (lane == i) c = v;
      }
      while (shorts) {
        unsigned at = 0;  // the four columns' lanes, a byte each
        int64_t bk[4];
        int lk[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const int l = shorts ? __ffs(shorts) - 1 : 0;
          bk[i] = __shfl_sync(0xffffffffu, b, l);
          lk[i] = __shfl_sync(0xffffffffu, len, l);
          lk[i] = shorts ? lk[i] : 0;
          at |= unsigned(shorts ? l : 255) << (8 * i);
          shorts &= shorts - 1;
        }
        const float v = dot4(bk, lk);
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const float vi = __shfl_sync(0xffffffffu, v, 8 * i);
          if (unsigned(lane) == ((at >> (8 * i)) & 255u)) c = vi;
        }
      }
      if (own) {
        if (UPDATE) {
          float dvs = sens[j];
          dvs += float(dvs == 0.f);
          const float xx = __fdiv_rn(__fmul_rn(x[j], c), dvs);
          out[j] = xx;
          sum += double(xx);
        } else {
          out[j] = c;
        }
      }
    }
    k = next ? warp_next(next, lane) : k + ((int64_t(gridDim.x) * blockDim.x) >> 5);
  }
  return sum;
}

}  // namespace raptr
