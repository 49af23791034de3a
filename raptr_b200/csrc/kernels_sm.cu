// System-matrix rows, ray endpoints and the enclosing-cylinder candidate
// search, for sm_100a.
//
// Row build (one CTA per channel row):
//   1. thread 0 builds the channel state (both crystal transforms from the
//      per-angle sine/cosine table, crystal centres, cylinder radius);
//   2. the row's rays (Philox keyed by (seed, channel)) are traced through the
//      grid.  A trace yields exactly the voxels whose intersection length with
//      the ray is positive, and that length with the same float operations as
//      the reference's intersectionLength (src/getSystemMatrixDeviceOnly.cu:129-174):
//      per-axis plane parameters (face - start)/(end - start), masked max of
//      the entry parameters, masked min of the exit parameters, and
//      (exit - entry) * |end - start|.  When the two crystals lie on opposite
//      sides of the grid along x or z, threads own slabs of the grid
//      (sm_slab_kernel); where the slabs' windows are too large for that
//      (crystals of many voxels) each ray is walked from plane to plane into
//      the windows (sm_window_kernel); the other rows walk their rays into an
//      open-addressing hash table keyed by voxel id (sm_table_kernel);
//   3. the sums are compacted keeping voxels that pass the exact cylinder
//      test (the reference only evaluates candidates,
//      src/getSystemMatrixDeviceOnly.cu:433-470), put in voxel-id order,
//      divided by the ray count and written to the row's staging slot.
// The rows are therefore emitted already in (row, column) order: no global
// COO sort (src/cooSort.hpp:75-99) and no coo->csr pass are needed; a scan
// of the row lengths and a gather place them into CSR.
//
// This translation unit is compiled with -fmad=false in addition to the
// explicit round-to-nearest intrinsics used on every exact path.
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdint>

#include "common.cuh"
#include "internal.h"

namespace raptr {

namespace {

constexpr int kProbeLimit = 128;

__device__ __forceinline__ float plane_alpha(float o, float d, int i, float r0, float dir) {
  return RFDIV(RFSUB(RFADD(o, RFMUL(float(i), d)), r0), dir);
}

// RN(a / b) from y = RN(1 / b): one correction of the product (the division with
// one multiplication and two fused multiply-adds of N. Brisebarre, J.-M. Muller
// and S. K. Raina, IEEE Trans. Computers 53(8), 2004, after P. Markstein's,
// IBM J. R&D 34(1), 1990).  Checked once for all 2^46 pairs of significands (16.8M
// random ones and those at the edges: tests/test_division.py), so it is
// the quotient wherever that and the remainder are normal floats.  (A second correction,
// for a first quotient off by more than one ulp, changes none and costs 10 % of the
// slab kernel: 10,000 rows of 70^3 x 1000 rays 2.29 against 2.07 ms.)
__device__ __forceinline__ float div_rcp(float a, float b, float y) {
  const float q = __fmul_rn(a, y);
  return __fmaf_rn(__fmaf_rn(-q, b, a), y, q);
}

// plane_alpha with the division by a precomputed reciprocal rc = RN(1/dir)
// (exact as RN(num/dir), see div_rcp); a dir whose reciprocal is not a
// normal float takes the division itself.
__device__ __forceinline__ float plane_alpha_r(float o, float d, int i, float r0, float dir, float rc) {
  const float num = RFSUB(RFADD(o, RFMUL(float(i), d)), r0);
  if (!(fabsf(dir) >= 1e-30f && fabsf(dir) <= 1e30f)) return RFDIV(num, dir);
  return div_rcp(num, dir, rc);
}

// Origin, pitch and size of axis k of the grid for a k known only at run
// time: selects, so that the by-value geometry stays in the constant bank
// instead of being copied to local memory for an indexed access.
__device__ __forceinline__ float axis_o(const DGeom& g, int k) { return k == 0 ? g.o[0] : (k == 1 ? g.o[1] : g.o[2]); }
__device__ __forceinline__ float axis_d(const DGeom& g, int k) { return k == 0 ? g.d[0] : (k == 1 ? g.d[1] : g.d[2]); }
__device__ __forceinline__ int axis_n(const DGeom& g, int k) { return k == 0 ? g.n[0] : (k == 1 ? g.n[1] : g.n[2]); }

// Shared-memory accumulation table: keys (voxel id, -1 = empty) and sums.
template <int H>
struct RowTable {
  int* keys;
  float* vals;
  int* overflow;

  __device__ __forceinline__ void add(int key, float v) const {
    constexpr int LOG2H = (H == 2048) ? 11 : (H == 4096) ? 12 : (H == 8192) ? 13 : 14;
    unsigned h = (unsigned(key) * 2654435761u) >> (32 - LOG2H);
#pragma unroll 1
    for (int p = 0; p < kProbeLimit; p++) {
      int k = reinterpret_cast<volatile int*>(keys)[h];
      if (k == key) {
        atomicAdd(&vals[h], v);
        return;
      }
      if (k < 0) {
        int old = atomicCAS(&keys[h], -1, key);
        if (old < 0 || old == key) {
          atomicAdd(&vals[h], v);
          return;
        }
      }
      h = (h + 1) & (H - 1);
    }
    *overflow = 1;
  }
};

// Where the step walk adds a voxel's length: the voxel id, added to the row's
// hash table.  begin() takes the ray's step directions, set() places the
// index at a voxel, advance() moves it one voxel along the axis the walk
// steps (x if ax, else y if ay, else z).
template <int H>
struct KeyIndex {
  const RowTable<H>* table;
  int nyz, nz;
  int key, k0, k1, k2;
  __device__ __forceinline__ void begin(const int step[3]) {
    k0 = step[0] * nyz;
    k1 = step[1] * nz;
    k2 = step[2];
  }
  __device__ __forceinline__ void set(int i0, int i1, int i2) { key = i0 * nyz + i1 * nz + i2; }
  __device__ __forceinline__ void advance(bool ax, bool ay) { key += ax ? k0 : (ay ? k1 : k2); }
  __device__ __forceinline__ void add(float L) const { table->add(key, L); }
};

// The same into the windows of a row with slab axis A (x or z): slot
// base[s] + iu * wv + iv for a voxel of slab s, which a step along A moves by
// dk[s] more than (u, v) do; no key is stored or compared.
template <int A>
struct WindowIndex {
  float* sums;
  const int* base;
  const int* dk;
  int wv, nslots;
  int slot, sa, ka, sta, ku, kv;
  __device__ __forceinline__ void begin(const int step[3]) {
    sta = step[A];
    ku = step[A == 0 ? 1 : 0] * wv;
    kv = step[A == 0 ? 2 : 1];
  }
  __device__ __forceinline__ void set(int i0, int i1, int i2) {
    sa = A == 0 ? i0 : i2;
    slot = A == 0 ? base[i0] + i1 * wv + i2 : base[i2] + i0 * wv + i1;
    ka = dk[sa];
  }
  __device__ __forceinline__ void advance(bool ax, bool ay) {
    if (A == 0) {
      slot += ax ? ka : (ay ? ku : kv);
      sa = ax ? sa + sta : sa;
    } else {
      slot += ax ? ku : (ay ? kv : ka);
      sa = (ax || ay) ? sa : sa + sta;
    }
    ka = dk[sa];
  }
  // a slot outside the windows is the spare one, which the row looks at afterwards
  __device__ __forceinline__ void add(float L) const {
    atomicAdd(&sums[unsigned(slot) < unsigned(nslots) ? slot : nslots], L);
  }
};

// Visits every grid voxel whose intersection length with ray r is positive.
// A ray that crosses the planes of all three axes takes the step loop,
// which adds the lengths through the index `ix`; any other ray takes the
// general loop, which adds through emit(ix, iy, iz, L): a ray parallel to
// the planes of some axis (start and end coordinate equal) leaves that axis
// unconstrained, as the reference's masked min/max does, and every
// candidate voxel along it gets the length.  Of those candidates the caller
// gets every k_step-th from k_first on, so that a block can share them.
template <bool OISO, class Emit, class Index>
__device__ __forceinline__ void walk_ray(const DGeom& g, const Channel& ch, const float r[6], int part, Emit& emit,
                                         Index& ix, int* bad_walk, int k_first, int k_step) {
  float dir[3];
  bool s[3];
#pragma unroll
  for (int d = 0; d < 3; d++) {
    dir[d] = RFSUB(r[3 + d], r[d]);
    s[d] = r[d] != r[3 + d];
  }
  if (!(s[0] || s[1] || s[2])) return;
  float rc[3];
#pragma unroll
  for (int d = 0; d < 3; d++) rc[d] = s[d] ? __frcp_rn(dir[d]) : 0.f;
  const float len = norm3_exact(dir[0], dir[1], dir[2]);
  int step[3] = {0, 0, 0};
  float amin_g = -INFINITY, amax_g = INFINITY;
#pragma unroll
  for (int d = 0; d < 3; d++) {
    if (s[d]) {
      step[d] = (r[3 + d] > r[d]) ? 1 : -1;
      float a0 = plane_alpha_r(g.o[d], g.d[d], 0, r[d], dir[d], rc[d]);
      float a1 = plane_alpha_r(g.o[d], g.d[d], g.n[d], r[d], dir[d], rc[d]);
      amin_g = fmaxf(amin_g, fminf(a0, a1));
      amax_g = fminf(amax_g, fmaxf(a0, a1));
    }
  }
  if (!(amin_g < amax_g)) return;
  int id[3];
  float lo[3], hi[3];
#pragma unroll
  for (int d = 0; d < 3; d++) {
    id[d] = 0;
    lo[d] = -INFINITY;
    hi[d] = INFINITY;
    if (s[d]) {
      const int n = g.n[d];
      float pos = r[d] + amin_g * dir[d];
      int i = int(floorf(__fdividef(pos - g.o[d], g.d[d])));  // a guess: corrected below
      i = min(max(i, 0), n - 1);
      // Exact correction against the plane parameters: find the voxel whose
      // interval [lo, hi) contains the entry parameter.
      float l, h;
#pragma unroll 1
      for (int guard = 0; guard < 64; guard++) {
        float pa = plane_alpha_r(g.o[d], g.d[d], i, r[d], dir[d], rc[d]);
        float pb = plane_alpha_r(g.o[d], g.d[d], i + 1, r[d], dir[d], rc[d]);
        l = step[d] > 0 ? pa : pb;
        h = step[d] > 0 ? pb : pa;
        if (!(h > amin_g)) {
          i += step[d];
        } else if (l > amin_g) {
          i -= step[d];
        } else {
          break;
        }
        if (i < 0 || i >= n) {
          *bad_walk = 1;
          return;
        }
      }
      id[d] = i;
      lo[d] = l;
      hi[d] = h;
    }
  }
  const bool all3 = s[0] && s[1] && s[2];
  const int guard_max = g.n[0] + g.n[1] + g.n[2] + 8;
  // The step loop computes plane parameters exactly as plane_alpha_r did
  // for the grid's bounding planes (same operations and reciprocals), which
  // keeps every step inside the grid; a direction component outside the
  // range where plane_alpha_r uses the reciprocal goes to the general loop.
  bool in_range = true;
#pragma unroll
  for (int d = 0; d < 3; d++) in_range = in_range && fabsf(dir[d]) >= 1e-30f && fabsf(dir[d]) <= 1e30f;
  if (all3 && in_range) {
    // One axis per step, chosen with selects (no runtime array index):
    // the axis whose next plane comes first.  Planes of two axes at the same
    // parameter take two steps; the voxel between them has zero length (its
    // reference value is zero) and is dropped when the row is compacted.
    int i0 = id[0], i1 = id[1], i2 = id[2];
    float lo0 = lo[0], lo1 = lo[1], lo2 = lo[2];
    float hi0 = hi[0], hi1 = hi[1], hi2 = hi[2];
    const float y0 = rc[0], y1 = rc[1], y2 = rc[2];
    ix.begin(step);
    ix.set(i0, i1, i2);
    // Staggered start: the walk begins at a plane of the dominant axis D,
    // part/256 of the way along the ray, runs to the exit, then wraps
    // around to the entry and runs up to that plane.  No voxel straddles a
    // plane of D, so every voxel is still visited once with the same
    // lengths, while the threads of a row -- nearly parallel rays of one
    // channel -- sit on different voxels at any step instead of adding to
    // the same shared-memory accumulator at once.
    const int s0 = i0, s1 = i1, s2 = i2;
    const Index six = ix;
    const float sl0 = lo0, sl1 = lo1, sl2 = lo2, sh0 = hi0, sh1 = hi1, sh2 = hi2;
    float stop = amax_g, a_split = amax_g;
    bool wrapped = true;
    if (part > 0) {
      const float dx = fabsf(dir[0]), dy = fabsf(dir[1]), dz = fabsf(dir[2]);
      const int D = (dx >= dy) ? ((dx >= dz) ? 0 : 2) : ((dy >= dz) ? 1 : 2);
      const float oD = D == 0 ? g.o[0] : (D == 1 ? g.o[1] : g.o[2]);
      const float pD = D == 0 ? g.d[0] : (D == 1 ? g.d[1] : g.d[2]);
      const float rD = D == 0 ? r[0] : (D == 1 ? r[1] : r[2]);
      const float dD = D == 0 ? dir[0] : (D == 1 ? dir[1] : dir[2]);
      const float cD = D == 0 ? rc[0] : (D == 1 ? rc[1] : rc[2]);
      const int stD = D == 0 ? step[0] : (D == 1 ? step[1] : step[2]);
      const int nD = D == 0 ? g.n[0] : (D == 1 ? g.n[1] : g.n[2]);
      const int iD = D == 0 ? i0 : (D == 1 ? i1 : i2);
      const float hD = D == 0 ? hi0 : (D == 1 ? hi1 : hi2);
      const int span = int(__fdividef(fabsf((amax_g - amin_g) * dD), pD)) + 1;
      const int k = (part * span) >> 8;
      const int is = iD + stD * k;
      if (k > 0 && is >= 0 && is < nD) {
        const float as = plane_alpha_r(oD, pD, stD > 0 ? is : is + 1, rD, dD, cD);
        if (as > hD && as < amax_g) {
          int ni[3];
          float nl[3], nh[3];
          bool ok = true;
#pragma unroll
          for (int d = 0; d < 3; d++) {
            if (d == D) {
              ni[d] = is;
              nl[d] = as;
              nh[d] = plane_alpha_r(oD, pD, stD > 0 ? is + 1 : is, rD, dD, cD);
            } else {
              // the voxel of axis d whose interval [lo, hi) holds as
              int i = int(floorf(__fdividef(r[d] + as * dir[d] - g.o[d], g.d[d])));
              i = min(max(i, 0), g.n[d] - 1);
              float l = 0.f, h = 0.f;
              bool found = false;
#pragma unroll 1
              for (int guard = 0; guard < 64 && !found; guard++) {
                const float pa = plane_alpha_r(g.o[d], g.d[d], i, r[d], dir[d], rc[d]);
                const float pb = plane_alpha_r(g.o[d], g.d[d], i + 1, r[d], dir[d], rc[d]);
                l = step[d] > 0 ? pa : pb;
                h = step[d] > 0 ? pb : pa;
                if (!(h > as))
                  i += step[d];
                else if (l > as)
                  i -= step[d];
                else
                  found = true;
                if (i < 0 || i >= g.n[d]) break;
              }
              ok = ok && found;
              ni[d] = i;
              nl[d] = l;
              nh[d] = h;
            }
          }
          if (ok) {
            i0 = ni[0];
            i1 = ni[1];
            i2 = ni[2];
            lo0 = nl[0];
            lo1 = nl[1];
            lo2 = nl[2];
            hi0 = nh[0];
            hi1 = nh[1];
            hi2 = nh[2];
            ix.set(i0, i1, i2);
            a_split = as;
            wrapped = false;
          }
        }
      }
    }
    // Loop state per axis: the parameter of the next plane (hi) and the index
    // of the plane after it times the step direction, as a float (exact
    // small integers), so that it grows by one per step on every axis; the
    // pitch carries the direction instead (q*pd = (-q)*(-pd) exactly).  The
    // entry parameter of the current voxel is the previous step's exit
    // (prev).
    const float ps0 = step[0] > 0 ? g.d[0] : -g.d[0];
    const float ps1 = step[1] > 0 ? g.d[1] : -g.d[1];
    const float ps2 = step[2] > 0 ? g.d[2] : -g.d[2];
    float q0 = float(step[0] > 0 ? i0 + 2 : 1 - i0);
    float q1 = float(step[1] > 0 ? i1 + 2 : 1 - i1);
    float q2 = float(step[2] > 0 ? i2 + 2 : 1 - i2);
    float prev = fmaxf(lo0, fmaxf(lo1, lo2));
    const float sq0 = float(step[0] > 0 ? s0 + 2 : 1 - s0);
    const float sq1 = float(step[1] > 0 ? s1 + 2 : 1 - s1);
    const float sq2 = float(step[2] > 0 ? s2 + 2 : 1 - s2);
    const float sprev = fmaxf(sl0, fmaxf(sl1, sl2));
#pragma unroll 1
    for (int it = 0; it < guard_max; it++) {
      const float a_hi = fminf(hi0, fminf(hi1, hi2));
      // A voxel between two planes at the same parameter gets length 0; it
      // is added all the same (no branch) and dropped with the other
      // zero sums when the row is compacted.
      ix.add(RFMUL(RFSUB(a_hi, prev), len));
      // The next plane lies before the exit, so it is not the grid's last
      // plane of its axis, and the step stays inside the grid.
      if (!(a_hi < stop)) {
        if (wrapped) return;
        // the second leg: from the entry up to the split plane
        q0 = sq0;
        q1 = sq1;
        q2 = sq2;
        hi0 = sh0;
        hi1 = sh1;
        hi2 = sh2;
        ix = six;
        prev = sprev;
        stop = a_split;
        wrapped = true;
        continue;
      }
      const bool ax = hi0 == a_hi;
      const bool ay = !ax && hi1 == a_hi;
      const float q = ax ? q0 : (ay ? q1 : q2);
      const float o = OISO ? g.o[0] : (ax ? g.o[0] : (ay ? g.o[1] : g.o[2]));
      const float pd = ax ? ps0 : (ay ? ps1 : ps2);
      const float r0 = ax ? r[0] : (ay ? r[1] : r[2]);
      const float dd = ax ? dir[0] : (ay ? dir[1] : dir[2]);
      const float yy = ax ? y0 : (ay ? y1 : y2);
      const float hn = div_rcp(RFSUB(RFADD(o, RFMUL(q, pd)), r0), dd, yy);
      const float qn = RFADD(q, 1.0f);
      ix.advance(ax, ay);
      q0 = ax ? qn : q0;
      q1 = ay ? qn : q1;
      q2 = (!ax && !ay) ? qn : q2;
      hi0 = ax ? hn : hi0;
      hi1 = ay ? hn : hi1;
      hi2 = (!ax && !ay) ? hn : hi2;
      prev = a_hi;
    }
    *bad_walk = 1;
    return;
  }
#pragma unroll 1
  for (int it = 0; it < guard_max; it++) {
    float a_lo = fmaxf(lo[0], fmaxf(lo[1], lo[2]));
    float a_hi = fminf(hi[0], fminf(hi[1], hi[2]));
    if (a_lo < a_hi) {
      float L = RFMUL(RFSUB(a_hi, a_lo), len);
      if (all3) {
        emit(id[0], id[1], id[2], L);
      } else {
        int r0[3], m[3];
#pragma unroll
        for (int d = 0; d < 3; d++) {
          r0[d] = s[d] ? id[d] : 0;
          m[d] = s[d] ? 1 : g.n[d];
        }
        for (int k = k_first; k < m[0] * m[1] * m[2]; k += k_step) {
          const int a = r0[0] + k / (m[1] * m[2]), b = r0[1] + k / m[2] % m[1], c = r0[2] + k % m[2];
          if (candidate_test(g, ch, a, b, c)) emit(a, b, c, L);
        }
      }
    }
    if (!(a_hi < amax_g)) return;
#pragma unroll
    for (int d = 0; d < 3; d++) {
      if (s[d] && hi[d] == a_hi) {
        id[d] += step[d];
        if (id[d] < 0 || id[d] >= g.n[d]) return;
        lo[d] = hi[d];
        hi[d] = plane_alpha(g.o[d], g.d[d], step[d] > 0 ? id[d] + 1 : id[d], r[d], dir[d]);
      }
    }
  }
  *bad_walk = 1;
}

// Block-wide exclusive scan of one int per thread; returns the prefix and
// sets *total.  `warp_sums` holds at least 32 ints.  Ends with a barrier.
template <int T>
__device__ __forceinline__ int block_exclusive_scan(int v, int* total, int* warp_sums) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_sums[warp] = x;
  __syncthreads();
  if (warp == 0) {
    int w = (lane < T / 32) ? warp_sums[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    if (lane < T / 32) warp_sums[lane] = w;  // inclusive
  }
  __syncthreads();
  int before = (warp > 0 ? warp_sums[warp - 1] : 0) + x - v;
  *total = warp_sums[T / 32 - 1];
  __syncthreads();
  return before;
}

// Bitonic sort of (keys, vals)[0, total) by key in shared memory (npad =
// the next power of two, padded with INT_MAX), then written to the row's
// staging slot and its length to *row_nnz.  Every thread of the CTA calls it.
template <int T>
__device__ void sort_and_write(int* keys, float* vals, int total, int32_t* __restrict__ st_col,
                               float* __restrict__ st_val, size_t base, int32_t* row_nnz) {
  const int tid = threadIdx.x;
  int npad = 1;
  while (npad < total) npad <<= 1;
  for (int i = total + tid; i < npad; i += T) keys[i] = INT_MAX;
  __syncthreads();
  for (int k = 2; k <= npad; k <<= 1) {
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int t = tid; t < (npad >> 1); t += T) {
        int i = ((t & ~(j - 1)) << 1) | (t & (j - 1));
        int p = i | j;
        bool asc = (i & k) == 0;
        int ki = keys[i], kp = keys[p];
        if ((ki > kp) == asc) {
          keys[i] = kp;
          keys[p] = ki;
          float vi = vals[i];
          vals[i] = vals[p];
          vals[p] = vi;
        }
      }
      __syncthreads();
    }
  }
  for (int i = tid; i < total; i += T) {
    st_col[base + i] = keys[i];
    st_val[base + i] = vals[i];
  }
  if (tid == 0) *row_nnz = total;
}

// ---------------------------------------------------------------------------
// Slab kernel: one thread owns one slab of the grid
// ---------------------------------------------------------------------------
//
// When both crystals of a row lie on opposite sides of the grid along x or z
// (the slab axis A), every ray of the row crosses the grid in the same
// direction along A.  A thread then owns kSlabs neighbouring slabs of A (the
// voxels between two planes of A) for one of G groups of the row's rays, and
// for each of its rays finds the segments inside its slabs on its own: the
// parameters of the slabs' planes, and in each slab of the one plane of each
// other axis (u < v) that the ray can cross there.  What bounds it is
// instruction issue (no HBM traffic but the finished row, no contraction):
//
//  * no order between the slabs of a ray is needed, so there is no walk state,
//    no choice of the next axis by selects, no divergence between long and
//    short rays (31 of 32 lanes active; 25 in a walk);
//  * u and v, and two planes of A, go through the same operations as packed
//    pairs (add/mul/fma.rn.f32x2, each result correctly rounded; 7 % faster
//    than the scalar operations);
//  * a thread's sums are its own (one shared-memory column per thread), so
//    they are plain loads and stores without bank conflicts: a shared-memory
//    float atomic is a compare-and-swap loop;
//  * three slabs share the ray's loads and their inner planes.
//
// A ray costs the same in any direction, while a walk takes one step per
// crossing (75 at 0 degrees, ~110 at 45 for 70^3 voxels).  Measured against
// the walk into dense windows with shared-memory atomics that it replaces:
// 60,000 rows of 70^3 x 1000 rays 21.9 -> 12.4 ms, 12,345 rows of 100^3 x 999
// rays 9.0 -> 4.1 ms (half of those rows did not fit the dense windows).
// Main loop, ~50 issue slots per (ray, slab) and as many again for half of
// the packed operations: 2/3 of the time; ray generation, set-up and
// compaction the rest.  The ray's 112 bytes matter too: with 128 or 144 (to save
// one operation per slab) three blocks no longer share an SM, or two rays' loads
// their banks, and the kernel is 12 to 15 % slower.
//
// Exactness.  The plane parameters are computed with the operations of
// walk_ray (and of the reference), so each is the same float.  A segment of
// a voxel lies between consecutive plane parameters in their float order,
// which are monotone in the plane index; a segment exists where they
// increase strictly.  Within a slab [lo, hi] a thread takes the first plane
// of u and of v that can come after lo: the index is computed from an
// approximate coordinate lowered by eps, a bound on its rounding error, so
// that every earlier plane's float parameter is at most lo.  That plane may
// lie before lo too (its segment is then empty), and a second plane of an
// axis may lie before hi: whenever that is possible (within 2 eps) the
// thread walks its slab plane by plane instead (slab_walk, 3 % of the time:
// planes within eps, and rays steeper than one voxel per slab).

using f32x2 = unsigned long long;

__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// Two quotients a / b, each as div_rcp: nb = -b, y = RN(1 / b).
__device__ __forceinline__ f32x2 div_rcp2(f32x2 a, f32x2 nb, f32x2 y) {
  const f32x2 q = mul2(a, y);
  return fma2(fma2(q, nb, a), y, q);
}

// A ray as the slab threads read it (16-byte broadcast loads), signed by the
// ray's step directions so that plane indices grow along it (q = step * i,
// and the pitch carries the sign back: q * p == i * d exactly).
struct alignas(16) SlabRay {
  float nr0a[2];        // -start along A, twice
  float rca[2];         // RN(1/direction) along A, twice
  float nda[2];         // -direction along A, twice
  float amin, amax;     // the ray's parameter range inside the grid (0, 0 if there is none)
  float g[2];           // voxels per unit parameter along u, v
  float f[2];           // signed coordinate at parameter 0, - eps + 1/2
  float p[2];           // signed pitch along u, v
  float nr0[2];         // -start along u, v
  float rc[2];          // RN(1/direction) along u, v
  float nd[2];          // -direction along u, v
  float w[2];           // parameter from one plane to the next, less 2 eps of it
  float len;            // |end - start|
  unsigned c;           // the ray's part of the byte offset (below)
  unsigned k[2];        // byte step of a voxel step along u, v
  float nzero[2];       // -0, twice: the plane's q * p is taken as fma(q, p, -0)
                        // (the assembler contracts mul.rn.f32x2 with the add.rn.f32x2
                        // after it into one rounding, unlike the scalar pair)
};
static_assert(sizeof(SlabRay) == 112, "seven 16-byte loads");

constexpr int kSlabs = 3;               // neighbouring slabs a thread owns (odd: an even number of planes)
constexpr float kIndexMagic = 12582912.f;  // 1.5 * 2^23: adding it rounds to an integer held in the low mantissa bits
constexpr unsigned kIndexBits = 0x4B400000u;

__device__ __forceinline__ float min3(float a, float b, float c) {
  float r;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// Adds the length `d * len` to the float `off` bytes into `acc`: one rounding
// (a positive length stays positive).
__device__ __forceinline__ void slab_add(unsigned char* acc, unsigned off, float d, float len) {
  float* p = reinterpret_cast<float*>(acc + off);
  *p = __fmaf_rn(d, len, *p);
}

// The slow path: ray R's segments in one slab between the parameters a0 and
// a1 of its planes, plane by plane.
__device__ __noinline__ void slab_walk(const SlabRay* __restrict__ R, float a0, float a1, unsigned off, float ou,
                                       float ov, unsigned spare, unsigned char* acc, int* bad_walk) {
  float cur = fmaxf(a0, R->amin);
  const float hi = fminf(a1, R->amax), len = R->len;
  const float mu = RFADD(__fmaf_rn(R->g[0], cur, R->f[0]), kIndexMagic);
  const float mv = RFADD(__fmaf_rn(R->g[1], cur, R->f[1]), kIndexMagic);
  float cu = RFSUB(mu, kIndexMagic), cv = RFSUB(mv, kIndexMagic);
  auto plane = [&](int k, float c, float o) {
    return div_rcp(RFADD(RFADD(RFMUL(c, R->p[k]), o), R->nr0[k]), -R->nd[k], R->rc[k]);
  };
  float hu = plane(0, cu, ou), hv = plane(1, cv, ov);
  off += unsigned(__float_as_int(mu)) * R->k[0] + unsigned(__float_as_int(mv)) * R->k[1] + R->c;
#pragma unroll 1
  for (int guard = 0; guard < 4096; guard++) {
    const float e = min3(hu, hv, hi);
    if (e > cur) {
      slab_add(acc, min(off, spare), RFSUB(e, cur), len);
      cur = e;
    }
    if (!(e < hi)) return;
    if (hu <= hv) {
      cu = RFADD(cu, 1.0f);
      off += R->k[0];
      hu = plane(0, cu, ou);
    } else {
      cv = RFADD(cv, 1.0f);
      off += R->k[1];
      hv = plane(1, cv, ov);
    }
  }
  *bad_walk = 1;
}

// The segments of ray R inside the thread's kSlabs slabs: pl = the planes
// before and after them in the ray's order, off0 = per slab the thread's part
// of the byte offset, o2 = the origin along (u, v), spare = the byte offset of
// the thread's spare slots, which take what an offset beyond the windows would
// hold (one per segment, `step` bytes apart, so that the three loads of a slab
// can go ahead of its stores).
__device__ __forceinline__ void slab_step(const SlabRay* __restrict__ R, const f32x2 (&pl)[(kSlabs + 2) / 2],
                                          const unsigned (&off0)[kSlabs], f32x2 o2, unsigned spare, unsigned step,
                                          unsigned char* acc, int* bad_walk) {
  const ulonglong2* q = reinterpret_cast<const ulonglong2*>(R);
  const ulonglong2 q0 = q[0], q1 = q[1], q2 = q[2], q3 = q[3], q4 = q[4], q5 = q[5], q6 = q[6];
  float a[kSlabs + 2], amin, amax, len, cf;
#pragma unroll
  for (int j = 0; j < (kSlabs + 2) / 2; j++) unpack2(div_rcp2(add2(pl[j], q0.x), q1.x, q0.y), a[2 * j], a[2 * j + 1]);
  unpack2(q1.y, amin, amax);
  unpack2(q5.y, len, cf);
#pragma unroll
  for (int j = 0; j <= kSlabs; j++) a[j] = fminf(fmaxf(a[j], amin), amax);
  const unsigned c = unsigned(__float_as_int(cf));
  const uint2 k = make_uint2(unsigned(q6.x), unsigned(q6.x >> 32));
  const f32x2 magic = pack2(kIndexMagic, kIndexMagic), nmagic = pack2(-kIndexMagic, -kIndexMagic);
  bool slow[kSlabs];
  float d1[kSlabs], d2[kSlabs], d3[kSlabs];
  unsigned o1[kSlabs], o2_[kSlabs], o3[kSlabs];
#pragma unroll
  for (int j = 0; j < kSlabs; j++) {
    // hi == lo where the slab is not inside the ray's range: three empty segments
    const float lo = a[j];
    float hi = a[j + 1];
    const f32x2 m = add2(fma2(q2.x, pack2(lo, lo), q2.y), magic);
    const f32x2 qi = add2(m, nmagic);
    const f32x2 h = div_rcp2(add2(add2(fma2(qi, q3.x, q6.y), o2), q3.y), q4.y, q4.x);
    float hu, hv, wu, wv, mu, mv;
    unpack2(h, hu, hv);
    unpack2(add2(h, q5.x), wu, wv);
    unpack2(m, mu, mv);
    const unsigned off = unsigned(__float_as_int(mu)) * k.x + (unsigned(__float_as_int(mv)) * k.y + (c + off0[j]));
    slow[j] = fminf(wu, wv) < hi;
    hi = slow[j] ? lo : hi;
    const float e1 = fmaxf(min3(hu, hv, hi), lo), e2 = fminf(max3(hu, hv, lo), hi);
    d1[j] = RFSUB(e1, lo);
    d2[j] = RFSUB(e2, e1);
    d3[j] = RFSUB(hi, e2);
    o1[j] = min(off, spare);
    o2_[j] = min(off + (hu <= hv ? k.x : k.y), spare + step);
    o3[j] = min(off + k.x + k.y, spare + 2 * step);
  }
#pragma unroll
  for (int j = 0; j < kSlabs; j++) {
    float* p1 = reinterpret_cast<float*>(acc + o1[j]);
    float* p2 = reinterpret_cast<float*>(acc + o2_[j]);
    float* p3 = reinterpret_cast<float*>(acc + o3[j]);
    const float v1 = *p1, v2 = *p2, v3 = *p3;
    *p1 = __fmaf_rn(d1[j], len, v1);
    *p2 = __fmaf_rn(d2[j], len, v2);
    *p3 = __fmaf_rn(d3[j], len, v3);
  }
  bool any = slow[0];
#pragma unroll
  for (int j = 1; j < kSlabs; j++) any = any || slow[j];
  if (any) {
    float ou, ov;
    unpack2(o2, ou, ov);
#pragma unroll
    for (int j = 0; j < kSlabs; j++)
      if (slow[j]) slab_walk(R, a[j], a[j + 1], off0[j], ou, ov, spare, acc, bad_walk);
  }
}

// Fills R for the ray r of the row (slab axis A, direction sdir along it);
// false where the row is to go to the table kernel: a direction component
// that is zero or out of the reciprocal's range, or coordinates so large
// against a voxel that eps would not be small.
__device__ __forceinline__ bool slab_ray(const DGeom& g, const float r[6], int A, int sdir, int wv, unsigned stride,
                                         SlabRay* R) {
  float dir[3], rc[3];
  float amin = -INFINITY, amax = INFINITY;
  bool ok = true;
#pragma unroll
  for (int d = 0; d < 3; d++) {
    dir[d] = RFSUB(r[3 + d], r[d]);
    ok = ok && fabsf(dir[d]) >= 1e-30f && fabsf(dir[d]) <= 1e30f;
  }
  float4 q[7];
  if (ok) {
#pragma unroll
    for (int d = 0; d < 3; d++) {
      rc[d] = __frcp_rn(dir[d]);
      const float a0 = div_rcp(RFSUB(RFADD(g.o[d], RFMUL(0.f, g.d[d])), r[d]), dir[d], rc[d]);
      const float a1 = div_rcp(RFSUB(RFADD(g.o[d], RFMUL(float(g.n[d]), g.d[d])), r[d]), dir[d], rc[d]);
      amin = fmaxf(amin, fminf(a0, a1));
      amax = fminf(amax, fmaxf(a0, a1));
    }
    const float da = A == 0 ? dir[0] : dir[2], ra = A == 0 ? r[0] : r[2], rca = A == 0 ? rc[0] : rc[2];
    ok = sdir > 0 ? da > 0.f : da < 0.f;
    q[0] = make_float4(-ra, -ra, rca, rca);
    // a ray that misses the grid: all its segments are empty, at its start (where
    // the indices are small, unlike at amin)
    const bool inside = amin < amax;
    q[1] = make_float4(-da, -da, inside ? amin : 0.f, inside ? amax : 0.f);
    float G[2], F[2], P[2], X[2], RC[2], ND[2], Wd[2];
    unsigned c = 0, K[2];
#pragma unroll
    for (int k = 0; k < 2; k++) {
      // u = y, v = z for A = x; u = x, v = y for A = z
      const float o = k == 0 ? (A == 0 ? g.o[1] : g.o[0]) : (A == 0 ? g.o[2] : g.o[1]);
      const float d = k == 0 ? (A == 0 ? g.d[1] : g.d[0]) : (A == 0 ? g.d[2] : g.d[1]);
      const int n = k == 0 ? (A == 0 ? g.n[1] : g.n[0]) : (A == 0 ? g.n[2] : g.n[1]);
      const float x = k == 0 ? (A == 0 ? r[1] : r[0]) : (A == 0 ? r[2] : r[1]);
      const float dk = k == 0 ? (A == 0 ? dir[1] : dir[0]) : (A == 0 ? dir[2] : dir[1]);
      const float rk = k == 0 ? (A == 0 ? rc[1] : rc[0]) : (A == 0 ? rc[2] : rc[1]);
      const bool up = dk > 0.f;
      const float inv = __fdividef(1.0f, d);
      const float f = (up ? x - o : o - x) * inv;
      G[k] = fabsf(dk) * inv;
      // the roundings of f + a*G and of the plane parameters, in voxels: at
      // most seven of 2^-24 of each of these magnitudes
      const float eps = 4.2e-7f * (2.f * fabsf(f) + G[k] + 2.f * fabsf(o) * inv + float(n) + 2.f);
      ok = ok && eps <= 0.01f;
      F[k] = (0.5f - eps) + f;
      P[k] = up ? d : -d;
      X[k] = -x;
      RC[k] = rk;
      ND[k] = -dk;
      Wd[k] = (1.0f - 2.f * eps) * (fabsf(rk) * d);
      const unsigned step = k == 0 ? stride * unsigned(wv) : stride;
      K[k] = up ? step : 0u - step;
      // the voxel before plane q is q - 1 going up, -q going down; the
      // indices come with kIndexBits on them
      c -= kIndexBits * K[k] + (up ? step : 0u);
    }
    q[2] = make_float4(G[0], G[1], F[0], F[1]);
    q[3] = make_float4(P[0], P[1], X[0], X[1]);
    q[4] = make_float4(RC[0], RC[1], ND[0], ND[1]);
    q[5] = make_float4(Wd[0], Wd[1], norm3_exact(dir[0], dir[1], dir[2]), __uint_as_float(c));
    q[6] = make_float4(__uint_as_float(K[0]), __uint_as_float(K[1]), -0.f, -0.f);
  }
  if (!ok) {
#pragma unroll
    for (int k = 0; k < 7; k++) q[k] = make_float4(0.f, 0.f, 0.f, 0.f);  // every parameter 0: empty segments only
  }
  float4* out = reinterpret_cast<float4*>(R);
#pragma unroll
  for (int k = 0; k < 7; k++) out[k] = q[k];
  return ok;
}

// i / d for i, d < 2^16 from m = div_magic(d): exact, since the magic number
// is off by less than d in 2^32 and i * d < 2^32.
__device__ __forceinline__ unsigned div_magic(int d) { return 0xffffffffu / unsigned(d) + 1u; }
__device__ __forceinline__ int div_by(int i, int d, unsigned m) { return d == 1 ? i : int(__umulhi(unsigned(i), m)); }

// Row status the slab kernel leaves: the row is to be built with the hash
// table, or by walks into its windows, which are too large for the slab kernel.
constexpr int kRowToTable = -2, kRowToWindows = -3;

constexpr int kMaxSlabs = 256;

constexpr int kSlabThreads = 192, kSlabBlocks = 3;  // most threads, blocks per SM

// Launch shape of the slab kernel on a grid: threads per block, floats of
// the sums and of the ray staging in dynamic shared memory.
struct SlabShape {
  int threads = 0;
  int acc_floats = 0;
  int stage_floats = 0;
  int batch = 0;  // rays staged at a time
  bool large_windows = false;  // some rows' windows may not fit
  size_t smem() const { return size_t(acc_floats + stage_floats) * 4; }
};
constexpr int kMostSlots = 64, kMostStage = 8192;  // planned for: voxels of a slab's window, floats of a finished row
// The most of any grid: the kernel's limit is always set to it, so that builds of
// different grids on two threads do not set it below each other's need.
constexpr int kSlabRayFloats = int(sizeof(SlabRay) / 4);
constexpr int kSlabSmem =
    ((kSlabs * kMostSlots + 3) * kSlabThreads +
     (kSlabThreads * kSlabRayFloats > kMostStage ? kSlabThreads * kSlabRayFloats : kMostStage)) * 4;
static_assert(kSlabSmem <= 220 * 1024, "fits a block");

// A row's crystals: boxes rotated about y, four corners in (x, z), two bounds in y.
struct Crystals {
  float x[2][4], z[2][4], y[2][2];
};

// The slab axis: of x and z, the one along which the crystals lie on opposite
// sides of the grid, the channel's dominant direction first; -1 if none.  *sdir =
// the rays' direction along it.
__device__ __forceinline__ int slab_axis(const DGeom& g, const float ab[3], const Crystals& c, int* sdir) {
  *sdir = 0;
  const int first = fabsf(ab[0]) >= fabsf(ab[2]) ? 0 : 2;
  for (int k = 0; k < 2; k++) {
    const int a = k == 0 ? first : 2 - first;
    if (axis_n(g, a) > kMaxSlabs) continue;
    const float* p = a == 0 ? c.x[0] : c.z[0];
    const float* q = a == 0 ? c.x[1] : c.z[1];
    const float plo = fminf(fminf(p[0], p[1]), fminf(p[2], p[3])), phi = fmaxf(fmaxf(p[0], p[1]), fmaxf(p[2], p[3]));
    const float qlo = fminf(fminf(q[0], q[1]), fminf(q[2], q[3])), qhi = fmaxf(fmaxf(q[0], q[1]), fmaxf(q[2], q[3]));
    const float c0 = axis_o(g, a), c1 = axis_o(g, a) + float(axis_n(g, a)) * axis_d(g, a);
    const float m = 1e-6f * (1.0f + fabsf(c0) + fabsf(c1));
    if (phi + m < c0 && qlo - m > c1) *sdir = 1;
    if (qhi + m < c0 && plo - m > c1) *sdir = -1;
    if (*sdir != 0) return a;
  }
  return -1;
}

// The window of slab sl of axis A: the first voxel and the number of voxels along
// u and v that the crystals' hull reaches at the slab's two faces, with `margin`
// voxels on each side.
__device__ __forceinline__ void slab_window(const DGeom& g, const Crystals& c, int A, int sl, float margin, int* u0,
                                            int* nu, int* v0, int* nv) {
  const float* pa = A == 0 ? c.x[0] : c.z[0];
  const float* qa = A == 0 ? c.x[1] : c.z[1];
  const float* pw = A == 0 ? c.z[0] : c.x[0];
  const float* qw = A == 0 ? c.z[1] : c.x[1];
  const float c0 = axis_o(g, A) + float(sl) * axis_d(g, A), c1 = axis_o(g, A) + float(sl + 1) * axis_d(g, A);
  float wlo = INFINITY, whi = -INFINITY, tlo = INFINITY, thi = -INFINITY;
#pragma unroll 4
  for (int ij = 0; ij < 16; ij++) {
    const int i = ij >> 2, j = ij & 3;
    const float inv = __fdividef(1.0f, qa[j] - pa[i]);
    const float t0 = (c0 - pa[i]) * inv, t1 = (c1 - pa[i]) * inv;
    const float w0 = pw[i] + t0 * (qw[j] - pw[i]), w1 = pw[i] + t1 * (qw[j] - pw[i]);
    wlo = fminf(wlo, fminf(w0, w1));
    whi = fmaxf(whi, fmaxf(w0, w1));
    tlo = fminf(tlo, fminf(t0, t1));
    thi = fmaxf(thi, fmaxf(t0, t1));
  }
  const float dy0 = c.y[1][0] - c.y[0][0], dy1 = c.y[1][1] - c.y[0][1];
  const float ylo = c.y[0][0] + fminf(tlo * dy0, thi * dy0);
  const float yhi = c.y[0][1] + fmaxf(tlo * dy1, thi * dy1);
  auto range = [&](int ax, float lo, float hi, int* first) {
    const int n = axis_n(g, ax);
    const float inv = __fdividef(1.0f, axis_d(g, ax));
    const int a = int(floorf((lo - axis_o(g, ax)) * inv - margin));
    const int b = int(floorf((hi - axis_o(g, ax)) * inv + margin));
    const int l = min(max(a, 0), n - 1);
    *first = l;
    return max(min(max(b, 0), n - 1) - l, 0) + 1;
  };
  int y0, w0;
  const int ny = range(1, ylo, yhi, &y0);
  const int nw = range(A == 0 ? 2 : 0, wlo, whi, &w0);
  *u0 = A == 0 ? y0 : w0;
  *nu = A == 0 ? ny : nw;
  *v0 = A == 0 ? w0 : y0;
  *nv = A == 0 ? nw : ny;
}

// One block per row.  The sums of the row's windows (per slab of A the
// voxels [ulo, ulo+wu) x [vlo, vlo+wv) that the crystals' hull can reach)
// are kept per thread: slot w of thread t at acc[w * S + t], S = the threads
// in use rounded up to a warp.  A row with more slots per slab than fit runs
// with fewer groups of rays; one whose slots do not fit one group gets row_nnz =
// kRowToWindows, one that has no slab axis or one of whose rays needs the general
// walk kRowToTable.
//
// The windows hold every voxel a ray visits: a ray lies in the convex hull
// of the two crystals, the windows are the hull's extents at the slab's two
// faces taken over all pairs of corners, with 0.02 voxel of margin against
// rounding (the rays' eps is at most 0.01 voxel; tests/test_slab_hull.py holds the
// rule against the exact walk).  The kernel rests on this: an offset that left its
// window sideways would be another voxel's slot of the thread.  What is looked at
// besides is no proof of it, but keeps the accesses in bounds and finds a gross
// mistake: an offset beyond the row's slots becomes the thread's spare slot (one per
// segment), and a sum there, or one that decodes outside the grid, sends the row to the
// table.  (Spare slots that no other segment's offset can reach take a
// compare and a select per offset: 60,000 rows of 70^3 x 1000 rays 13.25 ms
// instead of 12.65.)
__global__ void __launch_bounds__(kSlabThreads, kSlabBlocks)
    sm_slab_kernel(DGeom g, const float2* __restrict__ sincos, const int32_t* __restrict__ cnl_ids, int64_t row0,
                   int nrays, uint32_t seed, int H, int acc_floats, int stage_floats, int batch,
                   int32_t* __restrict__ st_col,
                   float* __restrict__ st_val, int32_t* __restrict__ row_nnz, int32_t* __restrict__ flags,
                   int32_t* __restrict__ reasons) {
  extern __shared__ __align__(16) unsigned char smem[];
  float* acc = reinterpret_cast<float*>(smem);
  float* stage = acc + acc_floats;  // the rays of a batch, then the row's sums
  SlabRay* rays = reinterpret_cast<SlabRay*>(stage);
  __shared__ Channel ch;
  __shared__ int bad_walk, to_table, outside, win_u, win_v;
  __shared__ Crystals cr;
  __shared__ int warp_sums[32];
  __shared__ short ulo[kMaxSlabs], vlo[kMaxSlabs];
  __shared__ int zbox[4];

  const int tid = threadIdx.x, T = blockDim.x, lane = tid & 31, warp = tid >> 5, NW = T >> 5;
  const int cnl = cnl_ids[row0 + blockIdx.x];
  if (cnl < 0 || cnl >= num_channels(g)) {
    if (tid == 0) {
      row_nnz[blockIdx.x] = -1;
      atomicOr(flags, 4);
    }
    return;
  }
  auto table = [&](int why) {  // called by every thread, or by one
    if (tid == 0) {
      row_nnz[blockIdx.x] = why == 1 ? kRowToWindows : kRowToTable;
      if (reasons && why != 1) atomicAdd(reasons + why, 1);
    }
  };
  if (warp == 0) {
    // The crystals are boxes rotated about y: four corners in (x, z), two bounds
    // in y.  Lanes 0-3 take the first crystal's corners, 4-7 the second's, each
    // with the crystal's transform (channel_setup does the same one after the
    // other in one thread).
    const ChannelIds id = channel_split(g, cnl);
    const float2 sc = sincos[id.ida];
    const int b = (lane >> 2) & 1, c = lane & 3;
    float m[12], p[3], mid[3];
    trafo_matrix(m, b == 0 ? g.pos0x : g.pos1x, b == 0 ? id.id0z : id.id1z, b == 0 ? id.id0y : id.id1y,
                 b == 0 ? g.n0y : g.n1y, b == 0 ? g.n0z : g.n1z, g.segx, g.segy, g.segz, sc.x, sc.y);
    trafo_apply(m, float(c & 1), float(c >> 1), float(c >> 1), p);
    trafo_apply(m, 0.5f, 0.5f, 0.5f, mid);
    if (lane < 8) {
      cr.x[b][c] = p[0];
      cr.z[b][c] = p[2];
      if ((c & 1) == 0) cr.y[b][c >> 1] = p[1];
    }
    if (lane < 8 && c == 0) {
      float* to = b == 0 ? ch.m0 : ch.m1;
#pragma unroll
      for (int k = 0; k < 12; k++) to[k] = m[k];
    }
#pragma unroll
    for (int d = 0; d < 3; d++) {
      const float other = __shfl_sync(0xffffffffu, mid[d], 4);
      if (lane == 0) {
        ch.c0[d] = mid[d];
        ch.ab[d] = RFSUB(other, mid[d]);
      }
    }
    if (lane == 0) {
      bad_walk = 0;
      to_table = 0;
      outside = 0;
      win_u = 0;
      win_v = 0;
      zbox[0] = zbox[2] = INT_MAX;
      zbox[1] = zbox[3] = INT_MIN;
    }
  } else {
    // the other warps clear the sums meanwhile
    float4* a4 = reinterpret_cast<float4*>(acc);
    for (int i = tid - 32; i < acc_floats / 4; i += T - 32) a4[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  __syncthreads();
  if (tid == T - 1) {  // what the cylinder test needs, for later
    ch.abs_ab = norm3_exact(ch.ab[0], ch.ab[1], ch.ab[2]);
    ch.radius = RFMUL(0.5f, RFADD(norm3_exact(g.d[0], g.d[1], g.d[2]), norm3_exact(g.segx, g.segy, g.segz)));
  }
  int sdir;
  const int A = slab_axis(g, ch.ab, cr, &sdir);
  if (A < 0) {
    table(0);
    return;
  }
  const int na = axis_n(g, A);
  if (na > T * kSlabs) {
    table(1);
    return;
  }
  const int iu_ax = A == 0 ? 1 : 0, iv_ax = A == 0 ? 2 : 1;
  {
    int wu_max = 0, wv_max = 0;
    for (int sl = tid; sl < na; sl += T) {
      int u0, nu, v0, nv;
      slab_window(g, cr, A, sl, 0.02f, &u0, &nu, &v0, &nv);
      wu_max = max(wu_max, nu);
      wv_max = max(wv_max, nv);
      ulo[sl] = short(u0);
      vlo[sl] = short(v0);
    }
    wu_max = __reduce_max_sync(0xffffffffu, wu_max);
    wv_max = __reduce_max_sync(0xffffffffu, wv_max);
    if (lane == 0 && wu_max > 0) {
      atomicMax(&win_u, wu_max);
      atomicMax(&win_v, wv_max);
    }
  }
  __syncthreads();
  // a voxel's offset and those one step on along u, v and both are four
  // different ones (slab_step loads three before it stores): wv is not 1
  const int wu = win_u, wv = max(win_v, 2), W = wu * wv;
  const int nt = (na + kSlabs - 1) / kSlabs;  // threads of a group
  int G = T / nt;
  G = min(G, batch);
  while (G > 0 && (long long)(kSlabs * W + 3) * ((G * nt + 31) & ~31) > (long long)acc_floats) G--;
  const int Wp = W | 1;  // odd: slots of neighbouring slabs fall into different banks
  if (G == 0 || (long long)na * Wp > (long long)stage_floats) {
    table(1);
    return;
  }
  const int S = (G * nt + 31) & ~31;
  const int grp = tid / nt, s0 = (tid - grp * nt) * kSlabs;

  // the thread's slabs, in the rays' order; those past the last have two
  // equal planes
  const bool works = grp < G;
  f32x2 pl[(kSlabs + 2) / 2];
  unsigned off0[kSlabs];
  {
    float p[kSlabs + 2];
    p[kSlabs + 1] = 0.f;
#pragma unroll
    for (int j = 0; j <= kSlabs; j++)
      p[j] = RFADD(axis_o(g, A), RFMUL(float(min(sdir > 0 ? s0 + j : s0 + kSlabs - j, na)), axis_d(g, A)));
#pragma unroll
    for (int j = 0; j < (kSlabs + 2) / 2; j++) pl[j] = pack2(p[2 * j], p[2 * j + 1]);
#pragma unroll
    for (int j = 0; j < kSlabs; j++) {
      const int k = sdir > 0 ? j : kSlabs - 1 - j, sl = min(s0 + k, na - 1);
      off0[j] = unsigned((k * W * S + tid) * 4) - unsigned(ulo[sl] * wv + vlo[sl]) * unsigned(S * 4);
    }
  }
  const unsigned spare = unsigned((kSlabs * W * S + (works ? tid : 0)) * 4);
  const f32x2 o2 = pack2(axis_o(g, iu_ax), axis_o(g, iv_ax));
  const int per = batch / G * G;  // as many rays for every group
  for (int base = 0; base < nrays; base += per) {
    const int cnt = min(per, nrays - base);
    __syncthreads();  // the batch before is done with
    for (int i = tid; i < cnt; i += T) {
      float r[6];
      make_ray(ch, seed, cnl, base + i, r);
      if (!slab_ray(g, r, A, sdir, wv, unsigned(S * 4), rays + i)) to_table = 1;
    }
    __syncthreads();
    if (works)
      for (int i = grp; i < cnt; i += G)
        slab_step(rays + i, pl, off0, o2, spare, unsigned(S * 4), smem, &bad_walk);
  }
  if (works)
    for (int k = 0; k < 3; k++)
      if (acc[(kSlabs * W + k) * S + tid] != 0.f) to_table = 1;
  __syncthreads();
  if (bad_walk) {
    if (tid == 0) {
      row_nnz[blockIdx.x] = -1;
      atomicOr(flags, 2);
    }
    return;
  }
  if (to_table) {
    table(2);
    return;
  }

  // The groups' sums per voxel, and the cylinder test: stage[s * Wp + w] =
  // the sum of a voxel of the row, 0 elsewhere.
  const unsigned m_wv = div_magic(wv), m_na = div_magic(na), m_wp = div_magic(Wp), m_ks = div_magic(kSlabs);
  auto voxel = [&](int s, int w, int* x, int* y, int* z) {
    const int u = div_by(w, wv, m_wv);
    const int iu = ulo[s] + u, iv = vlo[s] + (w - u * wv);
    *x = A == 0 ? s : iu;
    *y = A == 0 ? iu : iv;
    *z = A == 0 ? iv : s;
  };
  for (int i = tid; i < na * Wp; i += T) {
    const int w = div_by(i, na, m_na), s = i - w * na;
    float v = 0.f;
    if (w < W) {
      const int t = div_by(s, kSlabs, m_ks);
      const float* a = acc + ((s - t * kSlabs) * W + w) * S + t;
      for (int k = 0; k < G; k++) v += a[k * nt];
      if (v > 0.f) {
        int x, y, z;
        voxel(s, w, &x, &y, &z);
        if (x < g.n[0] && y < g.n[1] && z < g.n[2]) {
          if (!candidate_test(g, ch, x, y, z)) v = 0.f;
        } else {
          outside = 1;
        }
      }
    }
    stage[s * Wp + w] = v;
  }
  __syncthreads();
  if (outside) {
    table(3);
    return;
  }
  const float fr = float(nrays);
  const size_t out = size_t(blockIdx.x) * H;
  const int nz = g.n[2], nyz = g.n[1] * nz, n_out = na * Wp;
  if (A == 0) {
    // x slabs: slab-major, then y, z is column order; each warp takes a
    // contiguous run of slots, counts its voxels, and after a scan of the
    // counts writes them
    const int seg = ((n_out + NW - 1) / NW + 31) & ~31;
    const int b0 = min(warp * seg, n_out), b1 = min(b0 + seg, n_out);
    int cnt = 0;
    for (int b = b0 + lane; b - lane < b1; b += 32)
      cnt += __popc(__ballot_sync(0xffffffffu, b < b1 && stage[b] > 0.f));
    if (lane == 0) warp_sums[warp] = cnt;
    __syncthreads();
    int before = 0, total = 0;
    for (int k = 0; k < NW; k++) {
      before += k < warp ? warp_sums[k] : 0;
      total += warp_sums[k];
    }
    if (total > H) {
      if (tid == 0) {
        row_nnz[blockIdx.x] = -1;
        atomicOr(flags, 1);
      }
      return;
    }
    for (int b = b0 + lane; b - lane < b1; b += 32) {
      const float v = b < b1 ? stage[b] : 0.f;
      const unsigned m = __ballot_sync(0xffffffffu, v > 0.f);
      if (v > 0.f) {
        const int pos = before + __popc(m & ((1u << lane) - 1u));
        int x, y, z;
        const int s = div_by(b, Wp, m_wp);
        voxel(s, b - s * Wp, &x, &y, &z);
        st_col[out + pos] = x * nyz + y * nz + z;
        st_val[out + pos] = RFDIV(v, fr);
      }
      before += __popc(m);
    }
    if (tid == 0) row_nnz[blockIdx.x] = total;
    return;
  }
  // z slabs: column order is (x, y, z).  Per (x, y) of the box that holds
  // every slab's window, a bitmask of the z of the row's voxels; a voxel's
  // place is the number of bits of the (x, y) before its own and of the z
  // below its own.
  for (int s = tid; s < na; s += T) {
    atomicMin(&zbox[0], int(ulo[s]));
    atomicMax(&zbox[1], int(ulo[s]) + wu);
    atomicMin(&zbox[2], int(vlo[s]));
    atomicMax(&zbox[3], int(vlo[s]) + wv);
  }
  __syncthreads();
  const int x0 = zbox[0], y0 = zbox[2], wy = zbox[3] - y0;
  const int nkeys = (zbox[1] - x0) * wy, words = (nz + 31) >> 5;
  if ((long long)nkeys * (words + 1) > (long long)acc_floats) {
    table(1);
    return;
  }
  unsigned* mask = reinterpret_cast<unsigned*>(acc);   // [word][key]
  int* first = reinterpret_cast<int*>(acc) + words * nkeys;
  for (int i = tid; i < nkeys * words; i += T) mask[i] = 0u;
  __syncthreads();
  for (int i = tid; i < n_out; i += T)
    if (stage[i] > 0.f) {
      int x, y, z;
      const int s = div_by(i, Wp, m_wp);
      voxel(s, i - s * Wp, &x, &y, &z);
      atomicOr(&mask[(z >> 5) * nkeys + (x - x0) * wy + (y - y0)], 1u << (z & 31));
    }
  __syncthreads();
  int total = 0;
  {
    // exclusive scan of the keys' counts: each thread a run of keys
    const int pk = (nkeys + T - 1) / T;
    const int k0 = min(tid * pk, nkeys), k1 = min(k0 + pk, nkeys);
    int run = 0;
    for (int k = k0; k < k1; k++) {
      int c = 0;
      for (int w = 0; w < words; w++) c += __popc(mask[w * nkeys + k]);
      first[k] = c;
      run += c;
    }
    int incl = run;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    if (lane == 31) warp_sums[warp] = incl;
    __syncthreads();
    int off = incl - run;
    for (int k = 0; k < NW; k++) {
      off += k < warp ? warp_sums[k] : 0;
      total += warp_sums[k];
    }
    for (int k = k0; k < k1; k++) {
      const int c = first[k];
      first[k] = off;
      off += c;
    }
  }
  __syncthreads();
  if (total > H) {
    if (tid == 0) {
      row_nnz[blockIdx.x] = -1;
      atomicOr(flags, 1);
    }
    return;
  }
  for (int i = tid; i < n_out; i += T) {
    const float v = stage[i];
    if (v > 0.f) {
      int x, y, z;
      const int s = div_by(i, Wp, m_wp);
      voxel(s, i - s * Wp, &x, &y, &z);
      const int k = (x - x0) * wy + (y - y0), zw = z >> 5;
      int pos = first[k] + __popc(mask[zw * nkeys + k] & ((1u << (z & 31)) - 1u));
      for (int w = 0; w < zw; w++) pos += __popc(mask[w * nkeys + k]);
      st_col[out + pos] = x * nyz + y * nz + z;
      st_val[out + pos] = RFDIV(v, fr);
    }
  }
  if (tid == 0) row_nnz[blockIdx.x] = total;
}

// Blocks per SM the window and table kernels are compiled for: what their shared
// memory leaves (at H = 8192 the table kernel alone took 99 registers, two blocks:
// 4,000 rows x 300 of the caller's rays, 100^3 of 1.5 mm, 2.3 ms; so 1.75).
constexpr int rest_blocks(int H) { return H <= 2048 ? 8 : (H <= 4096 ? 4 : (H <= 8192 ? 3 : 1)); }

// Sums of a row that is walked into its windows: what leaves four blocks per SM
// their registers' share at H <= 4096, and no less than the entries take that are
// sorted in their place.
__host__ __device__ constexpr int window_floats(int H) { return H <= 4096 ? 3 * H : 2 * H; }

// Window kernel: the rows the slab kernel left for their windows' size
// (kRowToWindows).  A row's rays are walked, thread by thread, into one array of
// the windows' sums, by shared-memory atomics; a row that does not fit either, or one
// of whose rays leaves its windows, is left to the table kernel.  The windows have a
// margin of a voxel, since there is no bound eps on a ray's roundings here.  Bound by the
// walks' instructions and the atomics, as the slab kernel's forerunner was, but with no
// keys to look for: 4,000 rows x 300 rays of 70^3 voxels of 0.7 mm take 4.1 ms, with the
// table kernel 6.4; 100^3 of 1.5 mm seen by 8 mm crystals 3.5 and 5.2.
template <int H, int T, bool OISO>
__global__ void __launch_bounds__(T, rest_blocks(H))
    sm_window_kernel(DGeom g, const float2* __restrict__ sincos, const int32_t* __restrict__ cnl_ids, int64_t row0,
                     int64_t nrows, int nrays, uint32_t seed, int32_t* __restrict__ st_col,
                     float* __restrict__ st_val, int32_t* __restrict__ row_nnz, int32_t* __restrict__ flags,
                     int32_t* __restrict__ reasons) {
  extern __shared__ __align__(16) unsigned char smem[];
  float* sums = reinterpret_cast<float*>(smem);  // slots of the windows and the spare one
  __shared__ Channel ch;
  __shared__ Crystals cr;
  __shared__ int bad_walk, to_table, outside, win_u, win_v;
  __shared__ int warp_sums[32];
  __shared__ int ulo[kMaxSlabs], vlo[kMaxSlabs], base[kMaxSlabs], dk[kMaxSlabs];
  constexpr int NW = T / 32;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nz = g.n[2], nyz = g.n[1] * nz;
  for (int64_t bi = blockIdx.x; bi < nrows; bi += gridDim.x) {
    if (row_nnz[bi] != kRowToWindows) continue;
    // (called by every thread)
    auto error = [&](int flag) {
      if (tid == 0) {
        row_nnz[bi] = -1;
        atomicOr(flags, flag);
      }
    };
    auto table = [&](int why) {
      if (tid == 0) {
        row_nnz[bi] = kRowToTable;
        if (reasons) atomicAdd(reasons + why, 1);
      }
    };
    const int cnl = cnl_ids[row0 + bi];  // in range: the slab kernel has looked
    // (see sm_table_kernel)
    if (__syncthreads_or(tid == 0 && (*(volatile int32_t*)flags & 1) != 0)) break;
    if (tid == 0) {
      channel_setup(g, sincos, cnl, ch);
      bad_walk = to_table = outside = win_u = win_v = 0;
    }
    __syncthreads();
    if (tid < 8) {
      const int b = tid >> 2, c = tid & 3;
      float p[3];
      trafo_apply(b == 0 ? ch.m0 : ch.m1, float(c & 1), float(c >> 1), float(c >> 1), p);
      cr.x[b][c] = p[0];
      cr.z[b][c] = p[2];
      if ((c & 1) == 0) cr.y[b][c >> 1] = p[1];
    }
    __syncthreads();
    int sdir;
    const int A = slab_axis(g, ch.ab, cr, &sdir);
    if (A < 0) {
      table(0);
      continue;
    }
    const int na = axis_n(g, A);
    for (int sl = tid; sl < na; sl += T) {
      int u0, nu, v0, nv;
      slab_window(g, cr, A, sl, 1.0f, &u0, &nu, &v0, &nv);
      ulo[sl] = u0;
      vlo[sl] = v0;
      atomicMax(&win_u, nu);
      atomicMax(&win_v, nv);
    }
    __syncthreads();
    const int wu = win_u, wv = win_v, W = wu * wv;
    if ((long long)na * wu * wv >= (long long)window_floats(H)) continue;  // for the table kernel, which counts it
    const int nslots = na * W;
    for (int sl = tid; sl < na; sl += T) {
      auto at = [&](int k) { return k * W - ulo[k] * wv - vlo[k]; };
      const int next = sdir > 0 ? sl + 1 : sl - 1;
      base[sl] = at(sl);
      dk[sl] = next >= 0 && next < na ? at(next) - at(sl) : 0;
    }
    for (int i = tid; i <= nslots; i += T) sums[i] = 0.f;
    __syncthreads();

    auto emit = [&](int ix, int iy, int iz, float L) {
      const int s = A == 0 ? ix : iz;
      const int u = (A == 0 ? iy : ix) - ulo[s], v = (A == 0 ? iz : iy) - vlo[s];
      if (unsigned(u) < unsigned(wu) && unsigned(v) < unsigned(wv))
        atomicAdd(&sums[s * W + u * wv + v], L);
      else
        to_table = 1;
    };
    // start offsets: the thread index bit-reversed, so that neighbouring lanes
    // start far apart along the ray
    const int part = int(__brev(threadIdx.x) >> 24);
    auto walk = [&](auto index) {
      for (int ray = tid; ray < nrays; ray += T) {
        float r[6];
        make_ray(ch, seed, cnl, ray, r);
        const float da = A == 0 ? RFSUB(r[3], r[0]) : RFSUB(r[5], r[2]);
        // (the voxels of a ray parallel to an axis's planes: the table kernel's threads share them)
        if (!(sdir > 0 ? da > 0.f : da < 0.f) || r[0] == r[3] || r[1] == r[4] || r[2] == r[5]) {
          to_table = 1;
          break;
        }
        walk_ray<OISO>(g, ch, r, part, emit, index, &bad_walk, 0, 1);
      }
    };
    if (A == 0)
      walk(WindowIndex<0>{sums, base, dk, wv, nslots});
    else
      walk(WindowIndex<2>{sums, base, dk, wv, nslots});
    __syncthreads();
    if (bad_walk) {
      error(2);
      continue;
    }
    if (to_table || sums[nslots] != 0.f) {
      table(2);
      continue;
    }

    // each warp takes a run of slots: count those that are voxels of the row, clear
    // the others, and after a scan of the counts write them
    const int seg = ((nslots + NW - 1) / NW + 31) & ~31;
    const int b0 = min(warp * seg, nslots), b1 = min(b0 + seg, nslots);
    auto voxel = [&](int slot, int* x, int* y, int* z) {
      const int s = slot / W, u = (slot - s * W) / wv;
      const int iu = ulo[s] + u, iv = vlo[s] + (slot - s * W - u * wv);
      *x = A == 0 ? s : iu;
      *y = A == 0 ? iu : iv;
      *z = A == 0 ? iv : s;
    };
    int cnt = 0;
    for (int b = b0 + lane; b - lane < b1; b += 32) {
      bool keep = false;
      if (b < b1 && sums[b] > 0.f) {
        int x, y, z;
        voxel(b, &x, &y, &z);
        if (x < g.n[0] && y < g.n[1] && z < g.n[2])
          keep = candidate_test(g, ch, x, y, z);
        else
          outside = 1;
        if (!keep) sums[b] = 0.f;
      }
      cnt += __popc(__ballot_sync(0xffffffffu, keep));
    }
    if (lane == 0) warp_sums[warp] = cnt;
    __syncthreads();
    if (outside) {
      table(3);
      continue;
    }
    int before = 0, total = 0;
    for (int k = 0; k < NW; k++) {
      before += k < warp ? warp_sums[k] : 0;
      total += warp_sums[k];
    }
    if (total > H) {
      error(1);
      continue;
    }
    const float fr = float(nrays);
    const size_t out = size_t(bi) * H;
    for (int b = b0 + lane; b - lane < b1; b += 32) {
      const bool keep = b < b1 && sums[b] > 0.f;
      const unsigned m = __ballot_sync(0xffffffffu, keep);
      if (keep) {
        const int pos = before + __popc(m & ((1u << lane) - 1u));
        int x, y, z;
        voxel(b, &x, &y, &z);
        st_col[out + pos] = x * nyz + y * nz + z;
        st_val[out + pos] = RFDIV(sums[b], fr);
      }
      before += __popc(m);
    }
    if (A == 0) {  // slab by slab, then y, z: column order
      if (tid == 0) row_nnz[bi] = total;
      continue;
    }
    int* keys = reinterpret_cast<int*>(smem);
    float* vals = reinterpret_cast<float*>(keys + H);
    __syncthreads();  // the sums are done with, the entries written
    for (int i = tid; i < total; i += T) {
      keys[i] = st_col[out + i];
      vals[i] = st_val[out + i];
    }
    __syncthreads();
    sort_and_write<T>(keys, vals, total, st_col, st_val, out, row_nnz + bi);
  }
}

// Table kernel: its rays (generated, or given in `rays`) summed per voxel in
// an open-addressing hash table of H keys in shared memory, then the voxels
// with a positive sum that pass the cylinder test sorted into column order.
// Each CTA takes rows blockIdx.x, blockIdx.x + gridDim.x, ... of the nrows.
// With only_flagged it builds only the rows the other kernels left and leaves
// the others alone (launched then with a small grid: most workloads leave none,
// and the blocks only read the row states).
template <int H, int T, bool OISO>
__global__ void __launch_bounds__(T, rest_blocks(H)) sm_table_kernel(DGeom g, const float2* __restrict__ sincos,
                                                     const int32_t* __restrict__ cnl_ids, int64_t row0, int64_t nrows,
                                                     int nrays, uint32_t seed, const float* __restrict__ rays,
                                                     int32_t* __restrict__ st_col, float* __restrict__ st_val,
                                                     int32_t* __restrict__ row_nnz, int32_t* __restrict__ flags,
                                                     int32_t* __restrict__ reasons, int only_flagged) {
  extern __shared__ __align__(16) unsigned char smem[];
  int* keys = reinterpret_cast<int*>(smem);
  float* vals = reinterpret_cast<float*>(smem + H * sizeof(int));
  __shared__ Channel ch;
  __shared__ int overflow, bad_walk, n_parallel;
  __shared__ int warp_sums[32];
  // rays parallel to the planes of an axis: all candidates along that axis
  // get their lengths, which the block's threads share (one thread alone
  // takes 2-4 ms for one such ray, and a build of 20,000 rows meets about one)
  constexpr int kMaxParallel = 256;
  __shared__ int parallel[kMaxParallel];

  const int tid = threadIdx.x;
  const int nyz = g.n[1] * g.n[2];
  const int nz = g.n[2];
  for (int64_t bi = blockIdx.x; bi < nrows; bi += gridDim.x) {
    const int state = only_flagged ? row_nnz[bi] : kRowToTable;
    if (state > kRowToTable) continue;
    const int64_t li = row0 + bi;
    const int cnl = cnl_ids[li];
    if (cnl < 0 || cnl >= num_channels(g)) {
      if (tid == 0) {
        row_nnz[bi] = -1;
        atomicOr(flags, 4);
      }
      continue;
    }
    // the previous row's use of the shared memory is over; once a row has
    // overflowed, its whole chunk is built again a level up
    if (__syncthreads_or(tid == 0 && (*(volatile int32_t*)flags & 1) != 0)) break;
    if (tid == 0) {
      channel_setup(g, sincos, cnl, ch);
      overflow = 0;
      bad_walk = 0;
      n_parallel = 0;
      if (reasons && state == kRowToWindows) atomicAdd(reasons + 1, 1);
    }
    for (int i = tid; i < H; i += T) {
      keys[i] = -1;
      vals[i] = 0.f;
    }
    __syncthreads();
    {
      RowTable<H> table{keys, vals, &overflow};
      KeyIndex<H> kix{&table, nyz, nz};
      auto emit = [&](int ix, int iy, int iz, float L) { table.add(ix * nyz + iy * nz + iz, L); };
      const int part = int(__brev(threadIdx.x) >> 24);
      auto ray_ends = [&](int ray, float r[6]) {
        if (rays) {
          const float* src = rays + (li * int64_t(nrays) + ray) * 6;
#pragma unroll
          for (int k = 0; k < 6; k++) r[k] = src[k];
        } else {
          make_ray(ch, seed, cnl, ray, r);
        }
      };
#pragma unroll 1
      for (int shared = 0; shared < 2; shared++) {
        const int count = shared ? min(n_parallel, kMaxParallel) : nrays;
#pragma unroll 1
        for (int i = shared ? 0 : tid; i < count; i += shared ? 1 : T) {
          float r[6];
          ray_ends(shared ? parallel[i] : i, r);
          if (!shared && (r[0] == r[3] || r[1] == r[4] || r[2] == r[5])) {
            const int at = atomicAdd(&n_parallel, 1);
            if (at < kMaxParallel) {
              parallel[at] = i;
              continue;
            }
          }
          walk_ray<OISO>(g, ch, r, shared ? 0 : part, emit, kix, &bad_walk, shared ? tid : 0, shared ? T : 1);
        }
        __syncthreads();
      }
    }
    if (overflow || bad_walk) {
      if (tid == 0) {
        row_nnz[bi] = -1;
        atomicOr(flags, overflow ? 1 : 2);
      }
      continue;
    }
    // Compaction: keep voxels with a positive sum that pass the cylinder test.
    const float fr = float(nrays);
    constexpr int PER = H / T;
    int kr[PER];
    float vr[PER];
    int cnt = 0;
#pragma unroll
    for (int j = 0; j < PER; j++) {
      int slot = j * T + tid;
      int key = keys[slot];
      float v = vals[slot];
      bool ok = key >= 0 && v > 0.f;
      if (ok) {
        int ix = key / nyz;
        int rem = key - ix * nyz;
        int iy = rem / nz;
        int iz = rem - iy * nz;
        ok = candidate_test(g, ch, ix, iy, iz);
      }
      kr[j] = ok ? key : -1;
      vr[j] = ok ? RFDIV(v, fr) : 0.f;
      cnt += ok ? 1 : 0;
    }
    int total = 0;
    int pos = block_exclusive_scan<T>(cnt, &total, warp_sums);
#pragma unroll
    for (int j = 0; j < PER; j++) {
      if (kr[j] >= 0) {
        keys[pos] = kr[j];
        vals[pos] = vr[j];
        pos++;
      }
    }
    sort_and_write<T>(keys, vals, total, st_col, st_val, size_t(bi) * H, row_nnz + bi);
  }
}

struct Level {
  int H, T;
};
constexpr Level kLevels[] = {{2048, 128}, {4096, 256}, {8192, 256}, {16384, 512}};
constexpr int kNumLevels = 4;

// Threads and shared memory of the slab kernel on a grid.  192 threads and
// three blocks per SM for 2 mm voxels: the sums, kSlabs * W slots per thread,
// are what fills shared memory.  W is the window of the 4x4x20 mm crystals
// seen from any angle at the grid's pitch (16-24 slots for 75 % of the
// channels at 2 mm, 20-30 at 1.5 mm); a row with a larger one runs with fewer
// groups.  60,000 rows of 70^3 x 1000 rays / 12,345 of 100^3 x 999: 13.45 /
// 4.76 ms; with 96 threads 13.9 / 6.4, 256: 15.1 / 4.8, 288: 15.2 / 5.9; with
// room for four blocks (W = 16-18) 14.5-16.4 / 6.2-6.9, with two slabs per
// thread 15.0 / 4.8, with one 17.3 / 5.9.  With few rays a row's set-up and
// compaction are most of it, and more, smaller blocks overlap them: 142,805 rows
// of 40^3 x 100 rays 5.0 ms with 192 threads, 4.55 with 128 (at 300 rays 1.90 and
// 1.82 ms for 30,000 rows, at 1000 rays even or slower).
SlabShape slab_shape(const DGeom& g, int nrays) {
  SlabShape sh;
  const int most = nrays <= 256 ? 128 : kSlabThreads;
  // the most threads whose groups leave few of them idle
  double best = 0.0;
  for (int T = most; T >= 128; T -= 32) {
    double used = 0.0;
    for (int a = 0; a < 3; a += 2) {
      const int nt = (g.n[a] + kSlabs - 1) / kSlabs;
      if (g.n[a] <= kMaxSlabs && nt <= T) used += double(T / nt * nt) / T;
    }
    if (sh.threads == 0 || used > 1.1 * best) {
      best = used;
      sh.threads = T;
    }
  }
  const double wy = g.segy / g.d[1] + 2.1, wh = 1.5 * g.segz / std::min(g.d[0], g.d[2]) + 2.1;
  const int W = int(std::min(std::ceil(wy * wh), double(kMostSlots)));
  sh.acc_floats = (kSlabs * W + 3) * sh.threads;
  sh.batch = most;
  sh.stage_floats = std::max(sh.batch * kSlabRayFloats, std::min(50 * std::max(g.n[0], g.n[2]), kMostStage));
  // The largest windows are up to 1.7 times wy * wh (100^3 of 1.5 mm: no row of 49
  // slots and more of 29).  Where they surely fit, the window kernel's launch is
  // saved (2 us); a row that does not fit all the same takes the hash table.
  for (int a = 0; a < 3; a += 2) {
    const int nt = (g.n[a] + kSlabs - 1) / kSlabs, S = (nt + 31) & ~31;
    const double fit = std::min(double(sh.stage_floats) / g.n[a], (double(sh.acc_floats) / S - 3) / kSlabs);
    sh.large_windows = sh.large_windows || 1.7 * wy * wh > fit;
  }
  return sh;
}

template <int H, int T>
cudaError_t launch_level(const DGeom& g, const float2* d_sincos, const int32_t* d_cnl, int64_t row0, int64_t nrows,
                         int nrays, uint32_t seed, const float* d_rays, int32_t* st_col, float* st_val,
                         int32_t* row_nnz, int32_t* d_flags, int32_t* d_reasons, int parts, cudaStream_t s) {
  // A grid with the same origin on every axis (the usual centred cube) lets
  // the walk's step skip selecting the origin.
  const bool oiso = g.o[0] == g.o[1] && g.o[1] == g.o[2];
  auto table = oiso ? sm_table_kernel<H, T, true> : sm_table_kernel<H, T, false>;
  const size_t table_smem = size_t(H) * 8;
  cudaError_t e = cudaFuncSetAttribute(table, cudaFuncAttributeMaxDynamicSharedMemorySize, int(table_smem));
  if (e != cudaSuccess) return e;
  if (d_rays) {
    // caller-supplied rays: the table builds every row, one CTA each
    table<<<unsigned(nrows), T, table_smem, s>>>(g, d_sincos, d_cnl, row0, nrows, nrays, seed, d_rays, st_col,
                                                  st_val, row_nnz, d_flags, nullptr, 0);
    note_launches(1);
    return cudaGetLastError();
  }
  const SlabShape sh = slab_shape(g, nrays);
  if (parts & 1) {
    e = cudaFuncSetAttribute(sm_slab_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSlabSmem);
    if (e != cudaSuccess) return e;
    sm_slab_kernel<<<unsigned(nrows), unsigned(sh.threads), sh.smem(), s>>>(
        g, d_sincos, d_cnl, row0, nrays, seed, H, sh.acc_floats, sh.stage_floats, sh.batch, st_col, st_val, row_nnz,
        d_flags, d_reasons);
    note_launches(1);
  }
  if (parts & 2) {
    // the rows the slab kernel left (a few per million on the centred-cube
    // workloads), four blocks per SM looking through the row states
    const int64_t tb = std::min<int64_t>(nrows, 148 * 4);
    if (sh.large_windows) {
      auto window = oiso ? sm_window_kernel<H, T, true> : sm_window_kernel<H, T, false>;
      const size_t smem = size_t(window_floats(H)) * 4;
      static_assert(window_floats(H) >= 2 * H, "holds the entries to be sorted");
      e = cudaFuncSetAttribute(window, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
      if (e != cudaSuccess) return e;
      window<<<unsigned(tb), T, smem, s>>>(g, d_sincos, d_cnl, row0, nrows, nrays, seed, st_col, st_val, row_nnz,
                                           d_flags, d_reasons);
      note_launches(1);
    }
    table<<<unsigned(tb), T, table_smem, s>>>(g, d_sincos, d_cnl, row0, nrows, nrays, seed, nullptr, st_col,
                                              st_val, row_nnz, d_flags, d_reasons, 1);
    note_launches(1);
  }
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// CSR placement
// ---------------------------------------------------------------------------

template <typename TCount>
__global__ void __launch_bounds__(1024) rows_scan_kernel(const TCount* __restrict__ row_nnz, int64_t n,
                                                         int64_t* __restrict__ row_ptr, int64_t* __restrict__ d_base) {
  __shared__ long long warp_sums[32];
  __shared__ long long carry;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) carry = *d_base;
  __syncthreads();
  constexpr int U = 8;  // rows of a thread
  for (int64_t t0 = 0; t0 < n; t0 += 1024 * U) {
    const int64_t i = t0 + int64_t(tid) * U;
    long long c[U];
    long long v = 0;
#pragma unroll
    for (int u = 0; u < U; u++) {
      c[u] = i + u < n ? (long long)row_nnz[i + u] : 0;
      c[u] = c[u] < 0 ? 0 : c[u];
      v += c[u];
    }
    long long x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      long long y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    if (warp == 0) {
      long long w = warp_sums[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        long long y = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += y;
      }
      warp_sums[lane] = w;
    }
    __syncthreads();
    long long excl = carry + (warp > 0 ? warp_sums[warp - 1] : 0) + x - v;
#pragma unroll
    for (int u = 0; u < U; u++) {
      if (i + u < n) row_ptr[i + u] = excl;
      excl += c[u];
    }
    __syncthreads();
    if (tid == 0) carry += warp_sums[31];
    __syncthreads();
  }
  if (tid == 0) {
    row_ptr[n] = carry;
    *d_base = carry;
  }
}

__global__ void rows_gather_kernel(const int32_t* __restrict__ st_col, const float* __restrict__ st_val, int slot_cap,
                                   const int64_t* __restrict__ row_ptr, int64_t nrows, int64_t capacity,
                                   int32_t* __restrict__ col, float* __restrict__ val) {
  const int lane = threadIdx.x & 31;
  const int64_t w = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = (int64_t(gridDim.x) * blockDim.x) >> 5;
  for (int64_t r = w; r < nrows; r += nw) {
    const int64_t b = row_ptr[r], e = row_ptr[r + 1];
    const size_t src = size_t(r) * slot_cap;
    for (int64_t k = lane; k < e - b; k += 32) {
      if (b + k < capacity) {
        col[b + k] = st_col[src + k];
        val[b + k] = st_val[src + k];
      }
    }
  }
}

// For candidate k of row r (written by the workqueue fill in ascending
// voxel order), the value from the zero-free staged row, or 0.
__global__ void expand_kernel(const int32_t* __restrict__ st_col, const float* __restrict__ st_val, int slot_cap,
                              const int32_t* __restrict__ row_nnz, const int64_t* __restrict__ cand_ptr,
                              int64_t nrows, const int32_t* __restrict__ cand_vxl, float* __restrict__ out_val) {
  const int lane = threadIdx.x & 31;
  const int64_t w = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = (int64_t(gridDim.x) * blockDim.x) >> 5;
  for (int64_t r = w; r < nrows; r += nw) {
    const int64_t b = cand_ptr[r], e = cand_ptr[r + 1];
    const int32_t* rc = st_col + size_t(r) * slot_cap;
    const float* rv = st_val + size_t(r) * slot_cap;
    const int n = row_nnz[r];
    for (int64_t k = b + lane; k < e; k += 32) {
      int v = cand_vxl[k];
      int lo = 0, hi = n;
      while (lo < hi) {
        int mid = (lo + hi) >> 1;
        if (rc[mid] < v) lo = mid + 1;
        else hi = mid;
      }
      out_val[k] = (lo < n && rc[lo] == v) ? rv[lo] : 0.f;
    }
  }
}

__global__ void rays_kernel(DGeom g, const float2* __restrict__ sincos, const int32_t* __restrict__ cnl_ids,
                            int nrays, uint32_t seed, float* __restrict__ out) {
  __shared__ Channel ch;
  const int64_t li = blockIdx.x;
  const int cnl = cnl_ids[li];
  if (cnl < 0 || cnl >= num_channels(g)) {
    for (int64_t k = threadIdx.x; k < int64_t(nrays) * 6; k += blockDim.x) out[li * int64_t(nrays) * 6 + k] = NAN;
    return;
  }
  if (threadIdx.x == 0) channel_setup(g, sincos, cnl, ch);
  __syncthreads();
  for (int r = threadIdx.x; r < nrays; r += blockDim.x) {
    float v[6];
    make_ray(ch, seed, cnl, r, v);
    float* dst = out + (li * int64_t(nrays) + r) * 6;
#pragma unroll
    for (int k = 0; k < 6; k++) dst[k] = v[k];
  }
}

// ---------------------------------------------------------------------------
// Candidate search: one CTA per list entry.  The voxel rows (along z) that the
// cylinder can reach are flattened over the slabs; a thread takes a row, most of
// whose candidates follow from the row's intervals (row_cells), and tests the one
// or two voxels at each end that do not.  The fill lists the rows' voxels in
// order through shared memory.  Bound by the rows' arithmetic and, in the fill,
// by the 8 bytes per candidate.  (Testing every voxel of intervals widened by two
// voxels, 256 at a time with block scans per slab, took 0.61 ms a pass for 3,001
// channels of 70^3, 27M candidates; a whole call 1.30 ms, now 0.24.)
// ---------------------------------------------------------------------------

constexpr int kWqThreads = 128;
constexpr int kWqStage = 4096;  // candidates of a step listed through shared memory

template <bool FILL>
__global__ void __launch_bounds__(kWqThreads) wq_kernel(DGeom g, const float2* __restrict__ sincos,
                                                        const int32_t* __restrict__ list, int64_t li0,
                                                        int64_t start_vxl, int64_t* __restrict__ counts,
                                                        const int64_t* __restrict__ offsets, int64_t max_out,
                                                        int32_t* __restrict__ out_cnl, int32_t* __restrict__ out_vxl,
                                                        int32_t* __restrict__ flags) {
  constexpr int T = kWqThreads;
  __shared__ Channel ch;
  __shared__ int first_y[T], pre[T + 1];
  __shared__ int warp_sums[32];
  __shared__ int32_t stage[FILL ? kWqStage : 1];
  const int tid = threadIdx.x;
  const int cnl = list[li0 + blockIdx.x];
  if (cnl < 0 || cnl >= num_channels(g)) {
    if (tid == 0) {
      if (!FILL) counts[blockIdx.x] = 0;
      if (flags) atomicOr(flags, 4);
    }
    return;
  }
  const int64_t out0 = FILL ? offsets[blockIdx.x] : 0;
  if (FILL && out0 >= max_out) return;
  const int nx = g.n[0], ny = g.n[1], nz = g.n[2];
  const int64_t nyz = int64_t(ny) * nz;
  const int64_t start = (blockIdx.x == 0) ? start_vxl : 0;
  const int sx = int(start / nyz);
  const int sy = int((start % nyz) / nz);
  const int sz = int(start % nz);
  if (tid == 0) channel_setup(g, sincos, cnl, ch);
  __syncthreads();
  const CylinderRows cyl = cylinder_rows(ch);

  int64_t count = 0;  // FILL: candidates listed; else the thread's own
  for (int x0 = sx; x0 < nx; x0 += T) {
    int y0 = 0, y1 = -1;
    if (x0 + tid < nx && !slab_rows(g, ch, cyl, x0 + tid, &y0, &y1)) y1 = y0 - 1;
    int nrows;
    const int before = block_exclusive_scan<T>(max(y1 - y0 + 1, 0), &nrows, warp_sums);
    first_y[tid] = y0;
    pre[tid] = before;
    if (tid == 0) pre[T] = nrows;
    __syncthreads();
    for (int r0 = 0; r0 < nrows; r0 += T) {
      const int r = r0 + tid;
      int ix = 0, iy = 0, lo = 0, hi = -1, in0 = 0, in1 = -1, n = 0;
      if (r < nrows) {
        int a = 0, b = T;  // the last slab with pre <= r
        while (b - a > 1) {
          const int mid = (a + b) >> 1;
          if (pre[mid] <= r) a = mid;
          else b = mid;
        }
        ix = x0 + a;
        iy = first_y[a] + (r - pre[a]);
        if (!row_cells(g, ch, cyl, ix, iy, &lo, &hi, &in0, &in1)) hi = lo - 1;
        if (ix == sx && iy <= sy) {  // rows and voxels before the start
          lo = iy < sy ? nz : max(lo, sz);
          in0 = max(in0, lo);
        }
        n = max(in1 - in0 + 1, 0);
        for (int z = lo; z <= hi; z++) {
          if (z >= in0 && z <= in1) z = in1 + 1;
          if (z <= hi && candidate_test(g, ch, ix, iy, z)) n++;
        }
      }
      if (!FILL) {
        count += n;
        continue;
      }
      int total;
      const int at = block_exclusive_scan<T>(n, &total, warp_sums);
      const int64_t dst = out0 + count;
      const bool staged = total <= kWqStage;
      if (n > 0) {
        const int32_t v0 = int32_t(ix * nyz + int64_t(iy) * nz);
        int k = at;
        for (int z = lo; z <= hi; z++) {
          if ((z >= in0 && z <= in1) || candidate_test(g, ch, ix, iy, z)) {
            if (staged) {
              stage[k] = v0 + z;
            } else if (dst + k < max_out) {
              if (out_cnl) out_cnl[dst + k] = cnl;
              out_vxl[dst + k] = v0 + z;
            }
            k++;
          }
        }
      }
      __syncthreads();
      if (staged)
        for (int k = tid; k < total && dst + k < max_out; k += T) {
          if (out_cnl) out_cnl[dst + k] = cnl;
          out_vxl[dst + k] = stage[k];
        }
      count += total;
      __syncthreads();
      if (out0 + count >= max_out) return;
    }
    __syncthreads();
  }
  if (!FILL) {
    int total;
    block_exclusive_scan<T>(int(count), &total, warp_sums);
    if (tid == 0) counts[blockIdx.x] = total;
  }
}

}  // namespace

// ---------------------------------------------------------------------------
// Host launchers
// ---------------------------------------------------------------------------

int sm_num_levels() { return kNumLevels; }
int sm_level_capacity(int level) { return kLevels[level].H; }
int sm_level_threads(int level) { return kLevels[level].T; }

int sm_pick_level(const DGeom& g, int nrays) {
  long long span = (long long)g.n[0] + g.n[1] + g.n[2];
  if (nrays <= 128 && span <= 150) return 0;
  if (span <= 240) return 1;
  return 2;
}

cudaError_t launch_sm_rows(int level, const DGeom& g, const float2* d_sincos, const int32_t* d_cnl, int64_t row0,
                           int64_t nrows, int nrays, uint32_t seed, const float* d_rays, int32_t* st_col,
                           float* st_val, int32_t* row_nnz, int32_t* d_flags, cudaStream_t s,
                           int32_t* d_table_reasons, int parts) {
  if (nrows <= 0) return cudaSuccess;
  switch (level) {
    case 0: return launch_level<2048, 128>(g, d_sincos, d_cnl, row0, nrows, nrays, seed, d_rays, st_col, st_val, row_nnz, d_flags, d_table_reasons, parts, s);
    case 1: return launch_level<4096, 256>(g, d_sincos, d_cnl, row0, nrows, nrays, seed, d_rays, st_col, st_val, row_nnz, d_flags, d_table_reasons, parts, s);
    case 2: return launch_level<8192, 256>(g, d_sincos, d_cnl, row0, nrows, nrays, seed, d_rays, st_col, st_val, row_nnz, d_flags, d_table_reasons, parts, s);
    case 3: return launch_level<16384, 512>(g, d_sincos, d_cnl, row0, nrows, nrays, seed, d_rays, st_col, st_val, row_nnz, d_flags, d_table_reasons, parts, s);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_rows_scan(const int32_t* row_nnz, int64_t n, int64_t* row_ptr, int64_t* d_base, cudaStream_t s) {
  rows_scan_kernel<int32_t><<<1, 1024, 0, s>>>(row_nnz, n, row_ptr, d_base);
  note_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_rows_scan_i64(const int64_t* counts, int64_t n, int64_t* row_ptr, int64_t* d_base, cudaStream_t s) {
  rows_scan_kernel<int64_t><<<1, 1024, 0, s>>>(counts, n, row_ptr, d_base);
  note_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_rows_gather(const int32_t* st_col, const float* st_val, int slot_cap, const int64_t* row_ptr,
                               int64_t nrows, int64_t capacity, int32_t* col, float* val, cudaStream_t s) {
  if (nrows <= 0) return cudaSuccess;
  int64_t blocks = (nrows * 32 + 255) / 256;
  if (blocks > 148 * 64) blocks = 148 * 64;
  rows_gather_kernel<<<unsigned(blocks), 256, 0, s>>>(st_col, st_val, slot_cap, row_ptr, nrows, capacity, col, val);
  note_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_expand_candidates(const int32_t* st_col, const float* st_val, int slot_cap, const int32_t* row_nnz,
                                     const int64_t* cand_ptr, int64_t nrows, int32_t* cand_vxl, float* out_val,
                                     cudaStream_t s) {
  if (nrows <= 0) return cudaSuccess;
  int64_t blocks = (nrows * 32 + 255) / 256;
  if (blocks > 148 * 64) blocks = 148 * 64;
  expand_kernel<<<unsigned(blocks), 256, 0, s>>>(st_col, st_val, slot_cap, row_nnz, cand_ptr, nrows, cand_vxl,
                                                  out_val);
  note_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_rays(const DGeom& g, const float2* d_sincos, const int32_t* d_cnl, int64_t n, int nrays,
                        uint32_t seed, float* d_rays, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  rays_kernel<<<unsigned(n), 128, 0, s>>>(g, d_sincos, d_cnl, nrays, seed, d_rays);
  note_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_wq_count(const DGeom& g, const float2* d_sincos, const int32_t* d_list, int64_t li0, int64_t n,
                            int64_t start_vxl, int64_t* d_counts, int32_t* d_flags, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  wq_kernel<false><<<unsigned(n), kWqThreads, 0, s>>>(g, d_sincos, d_list, li0, start_vxl, d_counts, nullptr, 0,
                                                      nullptr, nullptr, d_flags);
  note_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_wq_fill(const DGeom& g, const float2* d_sincos, const int32_t* d_list, int64_t li0, int64_t n,
                           int64_t start_vxl, const int64_t* d_offsets, int64_t max_out, int32_t* d_cnl_out,
                           int32_t* d_vxl_out, int32_t* d_flags, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  wq_kernel<true><<<unsigned(n), kWqThreads, 0, s>>>(g, d_sincos, d_list, li0, start_vxl, nullptr, d_offsets,
                                                     max_out, d_cnl_out, d_vxl_out, d_flags);
  note_launches(1);
  return cudaGetLastError();
}

}  // namespace raptr
