// Device-side geometry, exact arithmetic and random numbers shared by the
// raptr_b200 kernels.
//
// Every float operation that decides the structure or the values of the
// system matrix is written with explicit round-to-nearest intrinsics
// (__fmul_rn, __fadd_rn, __fsub_rn, __fdiv_rn, __fsqrt_rn), in the order
// the reference evaluates it, so no multiply-add contraction can change a
// result: the candidate test, the crystal transforms and the per-voxel
// intersection lengths are bit-identical to the reference's float arithmetic.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "../../include/raptr_b200.h"

namespace raptr {

#define RFMUL(a, b) __fmul_rn((a), (b))
#define RFADD(a, b) __fadd_rn((a), (b))
#define RFSUB(a, b) __fsub_rn((a), (b))
#define RFDIV(a, b) __fdiv_rn((a), (b))
#define RFSQRT(a) __fsqrt_rn((a))

// Geometry as passed to kernels (by value).  Same fields as raptr_geom.
struct DGeom {
  float o[3];
  float d[3];
  int n[3];
  float pos0x, pos1x;
  int na, n0z, n0y, n1z, n1y;
  float da, segx, segy, segz;
};

inline DGeom to_dgeom(const raptr_geom& g) {
  DGeom d;
  for (int i = 0; i < 3; i++) {
    d.o[i] = g.grid_o[i];
    d.d[i] = g.grid_d[i];
    d.n[i] = g.grid_n[i];
  }
  d.pos0x = g.pos0x; d.pos1x = g.pos1x;
  d.na = g.na; d.n0z = g.n0z; d.n0y = g.n0y; d.n1z = g.n1z; d.n1y = g.n1y;
  d.da = g.da; d.segx = g.segx; d.segy = g.segy; d.segz = g.segz;
  return d;
}

__host__ __device__ inline int num_channels(const DGeom& g) { return g.na * g.n0z * g.n0y * g.n1z * g.n1y; }

// Channel id -> (ida, id0z, id0y, id1z, id1y), id1y fastest
// (src/MeasurementSetupLinIndex.hpp:82-91 and its inverse functors).
struct ChannelIds {
  int ida, id0z, id0y, id1z, id1y;
};

__host__ __device__ inline ChannelIds channel_split(const DGeom& g, int cnl) {
  ChannelIds c;
  int s1 = g.n1y, s2 = g.n1y * g.n1z, s3 = s2 * g.n0y, s4 = s3 * g.n0z;
  c.ida = cnl / s4;
  int t = cnl - c.ida * s4;
  c.id0z = t / s3;
  t -= c.id0z * s3;
  c.id0y = t / s2;
  t -= c.id0y * s2;
  c.id1z = t / s1;
  c.id1y = t - c.id1z * s1;
  return c;
}

// Per-channel state: both crystal transforms, the crystal centres, the
// centre-line direction and its length, the cylinder radius.
struct Channel {
  float m0[12];
  float m1[12];
  float c0[3];
  float ab[3];     // c1 - c0
  float abs_ab;    // |c1 - c0|
  float radius;    // 0.5*(|voxel diagonal| + |crystal diagonal|)
};

// Transform matrix of a crystal (src/MeasurementSetupTrafo2CartCoord.hpp:99-131):
// scale by the segment edges, translate into the crystal, rotate about y.
__device__ __forceinline__ void trafo_matrix(float m[12], float posx, int idz, int idy, int ny, int nz, float segx,
                                             float segy, float segz, float s, float c) {
  float pos1 = RFMUL(RFSUB(float(idy), RFMUL(0.5f, float(ny - 1))), segy);
  float pos2 = RFMUL(RFSUB(float(idz), RFMUL(0.5f, float(nz - 1))), segz);
  float hx = RFSUB(posx, RFMUL(0.5f, segx));
  float hz = RFSUB(pos2, RFMUL(0.5f, segz));
  m[0] = RFMUL(c, segx);
  m[1] = 0.f;
  m[2] = RFMUL(s, segz);
  m[3] = RFADD(RFMUL(c, hx), RFMUL(s, hz));
  m[4] = 0.f;
  m[5] = segy;
  m[6] = 0.f;
  m[7] = RFSUB(pos1, RFMUL(0.5f, segy));
  m[8] = RFMUL(-s, segx);
  m[9] = 0.f;
  m[10] = RFMUL(c, segz);
  m[11] = RFADD(RFMUL(-s, hx), RFMUL(c, hz));
}

// Matrix application (src/MeasurementSetupTrafo2CartCoord.hpp:134-147).
__device__ __forceinline__ void trafo_apply(const float* m, float u0, float u1, float u2, float out[3]) {
#pragma unroll
  for (int r = 0; r < 3; r++) {
    const float* q = m + 4 * r;
    out[r] = RFADD(RFADD(RFADD(RFMUL(q[0], u0), RFMUL(q[1], u1)), RFMUL(q[2], u2)), RFMUL(q[3], 1.0f));
  }
}

__device__ __forceinline__ float norm3_exact(float a, float b, float c) {
  return RFSQRT(RFADD(RFADD(RFMUL(a, a), RFMUL(b, b)), RFMUL(c, c)));
}

// Builds the channel state; `sincos` holds (sin, cos) per angle step,
// computed on the host with the same float expression the reference uses.
__device__ inline void channel_setup(const DGeom& g, const float2* sincos, int cnl, Channel& ch) {
  ChannelIds id = channel_split(g, cnl);
  float2 sc = sincos[id.ida];
  trafo_matrix(ch.m0, g.pos0x, id.id0z, id.id0y, g.n0y, g.n0z, g.segx, g.segy, g.segz, sc.x, sc.y);
  trafo_matrix(ch.m1, g.pos1x, id.id1z, id.id1y, g.n1y, g.n1z, g.segx, g.segy, g.segz, sc.x, sc.y);
  float c0[3], c1[3];
  trafo_apply(ch.m0, 0.5f, 0.5f, 0.5f, c0);
  trafo_apply(ch.m1, 0.5f, 0.5f, 0.5f, c1);
  for (int d = 0; d < 3; d++) {
    ch.c0[d] = c0[d];
    ch.ab[d] = RFSUB(c1[d], c0[d]);
  }
  ch.abs_ab = norm3_exact(ch.ab[0], ch.ab[1], ch.ab[2]);
  float rv = norm3_exact(g.d[0], g.d[1], g.d[2]);
  float rp = norm3_exact(g.segx, g.segy, g.segz);
  ch.radius = RFMUL(0.5f, RFADD(rv, rp));
}

// Enclosing-cylinder test of voxel (ix, iy, iz): distance of the voxel centre
// from the line through both crystal centres below the sum of radii
// (src/getSystemMatrixDeviceOnly.cu:78-117, src/distancePointLine.h:40-101).
__device__ __forceinline__ bool candidate_test(const DGeom& g, const Channel& ch, int ix, int iy, int iz) {
  float p0 = RFADD(g.o[0], RFMUL(RFADD(float(ix), 0.5f), g.d[0]));
  float p1 = RFADD(g.o[1], RFMUL(RFADD(float(iy), 0.5f), g.d[1]));
  float p2 = RFADD(g.o[2], RFMUL(RFADD(float(iz), 0.5f), g.d[2]));
  float ap0 = RFSUB(p0, ch.c0[0]), ap1 = RFSUB(p1, ch.c0[1]), ap2 = RFSUB(p2, ch.c0[2]);
  float cx = RFSUB(RFMUL(ch.ab[1], ap2), RFMUL(ch.ab[2], ap1));
  float cy = RFSUB(RFMUL(ch.ab[2], ap0), RFMUL(ch.ab[0], ap2));
  float cz = RFSUB(RFMUL(ch.ab[0], ap1), RFMUL(ch.ab[1], ap0));
  float dist = RFDIV(norm3_exact(cx, cy, cz), ch.abs_ab);
  return dist < ch.radius;
}

// The voxel rows (ix, iy, all z) of a channel's enclosing cylinder, from its
// centre line (unit direction u through c0) and squared radius.  A voxel whose
// squared distance from the line, in ordinary float arithmetic, is within
// `margin` of the radius's is decided by candidate_test; the others are settled
// by their row's intervals.  margin: 2e-3 of r2 (candidate_test itself rounds to
// 1e-5 of it) and 30 roundings of the squares that cancel in the distance.
struct CylinderRows {
  float ux, uy, uz, a2;  // a2 = ux^2 + uy^2
  float r2;
};

__device__ __forceinline__ CylinderRows cylinder_rows(const Channel& ch) {
  CylinderRows c;
  const float inv = 1.0f / ch.abs_ab;
  c.ux = ch.ab[0] * inv;
  c.uy = ch.ab[1] * inv;
  c.uz = ch.ab[2] * inv;
  c.a2 = c.ux * c.ux + c.uy * c.uy;
  c.r2 = ch.radius * ch.radius;
  return c;
}

// The rows [*y0, *y1] of slab ix that can hold candidates: a z with distance
// below R exists where |dy*ux - dx*uy| <= R*sqrt(a2).  One row of margin on
// each side.
__device__ __forceinline__ bool slab_rows(const DGeom& g, const Channel& ch, const CylinderRows& c, int ix, int* y0,
                                          int* y1) {
  *y0 = 0;
  *y1 = g.n[1] - 1;
  if (fabsf(c.ux) < 1e-3f) return true;
  const float dx = g.o[0] + (ix + 0.5f) * g.d[0] - ch.c0[0];
  const float mid = dx * c.uy / c.ux, half = 1.01f * ch.radius * sqrtf(c.a2) / fabsf(c.ux);
  const float lo = (mid - half + ch.c0[1] - g.o[1]) / g.d[1] - 0.5f, hi = (mid + half + ch.c0[1] - g.o[1]) / g.d[1] - 0.5f;
  const float e = 1.0f + 1e-5f * fabsf(mid) / g.d[1];
  *y0 = max(0, int(ceilf(fmaxf(lo - e, -1.0f))));
  *y1 = min(g.n[1] - 1, int(floorf(fminf(hi + e, float(g.n[1])))));
  return *y0 <= *y1;
}

// Row (ix, iy): its candidates lie in [*lo, *hi], and all voxels of [*in0, *in1]
// (empty where in0 > in1) are candidates.
__device__ __forceinline__ bool row_cells(const DGeom& g, const Channel& ch, const CylinderRows& c, int ix, int iy,
                                          int* lo, int* hi, int* in0, int* in1) {
  const int nz = g.n[2];
  const float dx = g.o[0] + (ix + 0.5f) * g.d[0] - ch.c0[0];
  const float dy = g.o[1] + (iy + 0.5f) * g.d[1] - ch.c0[1];
  const float q = dx * dx + dy * dy, w = dx * c.ux + dy * c.uy;
  const float margin = 2e-3f * c.r2 + 4e-6f * (q + w * w);
  const float rest = q - w * w;  // squared distance = rest + a2*dz^2 - 2*w*uz*dz
  *in0 = 0;
  *in1 = -1;
  if (c.a2 < 1e-6f) {  // along z: the squared distances of the row's voxels lie within +-s of each other
    const float z0 = g.o[2] - ch.c0[2], z1 = z0 + float(nz) * g.d[2], D = fmaxf(fabsf(z0), fabsf(z1));
    const float s = 2.f * fabsf(w) * D + c.a2 * D * D, m = margin + 4e-6f * s;
    if (rest - s > c.r2 + m) return false;
    *lo = 0;
    *hi = nz - 1;
    if (rest + s < c.r2 - m) {
      *in0 = 0;
      *in1 = nz - 1;
    }
    return true;
  }
  const float B = w * c.uz, inv = 1.0f / c.a2;
  const float outer = B * B - c.a2 * (rest - c.r2 - margin);
  if (outer < 0.f) return false;
  // z index of a distance dz from the crystal centre's z
  const float at = (ch.c0[2] - g.o[2]) / g.d[2] - 0.5f, scale = inv / g.d[2];
  const float so = sqrtf(outer), tol = 0.02f + 1e-5f * (fabsf(at) + (fabsf(B) + so) * scale);
  const float flo = fmaxf(at + (B - so) * scale - tol, -1.0f), fhi = fminf(at + (B + so) * scale + tol, float(nz));
  if (!(flo <= fhi)) return false;
  *lo = max(0, int(ceilf(flo)));
  *hi = min(nz - 1, int(floorf(fhi)));
  const float inner = B * B - c.a2 * (rest - c.r2 + margin);
  if (inner > 0.f) {
    const float si = sqrtf(inner);
    const float a = fmaxf(at + (B - si) * scale + tol, 0.0f), b = fminf(at + (B + si) * scale - tol, float(nz - 1));
    if (a <= b) {
      *in0 = int(ceilf(a));
      *in1 = int(floorf(b));
    }
  }
  return *lo <= *hi;
}

// ---------------------------------------------------------------------------
// Philox4x32-10 (Salmon, Moraes, Dror, Shaw, SC'11).  Key (seed, channel),
// counter (ray, half, 0, 0); 24 random bits -> float in (0, 1].
// ---------------------------------------------------------------------------
__host__ __device__ __forceinline__ void philox4x32_10(uint32_t c[4], uint32_t k0, uint32_t k1) {
#pragma unroll
  for (int r = 0; r < 10; r++) {
#ifdef __CUDA_ARCH__
    uint32_t hi0 = __umulhi(0xD2511F53u, c[0]), lo0 = 0xD2511F53u * c[0];
    uint32_t hi1 = __umulhi(0xCD9E8D57u, c[2]), lo1 = 0xCD9E8D57u * c[2];
#else
    uint64_t p0 = uint64_t(0xD2511F53u) * c[0], p1 = uint64_t(0xCD9E8D57u) * c[2];
    uint32_t hi0 = uint32_t(p0 >> 32), lo0 = uint32_t(p0), hi1 = uint32_t(p1 >> 32), lo1 = uint32_t(p1);
#endif
    uint32_t n0 = hi1 ^ c[1] ^ k0;
    uint32_t n2 = hi0 ^ c[3] ^ k1;
    c[0] = n0;
    c[1] = lo1;
    c[2] = n2;
    c[3] = lo0;
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
}

__host__ __device__ __forceinline__ float u01(uint32_t x) { return float((x >> 8) + 1u) * (1.0f / 16777216.0f); }

// Endpoints of ray `ray` of the channel: uniforms 0-2 into the first
// crystal, 3-5 into the second (src/RayGenerators.hpp:55-62).
__device__ __forceinline__ void make_ray(const Channel& ch, uint32_t seed, int cnl, int ray, float r[6]) {
  uint32_t a[4] = {uint32_t(ray), 0u, 0u, 0u};
  uint32_t b[4] = {uint32_t(ray), 1u, 0u, 0u};
  philox4x32_10(a, seed, uint32_t(cnl));
  philox4x32_10(b, seed, uint32_t(cnl));
  trafo_apply(ch.m0, u01(a[0]), u01(a[1]), u01(a[2]), &r[0]);
  trafo_apply(ch.m1, u01(a[3]), u01(b[0]), u01(b[1]), &r[3]);
}

// The warp's next work item: lane 0 draws it from the counter at `next`
// and broadcasts it.  Called by all 32 lanes together.  Draws from one
// address are served one after the other, ~1.5 ns each (343,000 draws of one
// short column each took 0.5 ms of a back pass that moves its bytes in 0.2),
// so an item is several rows or columns.
constexpr int kDrawWarps = 148 * 40;  // warps that draw
__device__ __forceinline__ int64_t warp_next(unsigned long long* next, int lane) {
  unsigned long long q = 0;
  if (lane == 0) q = atomicAdd(next, 1ull);
  return int64_t(__shfl_sync(0xffffffffu, q, 0));
}

// Whether the FP32 and FP16 forward passes draw their m rows over n voxels, or take them
// by a grid stride.  Below 47,360 rows (eight to a warp) the draws would take longer than
// the rows, and up to twice as many, each a draw of its own, they do where rows are
// short: 57,122 rows of 40^3 (438 entries) 73 us drawn, 51 strided; 94,000 of 70^3 (724) 131
// and 117; but of 100^3 (1535 entries) 57,122 155 and 158, 90,000 231 and 236.
inline bool rows_drawn(int64_t m, int64_t n) {
  const int64_t one = int64_t(kDrawWarps) * 8;
  return m >= 2 * one || (m >= one && n >= 600000);
}

// Rows a draw takes: 16 (one draw per row makes the forward pass of 5.14M rows
// twice as slow, one per 16 takes 7 % off the grid stride's time), fewer where
// that would leave less than eight draws to a warp (200,000 rows: 4).
__device__ __forceinline__ int draw_rows(int64_t m) {
  const int64_t c = m / (int64_t(kDrawWarps) * 8);
  return int(c < 1 ? 1 : (c > 16 ? 16 : c));
}

}  // namespace raptr
