// Binning building blocks shared by the single-job and the batched passes.
#pragma once

#include "fr_device.cuh"
#include "fr_kernels.h"

namespace frb {

// A traverse space by 16-byte loads where the caller's array allows them (it starts on a 16-byte
// boundary; a space is 7 x 16 bytes), else field by field.
__device__ __forceinline__ fr_traverse_space load_space(const fr_traverse_space *p)
{
  if (reinterpret_cast<uintptr_t>(p) & 15) return *p;
  fr_traverse_space s;
  const float4 *q = reinterpret_cast<const float4 *>(p);
  float4 *d = reinterpret_cast<float4 *>(&s);
#pragma unroll
  for (int k = 0; k < 7; ++k) d[k] = __ldg(q + k);
  return s;
}

template<typename T> __device__ __forceinline__ T pick3(int k, T a, T b, T c) { return k == 0 ? a : (k == 1 ? b : c); }

// Builds, for one space, the binning record (SpacePrep) and the insertion record (SpaceRec)
// relative to the volume centre (cx, cy, cz).  A space whose projectionIndex is outside the
// FFT payload is given direction -1, so it is never binned (never read); returns false then.
// Bound by latency -- a call has few spaces per SM: the FP64 part takes two quotients, and no
// array is indexed by the direction (13 -> 3.6 us for a thousand spaces).
__device__ __forceinline__ bool prep_space(const fr_traverse_space &s, float halfWidth, float xMin,
  float radius, int cx, int cy, int cz, int nProj, SpacePrep &p, SpaceRec &r)
{
  const int dir = s.dir;
  const int ua = dir == FR_DIR_YZ ? 1 : 0;
  const int va = dir == FR_DIR_XY ? 1 : 2;
  const int wa = dir == FR_DIR_XY ? 2 : (dir == FR_DIR_XZ ? 1 : 0);
  const int open = 1 << 30;
  for (int k = 0; k < 3; ++k) {
    p.t0[k] = s.transformInv[0][k];
    p.t2[k] = s.transformInv[2][k];
  }
  p.maxDist2 = s.maxDistanceSqr * 1.00001f + 1e-2f;
  p.halfWidth = halfWidth;
  p.xMin = xMin;
  p.lo[0] = wa == 0 ? -open : s.minX;
  p.lo[1] = wa == 1 ? -open : s.minY;
  p.lo[2] = wa == 2 ? -open : s.minZ;
  p.hi[0] = wa == 0 ? open : s.maxX;
  p.hi[1] = wa == 1 ? open : s.maxY;
  p.hi[2] = wa == 2 ? open : s.maxZ;
  const bool bad = s.projectionIndex < 0 || s.projectionIndex >= nProj;
  p.dir = bad ? -1 : dir;  // -1 matches no direction segment

  const int far = 1 << 24;  // floats hold every integer up to here
  r.lo0 = float(min(max(pick3(ua, s.minX, s.minY, s.minZ), -far), far));
  r.hi0 = float(min(max(pick3(ua, s.maxX, s.maxY, s.maxZ), -far), far));
  r.lo1 = float(min(max(pick3(va, s.minX, s.minY, s.minZ), -far), far));
  r.hi1 = float(min(max(pick3(va, s.maxX, s.maxY, s.maxZ), -far), far));
  for (int k = 0; k < 9; ++k) r.T[k] = s.transformInv[k / 3][k % 3];
  r.maxDist2 = s.maxDistanceSqr;
  r.weight = s.weight;
  r.proj = s.projectionIndex;
  const double cu = pick3(ua, cx, cy, cz), cv = pick3(va, cx, cy, cz), cw = pick3(wa, cx, cy, cz);
  const float (&t2)[3] = s.transformInv[2];
  const double nu = pick3(ua, t2[0], t2[1], t2[2]), nv = pick3(va, t2[0], t2[1], t2[2]), nw = pick3(wa, t2[0], t2[1], t2[2]);
  r.w0 = 0.f;  // degenerate normal: visit the whole column, the voxel checks decide
  r.wu = 0.f;
  r.wv = 0.f;
  r.hw = 1e9f;
  if (fabs(nw) > 1e-6) {
    const double inv = 1.0 / nw;
    r.w0 = float(cw + (nu * cu + nv * cv) * inv);
    r.wu = float(-nu * inv);
    r.wv = float(-nv * inv);
    r.hw = float(double(radius) * fabs(inv) + 2e-3);
  }
  // half-space x' >= -r, with a margin of 0.01 in x' (far above the float error of h at the
  // largest volume, 1.5e-3 in x')
  const float (&t0)[3] = s.transformInv[0];
  const double tu = pick3(ua, t0[0], t0[1], t0[2]), tv = pick3(va, t0[0], t0[1], t0[2]), tw = pick3(wa, t0[0], t0[1], t0[2]);
  r.h0 = -1e30f;
  r.hu = 0.f;
  r.hv = 0.f;
  if (fabs(tw) > 1e-3) {
    const double inv = 1.0 / tw;
    r.h0 = float(cw + (tu * cu + tv * cv - double(radius) - 0.01) * inv);
    r.hu = float(-tu * inv);
    r.hv = float(-tv * inv);
    if (tw < 0) r.hw = -r.hw;
  }
  r.sphere = s.maxDistanceSqr;
  r.nu = pick3(ua, s.unitNormal[0], s.unitNormal[1], s.unitNormal[2]);
  r.nv = pick3(va, s.unitNormal[0], s.unitNormal[1], s.unitNormal[2]);
  r.nw = pick3(wa, s.unitNormal[0], s.unitNormal[1], s.unitNormal[2]);
  r.bu = pick3(ua, s.bottomOrigin[0], s.bottomOrigin[1], s.bottomOrigin[2]);
  r.bv = pick3(va, s.bottomOrigin[0], s.bottomOrigin[1], s.bottomOrigin[2]);
  r.bw = pick3(wa, s.bottomOrigin[0], s.bottomOrigin[1], s.bottomOrigin[2]);
  r.pad[0] = r.pad[1] = 0;
  return !bad;
}

// Stores a record of 16-byte words.
template<typename R> __device__ __forceinline__ void store_record(R *dst, const R &r)
{
  static_assert(sizeof(R) % 16 == 0, "whole 16-byte words");
  const float4 *s = reinterpret_cast<const float4 *>(&r);
  float4 *d = reinterpret_cast<float4 *>(dst);
#pragma unroll
  for (int k = 0; k < int(sizeof(R) / 16); ++k) d[k] = s[k];
}

// One binning record through four 16-byte read-only loads.
__device__ __forceinline__ SpacePrep load_prep(const SpacePrep *p)
{
  const float4 *q = reinterpret_cast<const float4 *>(p);
  SpacePrep r;
  float4 *d = reinterpret_cast<float4 *>(&r);
  d[0] = __ldg(q);
  d[1] = __ldg(q + 1);
  d[2] = __ldg(q + 2);
  d[3] = __ldg(q + 3);
  return r;
}

// The (brick, direction) lists of up to kRowBricks bricks in a row along x (row `row` = y + nby z
// of the brick grid, bricks bx0 ...; `brickBase` is added to the brick indices, `spaceBase` to the
// listed space indices) by one 256-thread CTA.  A tile of 256 spaces at a time: every thread tests its
// space against all bricks of the row -- the y and z parts of the tests are shared by the row --
// and the hits go to shared memory as one bit mask per brick and warp; then FILL = false counts
// them per (brick, direction), FILL = true has each warp write the hits of its bricks, in
// ascending space order, into the bricks' three direction segments.  The next tile's records are
// loaded during the tests; the masks are double-buffered, so a tile takes one barrier.
//
// The tests are conservative: can any voxel of the brick [b0, b1] (inclusive voxel coordinates,
// relative to the reference's integer volume centre [a, e]) receive a contribution from the space?
// The traversal box, the slab's range over the box, the half-space's maximum and the distance of
// the box's nearest point decide.
//
// Bound by instruction issue (about 20 a space and brick).  A warp per brick testing the spaces
// that hit the union of its CTA's eight bricks, compacted with three barriers a tile, took
// 690 us per pass for 20,000 spaces at box 256 (now 180 counting, 325 filling) and 21 and 26 us for 1,013 at box 64 (now 5 and 9).
constexpr int kRowBricks = 32;

struct BinRow {
  BinGeom g;
  int row, bx0, n;            // n spaces from prep
  int brickBase, spaceBase, job;
  int cap;                    // the items' full capacity (ItemSplit)
  const SpacePrep *prep;
};

template<bool FILL>
__device__ __forceinline__ void bin_row(const BinRow &R, int *__restrict__ counts, const int *__restrict__ offsets,
  int *__restrict__ list, const BinBuffers &buf)
{
  __shared__ unsigned hits[2][kRowBricks][8];
  __shared__ unsigned dirs[2][8][3];
  const BinGeom &g = R.g;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nb = min(kRowBricks, g.nbx - R.bx0);
  const int by = R.row % g.nby, bz = R.row / g.nby;
  const int y0 = by * kBrick, z0 = bz * kBrick;
  const int y1 = min(y0 + kBrick, g.vy) - 1, z1 = min(z0 + kBrick, g.vz) - 1;
  const float ya = float(y0 - g.cy), ye = float(y1 - g.cy), za = float(z0 - g.cz), ze = float(z1 - g.cz);
  const float yc = fminf(fmaxf(0.f, ya), ye), zc = fminf(fmaxf(0.f, za), ze);
  const float yz2 = yc * yc + zc * zc;
  const int first = R.brickBase + (bz * g.nby + by) * g.nbx + R.bx0;  // the row's first brick
  int count = 0;          // FILL = false: thread 3 b + d counts (brick b, direction d)
  int at[4][3] = {};      // FILL = true: next list positions of bricks warp + 8 i
  if (FILL)
    for (int i = 0; i < 4; ++i)
      for (int d = 0; d < 3; ++d)
        if (warp + 8 * i < nb) at[i][d] = offsets[3 * (first + warp + 8 * i) + d];
  SpacePrep next{};
  if (tid < R.n) next = load_prep(R.prep + tid);
  for (int base = 0, t = 0; base < R.n; base += 256, t ^= 1) {
    const SpacePrep p = next;
    const bool live = base + tid < R.n;
    if (base + 256 + tid < R.n) next = load_prep(R.prep + base + 256 + tid);
    const bool row = live && y1 >= p.lo[1] && y0 <= p.hi[1] && z1 >= p.lo[2] && z0 <= p.hi[2];
    const float zl = fminf(p.t2[1] * ya, p.t2[1] * ye) + fminf(p.t2[2] * za, p.t2[2] * ze) - p.halfWidth;
    const float zh = fmaxf(p.t2[1] * ya, p.t2[1] * ye) + fmaxf(p.t2[2] * za, p.t2[2] * ze) + p.halfWidth;
    const float xh = fmaxf(p.t0[1] * ya, p.t0[1] * ye) + fmaxf(p.t0[2] * za, p.t0[2] * ze) - p.xMin;
    const float left = p.maxDist2 - yz2;
    for (int d = 0; d < 3; ++d) {
      const unsigned m = __ballot_sync(0xffffffffu, live && p.dir == d);
      if (lane == 0) dirs[t][warp][d] = m;
    }
    for (int b = 0; b < nb; ++b) {
      const int x0 = (R.bx0 + b) * kBrick, x1 = min(x0 + kBrick, g.vx) - 1;
      const float xa = float(x0 - g.cx), xe = float(x1 - g.cx);
      const float xc = fminf(fmaxf(0.f, xa), xe);
      const float u = p.t2[0] * xa, v = p.t2[0] * xe;
      const bool hit = row && x1 >= p.lo[0] && x0 <= p.hi[0] && zl + fminf(u, v) <= 0.f && zh + fmaxf(u, v) >= 0.f
                       && xh + fmaxf(p.t0[0] * xa, p.t0[0] * xe) >= 0.f && xc * xc <= left;
      const unsigned m = __ballot_sync(0xffffffffu, hit);
      if (lane == 0) hits[t][b][warp] = m;
    }
    __syncthreads();
    if (!FILL) {
      if (tid < 3 * nb) {
        const int b = tid / 3, d = tid - 3 * b;
#pragma unroll
        for (int w = 0; w < 8; ++w) count += __popc(hits[t][b][w] & dirs[t][w][d]);
      }
    } else {
      const unsigned before = (1u << lane) - 1u;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (warp + 8 * i >= nb) break;
        for (int w = 0; w < 8; ++w) {
          const unsigned m = hits[t][warp + 8 * i][w];
          if (m == 0) continue;
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            const unsigned md = m & dirs[t][w][d];
            if (md >> lane & 1u) list[at[i][d] + __popc(md & before)] = R.spaceBase + base + 32 * w + lane;
            at[i][d] += __popc(md);
          }
        }
      }
    }
  }
  if (!FILL) {
    if (tid < 3 * nb) counts[3 * first + tid] = count;
    return;
  }
  // the bricks' work items: at most the plan's capacity each (Kahan: R.cap where not cut), from the
  // plan's first item on
  for (int b = warp; b < nb; b += 8) {
    const int brick = first + b, beg = offsets[3 * brick], end = offsets[3 * brick + 3], item = buf.itemStart[brick];
    const int cap = buf.merge.slot && buf.merge.slot[brick] < 0 ? R.cap : *buf.itemCap;
    for (int q = lane; beg + q * cap < end; q += 32)
      buf.items[item + q] = { brick, beg + q * cap, min(end, beg + (q + 1) * cap), R.job };
  }
}

}// namespace frb
