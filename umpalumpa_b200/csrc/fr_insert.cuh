// The insertion kernel of the B200 Fourier-reconstruction engine.
//
// Why it is not the reference's ProcessKernel: the reference launches a 2D grid over the
// volume face and lets every CTA walk every traverse space, doing three global float
// atomics per voxel per projection (fr_cuda_kernels.cu:362-365,468-523).  Here the volume is
// cut into 16^3-voxel bricks.  The binning passes (fr_kernels.cu) list, per brick, the
// traverse spaces whose blob slab can touch it, grouped by traversal direction; this
// persistent kernel takes (brick, list range) work items, accumulates all their
// projections into shared-memory accumulators and adds the brick into the caller's volume
// once per item.
//
// The per-voxel arithmetic is the reference's ProcessVoxelBlob / ProcessVoxel
// (fr_cpu_kernels.hpp:18-152); the voxels visited are the reference's traversal
// (fr_cpu_kernels.hpp:154-240): for a space of direction XY the column (x, y) of the
// traversal AABB is walked along z across the blob slab, for XZ along y, for YZ along x.
//
// Work split: a CTA runs several independent 256-thread groups, each working on its own
// brick (Groups below); a batched launch (JOBS) takes the items of several jobs, each item
// naming its job in the job table.  Warp w of a group owns the 32 brick columns (U, V) = (tx, w + 8 ty),
// tx < 16, ty < 2, of the current direction.  Per projection each lane finds its column's voxel
// range; the warp deals the voxels of its projections, one projection after the other, to its
// lanes and runs them 32 at a time (insert_blobs), so that a step is full whatever the column
// lengths and wherever one projection's voxels end.  Within one
// direction a warp touches only its own columns, so projections need no synchronisation
// beyond __syncwarp; a group synchronises (named barrier) only when the direction changes.
//
// What bounds it (lookup, FP32, banded, 1,537-20,000 projections at box 256): the L1/shared data
// path (117 wavefronts per step of 32 voxels: 60 pixels and records; 34 table lookups, 13 accumulators
// and the lists, shuffles and flushes) at 80 % and instruction issue at 69 %, with the 24 warps that
// shared memory and registers allow.  Against steps that start anew for every projection (26 of 32 lanes filled, the source
// columns found by a binary search over shuffles), with one voxel body per direction instead of
// one for all: 18 % fewer instructions and 14 % fewer wavefronts; 20,000 projections
// 45.8 -> 36.3 ms (the whole call).
//
// Half-plane layouts (BANDED): the caller's row-major half-planes, or the same pixels in bands
// of four rows stored column by column (pixel (y, x) at (y / 4) * bandStride + 4 x + y % 4,
// band_projections in fr_kernels.cu).  A warp's 32 voxels map to a compact patch of the image;
// in bands a blob tap of the patch touches about 3 cache lines where rows take about 5, which
// cuts the L1 wavefronts of the pixel gathers by about a quarter.
#pragma once

#include "fr_device.cuh"
#include "fr_kernels.h"

namespace frb {

enum { kModeLut = 0, kModeKaiserPoly = 1, kModeKaiserTable = 2 };

// A brick's voxel (x, y, z) has the linear index 256 z + 16 y + x; its accumulators sit at that
// index with the low five bits -- the shared-memory bank -- rotated by 5 (y / 2) + 6 z, so that
// the voxels of a step (short runs along x, y or z in two rows of columns) spread over all 32
// banks: 2.1 wavefronts per access of a full step, where swizzling x by z + y / 2 alone, which
// keeps the rows y and y + 8 of a warp in the same 16 banks, took 3.6 (simulated over the dealing
// at box 256; the rotations with 5..9 in place of 5 and 6 are within 4 %).
__device__ __forceinline__ int acc_slot(int lin)
{
  return (lin & ~31) | ((lin + 5 * ((lin >> 5) & 7) + 6 * (lin >> 8)) & 31);
}

// Sizes and payloads of the job a work item belongs to.  A single-job launch builds it from
// the launch parameters (so the compiler reads them as constant operands); a batched launch
// loads it from the job table for every work item.
struct JobGeom {
  const void *fft;
  const float *scales;
  void *volume;
  float *weight;
  int fftX, fftY, vx, vy, vz, nbx, nby, cx, cy, cz;
  int genericTaps;
  int bandStride;  // banded half-planes: elements per 4-row band
};

__device__ __forceinline__ JobGeom geom_of(const InsertParams &P)
{
  JobGeom g;
  g.fft = P.fft;
  g.scales = P.scales;
  g.volume = P.volume;
  g.weight = P.weight;
  g.fftX = P.fftX;
  g.fftY = P.fftY;
  g.vx = P.vx;
  g.vy = P.vy;
  g.vz = P.vz;
  g.nbx = P.nbx;
  g.nby = P.nby;
  g.cx = P.cx;
  g.cy = P.cy;
  g.cz = P.cz;
  g.genericTaps = P.genericTaps;
  g.bandStride = P.bandStride;
  return g;
}

__device__ __forceinline__ JobGeom geom_of(const JobDesc &J)
{
  JobGeom g;
  g.fft = J.fft;
  g.scales = J.scales;
  g.volume = J.volume;
  g.weight = J.weight;
  g.fftX = J.fftX;
  g.fftY = J.fftY;
  g.vx = J.vx;
  g.vy = J.vy;
  g.vz = J.vz;
  g.nbx = J.nbx;
  g.nby = J.nby;
  g.cx = J.cx;
  g.cy = J.cy;
  g.cz = J.cz;
  g.genericTaps = J.genericTaps;
  g.bandStride = J.bandStride;
  return g;
}

struct Accum {
  float2 *v;              // brick accumulators: the complex values
  float *w;               // and the weights
  __nv_bfloat162 *cv;     // Kahan compensations (KAHAN only)
  __nv_bfloat16 *cw;
};

// Kahan-compensated add; returns the new sum.  The compensation -- the rounding error of the
// previous add, at most half an ulp of the sum -- is kept in BF16: its 8 significant bits leave
// each add at most 1/256 of plain FP32's rounding residual, and 18 instead of 24 bytes per voxel
// let the blob table stay in shared memory beside two brick groups.
__device__ __forceinline__ float kahan_add(float sum, float &comp, float v)
{
  const float y = __fsub_rn(v, comp);
  const float t = __fadd_rn(sum, y);
  comp = __fsub_rn(__fsub_rn(t, sum), y);
  return t;
}

template<bool KAHAN>
__device__ __forceinline__ void acc_add(const Accum &A, int i, float2 v, float w)
{
  float2 s = A.v[i];
  if (KAHAN) {
    float2 c = __bfloat1622float2(A.cv[i]);
    float cw = __bfloat162float(A.cw[i]);
    s.x = kahan_add(s.x, c.x, v.x);
    s.y = kahan_add(s.y, c.y, v.y);
    A.w[i] = kahan_add(A.w[i], cw, w);
    A.cv[i] = __floats2bfloat162_rn(c.x, c.y);
    A.cw[i] = __float2bfloat16_rn(cw);
  } else {
    s.x += v.x;
    s.y += v.y;
    A.w[i] += w;
  }
  A.v[i] = s;
}

// Voxels a warp's list holds (insert_blobs): an entry has at most 32 columns x 16, nearly always
// fewer than 120.  24 lists of 240 16-bit voxels leave three plain brick groups and a
// 10,000-entry table in the 196 KB shared-memory carve-out, so the L1 keeps its size.
constexpr int kVoxelList = 240;

__device__ __forceinline__ float approx_sqrt(float v)
{
  float r;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
}

// The fields of a SpaceRec a voxel needs (every voxel of a step may belong to another space).
struct VoxelRec {
  float T[9];
  float maxDist2, weight;
  int proj;
};

__device__ __forceinline__ VoxelRec load_voxel_rec(const SpaceRec *r)
{
  const float4 *q = reinterpret_cast<const float4 *>(r);
  const float4 f0 = __ldg(q), f1 = __ldg(q + 1), f2 = __ldg(q + 2);
  return { { f0.x, f0.y, f0.z, f0.w, f1.x, f1.y, f1.z, f1.w, f2.x }, f2.y, f2.z, __float_as_int(f2.w) };
}

// Coordinate of voxel i (0..15) of the brick relative to the volume centre, as a float: exact.
// `origin` is the brick's first coordinate relative to the centre less 2^23 (brick_origin), so
// that the integer is placed in the mantissa and one subtraction converts it.
__device__ __forceinline__ float brick_origin(int o, int c) { return float(o - c) - 8388608.f; }
__device__ __forceinline__ float voxel_coord(int i, float origin) { return __int_as_float(0x4b000000 | i) + origin; }

// FR<>::ProcessVoxelBlob (fr_cpu_kernels.hpp:70-152) for voxel (X, Y, Z): Kaiser-Bessel
// gather of the projection pixels within the blob radius.  The blob weights are summed raw
// and scaled by the space weight (and the storage scale) once at the end.  Returns false if
// the voxel is rejected.
template<int MODE, int TAPS, int STORAGE, bool GENERIC, bool JOBS, bool BANDED>
__device__ __forceinline__ bool voxel_blob(const InsertParams &P, const JobGeom &G, const VoxelRec &s,
  const typename Pixel<STORAGE>::T *__restrict__ img, int bandStride, float scale, const float *lut, float px,
  float py, float pz, float2 &ov, float &ow)
{
  const fr_constants &c = P.c;
  const float qx = add_(add_(mul_(s.T[0], px), mul_(s.T[1], py)), mul_(s.T[2], pz));
  const float qy0 = add_(add_(mul_(s.T[3], px), mul_(s.T[4], py)), mul_(s.T[5], pz));
  const float qz = add_(add_(mul_(s.T[6], px), mul_(s.T[7], py)), mul_(s.T[8], pz));
  const float r = c.cBlobRadius;
  const float qy = add_(qy0, float(G.cy));
  const float rSq = mul_(r, r);
  const float zSq = mul_(qz, qz);
  // The TAPS x TAPS window starts at (ceil(qx - r), ceil(qy - r)) shifted into the image, so
  // it covers the reference's clamped blob box [max(ceil(q - r), 0), min(floor(q + r), X-1)]
  // and lies inside the image; candidates outside the blob box have d2 > r^2, so d2 <= r^2
  // is the only per-tap test (FR::ProcessVoxelBlob's radius test, fr_cpu_kernels.hpp:128-134).
  // GENERIC (a half-plane narrower or shorter than the window) tests the blob box explicitly.
  // The origin stays a float (integer-valued, exact) for the distances and is converted once
  // for the addresses.
  float x0 = fmaxf(ceilf(sub_(qx, r)), 0.f);
  float y0 = fmaxf(ceilf(sub_(qy, r)), 0.f);
  if (!GENERIC) {
    x0 = fminf(x0, float(G.fftX - TAPS));
    y0 = fminf(y0, float(G.fftY - TAPS));
  }
  const float dx0 = sub_(qx, x0);
  // Outside the frequency sphere (integer-valued: exact), behind the image or off the slab, as
  // the reference rejects; and beyond the image's other edges, where no pixel lies within the
  // radius (which also rejects non-finite coordinates).  One predicate: the tests are independent.
  // The last three cost 0.3-0.9 % where no voxel lies out there (box 256 x 20,000 36.3 -> 36.5 ms),
  // but keep a voxel that can only add zeros out of the taps -- 2,000 half-planes cropped to
  // 33 x 64 into box 256 take 1.77 ms with them, 2.84 without -- and out of the sums, where the
  // zeros times an infinite or NaN weight would be NaN.  Either form is sound where the window is
  // shifted into the image; from the window's outer pixels, whose distances the taps use, is the faster
  // one beside the polynomial (box 256 x 6,000 12.49 -> 12.35 ms, box 96 FP16 x 777 383 -> 380 us) and
  // in batched launches, whose image size lies in shared memory (against the kernel without the tests,
  // six streamed jobs 0.992x -> 1.000x, twelve captured jobs 0.998x -> 1.003x); from the image's size
  // beside the table lookups of a single job (36.66 -> 36.54 ms).
  bool inside = !(px * px + py * py + pz * pz > s.maxDist2) & !(qx < -r) & !(zSq > rSq);
  if (GENERIC || (MODE == kModeLut && !JOBS))
    inside = inside & (qx <= float(G.fftX) + r) & (qy >= -r) & (qy <= float(G.fftY) + r);
  else
    inside = inside & (dx0 - float(TAPS - 1) <= r) & (sub_(qy, y0) >= -r) & (sub_(qy, add_(y0, float(TAPS - 1))) <= r);
  if (!inside) return false;
  const int minX = int(x0), minY = int(y0);
  const int maxX = min(int(floorf(add_(qx, r))), G.fftX - 1);  // GENERIC only
  const int maxY = min(int(floorf(add_(qy, r))), G.fftY - 1);
  // First pixel of window row ii.  Banded: rows o = minY % 4, o + 1, ... of the window's first
  // band; row ii lies (o + ii) / 4 bands further (at most one for 4 rows), where the same row
  // offset less 4 applies.
  using PT = typename Pixel<STORAGE>::T;
  const int o = BANDED ? minY & 3 : 0;
  const PT *w0 = BANDED ? img + size_t(unsigned(minY) >> 2) * unsigned(bandStride) + unsigned(o + 4 * minX)
                        : img + size_t(unsigned(minY)) * unsigned(G.fftX) + unsigned(minX);
  const PT *w1 = w0 + (bandStride - 4);
  auto window_row = [&](int ii) -> const PT * {
    if (!BANDED) return w0 + size_t(ii) * unsigned(G.fftX);
    if (TAPS == 4) return (o + ii >= 4 ? w1 : w0) + ii;
    return w0 + size_t(unsigned(o + ii) >> 2) * unsigned(bandStride - 4) + ii;
  };
  // Taps are evaluated in pairs with packed FP32x2 arithmetic: per pair one fused d2 and one
  // fused table position, per tap one fused complex accumulation.  Each lane rounds exactly
  // like the scalar fmaf it replaces.
  float2 dxp[TAPS / 2];
#pragma unroll
  for (int k = 0; k < TAPS / 2; ++k) dxp[k] = make_float2(dx0 - float(2 * k), dx0 - float(2 * k + 1));
  const float2 cI2 = make_float2(c.cIDeltaSqrt, c.cIDeltaSqrt);
  const float2 kt2 = make_float2(P.tableScale, P.tableScale);
  const float2 negInvR2 = make_float2(-c.cOneOverBlobRadiusSqr, -c.cOneOverBlobRadiusSqr);
  const float2 half2 = make_float2(0.5f, 0.5f);
  float2 acc = make_float2(0.f, 0.f);
  float w = 0.f;
  auto tap = [&](const PT *row, int ii, int jj, float d2, float pos) {
    const bool inBox = !GENERIC || (minY + ii <= maxY && minX + jj <= maxX);
    if (inBox && d2 <= rSq) {
      float wb;
      if (MODE == kModeLut) {
        // With at most 16,384 table entries (cIDeltaSqrt = (N-1)/r^2; the table in shared or,
        // beside Kahan accumulators, global memory), d2 <= r^2 bounds the position by
        // N - 1 + 0.5 + N * 2^-23 < N: no clamp needed.
        const int li = int(pos);
        wb = lut[GENERIC ? min(li, P.tableElems - 1) : li];
      } else if (MODE == kModeKaiserTable) {
        // pos = d2 (N-1) / r^2 in [0, N-1] (d2 <= r^2, rounding keeps it below N): node and
        // fraction, then value + slope * fraction
        const int li = GENERIC ? min(int(pos), P.tableElems - 1) : int(pos);
        const float2 e = reinterpret_cast<const float2 *>(lut)[li];
        wb = fmaf(e.y, pos - float(li), e.x);
      } else {
        wb = pos;  // the pair's weights, computed below with kaiser_poly2
      }
      const float2 v = Pixel<STORAGE>::load(row + (BANDED ? 4 * jj : jj));
      w += wb;
      acc = __ffma2_rn(v, make_float2(wb, wb), acc);
    }
  };
#pragma unroll
  for (int ii = 0; ii < TAPS; ++ii) {
    const float dy = sub_(qy, add_(y0, float(ii)));
    const float yz = add_(mul_(dy, dy), zSq);
    const float2 yz2 = make_float2(yz, yz);
    const PT *row = window_row(ii);
#pragma unroll
    for (int k = 0; k < TAPS / 2; ++k) {
      const float2 d2 = __ffma2_rn(dxp[k], dxp[k], yz2);
      // per tap: the table position, or the polynomial's blob weight
      const float2 pos = MODE == kModeLut           ? __ffma2_rn(d2, cI2, half2)
                         : MODE == kModeKaiserTable ? __fmul2_rn(d2, kt2)
                                                    : kaiser_poly2(d2, negInvR2, P.kaiser);
      tap(row, ii, 2 * k, d2.x, pos.x);
      tap(row, ii, 2 * k + 1, d2.y, pos.y);
    }
  }
  const float dw = mul_(s.weight, scale);
  ov = __fmul2_rn(acc, make_float2(dw, dw));
  ow = mul_(w, s.weight);
  return true;
}

// FR<>::ProcessVoxel (fr_cpu_kernels.hpp:18-68): nearest pixel.
template<int STORAGE, bool BANDED>
__device__ __forceinline__ bool voxel_nearest(const JobGeom &G, const VoxelRec &s,
  const typename Pixel<STORAGE>::T *__restrict__ img, int bandStride, float scale, float px, float py, float pz,
  float2 &ov, float &ow)
{
  if (px * px + py * py + pz * pz > s.maxDist2) return false;
  const float qx = add_(add_(mul_(s.T[0], px), mul_(s.T[1], py)), mul_(s.T[2], pz));
  const float qy = add_(add_(mul_(s.T[3], px), mul_(s.T[4], py)), mul_(s.T[5], pz));
  if (qx < 0.f) return false;
  const int imgX = min(max(int(add_(qx, 0.5f)), 0), G.fftX - 1);
  const int imgY = min(max(int(add_(add_(qy, 0.5f), float(G.cy))), 0), G.fftY - 1);
  const float2 v = Pixel<STORAGE>::load(BANDED ? img + size_t(imgY / 4) * size_t(bandStride) + 4 * imgX + imgY % 4
                                               : img + size_t(imgY) * G.fftX + imgX);
  const float w = s.weight;
  const float wt = mul_(w, scale);
  ov = make_float2(mul_(v.x, wt), mul_(v.y, wt));
  ow = w;
  return true;
}

// The brick at (ox, oy, oz) seen along one traversal direction (uniform across the group): the
// plane axes U, V and the column axis W (traverse_space.hpp:24-28; XY: x, y | z;  XZ: x, z | y;
// YZ: y, z | x), and this lane's column.
struct Column {
  float U, V;         // the column's volume coordinates
  int lin, sW;        // linear brick index of its voxel at W = 0 (before the brick), step along W
  bool in;            // inside the volume
  int oW, wHi;        // first coordinate of the brick along W, last one inside the volume
  float du, dv, cw;   // U, V relative to the centre; the centre along W
};

__device__ __forceinline__ Column column_of(const JobGeom &G, int dir, int ox, int oy, int oz, int warp, int lane)
{
  const bool xy = dir == FR_DIR_XY, yz = dir == FR_DIR_YZ;
  // warp w owns column rows w and w + 8: a slab that crosses part of the brick face spreads
  // over the warps instead of piling onto a few (2 % faster than adjacent rows)
  const int tu = lane & (kBrick - 1), tv = warp + 8 * (lane >> 4);
  const int U = (yz ? oy : ox) + tu, V = (xy ? oy : oz) + tv;
  Column c;
  c.U = float(U);
  c.V = float(V);
  c.in = U < (yz ? G.vy : G.vx) && V < (xy ? G.vy : G.vz);
  c.oW = xy ? oz : (yz ? ox : oy);
  c.wHi = min(c.oW + kBrick, xy ? G.vz : (yz ? G.vx : G.vy)) - 1;
  c.sW = xy ? 256 : (yz ? 1 : 16);
  c.lin = tu * (yz ? 16 : 1) + tv * (xy ? 16 : 256) - c.oW * c.sW;
  c.du = float(U - (yz ? G.cy : G.cx));
  c.dv = float(V - (xy ? G.cy : G.cz));
  c.cw = float(xy ? G.cz : (yz ? G.cx : G.cy));
  return c;
}

// All list entries [e0, e1) of one direction for the brick at (ox, oy, oz), blob insertion.
//
// The voxels of the entries form one stream per warp, in entry order: every lane lists its
// column's voxels of an entry in the warp's shared-memory list (at the prefix sum of the column
// lengths), the lanes from `n` on take them from there, and a step runs when all 32 lanes hold
// one (or the entries have ended).  A step that starts anew for every entry fills 26 of 32 lanes
// at box 256 (24 at box 64); the stream fills all of them, with 1.4 entries per step.  Two entries of a
// step may hold the same voxel, so their adds follow one another (`part` numbers the entries of
// the step).
template<int MODE, int TAPS, int STORAGE, bool KAHAN, bool JOBS, bool BANDED>
__device__ __forceinline__ void insert_blobs(const InsertParams &P, const JobGeom &G, const Accum &A,
  const float *lut, uint16_t *list, int ox, int oy, int oz, int dir, int warp, int lane, int e0, int e1)
{
  using PT = typename Pixel<STORAGE>::T;
  // a single-job launch reads the band stride as a constant operand of the launch parameters
  const int bandStride = JOBS ? G.bandStride : P.bandStride;
  const size_t plane = BANDED ? size_t((G.fftY + 3) / 4) * size_t(bandStride) : size_t(G.fftX) * size_t(G.fftY);
  const Column col = column_of(G, dir, ox, oy, oz, warp, lane);
  const float bx = brick_origin(ox, G.cx), by = brick_origin(oy, G.cy), bz = brick_origin(oz, G.cz);
  // the column inside the brick and the frequency sphere |p|^2 <= sphere (with a margin), kept
  // while the entries' spheres are alike -- as they are in a reconstruction
  float sphere = nanf(""), clipLo = 0.f, clipHi = 0.f;
  int n = 0, parts = 0;        // lanes that hold a voxel, entries they come from
  int voxel = 0, space = 0;    // this lane's: linear brick index | part << 12, space
  int at = 0, have = 0;        // the list: voxels taken, voxels listed
  int si = 0;                  // the space they belong to
  int listed = 0;              // voxels of entry e listed before (an entry longer than the list)
  for (int e = e0;;) {
    while (n < 32) {
      if (at == have) {  // list the next entry: this lane's column range
        if (e == e1) break;
        si = __ldg(P.list + e);
        const float4 *q = reinterpret_cast<const float4 *>(P.recs + si);
        const float4 box = __ldg(q + 3), slab = __ldg(q + 4), half = __ldg(q + 5);
        if (half.w != sphere) {  // uniform
          sphere = half.w;
          const float rem = sphere - col.du * col.du - col.dv * col.dv;
          const float sq = approx_sqrt(fmaxf(rem, 0.f)) + 8e-3f;
          const bool hit = col.in && rem >= 0.f;
          clipLo = hit ? fmaxf(col.cw - sq, float(col.oW)) : 1e9f;
          clipHi = hit ? fminf(col.cw + sq, float(col.wHi)) : -1e9f;
        }
        // slab |t2.p| <= r and image half-space t0.p >= -r, with margins; the voxel checks
        // decide exactly
        const float wc = fmaf(slab.y, col.U, fmaf(slab.z, col.V, slab.x));
        const float hb = fmaf(half.y, col.U, fmaf(half.z, col.V, half.x));
        float flo = fmaxf(wc - fabsf(slab.w), clipLo), fhi = fminf(wc + fabsf(slab.w), clipHi);
        if (slab.w > 0.f) flo = fmaxf(flo, hb);
        else fhi = fminf(fhi, hb);
        const int lo = int(ceilf(flo)), hi = int(floorf(fhi));
        const bool hit = col.U >= box.x && col.U <= box.y && col.V >= box.z && col.V <= box.w && lo <= hi;
        // prefix sum of the column lengths (0..16) by bit planes; a blob of radius < 2 gives at
        // most 7 voxels per column where the normal's component along W dominates
        const int cnt = hit ? hi - lo + 1 : 0;
        const unsigned before = (1u << lane) - 1u;
        const unsigned b0 = __ballot_sync(0xffffffffu, cnt & 1), b1 = __ballot_sync(0xffffffffu, cnt & 2),
                       b2 = __ballot_sync(0xffffffffu, cnt & 4), b3 = __ballot_sync(0xffffffffu, cnt & 24);
        int excl = __popc(b0 & before) + 2 * __popc(b1 & before) + 4 * __popc(b2 & before);
        int total = __popc(b0) + 2 * __popc(b1) + 4 * __popc(b2);
        int v = col.lin + lo * col.sW;
        if (b3 == 0 && total <= kVoxelList) {
          __syncwarp();  // the list's last voxels have been taken
#pragma unroll
          for (int j = 0; j < 7; ++j) {
            if (j < cnt) list[excl + j] = uint16_t(v);
            v += col.sW;
          }
          have = total;
          ++e;
        } else {  // long columns, or more voxels than the list takes: in rounds
          const unsigned c3 = __ballot_sync(0xffffffffu, cnt & 8), c4 = __ballot_sync(0xffffffffu, cnt & 16);
          excl += 8 * __popc(c3 & before) + 16 * __popc(c4 & before);
          total += 8 * __popc(c3) + 16 * __popc(c4);
          have = min(total - listed, kVoxelList);
          __syncwarp();
          for (int j = 0; j < cnt; ++j, v += col.sW) {
            const int k = excl + j - listed;
            if (k >= 0 && k < have) list[k] = uint16_t(v);
          }
          listed += have;
          if (listed == total) {
            listed = 0;
            ++e;
          }
        }
        __syncwarp();
        at = 0;
        continue;
      }
      const int k = at + lane - n;
      if (lane >= n && k < have) {
        voxel = list[k] | parts << 12;
        space = si;
      }
      const int took = min(32 - n, have - at);
      at += took;
      n += took;
      ++parts;
    }
    if (n == 0) break;
    float2 v;
    float w;
    bool ok = false;
    if (lane < n) {
      const VoxelRec s = load_voxel_rec(P.recs + space);
      const float px = voxel_coord(voxel & 15, bx), py = voxel_coord(voxel >> 4 & 15, by),
                  pz = voxel_coord(voxel >> 8 & 15, bz);
      const float scale = STORAGE == FR_STORAGE_FP32 ? 1.f : __ldg(G.scales + s.proj);
      const PT *img = reinterpret_cast<const PT *>(G.fft) + size_t(unsigned(s.proj)) * plane;
      if (G.genericTaps)
        ok = voxel_blob<MODE, TAPS, STORAGE, true, JOBS, BANDED>(P, G, s, img, bandStride, scale, lut, px, py, pz, v, w);
      else
        ok = voxel_blob<MODE, TAPS, STORAGE, false, JOBS, BANDED>(P, G, s, img, bandStride, scale, lut, px, py, pz, v, w);
    }
    const int slot = acc_slot(voxel & 4095);
    if (parts == 1) {  // two steps of three
      if (ok) acc_add<KAHAN>(A, slot, v, w);
      __syncwarp();  // the next step may revisit these voxels from other lanes
    } else {
      for (int p = 0; p < parts; ++p) {
        if (ok && voxel >> 12 == p) acc_add<KAHAN>(A, slot, v, w);
        __syncwarp();  // as may the next entry
      }
    }
    n = 0;
    parts = 0;
  }
}

// All list entries [e0, e1) of one direction, nearest-pixel insertion: at most one voxel per
// column and projection, which the column's lane inserts itself (no lane touches another's column,
// so no synchronisation either).  The next entry's record is fetched while this one's voxel is
// inserted: the loads' latency, one after the other, is what an entry waits for (box 256 x 8,192:
// 4.8 -> 3.9 ms; adding each pixel one entry after its load was issued gained nothing more).
template<int STORAGE, bool KAHAN, bool JOBS, bool BANDED>
__device__ __forceinline__ void insert_nearest(const InsertParams &P, const JobGeom &G, const Accum &A, int ox,
  int oy, int oz, int dir, int warp, int lane, int e0, int e1)
{
  using PT = typename Pixel<STORAGE>::T;
  const int bandStride = JOBS ? G.bandStride : P.bandStride;
  const size_t plane = BANDED ? size_t((G.fftY + 3) / 4) * size_t(bandStride) : size_t(G.fftX) * size_t(G.fftY);
  const Column col = column_of(G, dir, ox, oy, oz, warp, lane);
  const float bx = brick_origin(ox, G.cx), by = brick_origin(oy, G.cy), bz = brick_origin(oz, G.cz);
  if (!col.in) e0 = e1;
  int next = e0 < e1 ? __ldg(P.list + e0) : 0;
  float4 box, n, b;
  auto fetch = [&](int space) {
    const float4 *q = reinterpret_cast<const float4 *>(P.recs + space);
    box = __ldg(q + 3);
    n = __ldg(q + 6);
    b = __ldg(q + 7);
  };
  if (e0 < e1) fetch(next);
  for (int e = e0; e < e1; ++e) {
    const int si = next;
    const float4 cbox = box, cn = n, cb = b;
    if (e + 1 < e1) {
      next = __ldg(P.list + e + 1);
      fetch(next);
    }
    if (col.U < cbox.x || col.U > cbox.y || col.V < cbox.z || col.V > cbox.w) continue;
    // the reference's rounded plane hit
    const int W = int(add_(plane_hit(col.U, col.V, cn.x, cn.y, cn.z, cn.w, cb.x, cb.y), 0.5f));
    if (W < col.oW || W > col.wHi) continue;
    const int lin = col.lin + W * col.sW;
    const VoxelRec s = load_voxel_rec(P.recs + si);
    const float scale = STORAGE == FR_STORAGE_FP32 ? 1.f : __ldg(G.scales + s.proj);
    const PT *img = reinterpret_cast<const PT *>(G.fft) + size_t(unsigned(s.proj)) * plane;
    float2 v;
    float w;
    if (voxel_nearest<STORAGE, BANDED>(G, s, img, bandStride, scale, voxel_coord(lin & 15, bx),
          voxel_coord(lin >> 4 & 15, by), voxel_coord(lin >> 8, bz), v, w))
      acc_add<KAHAN>(A, acc_slot(lin), v, w);
  }
  __syncwarp();
}

// Shared-memory groups per CTA: one 256-thread group per brick in flight.  The groups of a CTA
// share one copy of the blob table, so three plain-accumulator groups (3 x 48 KB + 40 KB)
// fit on an SM where three separate CTAs would not.  Kahan accumulators (72 KB: FP32 sums and
// BF16 compensations) allow two groups beside the table.
// Nearest-pixel insertion needs no table, which makes room for one group more (box 256 x 8,192:
// 5.9 -> 4.8 ms).
// This is the most a CTA may hold; the launch picks 1..value groups (blockDim.x / 256).
template<bool KAHAN, bool FAST> struct Groups { static constexpr int value = (KAHAN ? 2 : 3) + FAST; };

__device__ __forceinline__ void group_sync(int group)
{
  asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "r"(kThreads) : "memory");
}

template<int MODE, int TAPS, bool FAST, int STORAGE, bool KAHAN, bool JOBS, bool BANDED>
__global__ void __launch_bounds__(kThreads *Groups<KAHAN, FAST>::value, 1) insert_kernel(InsertParams P)
{
  constexpr int kMaxGroups = Groups<KAHAN, FAST>::value;
  constexpr int kAccFloats = (KAHAN ? 9 * kBrickVox / 2 : 3 * kBrickVox);  // 32-bit words
  const int nGroups = int(blockDim.x) / kThreads;  // launch shape: 1..kMaxGroups
  extern __shared__ float4 smem4[];
  float *smem = reinterpret_cast<float *>(smem4);
  __shared__ int sItem[kMaxGroups];
  __shared__ int sLast[KAHAN ? kMaxGroups : 1];  // the item ends a merged brick
  __shared__ uint16_t sVoxels[FAST ? 1 : kMaxGroups * (kThreads / 32)][kVoxelList];
  // Batched launches: the current job's geometry, one copy per group in shared memory.  Held
  // in registers (as the single-job kernel may, where the values are constant operands of the
  // launch parameters) its 20 words spilled 80 bytes at the register cap.
  __shared__ JobGeom sGeom[kMaxGroups];
  const int group = threadIdx.x / kThreads;
  const int tid = threadIdx.x % kThreads;
  const int warp = tid >> 5, lane = tid & 31;
  float *acc = smem + group * kAccFloats;
  Accum A;
  A.v = reinterpret_cast<float2 *>(acc);
  A.w = acc + 2 * kBrickVox;
  A.cv = reinterpret_cast<__nv_bfloat162 *>(acc + 3 * kBrickVox);
  A.cw = reinterpret_cast<__nv_bfloat16 *>(A.cv + kBrickVox);
  float *lutS = smem + nGroups * kAccFloats;

  const float *lut = P.table;
  if ((MODE == kModeLut || MODE == kModeKaiserTable) && !FAST && P.lutInSmem) {
    const int nf = MODE == kModeKaiserTable ? 2 * P.tableElems : P.tableElems;  // float2 entries
    for (int i = threadIdx.x; i < nf; i += int(blockDim.x)) lutS[i] = __ldg(P.table + i);
    lut = lutS;
  }
  for (int i = tid; i < kAccFloats; i += kThreads) acc[i] = 0.f;  // the flush leaves zeros behind
  if (tid == 0) sItem[group] = atomicAdd(P.workCounter, 1);
  __syncthreads();
  const int nItems = *P.nItems;

  for (;;) {
    group_sync(group);  // the flush is finished, the next item's index is there
    const int itIdx = sItem[group];
    if (itIdx >= nItems) break;
    const WorkItem it = P.items[itIdx];
    int next = 0;  // fetched while this item is inserted
    if (tid == 0) next = atomicAdd(P.workCounter, 1);
    if (JOBS) {
      if (tid == 0) sGeom[group] = geom_of(P.jobs[it.job]);
      group_sync(group);
    }
    JobGeom Gl;
    if (!JOBS) Gl = geom_of(P);
    const JobGeom &G = JOBS ? sGeom[group] : Gl;
    // batch-wide brick index; offsets and lists are batch-wide
    const int brick = it.brick - (JOBS ? P.jobs[it.job].brickBase : 0);
    const int bx = brick % G.nbx, by = (brick / G.nbx) % G.nby, bz = brick / (G.nbx * G.nby);
    const int ox = bx * kBrick, oy = by * kBrick, oz = bz * kBrick;
    const int base = 3 * it.brick;
    for (int dir = 0; dir < 3; ++dir) {
      const int e0 = max(it.begin, P.offsets[base + dir]);
      const int e1 = min(it.end, P.offsets[base + dir + 1]);
      if (e0 >= e1) continue;  // uniform across the group
      if (FAST)
        insert_nearest<STORAGE, KAHAN, JOBS, BANDED>(P, G, A, ox, oy, oz, dir, warp, lane, e0, e1);
      else
        insert_blobs<MODE, TAPS, STORAGE, KAHAN, JOBS, BANDED>(P, G, A, lut, sVoxels[threadIdx.x >> 5], ox, oy, oz, dir,
          warp, lane, e0, e1);
      group_sync(group);  // the next direction maps warps to other voxels
    }
    // add the brick into the caller's volume -- Kahan: a cut brick into its FP64 sums, which the
    // last of its items adds to the volume -- and clear it (an item has at least one entry, so a
    // barrier lies between the reads of sItem above and its new value)
    double *sums = nullptr;
    if (KAHAN && P.merge.slot) {
      const int slot = P.merge.slot[it.brick];  // uniform across the group
      if (slot >= 0) sums = P.merge.sums + size_t(slot) * (3 * kBrickVox);
    }
    for (int lin = tid; lin < kBrickVox; lin += kThreads) {
      const int i = acc_slot(lin);
      float2 v = A.v[i];
      float w = A.w[i];
      A.v[i] = make_float2(0.f, 0.f);
      A.w[i] = 0.f;
      if (KAHAN) {
        const float2 c = __bfloat1622float2(A.cv[i]);
        const float cw = __bfloat162float(A.cw[i]);
        A.cv[i] = __floats2bfloat162_rn(0.f, 0.f);
        A.cw[i] = __float2bfloat16_rn(0.f);
        if (sums) {
          const double x = double(v.x) - c.x, y = double(v.y) - c.y, z = double(w) - cw;
          if (x != 0.0) atomicAdd(sums + lin, x);
          if (y != 0.0) atomicAdd(sums + kBrickVox + lin, y);
          if (z != 0.0) atomicAdd(sums + 2 * kBrickVox + lin, z);
          continue;
        }
        v.x = __fsub_rn(v.x, c.x);
        v.y = __fsub_rn(v.y, c.y);
        w = __fsub_rn(w, cw);
      }
      const int X = ox + (lin & 15), Y = oy + (lin >> 4 & 15), Z = oz + (lin >> 8);
      if (X >= G.vx || Y >= G.vy || Z >= G.vz) continue;
      if (__float_as_uint(v.x) == 0u && __float_as_uint(v.y) == 0u && __float_as_uint(w) == 0u) continue;
      const size_t g = (size_t(Z) * G.vy + Y) * G.vx + X;
      atomicAdd(reinterpret_cast<float2 *>(G.volume) + g, v);
      atomicAdd(G.weight + g, w);
    }
    if (KAHAN && sums) {
      __threadfence();    // this thread's adds before the count of the items still to come
      group_sync(group);
      if (tid == 0) sLast[group] = atomicSub(P.merge.left + it.brick, 1) == 1;
      group_sync(group);
      if (sLast[group]) {
        __threadfence();  // the other items' adds after the count
        // bound by the latency of its loads: four voxels in flight per thread (one: 5 us more
        // per call, eight: the same)
        constexpr int kAhead = 4;
        for (int l0 = tid; l0 < kBrickVox; l0 += kAhead * kThreads) {
          double m[kAhead][3];
#pragma unroll
          for (int k = 0; k < 3 * kAhead; ++k)
            m[k / 3][k % 3] = __ldcg(sums + (k % 3) * kBrickVox + l0 + (k / 3) * kThreads);
#pragma unroll
          for (int k = 0; k < kAhead; ++k) {
            const int lin = l0 + k * kThreads;
            const float x = float(m[k][0]), y = float(m[k][1]), z = float(m[k][2]);
            sums[lin] = sums[kBrickVox + lin] = sums[2 * kBrickVox + lin] = 0.0;
            const int X = ox + (lin & 15), Y = oy + (lin >> 4 & 15), Z = oz + (lin >> 8);
            if (X >= G.vx || Y >= G.vy || Z >= G.vz || (x == 0.f && y == 0.f && z == 0.f)) continue;
            const size_t g = (size_t(Z) * G.vy + Y) * G.vx + X;
            atomicAdd(reinterpret_cast<float2 *>(G.volume) + g, make_float2(x, y));
            atomicAdd(G.weight + g, z);
          }
        }
      }
    }
    if (tid == 0) sItem[group] = next;
  }
}

template<int MODE, bool FAST, int STORAGE, bool KAHAN, bool JOBS, bool BANDED>
static InsertFn pick_taps(int taps)
{
  if (taps <= 4) return insert_kernel<MODE, 4, FAST, STORAGE, KAHAN, JOBS, BANDED>;
  return insert_kernel<MODE, 8, FAST, STORAGE, KAHAN, JOBS, BANDED>;
}

template<int STORAGE, bool KAHAN, bool JOBS, bool BANDED>
static InsertFn pick_mode(const InsertConfig &cfg)
{
  if (cfg.fast) return insert_kernel<kModeLut, 4, true, STORAGE, KAHAN, JOBS, BANDED>;
  switch (cfg.mode) {
  case kModeLut: return pick_taps<kModeLut, false, STORAGE, KAHAN, JOBS, BANDED>(cfg.taps);
  case kModeKaiserPoly: return pick_taps<kModeKaiserPoly, false, STORAGE, KAHAN, JOBS, BANDED>(cfg.taps);
  default: return pick_taps<kModeKaiserTable, false, STORAGE, KAHAN, JOBS, BANDED>(cfg.taps);
  }
}

// Single-job kernels (accumulation plain or Kahan) over row-major or banded half-planes.
template<int STORAGE, bool BANDED>
static InsertFn pick_storage(const InsertConfig &cfg)
{
  return cfg.kahan ? pick_mode<STORAGE, true, false, BANDED>(cfg) : pick_mode<STORAGE, false, false, BANDED>(cfg);
}

// Batched kernels (work items of several jobs in one launch); a batch always reads banded
// half-planes (fr_batch_execute copies every job's projections into bands).
template<int STORAGE>
static InsertFn pick_storage_jobs(const InsertConfig &cfg)
{
  return cfg.kahan ? pick_mode<STORAGE, true, true, true>(cfg) : pick_mode<STORAGE, false, true, true>(cfg);
}

}// namespace frb
