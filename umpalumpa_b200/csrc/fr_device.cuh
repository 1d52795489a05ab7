// Device-side building blocks of the B200 Fourier-reconstruction engine: layouts shared by
// the kernels, the Kaiser-Bessel blob math and the slab geometry.  Reference citations are
// path:line relative to the Umpalumpa project root.
#pragma once

#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>

#include "fr_kernels.h"
#include "umpalumpa_fr.h"

namespace frb {

static_assert(sizeof(fr_traverse_space) == 112, "TraverseSpace must stay 112 bytes");
static_assert(sizeof(fr_constants) == 32, "Constants must stay 32 bytes");

constexpr int kThreads = 256;     // insertion CTA: 16 x 16 columns of one brick face
constexpr int kBrick = 16;        // brick edge in voxels (16^3 voxels = 48 KB of accumulators)
constexpr int kBrickVox = kBrick * kBrick * kBrick;
constexpr int kLutSmemMax = 16384;// blob tables up to 64 KB live in shared memory
// Dynamic interpolation's Kaiser table for alpha > 15: (value, slope) at nodes equally spaced
// in d^2 over [0, r^2], interpolated linearly (32 KB; at r 1.9 its error is 5.4e-7 of the
// peak weight at alpha 18, 1.1e-6 at alpha 25, 2.8e-6 at alpha 40).
constexpr int kKaiserTableElems = 4096;

// Compact per-space record used by the binning passes (64 bytes).  t0/t2 are rows 0 and 2
// of transformInv: t0.p is the image x of voxel offset p, t2.p its distance from the
// projection plane.  lo/hi are the traversal-AABB limits on the two axes the reference's
// traversal constrains for this direction (fr_cpu_kernels.hpp:166-238); the third axis is
// left open.  All thresholds carry a small outward margin so the test is conservative.
struct SpacePrep {
  float t0[3];
  float maxDist2;
  float t2[3];
  float halfWidth;
  int lo[3];
  int dir;
  int hi[3];
  float xMin;
};
static_assert(sizeof(SpacePrep) == 64, "SpacePrep is 64 bytes");

// Per-space record read by the insertion kernel (128 bytes = eight 16-byte loads), built
// once per space by the binning prep pass.  The axes U, V are the traversal plane of the
// space's direction and W its column axis (XY: x, y | z;  XZ: x, z | y;  YZ: y, z | x).
//  - T, maxDist2, weight, proj: as in the TraverseSpace (the voxels' part, three loads).
//  - lo0/hi0/lo1/hi1: the traversal AABB on U and V (fr_cpu_kernels.hpp:166-238), as floats
//    (clamped to 2^24, beyond every volume).
//  - w0, wu, wv, hw (blob mode): the slab |t2.(q - c)| <= r crosses column (U, V) at
//    W = w0 + wu U + wv V with half-width |hw| along W (plus a margin).  A voxel contributes
//    only if its float |t2.(q - c)| <= r, and the reference's column range
//    [floor(min(z1,z2)), ceil(max(z1,z2))] always contains every such voxel, so visiting
//    [ceil(wc - hw), floor(wc + hw)] instead yields the same contributing voxels.
//  - h0, hu, hv (blob mode): a voxel contributes only if its image x' = t0.(q - c) >= -r, which
//    bounds column (U, V) at W = h0 + hu U + hv V: from below where hw is positive, from
//    above where it is negative; h0 = -1e30 where t0 has no component along W.  sphere = maxDist2.
//  - nu, nv, nw, bu, bv, bw (nearest mode): the plane normal and bottom origin on U, V, W,
//    for the reference's exact rounded plane hit.
struct SpaceRec {
  float T[9];
  float maxDist2;
  float weight;
  int proj;
  float lo0, hi0, lo1, hi1;
  float w0, wu, wv, hw;
  float h0, hu, hv, sphere;
  float nu, nv, nw, bu, bv, bw;
  int pad[2];
};
static_assert(sizeof(SpaceRec) == 128, "SpaceRec is 128 bytes");

// One unit of insertion work: a brick and a range [begin, end) of its binned list; in a
// batched launch also the job the brick belongs to.
struct WorkItem {
  int brick;
  int begin;
  int end;
  int job;
};

// One job of a batched launch (128 bytes): its payloads, sizes, brick grid and the offsets
// of its traverse spaces and bricks in the batch-wide arrays.
struct JobDesc {
  const void *fft;
  const float *scales;
  void *volume;
  float *weight;
  int nProj, fftX, fftY, vx;
  int vy, vz, nbx, nby;
  int nbz, cx, cy, cz;
  int genericTaps, spaceBase, nSpaces, brickBase;
  int nBricks, groupBase;              // bricks; first binning CTA of the job (bin_groups)
  const fr_traverse_space *spaces;     // the job's traverse spaces (device memory)
  const void *src;                     // the caller's row-major half-planes (fft: their bands)
  int bandStride;                      // elements per 4-row band of fft
  int unitBase;                        // the job's first band in the batch's band copy
};
static_assert(sizeof(JobDesc) == 128, "JobDesc is 128 bytes");

// ------------------------------------------------------------------------------------
// Exact-rounding helpers.  The reference's geometry is evaluated without fused
// multiply-adds (its ISO-mode host build); the helpers keep nvcc from contracting them so
// slab bounds and blob boxes round the same way.
// ------------------------------------------------------------------------------------
__device__ __forceinline__ float mul_(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float add_(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float sub_(float a, float b) { return __fsub_rn(a, b); }

// Plane intersection along one axis: from n.(q - p0) = 0 solve for the free coordinate
// (libumpalumpa/math/geometry.hpp:11-33).  (u, v) are the two fixed coordinates, nu/nv
// their normal components, nw the normal component of the solved axis.
__device__ __forceinline__ float plane_hit(float u, float v, float nu, float nv, float nw,
  float pu, float pv, float pw)
{
  float a = mul_(-nu, sub_(u, pu));
  float b = mul_(nv, sub_(v, pv));
  return add_(__fdiv_rn(sub_(a, b), nw), pw);
}

__device__ __forceinline__ float clampf_(float v, float lo, float hi)
{
  float r = (v > hi) ? hi : v;
  return (r < lo) ? lo : r;
}

// ------------------------------------------------------------------------------------
// Bessel functions.  I0/I1 by the polynomial approximations of Abramowitz & Stegun
// 9.8.1-9.8.4 and I2..I4 by upward recurrence -- the reference's choice
// (libumpalumpa/math/bessier.hpp:9-63 in double; fr_common_kernels.hpp:55-127 in float).
// The double forms use explicit round-to-nearest operations in the reference's
// evaluation order so the blob table matches the reference's host table.
// ------------------------------------------------------------------------------------
__device__ __forceinline__ double dm(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double da(double a, double b) { return __dadd_rn(a, b); }

__device__ inline double bessel_i0_d(double x)
{
  double ax = fabs(x);
  if (ax < 3.75) {
    double t = x / 3.75;
    t = dm(t, t);
    double p = 0.45813e-2;
    p = da(0.360768e-1, dm(t, p));
    p = da(0.2659732, dm(t, p));
    p = da(1.2067492, dm(t, p));
    p = da(3.0899424, dm(t, p));
    p = da(3.5156229, dm(t, p));
    return da(1.0, dm(t, p));
  }
  double t = 3.75 / ax;
  double p = 0.392377e-2;
  p = da(-0.1647633e-1, dm(t, p));
  p = da(0.2635537e-1, dm(t, p));
  p = da(-0.2057706e-1, dm(t, p));
  p = da(0.916281e-2, dm(t, p));
  p = da(-0.157565e-2, dm(t, p));
  p = da(0.225319e-2, dm(t, p));
  p = da(0.1328592e-1, dm(t, p));
  p = da(0.39894228, dm(t, p));
  return dm(exp(ax) / sqrt(ax), p);
}

__device__ inline double bessel_i1_d(double x)
{
  double ax = fabs(x), r;
  if (ax < 3.75) {
    double t = x / 3.75;
    t = dm(t, t);
    double p = 0.32411e-3;
    p = da(0.301532e-2, dm(t, p));
    p = da(0.2658733e-1, dm(t, p));
    p = da(0.15084934, dm(t, p));
    p = da(0.51498869, dm(t, p));
    p = da(0.87890594, dm(t, p));
    p = da(0.5, dm(t, p));
    r = dm(ax, p);
  } else {
    double t = 3.75 / ax;
    double q = __dsub_rn(0.1787654e-1, dm(t, 0.420059e-2));
    q = da(-0.2895312e-1, dm(t, q));
    q = da(0.2282967e-1, dm(t, q));
    double p = da(-0.1031555e-1, dm(t, q));
    p = da(0.163801e-2, dm(t, p));
    p = da(-0.362018e-2, dm(t, p));
    p = da(-0.3988024e-1, dm(t, p));
    p = da(0.39894228, dm(t, p));
    r = dm(p, exp(ax) / sqrt(ax));
  }
  return x < 0.0 ? -r : r;
}

__device__ inline double bessel_in_d(int order, double x)
{
  if (order == 0) return bessel_i0_d(x);
  if (order == 1) return bessel_i1_d(x);
  if (x == 0) return 0;
  double im1 = bessel_i0_d(x), i = bessel_i1_d(x);
  for (int k = 1; k < order; ++k) {
    double nx = __dsub_rn(im1, dm((2.0 * k) / x, i));
    im1 = i;
    i = nx;
  }
  return i;
}

// The dynamic blob for alpha <= 15 (fr_common_kernels.hpp:163-170: bessi0Fast(alpha sqrt(1 - d2/r^2))
// / I0(alpha) * cIw0) for two taps at once, for the insertion's tap pairs: a polynomial of degree
// kKaiserDegree in u = 1 - d2/r^2 by Horner's rule in packed FP32x2.  The weight is a power series
// in u (I0(alpha sqrt u) = sum (alpha^2 u / 4)^k / (k!)^2), so no square root and no quotient is
// needed; kaiser_polynomial (fr_capi.cu) interpolates it in FP64 for the settings' alpha.  At
// alpha 15, evaluated in FP32 over d2 in [0, r^2]: 1.5e-7 relative L2, 3.8e-7 of the peak and
// 1.5e-6 relative at most, against 2.2e-7, 5.7e-7 and 3.0e-6 for the rational approximation of Blair
// & Edwards (the reference's bessi0Fast) with a fast divide, which took 27 instructions and two
// reciprocals per pair instead of 13 (box 256 x 6,000: 14.4 -> 12.6 ms).
// A tap beyond r^2 gets a meaningless value; the caller does not use it.
__device__ __forceinline__ float2 kaiser_poly2(float2 d2, float2 negInvR2, const float2 (&c)[kKaiserDegree + 1])
{
  const float2 u = __ffma2_rn(d2, negInvR2, make_float2(1.f, 1.f));
  float2 h = c[kKaiserDegree];
#pragma unroll
  for (int k = kKaiserDegree - 1; k >= 0; --k) h = __ffma2_rn(h, u, c[k]);
  return h;
}

// ------------------------------------------------------------------------------------
// Projection storage: complex64, or 2 x 16-bit complex with a per-projection scale.
// ------------------------------------------------------------------------------------
template<int STORAGE> struct Pixel;

template<> struct Pixel<FR_STORAGE_FP32> {
  using T = float2;
  static constexpr int kBytes = 8;
  __device__ __forceinline__ static float2 load(const T *p) { return __ldg(p); }
};

template<> struct Pixel<FR_STORAGE_BF16> {
  using T = __nv_bfloat162;
  static constexpr int kBytes = 4;
  // A BF16 value is the upper half of the FP32 one: the pair's low half (re) shifted up, the
  // high half (im) masked -- two integer operations (2.3 % faster insertion than the library
  // conversion at box 256).
  __device__ __forceinline__ static float2 load(const T *p)
  {
    const unsigned u = __ldg(reinterpret_cast<const unsigned *>(p));
    return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u));
  }
};

template<> struct Pixel<FR_STORAGE_FP16> {
  using T = __half2;
  static constexpr int kBytes = 4;
  __device__ __forceinline__ static float2 load(const T *p) { return __half22float2(__ldg(p)); }
};

}// namespace frb
