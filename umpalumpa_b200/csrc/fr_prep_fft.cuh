// Fused input preparation for square images of side N = 64, 96, 128, 192, 256, 320 or 384: the
// real-to-complex 2D FFT and the reference's Fourier processing in one kernel that reads each
// image once and writes its finished half-plane once.
//
// The reference runs AFFT (batched cuFFT R2C, fourier_transformation/fft_cuda.cpp:92-95), whose
// spectra go to a buffer, and AFP (scaleFFT2DKernel, fourier_processing/fp_cuda_kernels.cu:9-61),
// which reads that buffer and writes a second one.  Here persistent CTAs take images in turn:
//   1. column pass: two adjacent image columns form one complex sequence z_y = I[y][2m] + i I[y][2m+1]
//      (one 8-byte load per point, 128 contiguous bytes per 16 lanes); its N-point DFT Z_m goes,
//      row by row, to the CTA's own scratch S[ky][m] (N rows of N/2 values, read back from L2).
//   2. row pass: the column spectra of row ky come out of the rows ky and N - ky of S,
//      C_2m = (Z_m[ky] + conj Z_m[N - ky]) / 2, C_2m+1 = (Z_m[ky] - conj Z_m[N - ky]) / 2i, and
//      their N-point DFT over x gives F[ky][kx] for all kx -- and with it, as the image is real,
//      F[N - ky][kx] = conj F[ky][N - kx]: N/2 - 1 row DFTs yield both halves.  The rows 0 and N/2,
//      whose column spectra are real, share one DFT (real and imaginary part) and are separated
//      afterwards.  The values are processed exactly like ScaleFFT2DCPU (fp_cpu_kernels.hpp:24-36,
//      crop / normalise / centre / row shift, each product rounded separately) and stored from the
//      registers, in the order of lanes that fills the rows' or the bands' sectors.  For 16-bit
//      storage they go back to S while the largest |re|, |im| is reduced, and a last pass quantises
//      them exactly like fr_quantize_projections.
// A DFT of N = 16 TT points is two steps with an exchange through shared memory between them
// (n = j + TT q, k = k1 + 16 k2): 16-point DFTs over q, twiddles e^{-2 pi i j k1 / N} from a table
// built in double precision on the host, TT-point DFTs over j.  A pass runs 16 DFTs.
//
// What bounds it: latency and instruction issue at the 16 warps per SM its registers allow (N = 256;
// the HBM floor, one read and one write, is 80 ns per image).  Measured per image, FP32 / BF16
// rows, against cuFFT and a processing pass: N = 64 13 / 19 (23 / 30) ns, 96 24 / 31 (78 / 90),
// 128 39 / 59 (79 / 99), 192 103 / 128 (211 / 254), 256 189 / 251 (329 / 436), 320 343 / 475
// (839 / 1010), 384 556 / 738 (1216 / 1474) -- and against the kernel before, which took row pairs first,
// separated and staged them in shared memory with four barriers a pass, 355 ns at N = 256.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "umpalumpa_fr.h"

namespace frb {
namespace prepfft {

// ---- small DFTs in registers ------------------------------------------------------------------

// cos and sin of 2 pi e / S at compile time: exact at the quarter turns, else the Taylor series
// of the angle reduced to at most a quarter turn, in double.
__host__ __device__ constexpr double series(double x, bool sine)
{
  double term = sine ? x : 1.0, sum = term;
  for (int k = sine ? 3 : 2; k < 30; k += 2) {
    term *= -x * x / double(k * (k - 1));
    sum += term;
  }
  return sum;
}

__host__ __device__ constexpr double turn_cos(int e, int s)
{
  e %= s;
  if (2 * e > s) e = s - e;                       // cos(-a) = cos a
  if (4 * e > s) return -turn_cos(s - 2 * e, 2 * s);  // cos(pi - a) = -cos a
  if (4 * e == s) return 0.0;
  return series(6.283185307179586476925287 * double(e) / double(s), false);
}

__host__ __device__ constexpr double turn_sin(int e, int s)
{
  e %= s;
  if (2 * e > s) return -turn_sin(s - e, s);
  if (4 * e > s) return turn_sin(s - 2 * e, 2 * s);
  if (4 * e == s) return 1.0;
  return series(6.283185307179586476925287 * double(e) / double(s), true);
}

__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
__device__ __forceinline__ float2 cmul(float2 a, float2 w)
{
  return make_float2(fmaf(a.x, w.x, -a.y * w.y), fmaf(a.x, w.y, a.y * w.x));
}

// a * e^{-2 pi i E / S}
template<int E, int S> __device__ __forceinline__ float2 rotate(float2 a)
{
  constexpr int e = E % S;
  if constexpr (e == 0) return a;
  else if constexpr (4 * e == S) return make_float2(a.y, -a.x);
  else if constexpr (2 * e == S) return make_float2(-a.x, -a.y);
  else if constexpr (4 * e == 3 * S) return make_float2(-a.y, a.x);
  else {
    constexpr float c = float(turn_cos(e, S)), s = float(-turn_sin(e, S));
    return make_float2(fmaf(a.x, c, -a.y * s), fmaf(a.x, s, a.y * c));
  }
}

template<int S> __device__ __forceinline__ void dft(float2 (&v)[S]);

// v[I] for compile-time loops
template<int A, int B, int N2, int K1> __device__ __forceinline__ void twiddle_column(float2 (&u)[A])
{
  if constexpr (K1 < A) {
    u[K1] = rotate<N2 * K1, A * B>(u[K1]);
    twiddle_column<A, B, N2, K1 + 1>(u);
  }
}

template<int A, int B, int N2> __device__ __forceinline__ void inner_dfts(float2 (&v)[A * B])
{
  if constexpr (N2 < B) {
    float2 u[A];
#pragma unroll
    for (int n1 = 0; n1 < A; ++n1) u[n1] = v[B * n1 + N2];
    dft<A>(u);
    twiddle_column<A, B, N2, 1>(u);
#pragma unroll
    for (int k1 = 0; k1 < A; ++k1) v[B * k1 + N2] = u[k1];
    inner_dfts<A, B, N2 + 1>(v);
  }
}

// A x B points, n = B n1 + n2, k = k1 + A k2: A-point DFTs over n1, twiddles, B-point DFTs over n2.
template<int A, int B> __device__ __forceinline__ void composite(float2 (&v)[A * B])
{
  inner_dfts<A, B, 0>(v);
  float2 o[A * B];
#pragma unroll
  for (int k1 = 0; k1 < A; ++k1) {
    float2 u[B];
#pragma unroll
    for (int n2 = 0; n2 < B; ++n2) u[n2] = v[B * k1 + n2];
    dft<B>(u);
#pragma unroll
    for (int k2 = 0; k2 < B; ++k2) o[k1 + A * k2] = u[k2];
  }
#pragma unroll
  for (int k = 0; k < A * B; ++k) v[k] = o[k];
}

// Forward DFT (e^{-2 pi i n k / S}) of S points in registers, natural order in and out.
template<int S> __device__ __forceinline__ void dft(float2 (&v)[S])
{
  if constexpr (S == 2) {
    const float2 a = v[0], b = v[1];
    v[0] = cadd(a, b);
    v[1] = csub(a, b);
  } else if constexpr (S == 3) {
    constexpr float h = float(turn_sin(1, 3));
    const float2 t = cadd(v[1], v[2]), d = csub(v[1], v[2]);
    const float2 m = __ffma2_rn(t, make_float2(-0.5f, -0.5f), v[0]);
    v[0] = cadd(v[0], t);
    v[1] = make_float2(fmaf(h, d.y, m.x), fmaf(-h, d.x, m.y));
    v[2] = make_float2(fmaf(-h, d.y, m.x), fmaf(h, d.x, m.y));
  } else if constexpr (S == 4) {
    const float2 a0 = cadd(v[0], v[2]), a1 = csub(v[0], v[2]), b0 = cadd(v[1], v[3]), b1 = csub(v[1], v[3]);
    v[0] = cadd(a0, b0);
    v[2] = csub(a0, b0);
    v[1] = make_float2(a1.x + b1.y, a1.y - b1.x);  // a1 - i b1
    v[3] = make_float2(a1.x - b1.y, a1.y + b1.x);  // a1 + i b1
  } else if constexpr (S == 5) {
    constexpr float c1 = float(turn_cos(1, 5)), c2 = float(turn_cos(2, 5));
    constexpr float s1 = float(turn_sin(1, 5)), s2 = float(turn_sin(2, 5));
    const float2 t1 = cadd(v[1], v[4]), t2 = cadd(v[2], v[3]), d1 = csub(v[1], v[4]), d2 = csub(v[2], v[3]);
    const float2 m1 = __ffma2_rn(t2, make_float2(c2, c2), __ffma2_rn(t1, make_float2(c1, c1), v[0]));
    const float2 m2 = __ffma2_rn(t2, make_float2(c1, c1), __ffma2_rn(t1, make_float2(c2, c2), v[0]));
    const float2 n1 = __ffma2_rn(d2, make_float2(s2, s2), __fmul2_rn(d1, make_float2(s1, s1)));
    const float2 n2 = __ffma2_rn(d2, make_float2(-s1, -s1), __fmul2_rn(d1, make_float2(s2, s2)));
    v[0] = cadd(v[0], cadd(t1, t2));
    v[1] = make_float2(m1.x + n1.y, m1.y - n1.x);
    v[4] = make_float2(m1.x - n1.y, m1.y + n1.x);
    v[2] = make_float2(m2.x + n2.y, m2.y - n2.x);
    v[3] = make_float2(m2.x - n2.y, m2.y + n2.x);
  } else if constexpr (S % 4 == 0) {
    composite<4, S / 4>(v);
  } else {
    static_assert(S == 6, "2, 3, 4, 5, 6 or a multiple of 4 points");
    composite<2, 3>(v);
  }
}

// ---- the kernel -------------------------------------------------------------------------------

struct Args {
  const float *images;   // [n][N][N]
  int n;
  float2 *scratch;       // per CTA: [l2Rows][pitch]
  const float2 *tw;      // [16][N / 16]: e^{-2 pi i j k1 / N}
  int outX, outY;
  int normalize, center, shift, crop;
  float maxFreq, norm;
  void *out;             // [n][outY][outX] in the storage type, or n banded planes
  float *scales;
  int bandStride;        // banded output: elements per 4-row band (frb::band_stride); rows: 0
  int64_t outPlane;      // elements per output plane
};

// Idx2Freq (fourier_processing/fp_common_kernels.hpp:13-20)
__device__ __forceinline__ float idx2freq_(int idx, int size)
{
  if (size <= 1) return 0.f;
  const float t = idx <= size / 2 ? float(idx) : __fsub_rn(float(idx), float(size));
  return __fdiv_rn(t, float(size));
}

template<int N> struct Side { static constexpr int value = N; };

template<int N> struct Shape {
  static constexpr int TT = N / 16;
  static constexpr int threads = 16 * (TT > 16 ? TT : 16);  // both steps of a pass in one go
  static constexpr int pitch = N / 2 + 4;                   // scratch row (16-bit storage: N/2 + 1 values)
  static constexpr int rowBuf = 16 * (TT + 1) + 4;          // exchange of one row DFT: 4 rows x 4 lanes conflict-free
  static constexpr int buf = 16 * (rowBuf > 16 * TT ? rowBuf : 16 * TT);
  static constexpr int ctas = N <= 64 ? 6 : N <= 128 ? 4 : N <= 192 ? 3 : N <= 256 ? 2 : 1;  // per SM
  // The first rows of S, sixteen at a time, live in the shared memory the exchange leaves free
  // under a carve-out of 164 KB; the rest of S, of all CTAs, has to stay in L2 beside the images
  // that stream through.  N = 256: 189 ns per image, 202 with all rows in L2, 200 with a carve-out of
  // 228 KB, whose L1 is too small for the row pass.
  static constexpr int room = 164 * 1024 / ctas - 1024 - 128 - int((N + buf + N) * sizeof(float2));
  static constexpr int fit = room > 0 ? room / int(16 * pitch * sizeof(float2)) : 0;
  static constexpr int smemRows = 16 * (fit < TT ? fit : TT);
  static constexpr int l2Rows = N - smemRows;
  static constexpr size_t smem = (size_t(N + buf + N) + size_t(smemRows) * pitch) * sizeof(float2);
  // Whether the next columns' points are loaded during a pass: they fit the registers beside it
  // (128 and more per thread) from N = 256 on (208 -> 189 ns); below, they spill or cost a CTA
  // (N = 128: 39 -> 47 ns).
  static constexpr bool ahead = N >= 256;
};

// CTAs an image is split between in a call of few images: FP32 sides from 192 on, where one CTA per
// image is slower than cuFFT up to 2 (192), 8 (256) or 12 images (320, 384).  It is the latency of the
// passes' N / 32 rounds, which the CTAs of a cluster share: 1, 8, 32 and 37 images of side 320 take 19,
// 19, 21 and 33 us (one CTA each 51; cuFFT 43, 48, 64 and 68), of side 384 21, 21, 23 and 41 (70; 56,
// 62, 86 and 88); 1, 32 and 74 of side 256 12, 13 and 25 (35; 29, 38 and 45); 1, 32 and 111 of side 192
// 11, 12 and 22 (25 to 27; 23, 27 and 41).  At the smaller sides, and with 16-bit output, one CTA per
// image is faster than cuFFT at every number of images (side 128 14.5 against 16.5 us, BF16 side 384 92
// against 106).
constexpr int kSplit = 4;
template<int N, int STORAGE> constexpr bool kSplits = N >= 192 && STORAGE == FR_STORAGE_FP32;

template<int N, int SPLIT> constexpr int kNearRows = SPLIT > 1 ? 0 : Shape<N>::smemRows;
template<int N, int SPLIT> constexpr size_t kSmem =
  Shape<N>::smem - size_t(Shape<N>::smemRows - kNearRows<N, SPLIT>) * Shape<N>::pitch * sizeof(float2);

// BANDED: FP32 output in bands (16-bit output takes its layout in the last pass).
// SPLIT > 1: clusters of SPLIT CTAs take one image each (gridDim.x = SPLIT n), all of S in L2, the
// rounds of the passes dealt between the CTAs; the values are the same bit for bit.
template<int N, int STORAGE, bool BANDED, int SPLIT>
__global__ void __launch_bounds__(Shape<N>::threads, Shape<N>::ctas) prep_fft_kernel(Args a)
{
  static_assert(SPLIT == 1 || STORAGE == FR_STORAGE_FP32, "the CTAs of an image share no maximum");
  using Sh = Shape<N>;
  constexpr int nearRows = kNearRows<N, SPLIT>;
  const int group = int(blockIdx.x) / SPLIT, groups = int(gridDim.x) / SPLIT;
  const int first = 16 * (int(blockIdx.x) % SPLIT);  // of the CTA's rounds, 16 columns or rows each
  constexpr int TT = Sh::TT, H = N / 2;
  extern __shared__ float2 sm[];
  float2 *tw = sm;            // [16][TT]
  float2 *buf = tw + N;
  float2 *edge = buf + Sh::buf;  // the DFT shared by the rows 0 and N/2
  float2 *near = edge + N;       // rows of S in shared memory, the others in L2
  __shared__ float red[Sh::threads / 32];
  const int tid = threadIdx.x;
  for (int i = tid; i < N; i += Sh::threads) tw[i] = a.tw[i];
  float2 *far = a.scratch + size_t(group) * (N - nearRows) * Sh::pitch;
  auto S = [&](int row) -> float2 * {
    return row < nearRows ? near + row * Sh::pitch : far + size_t(row - nearRows) * Sh::pitch;
  };
  const bool pairs = (reinterpret_cast<uintptr_t>(a.images) & 7) == 0;
  __syncthreads();

  for (int img = group; img < a.n; img += groups) {
    const float *I = a.images + size_t(img) * N * N;
    // ---- 1. column pass, 16 column pairs at a time, the next ones' points in flight
    const int m = tid & 15, cj = tid >> 4;
    float2 v[16];
    auto load_columns = [&](int m0) {
      const float *p = I + size_t(cj) * N + 2 * (m0 + m);
      if (pairs) {
#pragma unroll
        for (int q = 0; q < 16; ++q) v[q] = __ldcs(reinterpret_cast<const float2 *>(p + size_t(TT * q) * N));
      } else {
#pragma unroll
        for (int q = 0; q < 16; ++q)
          v[q] = make_float2(__ldcs(p + size_t(TT * q) * N), __ldcs(p + size_t(TT * q) * N + 1));
      }
    };
    if (Sh::ahead && cj < TT) load_columns(first);
    for (int m0 = first; m0 < H; m0 += 16 * SPLIT) {
      if (cj < TT) {
        if (!Sh::ahead) load_columns(m0);
        dft<16>(v);
#pragma unroll
        for (int k1 = 0; k1 < 16; ++k1)
          buf[(k1 * TT + cj) * 16 + m] = k1 ? cmul(v[k1], tw[k1 * TT + cj]) : v[0];
        if (Sh::ahead && m0 + 16 * SPLIT < H) load_columns(m0 + 16 * SPLIT);
      }
      __syncthreads();
      if (tid < 256) {
        const int k1 = cj;
        float2 u[TT];
#pragma unroll
        for (int i = 0; i < TT; ++i) u[i] = buf[(k1 * TT + i) * 16 + m];
        dft<TT>(u);
#pragma unroll
        for (int k2 = 0; k2 < TT; ++k2) {
          if (16 * k2 < nearRows) near[(k1 + 16 * k2) * Sh::pitch + m0 + m] = u[k2];
          else far[(k1 + 16 * k2 - nearRows) * Sh::pitch + m0 + m] = u[k2];
        }
      }
      __syncthreads();
    }
    // the cluster's column spectra, written to global memory, before any of its CTAs reads them
    if (SPLIT > 1)
      asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    // the first columns of the CTA's next image, on their way to L2 during the row pass
    if (img + groups < a.n && tid < N)
      asm volatile("prefetch.global.L2 [%0];" ::"l"(I + size_t(groups) * N * N + size_t(tid) * N));
    // ---- 2. row pass, 16 rows ky (with their mirrors N - ky) at a time
    float amax = 0.f;
    // The processed value F[origY][x] (twice: the separations leave their halves out) of output
    // row y goes to element x of row_start(y, origY): ScaleFFT2DCPU's normalisation and centring
    // are one product -- the halves and signs are exact -- whose factor is the same for all of a
    // thread's values of a row and its mirror (x and y keep their parities).
    constexpr int kStep = BANDED ? 4 : 1;
    float2 *const O = static_cast<float2 *>(a.out) + size_t(img) * a.outPlane;
    auto row_start = [&](int y, int origY) -> float2 * {
      if (STORAGE != FR_STORAGE_FP32) return S(origY);  // its column spectra have been read whole
      const int t = y + a.outY / 2;
      const int row = a.shift ? (t >= a.outY ? t - a.outY : t) : y;
      return BANDED ? O + size_t(row >> 2) * a.bandStride + (row & 3) : O + size_t(row) * a.outX;
    };
    auto factor_of = [&](int x, int y) {
      const float f = a.normalize ? 0.5f * a.norm : 0.5f;
      return a.center && ((x + y) & 1) ? -f : f;
    };
    auto cropped = [&](int x, int origY) {
      const float fx = idx2freq_(x, N), fy = idx2freq_(origY, N);
      return __fadd_rn(__fmul_rn(fx, fx), __fmul_rn(fy, fy)) > a.maxFreq;
    };
    auto emit = [&](float2 w, float f, float2 *row, int origY, int x) {
      if (a.crop && cropped(x, origY)) w = make_float2(0.f, 0.f);
      w = make_float2(w.x * f, w.y * f);
      if (STORAGE == FR_STORAGE_FP32) {
        __stcs(row + kStep * x, w);
      } else {
        amax = fmaxf(amax, fmaxf(fabsf(w.x), fabsf(w.y)));
        row[x] = w;
      }
    };
    const int half = a.outY / 2;  // rows 0..half and N - (half - 1)..N - 1 are wanted
    for (int r0 = first; r0 < H && r0 <= half; r0 += 16 * SPLIT) {
      {
        const int r = tid / TT, j = tid - r * TT, ky = r0 + r;
        if (r < 16) {
          float2 v[16];
          const float2 *za = S(ky) + (j >> 1), *zb = S(ky ? N - ky : H) + (j >> 1);
          const bool odd = j & 1;  // x = j + TT q, TT even
#pragma unroll
          for (int q = 0; q < 16; ++q) {
            const float2 A = za[(TT / 2) * q], B = zb[(TT / 2) * q];
            if (ky == 0) v[q] = odd ? make_float2(A.y, B.y) : make_float2(A.x, B.x);
            else v[q] = odd ? make_float2(A.y + B.y, B.x - A.x) : make_float2(A.x + B.x, A.y - B.y);
          }
          dft<16>(v);
#pragma unroll
          for (int k1 = 0; k1 < 16; ++k1)
            buf[r * Sh::rowBuf + k1 * (TT + 1) + j] = k1 ? cmul(v[k1], tw[k1 * TT + j]) : v[0];
        }
      }
      __syncthreads();
      if (tid < 256) {
        // lanes: four rows x eight k1, so that eight columns of a band are stored whole
        const int r = (tid & 3) | (tid >> 6) << 2, k1 = (tid >> 2) & 15, ky = r0 + r;
        float2 u[TT];
#pragma unroll
        for (int i = 0; i < TT; ++i) u[i] = buf[r * Sh::rowBuf + k1 * (TT + 1) + i];
        dft<TT>(u);
        if (ky == 0) {
#pragma unroll
          for (int k2 = 0; k2 < TT; ++k2) edge[k1 + 16 * k2] = u[k2];
        } else {
          // columns kx <= N/2 of row ky, and of its mirror from kx >= N/2 (and 0)
          const float f = factor_of(k1, ky);
          float2 *const low = row_start(ky, ky), *const high = row_start(a.outY - ky, N - ky);
          if (ky <= half) {
#pragma unroll
            for (int k2 = 0; k2 <= TT / 2; ++k2) {
              const int x = k1 + 16 * k2;
              if (x <= H && x < a.outX) emit(u[k2], f, low, ky, x);
            }
          }
          if (ky < half) {
#pragma unroll
            for (int k2 = 0; k2 < TT; ++k2) {
              if (k2 > 0 && k2 < TT / 2) continue;
              const int kx = k1 + 16 * k2, x = kx ? N - kx : 0;
              if (x <= H && x < a.outX) emit(make_float2(u[k2].x, -u[k2].y), f, high, N - ky, x);
            }
          }
        }
      }
      __syncthreads();
      if (r0 == 0) {  // rows 0 and N/2 out of their common DFT
        for (int x = tid; x < a.outX; x += Sh::threads) {
          const float2 z = edge[x], zr = edge[x ? N - x : 0];
          emit(make_float2(z.x + zr.x, z.y - zr.y), factor_of(x, 0), row_start(0, 0), 0, x);
          if (half == H) emit(make_float2(z.y + zr.y, zr.x - z.x), factor_of(x, H), row_start(H, H), H, x);
        }
      }
    }
    if (STORAGE != FR_STORAGE_FP32) {
      for (int s = 16; s > 0; s >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, s));
      if ((tid & 31) == 0) red[tid >> 5] = amax;
      __syncthreads();
      float m = 0.f;
      for (int w = 0; w < Sh::threads / 32; ++w) m = fmaxf(m, red[w]);
      const float scale = m > 0.f ? m / 16384.f : 1.f;
      const float inv = 1.f / scale;
      if (tid == 0) a.scales[img] = scale;
      // four output rows at a time, eight loads in flight: a warp stores 2 x 32 columns of each
      // (rows) or of the band
      const int bands = (a.outY + 3) / 4, tiles = (a.outX + 63) / 64;
      const size_t base = size_t(img) * a.outPlane;
      for (int t = tid >> 5; t < bands * tiles; t += Sh::threads / 32) {
        const int b = t / tiles, x0 = 64 * (t - b * tiles) + (tid & 31);
        float2 w[2][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int row = min(4 * b + i, a.outY - 1);
          const int y = a.shift ? (row >= half ? row - half : row + half) : row;
          const float2 *src = S(y <= half ? y : N - (a.outY - y));
#pragma unroll
          for (int h = 0; h < 2; ++h) w[h][i] = src[min(x0 + 32 * h, a.outX - 1)];
        }
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int row = 4 * b + i, x = x0 + 32 * h;
            if (x >= a.outX || row >= a.outY) continue;
            const size_t d = base + (a.bandStride ? size_t(b) * a.bandStride + 4 * x + i : size_t(row) * a.outX + x);
            if (STORAGE == FR_STORAGE_BF16)
              static_cast<__nv_bfloat162 *>(a.out)[d] = __floats2bfloat162_rn(w[h][i].x * inv, w[h][i].y * inv);
            else
              static_cast<__half2 *>(a.out)[d] = __floats2half2_rn(w[h][i].x * inv, w[h][i].y * inv);
          }
      }
      __syncthreads();
    }
  }
}

}// namespace prepfft
}// namespace frb
