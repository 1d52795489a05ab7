// Internal interface between the host engine (fr_capi.cu) and the kernels (fr_kernels.cu).
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "umpalumpa_fr.h"

namespace frb {

struct SpacePrep;
struct SpaceRec;
struct WorkItem;
struct JobDesc;

// Brick grid over the volume and the reference's integer volume centre
// (cMaxVolumeIndex / 2, fr_cpu_kernels.hpp:34-36).
struct BinGeom {
  int vx, vy, vz;
  int nbx, nby, nbz, n_bricks;
  int cx, cy, cz;
};

// Scratch of one binning + insertion chunk.
// Kahan accumulation: the items of a brick that is cut for idle groups are summed in FP64 before
// the volume sees them, so that the cut leaves the sums as accurate as one item's (MergeBuffers.sums).
struct MergeBuffers {
  int *slot;     // [n_bricks] the brick's entry of `sums`, -1: not cut (nullptr: nothing is merged)
  int *left;     // [n_bricks] items of the brick still to come
  double *sums;  // [slots][3][kBrickVox] re, im, weight; zero between launches
  int slots;
};

struct BinBuffers {
  SpacePrep *prep;        // [chunk capacity]
  SpaceRec *rec;          // [chunk capacity]
  int *counts;            // [3 * n_bricks]; after the plan itemStart's memory
  int *offsets;           // [3 * n_bricks + 1]
  int *list;              // [listCap] space indices, grouped by (brick, direction)
  const int *order;       // [n_bricks] brick visiting order (heaviest expected first)
  WorkItem *items;        // [itemsCap]
  int *itemStart;         // [n_bricks] first work item of each brick
  int *nItems;            // [1]
  int *status;            // [1] sticky FR_E_* of device-side failures
  int *workCounter;       // [1] next work item of the insertion
  int *itemCap;           // [1] list entries per work item
  MergeBuffers merge;
  unsigned long long *stats;  // [4] pairs, items, chunks of the call
  int64_t listCap;
  int64_t itemsCap;
};

// How the plan cuts the binned lists into work items: at most `cap` list entries per item and,
// where `want` > 0, so few that the launch's brick groups get about `want` items between them,
// but at least `least` entries, and (`perBrick` > 0: Kahan accumulation) no brick is cut into more
// than `perBrick` items for it, and none without an entry of MergeBuffers.sums.
struct ItemSplit {
  int cap;
  int want;
  int least;
  int perBrick;
};

// The default item capacity.
constexpr int kItemCapacity = 512;
constexpr int kItemsPerGroup = 4;
constexpr int kFastItemsPerGroup = 1;  // nearest pixel: an entry costs a tenth of a blob entry

// Degree of the dynamic blob's polynomial (alpha <= 15).
constexpr int kKaiserDegree = 12;

struct InsertParams {
  const JobDesc *jobs;  // batched launches: the job table (the per-job fields below unused)
  void *volume;
  float *weight;
  const void *fft;
  const float *scales;
  const SpaceRec *recs;
  const int *list;
  const int *offsets;
  const WorkItem *items;
  const int *nItems;
  int *workCounter;
  MergeBuffers merge;
  const float *table;  // lookup: the blob table; dynamic: the Kaiser (value, slope) table
  int tableElems;      // entries (float2 entries for the Kaiser table)
  float tableScale;    // Kaiser table: nodes per unit of d^2, (N - 1) / r^2
  float2 kaiser[kKaiserDegree + 1];  // dynamic, alpha <= 15: kaiser_polynomial, each coefficient twice
  int lutInSmem;
  int genericTaps;  // bounds-checked taps with a clamped table index: half-plane narrower or
                    // shorter than the blob window, or a blob table above kLutSmemMax entries
  fr_constants c;
  int nProj;
  int fftX, fftY;
  int vx, vy, vz;
  int nbx, nby, nbz;
  int cx, cy, cz;
  int bandStride;  // banded half-planes: elements per 4-row band (band_stride); row-major: 0
};

// Which insertion kernel variant runs.
struct InsertConfig {
  int mode;     // 0 lookup table, 1 the blob's polynomial (alpha <= 15), 2 Kaiser of any order from
                // the interpolated (value, slope) table (alpha > 15)
  int taps;     // blob footprint per axis: floor(2 r) + 1
  bool fast;    // nearest-pixel insertion (Settings::Type::kFast)
  int storage;  // FR_STORAGE_*
  bool kahan;   // Kahan-compensated brick accumulators
  bool jobs;    // batched launch over a job table
  int groups;   // 256-thread groups per CTA (launch shape); 0 = the most that fit
  bool banded;  // half-planes in 4-row bands (always for a batch); else row-major
};

// The split of a launch of `brickGroups` groups (0: the capacity as given).
ItemSplit item_split(int itemCapacity, int brickGroups, const InsertConfig &cfg);

using InsertFn = void (*)(InsertParams);
// One insertion-kernel variant per storage type and layout, each in its own translation unit.
InsertFn pick_insert_fp32(const InsertConfig &cfg);
InsertFn pick_insert_bf16(const InsertConfig &cfg);
InsertFn pick_insert_fp16(const InsertConfig &cfg);
InsertFn pick_insert_band_fp32(const InsertConfig &cfg);
InsertFn pick_insert_band_bf16(const InsertConfig &cfg);
InsertFn pick_insert_band_fp16(const InsertConfig &cfg);
InsertFn pick_insert_batch_fp32(const InsertConfig &cfg);
InsertFn pick_insert_batch_bf16(const InsertConfig &cfg);
InsertFn pick_insert_batch_fp16(const InsertConfig &cfg);

// Coefficients, constant first, of the polynomial in u = 1 - d2 / r^2 that interpolates
// ks I0(alpha sqrt(u)), 0 < alpha <= 15 (cIw0, and so ks, is NaN for any other below).
void kaiser_polynomial(float alpha, float ks, float2 (&c)[kKaiserDegree + 1]);
// Dynamic interpolation's Kaiser (value, slope) table: kKaiserTableElems float2 entries.
cudaError_t launch_kaiser_table(float *table, int order, float alpha, float radius, float iw0, cudaStream_t st);
cudaError_t launch_blob_table(float *table, int64_t n, int order, float alpha, float radius,
  float iw0, cudaStream_t st);
cudaError_t launch_traverse_spaces(const float *rot, int64_t n, uint32_t imgX, uint32_t imgY,
  uint32_t maxVX, uint32_t maxVYZ, int useFast, float radius, float weight, int32_t first,
  fr_traverse_space *out, cudaStream_t st);
cudaError_t launch_traverse_spaces_sym(const float *rot, int64_t n, const float *sym, int nSym, uint32_t imgX,
  uint32_t imgY, uint32_t maxVX, uint32_t maxVYZ, int useFast, float radius, float weight, int32_t first,
  fr_traverse_space *out, cudaStream_t st);
cudaError_t launch_quantize(const void *in, int64_t n, int64_t elems, int storage, void *out, float *scales,
  cudaStream_t st);

// Banded half-planes: rows grouped in bands of four, each band stored column by column, the
// band pitch rounded up to 8 columns (whole 128-byte lines for 8- and 4-byte pixels).
__host__ __device__ inline int band_pitch(int fftX) { return (fftX + 7) & ~7; }
__host__ __device__ inline int band_stride(int fftX) { return 4 * band_pitch(fftX); }
__host__ __device__ inline int64_t band_plane_elems(int fftX, int fftY)
{
  return int64_t((fftY + 3) / 4) * band_stride(fftX);
}
// Copies n row-major half-planes [n][fftY][fftX] of elemBytes-byte pixels (8: complex64, 4: a
// 16-bit pair) into bands; padding columns and rows are written as zeros.
cudaError_t launch_band_projections(const void *src, void *dst, int64_t n, int fftX, int fftY, int elemBytes,
  cudaStream_t st);
// The same for every job of a batch: job j's projections go from its `src` to its `fft`, its
// bands numbered from its `unitBase` (totalUnits bands in all).
cudaError_t launch_batch_band(const JobDesc *jobs, int nJobs, int64_t totalUnits, int elemBytes, cudaStream_t st);
// Engine scratch's small words, one device block mirrored by one pinned host block.
constexpr int kMiscStatus = 1, kMiscStats = 4;  // word indices: status; stats (4 x 64 bits)
constexpr size_t kMiscBytes = 48;
void set_misc(BinBuffers &b, int *misc);
// Brick sums a Kahan call of this split can need (fewer than `want` bricks are longer than the
// total / want entries of an item), and their bytes.
inline int merge_slots(const ItemSplit &split, int64_t nBricks)
{
  return split.perBrick > 0 ? int(nBricks < split.want ? nBricks : split.want) : 0;
}
constexpr size_t kMergeSlotBytes = size_t(3) * 16 * 16 * 16 * sizeof(double);
// Sets the carve-out preference of the kernels that run beside one another (fr_create).
void prefer_shared_carveout();

// Binning and planning of one chunk of a call's spaces (`first`: its first chunk, which starts the
// call's statistics).  `split`: see ItemSplit.
cudaError_t launch_binning(const BinGeom &g, const fr_traverse_space *spaces, int n, int nProj,
  bool fast, float radius, const BinBuffers &b, const ItemSplit &split, bool first, cudaStream_t st);
// Brick rows of a volume the binning takes one CTA for (fr_binning.cuh, bin_row).
__host__ __device__ inline int bin_groups(int nbx, int nby, int nbz) { return (nbx + 31) / 32 * nby * nbz; }
// Binning of a batch: jobs (device job table, nJobs entries) with totalSpaces spaces,
// totalBricks bricks and totalGroups binning CTAs (bin_groups) in all.
cudaError_t launch_batch_binning(const JobDesc *jobs, int nJobs, int totalSpaces, int totalBricks,
  int totalGroups, bool fast, float radius, const BinBuffers &b, const ItemSplit &split, cudaStream_t st);
cudaError_t launch_insert(const InsertParams &P, const InsertConfig &cfg, int grid, cudaStream_t st);
size_t insert_smem_bytes(const InsertConfig &cfg, int tableElems);
cudaError_t allow_insert_smem(const InsertConfig &cfg);  // lets the kernel be launched with as much
int insert_groups(const InsertConfig &cfg);      // 256-thread groups per insertion CTA
int insert_max_groups(const InsertConfig &cfg);  // the most groups a CTA of this variant holds
// Whether the kernel's table goes to shared memory beside the launch's brick accumulators (a
// lookup table of at most kLutSmemMax entries, or the Kaiser table, with room left); else it
// is read from global memory.
bool insert_lut_in_smem(const InsertConfig &cfg, int tableElems);
const void *insert_kernel_ptr(const InsertConfig &cfg);

// Records `msg` as the calling thread's fr_last_error() and returns `code`.
int set_last_error(int code, const char *msg);

constexpr size_t kSpacePrepBytes = 64;
constexpr size_t kSpaceRecBytes = 128;
constexpr size_t kWorkItemBytes = 16;

}// namespace frb
