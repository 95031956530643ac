// Internal declarations shared by the CUDA translation units of
// libvoroffset_gpu.so. Not part of the public ABI (include/voroffset_gpu.h).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <functional>
#include <string>
#include <vector>

#include "voroffset_gpu.h"

namespace vo {

// Per-thread capacities of the in-register/local-memory working lists. A
// column that needs more is flagged and re-run by the large-capacity variant
// of the same kernel, whose lists live in global scratch.
constexpr int kCapSmall = 32;    // pass-1 touching-merged piece list / pass-2 union
constexpr int kScanExtra = 16;   // ints that a scan's synchronisation may read back besides its total
constexpr int kCapLarge = 2048;  // overflow re-run capacity per column

// Radius tables, computed on the host with the reference's own FP64
// expressions (so device results match bit for bit) and uploaded once per
// (radius, grid extent).
struct Tables {
  double R = 0;
  int Dy = 0;                 // max pass-1 lattice distance (floor(R))
  int W = 0;                  // Dx[0] + 1 (row stride of H)
  std::vector<double> r1;     // [Dy+1] pass-1 radius per label
  std::vector<int> Dx;        // [Dy+1] max |dx| per label
  std::vector<double> H;      // [(Dy+1)*W] sqrt(r1*r1 - dx*dx), NaN beyond Dx
  // FP32 rounding of H for patches of columns: rows 0 .. Dy + 2 kPatchY - 1 of
  // stride hs >= W + kPatchX + 2, -inf beyond the disc (the distances between
  // the columns of a patch and of a 4 x 4 tile within its reach). hs is 8 or 24 modulo 32,
  // so that the 4 rows of 8 consecutive entries that a warp reads fall into 32
  // different banks.
  int hs = 0;
  std::vector<float> Hp;
  std::vector<double> HB;     // [(Dy+1)^2] brute force sqrt(R*R - dx^2 - dy^2), NaN outside
};

// Device view of the tables (kernel argument by value).
struct DevTables {
  int Dy, W;
  const double *H;
  const int *Dx;
  const double *HB;
};

// Builds tables for radius R serving sweep indices 0..kmax-1; returns VO_OK,
// VO_EINVAL or VO_ERADIUS.
int build_tables(double R, int kmax, Tables &t);

constexpr int kDomLevels = 11;  // growths of H whose dominance masks are kept (15 in a pair record: none)
struct DomLevels {
  float t[kDomLevels];
};

struct DeviceTables {
  double R = -1;
  int kmax = 0;
  double *H = nullptr;
  float *Hp = nullptr;
  int *Dx = nullptr;
  double *HB = nullptr;
  // for the per-column kernel, made when it is first used (column_tables)
  float4 *prec = nullptr;
  int npairs = 0;
  DomLevels dom{};
  Tables host;
  DevTables view() const { return DevTables{host.Dy, host.W, H, Dx, HB}; }
};

}  // namespace vo

struct vo_volume {
  vo_grid grid;
  int64_t nseg = 0;      // host-known segment count
  // Whether some pair has z1 > z2 (an inverted pair left by complementing a
  // column whose values exceed [zmin, zmax]): 0 no, 1 yes, -1 not yet known.
  mutable int inverted = -1;
  int32_t *offs = nullptr;  // device [nx*ny+1]
  double2 *z = nullptr;     // device [nseg]
  bool owns = true;
  // Copies on the context's copy stream (vo_volume_upload_async /
  // vo_volume_download_async): `ready` completes when the upload has landed,
  // `copied` when the last download has left; null when none was made.
  mutable cudaEvent_t ready = nullptr, copied = nullptr;
};

struct vo_ctx {
  int device = 0;
  cudaStream_t stream = nullptr;
  cudaStream_t copy_stream = nullptr;  // asynchronous uploads and downloads
  cudaEvent_t ev_order = nullptr;      // orders the copy stream after the compute stream
  std::string err;
  std::vector<vo::DeviceTables *> tables;  // small cache keyed by (R, kmax)
  cudaEvent_t ev[8] = {};
  int launches = 0;  // kernel launches of the current call
  int ovf_cols = 0;
  // persistent small device scratch
  int *d_flags = nullptr;  // [0]: overflow count, [1..]: misc status
  long long *d_total = nullptr;
  long long *h_total = nullptr;  // pinned, written by the scan's kernels: its total, then up to kScanExtra ints
  vo_sizer *sizer = nullptr;     // learned sizing for the batched executor (not owned)
  int64_t dexel_odd_columns = -1;  // odd-hit columns of the last vo_dexelize (-1: none yet)
  std::vector<std::pair<long long, int>> tune_cache;  // batch autotuner: shape key -> lanes per column
};

namespace vo {

// Orders the context's stream after the asynchronous upload of v, if any (every
// entry point that reads a volume calls it first).
void vol_wait(vo_ctx *ctx, const vo_volume *v);

// Error helpers: set ctx->err and return a status.
int set_error(vo_ctx *ctx, int code, const std::string &msg);
int cuda_error(vo_ctx *ctx, cudaError_t e, const char *where);

#define VO_CK(ctx, call)                                 \
  do {                                                   \
    cudaError_t e_ = (call);                             \
    if (e_ != cudaSuccess) return vo::cuda_error((ctx), e_, #call); \
  } while (0)

// Stream-ordered allocation helpers on ctx->stream.
template <typename T>
int dalloc(vo_ctx *ctx, T **p, size_t n) {
  *p = nullptr;
  if (n == 0) n = 1;
  cudaError_t e = cudaMallocAsync((void **)p, n * sizeof(T), ctx->stream);
  if (e != cudaSuccess) return cuda_error(ctx, e, "cudaMallocAsync");
  return VO_OK;
}
void dfree(vo_ctx *ctx, void *p);

// Tables for radius R, cached in the context.
int get_tables(vo_ctx *ctx, double R, int kmax, const DeviceTables **out);

// Exclusive scan of int32 counts into int32 offsets (n+1 entries); the total
// is returned through ctx->h_total (synchronising read). Returns VO_ERANGE if
// the total exceeds INT32_MAX. With extra_n > 0 that many ints at extra_dev are
// read back by the same synchronisation.
// (at most kScanExtra). With `ends` the counts are ends[i] - counts[i].
int scan_counts(vo_ctx *ctx, const int32_t *counts, int32_t *offs, int n, long long *total,
                const int *extra_dev = nullptr, int *extra_host = nullptr, int extra_n = 0,
                const int32_t *ends = nullptr);
// The separable scheme in its sweeping envelope form, FP64 (vo_env.cu).
// Returns VO_OK, an error, or 1 when the volume exceeds the kernels' working
// capacities and must take the painter form (VO_METHOD_SEPARABLE).
int dilate_envelope(vo_ctx *ctx, double R, const vo_volume *in, vo_volume **out, vo_timings *tm);

// Exact FP32-guarded separable dilation (vo_fast.cu).
int dilate_fast(vo_ctx *ctx, double R, const vo_volume *in, vo_volume **out, vo_timings *tm);

// Rewrites inverted pairs as their two endpoints (points) and re-sorts / merges
// the affected columns (vo_morph.cu). *out is a new volume, or nullptr when
// `in` has no inverted pair.
int normalize_inverted(vo_ctx *ctx, const vo_volume *in, vo_volume **out);

// Morphology drivers (vo_morph.cu).
int dilate(vo_ctx *ctx, int method, double R, const vo_volume *in, vo_volume **out,
           vo_timings *tm);
int erode(vo_ctx *ctx, int method, double R, const vo_volume *in, vo_volume **out,
          vo_timings *tm);

// Slot volume: column c holds z[beg[c], end[c]). slot_alloc gives the
// fixed-capacity layout beg[c] = c*cap; a CSR volume is viewed as one with
// beg = offs, end = offs + 1; batch dilations write per-tile layouts. `cap`
// bounds every column's count, `entries` is the length of z.
struct SlotVol {
  vo_grid grid{};
  int cap = 0;
  int64_t entries = 0;
  int32_t *beg = nullptr, *end = nullptr;
  double2 *z = nullptr;
  bool owns = false;
};
int slot_alloc(vo_ctx *ctx, const vo_grid &g, int cap, SlotVol &v);
void slot_free(vo_ctx *ctx, SlotVol &v);
SlotVol slot_view(const vo_volume *in, int cap);
// Complement with a one-column border (negate), normalisation of inverted
// pairs, and complement back on the inner range (negate_inv), as launches into
// already allocated slot outputs (batch plans record them for graph capture).
void slot_negate_launch(cudaStream_t st, const SlotVol &in, const SlotVol &out, int *overflow);
void slot_normalize_launch(cudaStream_t st, const SlotVol &in, const SlotVol &out, int *overflow);
void slot_negate_inv_launch(cudaStream_t st, const SlotVol &in, const vo_grid &g, const SlotVol &out,
                            int *overflow);
int slot_max_count(vo_ctx *ctx, const SlotVol &v, int *d_max);
// CSR volume of a slot volume; extra_*: see scan_counts.
int slot_to_volume(vo_ctx *ctx, const SlotVol &v, vo_volume **out, const int *extra_dev = nullptr,
                   int *extra_host = nullptr, int extra_n = 0);

// Scalars of a dilation's FP32 arithmetic, from the range of its input
// (set_par in vo_fast.cu): FP32 values are relative to base, E is the guard
// band, 1 / inv_w the bin width, thr the least length of a long interval, and
// lo and hi bound the FP32 values (infinite ones are brought there).
struct FastPar {
  double base;
  float E, inv_w, thr;
  int nbins;
  float lo, hi;
  float q;  // bounds the error of a difference of two values less the base
};

// Columns of a warp of the FP32 kernel: a kPatchX x kPatchY patch, lane l at
// (l % kPatchX, l / kPatchX).
constexpr int kPatchX = 8, kPatchY = 4;

// Arguments of the FP32-guarded dilation of one volume (vo_fast.cu).
struct FastArgs {
  int nx, ny, W, Dy, hs;
  const int32_t *beg, *end;  // segments [beg[c], end[c]) of column c as given (CSR or slots)
  const double *zd;          // FP64 values as given
  // Packed by 4 x 4 tiles of columns (k_pack in vo_fast.cu): FP32 values
  // relative to FastPar::base, column in the tile (bits 24 .. 27) with widths (k_widths), FP64 values; the clusters
  // and their offsets [tile rows][tiles per row + 1].
  const float2 *zf;
  const uint2 *code;
  const double *zx;
  const float4 *cl;
  const int32_t *coff;
  const float *Hp;      // [(Dy + 2 kPatchY)][hs], -inf beyond the disc
  const double *H64;    // [(Dy + 1) * W]
  const int *Dx;        // [Dy + 1], then the growth of H over a step inwards (Tables::Dx)
  const FastPar *par;
  // small radii (k_widths): per segment what k_direct needs and its FP64 values, contiguous by rows;
  // [rbeg[c], rend[c]) of column c
  const uint4 *rec;
  const double2 *rz;
  const int32_t *rbeg, *rend;
  double off;  // value_offset of the grid
};

// Arguments of the per-column kernel for one volume (vo_column.cu).
struct ColumnArgs {
  int nx, ny, W, npairs, mask_bits, unused;
  const int32_t *beg, *end;  // segments [beg[c], end[c]) of column c (CSR or slots)
  const double *zd;          // FP64 values
  const float *zf;           // FP32 copies relative to FastPar::base
  const double *H64;         // [(Dy + 1) * W]
  const float4 *prec;        // pair records (column_pairs)
  const FastPar *par;
  // (beg, end, widths x- | x+ << 16, y- | y+ << 16 as FP16) per column
  const int4 *col;
  // Segment dominance masks [4 directions][kDomLevels][ncols] of mask_bits bits: bit j of a column with at most
  // mask_bits segments is set when its segment j lies in a neighbour segment widened by the level's threshold.
  const void *dmask;
};

constexpr int kSizerTile = 32;     // side of a sizing tile (columns)
constexpr int kUnionCap = 32;      // output slots per column of a batch dilation without a sizer
constexpr int kUnionCapMid = 128;  // most output slots per column of a sized tile
constexpr int kUnionLarge = 63;    // intervals of the first tiers' largest unions
// One dilation of a launch (device array element).
struct BatchVol {
  FastArgs A;
  int32_t *obeg, *oend;  // output slot arrays, written for every column
  double2 *oz;           // output values: tile slots, then the spill region
  const int32_t *tcap;   // per sizing tile capacity, or nullptr: `cap` for all
  const int32_t *toff;   // per sizing tile offset into oz
  int cap;
  int tiles32_x;
  int item0, item1;      // its patches in the launch's queue
  unsigned spill_base, spill_cap;
  unsigned *spill_used;
  int *big_list, *big_count;  // columns for the last tier (FP64)
  int *ovf;  // flags: 1 a union beyond the FP64 list, 4 spill region exhausted, 8 more unions beyond the lists than the tiers take
  // The per-column kernel: its arguments, and the columns for k_column_list: those with more intervals than it holds,
  // or those of the first tier that the caller lists there.
  const ColumnArgs *column;
  int *over_list, *over_count;
  // More columns (k_direct) or patches (k_patch) than this beyond the first tier's lists: the rest of the dilation
  // is left undone, for the caller to do it all by columns.
  int *listed, most;
  int *large;  // columns of the later tiers with more than kUnionLarge intervals
  // k_direct: kFewColumns lists of kPoolCap intervals for columns beyond its own, shared by the launch's dilations
  // (how many are taken: pool_used); nullptr: those columns are listed.
  double2 *pool;
  int *pool_used;
};
constexpr int kPoolCap = 1024;

// Masks of 16 bits per column and level where the input averages at most this many segments per column, else of
// 32; a column with more segments than bits takes part with all of them (2048^2 spheres + cylinders: 0.02 % of the
// columns have more than 16).
constexpr double kMask16MeanSegs = 8.0;

// Working memory of column_prepare.
struct ColumnPrep {
  int mask_bits = 16;
  float2 *zf = nullptr;
  int4 *col = nullptr;
  void *dmask = nullptr;
  FastPar *par = nullptr;
  unsigned long long *mm = nullptr;
};
// Allocates it for a grid with an input of `entries` segments (unused slots included), by alloc(pointer, bytes).
int column_alloc(const vo_grid &g, size_t entries, double mean_segs, const std::function<int(void **, size_t)> &alloc,
                 ColumnPrep &P);
ColumnArgs column_args(int nx, int ny, const DeviceTables &T, const int32_t *beg, const int32_t *end, const double2 *z,
                       const ColumnPrep &P);
void column_prepare(cudaStream_t st, const ColumnArgs &A, float R, const DomLevels &L, const ColumnPrep &P);
// The launch over the nv dilations vols, items as patches (patch_count with split 1), and the one over the columns
// that they list. A: of the first one.
int column_slots(double mean_segs);
void column_launch(cudaStream_t st, const BatchVol *vols, int nv, int blocks, int slots, const ColumnArgs &A);
void column_list_launch(cudaStream_t st, const BatchVol *vols, int nv);
// A radius' pair records and dominance levels (DeviceTables::prec, ::dom).
std::vector<float4> column_pairs(const Tables &h, DomLevels &L);
int column_tables(vo_ctx *ctx, const DeviceTables *T);
// Whether a dilation by that radius is to take the per-column kernel first: where the sizes leave it open, a sample of
// the input, there after ready(), decides (synchronising).
int column_choice(vo_ctx *ctx, const vo_grid &g, const DeviceTables &T, double mean_segs, const int32_t *beg,
                  const int32_t *end, const double2 *z, const std::function<void()> &ready, bool *columns);

// Queue of a launch. count: the first tier's next item, the items it listed
// for the second tier, that tier's next one, columns of the listed items.
struct PatchQueue {
  int *count = nullptr, *list = nullptr;
};
// Global working memory of a tier's warps.
struct PatchScratch {
  float2 *sv = nullptr;
  int2 *ids = nullptr;
  float2 *cv = nullptr;
  int2 *cids = nullptr;
  float4 *shorts = nullptr;
};
// A launch and its second tier (index 1).
struct PatchPlan {
  int nitems = 0, split = 1, hs_max = 0, grid[2] = {0, 0};
  PatchQueue Q;
  PatchScratch scratch[2];
};
// Lanes per column for a launch over the given grids (1, or more for small
// ones), and the patches of a grid with that many.
int patch_split(const vo_grid *const *grids, int n);
// Small radii: whether a dilation meets its candidates column by column
// (k_direct; its prepared inputs are not needed then), the launch over the nv
// dilations vols and its blocks for a grid. launch_cols: columns of all of them;
// shift: whether one of them has an offset (FastArgs::off).
bool direct_choice(const vo_grid &g, const DeviceTables &T, double mean_segs);
double reach_columns(const vo_grid &g, const DeviceTables &T);  // source columns in reach of a column, on average
int direct_blocks(const vo_grid &g, int64_t launch_cols);
size_t direct_smem(const FastArgs &A);
void direct_launch(cudaStream_t st, const BatchVol *vols, int nv, int blocks, int64_t launch_cols, size_t smem, bool shift);
int64_t patch_total(const vo_grid *const *grids, int n);  // with one lane per column
int patch_count(const vo_grid &g, int split);
// Grids of a launch over nitems patches; the working memory of each tier is
// given by patch_scratch_bytes / patch_scratch_set.
int patch_plan(vo_ctx *ctx, int nitems, int split, int hs_max, PatchPlan &P);
size_t patch_scratch_bytes(const PatchPlan &P, bool big);
void patch_scratch_set(PatchPlan &P, bool big, void *mem);
void patch_launch(bool big, const PatchPlan &P, cudaStream_t st, const BatchVol *vols);
// Last tier (FP64) over the dilations vols[0..nv), with unions of up to `cap` intervals; scratch holds
// big_scratch_elems(blocks, cap) of them. big_blocks: for up to so many columns.
int big_blocks(int64_t columns);
size_t big_scratch_elems(int blocks, int cap);
void big_launch(cudaStream_t st, const BatchVol *vols, int nv, double2 *scratch, int blocks, int cap);
// Outputs of the packing step, each as long as the input's segment array
// (with its unused slots), coff pack_offsets(grid).
struct PackOut {
  float2 *zf = nullptr;
  uint2 *code = nullptr, *wide = nullptr;  // wide: widths in the input's order (k_widths)
  double2 *zx = nullptr;
  float4 *cl = nullptr;
  int32_t *coff = nullptr;
  FastPar *par = nullptr;
  uint4 *rec = nullptr;     // small radii: instead of all the others; for slots zx and rbeg (2 x columns) too
  int32_t *rbeg = nullptr;
};
size_t pack_offsets(const vo_grid &g);
// Prepares the input of k_direct (pk.rec).
void direct_prepare(cudaStream_t st, const FastArgs &A, const PackOut &out);
FastArgs fast_args(const vo_grid &g, const DeviceTables &T, const int32_t *beg, const int32_t *end, const double2 *z,
                   const PackOut &out);
// Packs the input of a dilation (CSR or slots in column order). mm: four words of scratch.
void fast_prepare(cudaStream_t st, const FastArgs &A, float R, double mean_segs, unsigned long long *mm,
                  const PackOut &out);

// What a launch of one of them is like: lanes that share a column, union slots per column, registers per thread.
struct KernelShape {
  int lanes = 0, slots = 0, regs = 0;
};
KernelShape patch_shape(int split);
KernelShape direct_shape(int64_t launch_cols, bool shift);
KernelShape column_shape(int slots, bool single);

// Which kernel a dilation takes first: k_direct, k_patch or k_column.
enum class Engine { kDirect, kPatches, kColumns };
constexpr int kFewColumns = 4096;  // columns beyond k_direct's list up to which the FP64 tier takes them as they are
constexpr int kFewPatches = 608;   // patches that the patch kernel's second tier takes (eight rounds of its warps)

// Batch plans (vo_batch.cu).
int morph_batched_fast(vo_ctx *ctx, int n, const int *ops, const double *radii, const vo_volume *const *ins,
                       vo_volume **outs, vo_timings *tm);

// Learned sizing (vo_sizer.cu): tile features of a slot volume into a device
// array of ntiles x VO_SIZER_FEATURES, and predictions (ntiles x 4, three used).
int sizer_features_device(vo_ctx *ctx, const SlotVol &in, double radius, float *feats, int *ntiles);
int sizer_predict_device(vo_ctx *ctx, const vo_sizer *s, const float *feats, int n, float *out4);

// A value near those of a volume over the grid, from its origin: 0 below the magnitude from which taking it off pays
// (1024^2 spheres, r = 32, at 1e4: 3.83 ms without and 4.02 with it, at 1e5 4.17 and 4.01). It only makes filters
// sharper, never decides a result.
inline double value_offset(const vo_grid &g) {
  const double z = g.origin[2] / g.spacing;
  return z >= 32768.0 || z <= -32768.0 ? (z >= 1e15 || z <= -1e15 ? 0.0 : (double)(long long)z) : 0.0;
}

// Volume allocation (vo_api.cu).
int volume_alloc(vo_ctx *ctx, const vo_grid &g, int64_t nseg, vo_volume **out);

#ifdef __CUDACC__
// Output slot of column (x, y) for an n-interval union: the column's own slot
// when its capacity allows, else spill space, else false (the dilation's
// overflow flag is then set). Slot indices are unsigned 32-bit.
static __device__ __forceinline__ bool place_union(const BatchVol &V, int x, int y, int n, unsigned &dst) {
  const int nx = V.A.nx;
  int cap = V.cap;
  if (V.tcap) {
    const int tx = x / kSizerTile, ty = y / kSizerTile, t = tx + V.tiles32_x * ty;
    const int w = min(kSizerTile, nx - tx * kSizerTile);
    cap = V.tcap[t];
    dst = (unsigned)V.toff[t] + (unsigned)(((x - tx * kSizerTile) + w * (y - ty * kSizerTile)) * cap);
  } else {
    dst = (unsigned)(x + nx * y) * (unsigned)cap;
  }
  if (n > cap) {
    const unsigned off = atomicAdd(V.spill_used, (unsigned)n);
    if (off + (unsigned)n <= V.spill_cap) {
      dst = V.spill_base + off;
      return true;
    }
    atomicOr(V.ovf, 4);  // spill region exhausted
    return false;
  }
  return true;
}

// The FP64 methods compare and select values far more often than they add them,
// and an FP64 comparison occupies the SM for as long as sixteen integer ones.
// So they hold ends as signed integers of the same order: the bit pattern, its
// lower 63 bits flipped for negative values, -0 as 0.
using Key = long long;
using Key2 = longlong2;
constexpr Key kKeyMin = -0x7fffffffffffffffll - 1, kKeyMax = 0x7fffffffffffffffll;

__device__ __forceinline__ Key key_of(double v) {
  const Key b = __double_as_longlong(v);
  const Key k = b ^ ((b >> 63) & 0x7fffffffffffffffll);
  return k == -1 ? 0 : k;  // -0
}
__device__ __forceinline__ double value_of(Key k) {
  return __longlong_as_double(k ^ ((k >> 63) & 0x7fffffffffffffffll));
}
__device__ __forceinline__ Key2 key2_of(double2 v) { return make_longlong2(key_of(v.x), key_of(v.y)); }
// A double's bits, or a key's value, as FP32, rounded towards zero (NaN beyond
// its range): integer operations only, within 2^-23 of the magnitude for normal
// values, 0 for smaller ones.
__device__ __forceinline__ float trunc32_bits(Key b) {
  const unsigned hi = (unsigned)(b >> 32), lo = (unsigned)b, e = hi & 0x7fffffffu;
  unsigned f = e < 0x38100000u ? 0u : ((e - 0x38000000u) << 3) | (lo >> 29);
  if (e >= 0x47f00000u) f = 0x7fc00000u;
  return __uint_as_float((hi & 0x80000000u) | f);
}
__device__ __forceinline__ float trunc32(Key k) { return trunc32_bits(k ^ ((k >> 63) & 0x7fffffffffffffffll)); }
// The same of the value less `off` (value_offset): FP32 margins are parts of the
// magnitude, and values far from zero leave none at all of a filter without it
// (1024^2 spheres, r = 5: 2.8 ms at z = 0, 6.2 at 1e6). The difference is within
// 2^-53 of itself, which the margins cover. Without an offset, integer operations only.
__device__ __forceinline__ float trunc32_bits(Key b, double off) {
  return trunc32_bits(off == 0.0 ? b : __double_as_longlong(__dsub_rn(__longlong_as_double(b), off)));
}
__device__ __forceinline__ float trunc32(Key k, double off) {
  return trunc32_bits(k ^ ((k >> 63) & 0x7fffffffffffffffll), off);
}
__device__ __forceinline__ Key kmax(Key a, Key b) { return a > b ? a : b; }
__device__ __forceinline__ Key kmin(Key a, Key b) { return a < b ? a : b; }

// Inserts [lo, hi] into a sorted list of n disjoint closed intervals, merging
// overlapping or touching ones. One function, not inlined: its callers use it
// in several places, and copies would crowd the instruction cache. Returns the
// position of the interval that now holds [lo, hi] (-1 beyond `cap`) and the
// list's new length.
static __device__ __noinline__ int2 union_insert_keys(Key2 *A, int n, int cap, Key lo, Key hi) {
  int l = 0, r = n;
  while (l < r) {
    const int m = (l + r) >> 1;
    if (A[m].y >= lo)
      r = m;
    else
      l = m + 1;
  }
  if (l == n || A[l].x > hi) {
    if (n >= cap) return make_int2(-1, n);
    for (int k = n; k > l; --k) A[k] = A[k - 1];
    A[l] = make_longlong2(lo, hi);
    return make_int2(l, n + 1);
  }
  int j = l;
  while (j + 1 < n && A[j + 1].x <= hi) ++j;
  A[l] = make_longlong2(kmin(A[l].x, lo), kmax(A[j].y, hi));
  if (j > l) {
    const int sh = j - l;
    for (int k = l + 1; k + sh < n; ++k) A[k] = A[k + sh];
    n -= sh;
  }
  return make_int2(l, n);
}

// Moves the columns' segments from src(c) to oz[ooffs[c] ..): a warp per 32
// columns, whose lanes share out the segments, so that few per column leave no
// lane idle and the writes are contiguous (a warp per column took 0.13 ms for
// 810,000 columns of 1.6 segments).
template <typename Src>
__device__ __forceinline__ void compact_columns(int ncols, const int32_t *__restrict__ ooffs,
                                                double2 *__restrict__ oz, Src src) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;
  if (c - lane >= ncols) return;
  const int off = ooffs[min(c, ncols)];
  const long long from = c < ncols ? reinterpret_cast<long long>(src(c)) : 0;
  // in 64 bits: totals reach 2^31 - 1, and the last turn's positions lie beyond
  const long long first = __shfl_sync(0xffffffffu, off, 0), end = ooffs[min(c - lane + 32, ncols)];
  for (long long k0 = first; k0 < end; k0 += 32) {
    const long long k = k0 + lane;
    int l = 0;  // the last column that starts at or before k (of those that do, the one with segments)
    for (int o = 16; o > 0; o >>= 1)
      if (__shfl_sync(0xffffffffu, off, l + o) <= k) l += o;
    const double2 *p = reinterpret_cast<const double2 *>(__shfl_sync(0xffffffffu, from, l));
    const long long at = k - __shfl_sync(0xffffffffu, off, l);
    if (k < end) oz[k] = p[at];
  }
}
#endif

}  // namespace vo
