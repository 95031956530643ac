// Exact separable dilation with FP32 arithmetic and an FP64 guard
// (VO_METHOD_FAST, and the engine of batch plans).
//
// The separable scheme of the reference (VoronoiVorPower.cpp:24-96: a y-pass
// giving each z the nearest covering row distance d with radius
// r(d) = sqrt(R^2 - d^2), then an x-pass dilating by sqrt(r(d)^2 - dx^2))
// produces, per output column (x, y), the union of the candidate intervals
//     [z1 - H[|dy|][|dx|], z2 + H[|dy|][|dx|]]
// over the input segments [z1, z2] of every column (x+dx, y+dy) with
// |dx| <= Dx[|dy|], where H[d][a] = sqrt(r(d)*r(d) - a*a) is the reference's
// own FP64 value (pass-1 pieces are sub-intervals of these segments whose
// candidates tile them, so both unions are the same set, bit for bit).
//
// One warp computes an 8 x 4 patch of output columns (one per lane) in two
// sweeps over the clusters of source segments within reach, one per lane:
//
// 1. Cover. H at the patch column farthest from the source bounds H from
//    below for all 32 columns, so [z1 - Hmin, z2 + Hmin] is covered in every
//    one of them. The union of these intervals (the cover) is taken without
//    sorting: bins of the lower end hold the smallest lower and the largest
//    upper end of their intervals; intervals of at least a bin's width overlap
//    every other one of their bin, so a component ends exactly where the
//    running maximum of the upper ends stops short of the next bin's smallest
//    lower end. This sweep takes clusters whole: their segments' union is one
//    interval, and so it stays when every segment is widened by Hmin.
// 2. Filter and merge. A cluster, and then a segment, whose interval at the
//    nearest column (Hmax) lies inside one component of the cover cannot
//    change any of the 32 unions and is dropped (2048^2 spheres + cylinders,
//    r = 32, modelled: 2,083 clusters of 22,266 segments in reach of a patch;
//    393 clusters of 4,511 segments pass the first test, 3,001 segments the
//    second). So is one that the candidate of a neighbour between it and the
//    patch holds in every column (k_widths). The others are queued in shared memory, and each is merged by
//    all lanes at once, one column each: the lane looks up the bin of its
//    lower end and, only when the interval reaches beyond what its entry for
//    that bin holds, updates it. Entries (smallest lower and largest upper
//    end, per lane) exist only for bins that some queued segment can fall
//    into; bins wholly inside a component of the cover share one entry that
//    starts at the component's end.
//
// The segments are packed beforehand by 4 x 4 tiles of columns into clusters
// of up to 16 overlapping segments (k_pack), a surface patch typically: the
// sweeps then load contiguous records, one per lane, and no lane idles over
// columns of uneven counts.
//
// A last pass over the entries in bin order yields the union's intervals.
// Intervals shorter than a bin (near the rim of the disc) that their entry
// does not hold are kept aside and inserted into the finished union.
//
// Exactness: candidates are formed in FP32 (copies of the inputs relative to
// a base below them, and of H). E bounds the FP32 error of a comparison: the
// filter drops a segment only when it is inside by more than E, and every
// comparison of the merge within E is re-evaluated in FP64 from the
// candidates' identities (value index, d, a), kept beside each entry. Output
// endpoints are always recomputed in FP64 from their identities, so results
// are bit-identical to the FP64 oracle. Nothing in the cover enters a result:
// a segment that reaches a component's ends is never dropped but for a neighbour
// whose candidate holds its own, which then reaches them too; and being long they
// overlap the stretch that its shared entry stands for.
//
// What bounds it: dependent latency at 20 warps per SM, with half of the issue
// slots used (1024^2 spheres, r = 32: 3.1 ms, IPC 2.1, 27 of 32 lanes; 2048^2
// spheres + cylinders 21.6 ms, 3,098 warp instructions per column). A thread per
// column, with masks of the segments that a neighbour's candidate holds at each
// of eleven growths, took 26.9 and 183 ms. The bins' width is
// a power of two, so that binning is exact (one fused multiply-add that
// rounds to an integer).
//
// Small radii take another way (k_direct).
//
// Capacities: a patch that needs more entries, kept-aside intervals or union
// intervals than the launch has re-runs with larger lists (second tier), if those
// are few; if they are many their columns go to the per-column kernel
// (vo_column.cu), and if they are most, all of the dilation does: patches of
// scattered short intervals spend their time on intervals kept aside. A column
// that outgrows the larger lists too goes to an FP64 kernel with an
// 8,192-interval list.
#include <algorithm>
#include <cmath>
#include <cstddef>
#include <cstring>
#include <vector>

#include <cuda_fp16.h>

#include "vo_internal.cuh"
#include "vo_range.cuh"
#include "vo_slots.h"

namespace vo {
namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kCoverBins = 512;   // bins of the cover: the same, or two in one for inputs that use more
constexpr int kTile = 4;          // side of a source tile (columns), equal to the patch's height
constexpr int kGroup = 16;        // most segments of a cluster (half a warp)
constexpr int kPackSort = 4096;   // segments that a packing block sorts at a time (its warps share them evenly)
constexpr int kPairs = 3;         // pairs of clusters expanded at a time
constexpr int kQueue = 32 + 32 * kPairs;  // queued segments of a patch: flushed above 32
constexpr int kSplit = 4;         // lanes per column of the split form
constexpr int kPad = 4 * kSplit;  // padding of the queue
constexpr int kClusters = 96;     // clusters of a tile row to expand: expanded above 32
constexpr int kEntries = 512;     // entries of a patch (bins and components of the cover together)
constexpr int kComps = 63;        // components of the cover that are used
constexpr int kUnion = 64;        // union intervals per column, plus one
constexpr int kShort = 1024;      // kept-aside segments of a patch
constexpr int kEntriesBig = 1600; // the same for the second tier
constexpr int kUnionBig = 1024;
constexpr int kShortBig = 8192;
constexpr double kDirectWork = 450;            // candidates per column up to which k_direct takes a dilation
constexpr int64_t kDirectSplitCols = 1 << 16;  // columns of a launch up to which kSplit threads share one there
constexpr int kStep = 8;          // segments that k_direct loads at a time
constexpr int kPrepThreads = 256;
constexpr int kList = 16;         // intervals that it keeps at hand, unordered
constexpr int kHot = 2;           // intervals that each candidate is compared with at once
constexpr int kDirectCap = 48;    // union intervals per column there
constexpr int kBigCap = 8192;     // last tier (FP64): intervals of a column's working list
constexpr int kBigThreads = 32;
constexpr int kPatchBigBlocks = 76; // second tier: warps
static_assert(kTile == kPatchY && kPatchX % kTile == 0, "tiles and patches are aligned to each other");

// ------------------------------------------------------------ preparation

// Packs the segments by 4 x 4 tiles of columns into clusters: runs of at most
// kGroup segments, in order of their lower ends, whose union is one interval
// (each starts at or below the largest upper end so far). A block per row of
// tiles, a warp per tile. Tile row T's clusters and segments start at
// beg[first column of its first row], which leaves room for all of them in
// CSR and slot layouts alike. Written per cluster: (union's ends, first
// segment, count | tile << 5); per segment: FP32 values relative to the base,
// its column in the tile, and its FP64 values.
// A warp sorts up to kPackSort / WARPS segments, by counting for each those
// before it (a few dozen per tile); a tile of more keeps every segment a
// cluster. More warps for sparse inputs: a block's steps are chains of
// dependent loads, and what bounds it is how many tiles it has in flight.
template <int WARPS>
__global__ void __launch_bounds__(32 * WARPS) k_pack(int nx, int ny, const int32_t *__restrict__ beg,
                                                     const int32_t *__restrict__ end, const double2 *__restrict__ z,
                                                     const FastPar *__restrict__ par, float2 *__restrict__ zf,
                                                     const uint2 *__restrict__ wide, uint2 *__restrict__ code,
                                                     double2 *__restrict__ zx,
                                                     float4 *__restrict__ cl, int32_t *__restrict__ coff) {
  constexpr int CAP = kPackSort / WARPS;
  __shared__ __align__(16) int s_key[WARPS][CAP];  // bit patterns of the lower ends (none is negative)
  __shared__ float s_hi[WARPS][CAP];
  __shared__ unsigned short s_ord[WARPS][CAP];  // segment of rank r
  __shared__ unsigned char s_col[WARPS][CAP];
  __shared__ int s_src[WARPS][16];  // per column: its segments' index in z minus their position here
  __shared__ int s_ns[WARPS], s_nc[WARPS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tiles_x = (nx + kTile - 1) / kTile, T = blockIdx.x;
  const double base = par->base;
  const float least = par->lo, most = par->hi;
  auto in_fp32 = [=](double v) { return fminf(fmaxf(__double2float_rn(__dsub_rn(v, base)), least), most); };
  int seg0 = beg[T * kTile * nx], cl0 = seg0;  // next free segment and cluster of the tile row
  for (int t0 = 0; t0 < tiles_x; t0 += WARPS) {
    const int tx = t0 + warp;
    // two lanes per column: its segments alternate between them
    const int c4 = lane >> 1, x = tx * kTile + (c4 & 3), y = T * kTile + (c4 >> 2);
    int k0 = 0, n = 0;
    if (tx < tiles_x && x < nx && y < ny) {
      k0 = beg[x + nx * y];
      n = end[x + nx * y] - k0;
    }
    int pre = lane & 1 ? 0 : n;  // exclusive prefix over the columns
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(kFull, pre, o);
      if (lane >= o) pre += v;
    }
    const int m = __shfl_sync(kFull, pre, 31);
    pre -= n;  // both lanes of a column: the segments before it
    if (lane == 0) s_ns[warp] = m;
    const bool sort = m <= CAP;
    int nc = m;
    unsigned starts[CAP / 32];  // per 32 ranks: where the clusters start
    if (sort) {
      if ((lane & 1) == 0) s_src[warp][c4] = k0 - pre;
      for (int i = lane & 1; i < n; i += 2) {
        const double2 v = z[k0 + i];
        s_key[warp][pre + i] = __float_as_int(in_fp32(v.x));
        s_hi[warp][pre + i] = in_fp32(v.y);
        s_col[warp][pre + i] = (unsigned char)c4;
      }
      // padding up to the next 32: after every segment
      const int full = (m + 31) & ~31;
      if (m + lane < full) s_key[warp][m + lane] = 0x7fffffff;
      __syncwarp();
      for (int i0 = 0; i0 < m; i0 += 32) {
        const int v = i0 + lane < m ? s_key[warp][i0 + lane] : 0;
        int r = 0;
        for (int j0 = 0; j0 < full; j0 += 32) {
          // equal ends keep their order: earlier blocks count them, later ones do not
          if (j0 == i0) {
            for (int j = 0; j < 32; ++j) {
              const int u = s_key[warp][j0 + j];
              r += u < v || (u == v && j < lane) ? 1 : 0;
            }
          } else if (j0 < i0) {
#pragma unroll
            for (int j = 0; j < 32; j += 4) {
              const int4 u = *reinterpret_cast<const int4 *>(&s_key[warp][j0 + j]);
              r += (u.x <= v) + (u.y <= v) + (u.z <= v) + (u.w <= v);
            }
          } else {
#pragma unroll
            for (int j = 0; j < 32; j += 4) {
              const int4 u = *reinterpret_cast<const int4 *>(&s_key[warp][j0 + j]);
              r += (u.x < v) + (u.y < v) + (u.z < v) + (u.w < v);
            }
          }
        }
        if (i0 + lane < m) s_ord[warp][r] = (unsigned short)(i0 + lane);
      }
      __syncwarp();
      // where the clusters break: one step per segment, the same in every lane
      nc = 0;
      float hi = 0.f;
      int cnt = kGroup;
#pragma unroll
      for (int b = 0; b < CAP / 32; ++b) {
        starts[b] = 0;
        if (32 * b >= m) continue;
        const int i = s_ord[warp][min(32 * b + lane, m - 1)];
        const float va = __int_as_float(s_key[warp][i]), vb = s_hi[warp][i];
        const int e = min(32, m - 32 * b);
        for (int j = 0; j < e; ++j) {
          const float lo = __shfl_sync(kFull, va, j), up = __shfl_sync(kFull, vb, j);
          if (cnt == kGroup || !(lo <= hi)) {
            starts[b] |= 1u << j;
            cnt = 0;
            hi = up;
          }
          ++cnt;
          hi = fmaxf(hi, up);
        }
        nc += __popc(starts[b]);
      }
    }
    if (lane == 0) s_nc[warp] = nc;
    __syncthreads();
    int sb = seg0, seg_all = 0, cb = cl0, cl_all = 0;
    {
      int a = lane < WARPS ? s_ns[lane] : 0, c = lane < WARPS ? s_nc[lane] : 0;
      sb += __reduce_add_sync(kFull, lane < warp ? a : 0);
      cb += __reduce_add_sync(kFull, lane < warp ? c : 0);
      seg_all = __reduce_add_sync(kFull, a);
      cl_all = __reduce_add_sync(kFull, c);
    }
    if (tx < tiles_x && lane == 0) coff[(size_t)T * (tiles_x + 1) + tx] = cb;
    if (sort) {
      int g = cb;  // clusters before this block of ranks
#pragma unroll
      for (int b = 0; b < CAP / 32; ++b) {
        if (32 * b >= m) continue;
        const int r = 32 * b + lane;
        if (r < m) {
          const int i = s_ord[warp][r], col = s_col[warp][i];
          const float a = __int_as_float(s_key[warp][i]);
          zf[sb + r] = make_float2(a, s_hi[warp][i]);
          const uint2 w = wide[s_src[warp][col] + i];
          code[sb + r] = make_uint2(w.x | (unsigned)col << 24, w.y);
          zx[sb + r] = z[s_src[warp][col] + i];
          if (starts[b] >> lane & 1) {
            // the cluster's end: the next start, in this block of ranks or the next one
            const unsigned after = lane < 31 ? starts[b] >> (lane + 1) : 0u;
            int e = after ? r + __ffs(after) : 32 * (b + 1);
            if (!after && b + 1 < CAP / 32) e += starts[b + 1 < CAP / 32 ? b + 1 : b] ? __ffs(starts[b + 1 < CAP / 32 ? b + 1 : b]) - 1 : 32;
            e = min(e, m);
            float top = 0.f;
            for (int q = r; q < e; ++q) top = fmaxf(top, s_hi[warp][s_ord[warp][q]]);
            cl[g + __popc(starts[b] & ((1u << lane) - 1u))] =
                make_float4(a, top, __int_as_float(sb + r), __int_as_float((e - r) | (tx << 5)));
          }
        }
        g += __popc(starts[b]);
      }
    } else {
      for (int i = lane & 1; i < n; i += 2) {
        const double2 v = z[k0 + i];
        const float2 f = make_float2(in_fp32(v.x), in_fp32(v.y));
        const int r = pre + i;
        zf[sb + r] = f;
        code[sb + r] = make_uint2(wide[k0 + i].x | (unsigned)c4 << 24, wide[k0 + i].y);
        zx[sb + r] = v;
        cl[cb + r] = make_float4(f.x, f.y, __int_as_float(sb + r), __int_as_float(1 | (tx << 5)));
      }
    }
    seg0 += seg_all;
    cl0 += cl_all;
    __syncthreads();
  }
  if (threadIdx.x == 0) coff[(size_t)T * (tiles_x + 1) + tiles_x] = cl0;
}

// ------------------------------------------------------------ exact comparisons

// An endpoint's identity: (value index, d | a << 8), index < 0 for none.
__device__ __forceinline__ double exact_val(const double *H, int W, const double *z, int2 id, bool plus) {
  const double h = H[(id.y & 255) * W + (id.y >> 8)];
  const double v = z[max(id.x, 0)];
  return plus ? __dadd_rn(v, h) : __dsub_rn(v, h);
}
__device__ __noinline__ bool exact_less(const double *H, int W, const double *z, int2 a, bool ap, int2 b, bool bp) {
  return exact_val(H, W, z, a, ap) < exact_val(H, W, z, b, bp);
}

// x < y for FP32 values with t = y - x, decided exactly inside the guard band
#define GUARD(t, E, exact) ((t) > (E) ? true : ((t) < -(E) ? false : (exact)))

// ------------------------------------------------------------ one patch

// The working memory of one warp. Entry e of column c is at [COLS * e + c]. The
// entries are read once per queued segment and column; they sit in global
// memory, where L1 holds them: in shared memory they took 256 bytes each for
// the most that a patch may need (2048^2, r = 32: 36 on average, 65 at most;
// r = 16: 86 and 146), and 10 warps per SM instead of 16 ran (81 against 63 ms
// at r = 32, 244 against 91 ms at r = 16).
struct PatchMem {
  float2 *sv;             // entries: smallest lower end + E, largest upper end - E
  float2 *ml;             // bins of the cover
  unsigned short *cmap;   // entry of each bin (0: none)
  float2 *bnd;            // entries 1 .. S.nbnd - 1: the component of the cover that their bins' segments may lie in
  float *hrow1;           // first sweep: H for the current tile row, at the farthest row of the patch
  float *hrow;            // second sweep: H for the current tile row, 7 rows (see hrow_row)
  float4 *queue;          // queued segments (z1, z2, x - X0, row of the tile), and their indices
  int *qk;
  int2 *clist;            // clusters to expand (first segment, count | tile << 5)
  float4 *shorts;         // kept-aside segments (z1, z2, index, x - X0 and y - Y0)
  int2 *idl, *idh;        // identities of the entries' ends
  float2 *cv;             // finished intervals and the identities of their ends
  int2 *cl, *ch;
  int ne, nunion, nshort; // capacities
};

// How a warp's lanes are spread: G segments at a time for the kPatchX / G x
// kPatchY columns of its patch; lane l takes column l % COLS (cell), segment
// l / COLS of the group.
template <int G>
struct Shape {
  static constexpr int PX = kPatchX / G, COLS = PX * kPatchY;
};

struct PatchState {
  int X0, Y0, lx, ly, lane, col, g;
  int nent;               // entries in use, the dummy entry 0 included
  int nbnd;               // entries with a component of the cover, entry 0 included
  int ns;                 // kept-aside segments
  int qn, cn;             // queued segments, clusters to expand
  float E, inv_w, thr;
  int cshift;             // cover bins: bins >> cshift
  float cthr;             // least length of an interval of the cover
};

// Bin of a lower end: rounds lo / w to an integer (exact scaling, one
// rounding), masked below kBins so that no value, NaN included (kBins - 1), can
// index cmap out of range. The cover has fewer bins: cover_bin_of.
__device__ __forceinline__ unsigned bin_of(float lo, float inv_w) {
  return __float_as_uint(__fmaf_rn(lo, inv_w, 8388608.f)) & (kBins - 1);
}

// Bin of the cover for a lower end. Those of numbers lie below kCoverBins (the cover's bins are two in one
// where the input uses more); a NaN's, which k_widths leaves out of the range, is brought there.
__device__ __forceinline__ unsigned cover_bin_of(float lo, float inv_w, int cshift) {
  return min(bin_of(lo, inv_w) >> cshift, (unsigned)kCoverBins - 1);
}

// New entry for bin b (uniform). False when the entries are used up.
template <int G>
__device__ __forceinline__ bool new_entry(const PatchMem &M, PatchState &S, int b) {
  const int e = S.nent;
  if (e >= M.ne) return false;
  ++S.nent;
  if (S.lane == 0) M.cmap[b] = (unsigned short)e;
  if (S.g == 0) {
    const int a = Shape<G>::COLS * e + S.col;
    M.sv[a] = make_float2(INFINITY, -INFINITY);
    M.idl[a] = make_int2(-1, 0);
    M.idh[a] = make_int2(-1, 0);
  }
  __syncwarp();
  return true;
}

// The component of the cover that an interval with lower end lo may lie in.
__device__ __forceinline__ float2 component_of(const PatchMem &M, const PatchState &S, float lo) {
  const int e = M.cmap[bin_of(lo, S.inv_w)];
  return M.bnd[e < S.nbnd ? e : 0];
}

// Row of hrow for |dy| between row sy of the tile row k (relative to the
// patch's) and row ly of the patch: the rows hold 4 |k| - 3 .. 4 |k| + 3 for
// k != 0, and 3, 2, 1, 0, 1, 2, 3 for k = 0.
__device__ __forceinline__ int hrow_row(int k, int sy, int ly) {
  return k < 0 ? kTile - 1 + ly - sy : kTile - 1 + sy - ly;
}
// distances of a column t = x - X0 to the nearest and the farthest column of the patch
template <int G>
__device__ __forceinline__ int near_dx(int t) {
  return max(0, max(-t, t - (Shape<G>::PX - 1)));
}
template <int G>
__device__ __forceinline__ int far_dx(int t) {
  return max(t, Shape<G>::PX - 1 - t);
}

// Merges the segments of `todo` (bits 0 .. 3: queue positions G apart) into
// this lane's column with every comparison inside the guard band decided in FP64.
// Closings bring such ties in numbers: every column under one ball of the
// first dilation gives the second one the same end up to rounding. All loads
// of a segment go out together (identities and candidate, then the entry's
// values). Not inlined: the merge loop has to stay in the instruction cache.
template <int G>
__device__ __noinline__ void merge_exact(const double *__restrict__ H, int W, const double2 *__restrict__ zx,
                                         const float4 *queue, const int *qk, const float *hl, int step,
                                         const unsigned short *cmap, float2 *sv, int2 *idl, int2 *idh, int lx, int dy0,
                                         float E, float inv_w, unsigned todo) {
  const double *z = reinterpret_cast<const double *>(zx);
  for (; todo; todo &= todo - 1) {
    const int i = __ffs(todo) - 1;
    const float4 u = queue[G * i];
    const int key = qk[G * i], sy = __float_as_int(u.w), dx = abs(__float_as_int(u.z) - lx), dy = abs(dy0 + sy);
    const float g = hl[sy * step + dx];
    const float l = u.x - g, r = u.y + g;
    const int en = Shape<G>::COLS * cmap[bin_of(l, inv_w)];
    const int2 il = idl[en], ih = idh[en];
    float2 w = sv[en];
    const double2 zc = zx[key];
    const double hc = H[dy * W + dx];
    const double zl = z[max(il.x, 0)], zh = z[max(ih.x, 0)];
    const double hl64 = H[(il.y & 255) * W + (il.y >> 8)], hh64 = H[(ih.y & 255) * W + (ih.y >> 8)];
    const int da = dy | (dx << 8);
    const float tl = (w.x - E) - l, th = r - (w.y + E);
    if (GUARD(tl, E, il.x < 0 || __dsub_rn(zc.x, hc) < __dsub_rn(zl, hl64))) {
      w.x = l + E;
      idl[en] = make_int2(2 * key, da);
    }
    if (GUARD(th, E, ih.x < 0 || __dadd_rn(zh, hh64) < __dadd_rn(zc.y, hc))) {
      w.y = r - E;
      idh[en] = make_int2(2 * key + 1, da);
    }
    sv[en] = w;
  }
}

// Merges the queued segments of tile row k (relative to the patch's) into
// every column's entries. Returns false when a capacity is exceeded.
template <int G>
__device__ __forceinline__ bool flush_queue(const FastArgs &A, const PatchMem &M, PatchState &S, int k) {
  const int lane = S.lane, qn = S.qn, hs = A.hs;
  const float E = S.E, inv_w = S.inv_w;
  constexpr int COLS = Shape<G>::COLS;
  if (lane < 4 * G) M.queue[qn + lane] = make_float4(INFINITY, -INFINITY, 0.f, 0.f);  // padding: no candidate
  __syncwarp();
  // entries for every bin that a queued segment's lower end can fall into in some column
  for (int q0 = 0; q0 < qn; q0 += 32) {
    int b = 1, b1 = 0;
    if (q0 + lane < qn) {
      const float4 c = M.queue[q0 + lane];
      const int t = __float_as_int(c.z), sy = __float_as_int(c.w);
      const int near = k > 0 ? kPatchY - 1 : k < 0 ? 0 : sy;
      const int far = k > 0 || (k == 0 && sy >= kPatchY / 2) ? 0 : kPatchY - 1;
      b = (int)bin_of(c.x - M.hrow[hrow_row(k, sy, near) * hs + near_dx<G>(t)], inv_w);
      b1 = (int)bin_of(c.x - fmaxf(M.hrow[hrow_row(k, sy, far) * hs + far_dx<G>(t)], 0.f), inv_w);
    }
    for (;;) {
      while (b <= b1 && M.cmap[b] != 0) ++b;
      const unsigned w = __ballot_sync(kFull, b <= b1);
      if (!w) break;
      if (!new_entry<G>(M, S, __shfl_sync(kFull, b, __ffs(w) - 1))) return false;
    }
  }
  // row sy of the tile row: hl[sy * step]
  const float *hl = M.hrow + hrow_row(k, 0, S.ly) * hs;
  const int step = k < 0 ? -hs : hs;
  float2 *const sv = M.sv + S.col;
  int2 *const idl = M.idl + S.col, *const idh = M.idh + S.col;
  const float E2 = 2.f * E;
  for (int q = 0; q < qn; q += 4 * G) {
    // Four segments per lane at a time in stages, so that their dependent loads (segment, H, bin, entry)
    // overlap: one after the other they took 462 cycles each, staged 210 (2048^2, r = 32).
    unsigned need = 0;
    float4 c[4];
    float h[4], lo[4], hi[4];
    int e[4];
    float2 v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) c[i] = M.queue[q + G * i + S.g];
#pragma unroll
    for (int i = 0; i < 4; ++i) h[i] = hl[__float_as_int(c[i].w) * step + abs(__float_as_int(c[i].z) - S.lx)];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      lo[i] = c[i].x - h[i];
      hi[i] = c[i].y + h[i];
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) e[i] = COLS * M.cmap[bin_of(lo[i], inv_w)];
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = sv[e[i]];
#pragma unroll
    for (int i = 0; i < 4; ++i) need |= lo[i] < v[i].x || hi[i] > v[i].y ? 1u << i : 0u;
    // segments with which some column's union may grow: the entry is updated where the comparison is
    // clear of the guard band; short intervals are kept aside, the others left to the exact merge
    const unsigned any = __ballot_sync(kFull, need != 0);
    if (!any) continue;
    unsigned unclear = 0, shorts = 0;
#pragma unroll
    for (int s = 0; s < G; ++s) {  // one lane of a column after the other
      if (G == 1 || (any >> (COLS * s) & (0xffffffffu >> (32 - COLS)))) {
        if (G == 1 || (S.g == s && need)) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            if (G > 1) {
              v[i] = sv[e[i]];
            } else {
#pragma unroll
              for (int j = 0; j < i; ++j)
                if (e[j] == e[i]) v[i] = v[j];  // as the segments before left it
            }
            const bool gl = lo[i] < v[i].x, gh = hi[i] > v[i].y;
            const bool cl = lo[i] < v[i].x - E2, ch = hi[i] > v[i].y + E2;
            const bool grow = gl || gh, brief = hi[i] - lo[i] < S.thr, clear = gl == cl && gh == ch;
            if (grow && brief) shorts |= 1u << (G * i + S.g);
            if (grow && !brief && !clear) unclear |= 1u << i;
            if (grow && !brief && clear) {
              const int key = M.qk[q + G * i + S.g];
              const int da = abs(kTile * k - S.ly + __float_as_int(c[i].w)) | (abs(__float_as_int(c[i].z) - S.lx) << 8);
              if (cl) {
                v[i].x = lo[i] + E;
                idl[e[i]] = make_int2(2 * key, da);
              }
              if (ch) {
                v[i].y = hi[i] - E;
                idh[e[i]] = make_int2(2 * key + 1, da);
              }
              sv[e[i]] = v[i];
            }
          }
        }
        if (G > 1) __syncwarp();
      }
    }
    for (unsigned todo = __reduce_or_sync(kFull, shorts); todo; todo &= todo - 1) {
      const int i = __ffs(todo) - 1;
      if (S.ns >= M.nshort) return false;
      if (lane == 0) {
        const float4 u = M.queue[q + i];
        const int at = (__float_as_int(u.z) + 1024) | ((kTile * k + __float_as_int(u.w) + 1024) << 16);
        M.shorts[S.ns] = make_float4(u.x, u.y, __int_as_float(M.qk[q + i]), __int_as_float(at));
      }
      ++S.ns;
    }
    if (__any_sync(kFull, unclear != 0)) {
      for (int s = 0; s < G; ++s) {
        if (S.g == s && unclear)
          merge_exact<G>(A.H64, A.W, reinterpret_cast<const double2 *>(A.zx), M.queue + q + S.g, M.qk + q + S.g, hl,
                         step, M.cmap, sv, idl, idh, S.lx, kTile * k - S.ly, E, inv_w, unclear);
        __syncwarp();
      }
    }
  }
  S.qn = 0;
  __syncwarp();
  return true;
}

// Expands the listed clusters of tile row k: their segments that no component
// of the cover holds are queued (half a warp per cluster, kPairs pairs at a
// time so that their loads overlap), and the queue is flushed when it fills
// up and, with `last`, at the end of the tile row.
template <int G>
__device__ __forceinline__ bool expand_clusters(const FastArgs &A, const PatchMem &M, PatchState &S, int k,
                                                bool last) {
  const int lane = S.lane, hs = A.hs, cn = S.cn;
  __syncwarp();
  for (int q = 0;; q += 2 * kPairs) {
    float2 z[kPairs];
    int key[kPairs], t[kPairs];
    uint2 code[kPairs];
    bool ok[kPairs];
#pragma unroll
    for (int i = 0; i < kPairs; ++i) {
      const int p = q + 2 * i + (lane >> 4);
      const int2 c = p < cn ? M.clist[p] : make_int2(0, 0);
      ok[i] = (lane & 15) < (c.y & 31);
      key[i] = c.x + (lane & 15);
      t[i] = (c.y >> 5) * kTile - S.X0;
      z[i] = ok[i] ? __ldcg(A.zf + key[i]) : make_float2(0.f, 0.f);
      code[i] = ok[i] ? __ldcg(A.code + key[i]) : make_uint2(0u, 0u);
    }
#pragma unroll
    for (int i = 0; i < kPairs; ++i) {
      const int sy = code[i].x >> 26, near = k > 0 ? kPatchY - 1 : k < 0 ? 0 : sy;
      t[i] += code[i].x >> 24 & 3;
      const int row = hrow_row(k, sy, near);
      // held, for every column of the patch, by the candidate of a neighbour between it and the patch
      bool held = false;
      {
        const int a = near_dx<G>(t[i]), d = abs(kTile * k + sy - near);
        if (ok[i] && d <= A.Dy && a < A.W) {
          const int g = A.Dx[A.Dy + 1 + d * A.W + a];
          const unsigned wx = t[i] < 0 ? code[i].x >> 12 : code[i].x, wy = k < 0 ? code[i].y >> 12 : code[i].y;
          held = (a > 0 && (int)(wx & 0xfff) << 3 <= (short)g) || (d > 0 && (int)(wy & 0xfff) << 3 <= g >> 16);
        }
      }
      const float h = M.hrow[row * hs + (ok[i] ? near_dx<G>(t[i]) : 0)];
      const float lo = z[i].x - h, hi = z[i].y + h;
      const float2 b = component_of(M, S, lo);
      const bool keep = ok[i] && !held && !(b.x <= lo && hi <= b.y);
      const unsigned w = __ballot_sync(kFull, keep);
      if (keep) {
        const int p = S.qn + __popc(w & ((1u << lane) - 1u));
        M.queue[p] = make_float4(z[i].x, z[i].y, __int_as_float(t[i]), __int_as_float(sy));
        M.qk[p] = key[i];
      }
      S.qn += __popc(w);
    }
    const bool end = q + 2 * kPairs >= cn;
    if (S.qn > (end && last ? 0 : 32))
      if (!flush_queue<G>(A, M, S, k)) return false;
    if (end) break;
  }
  S.cn = 0;
  __syncwarp();
  return true;
}

// One sweep over the tile rows within reach: PASS 1 builds the cover's bins
// from the clusters, PASS 2 filters the clusters and merges what is left.
template <int PASS, int G>
__device__ __forceinline__ bool sweep(const FastArgs &A, const PatchMem &M, PatchState &S) {
  const int lane = S.lane, X0 = S.X0, T0 = S.Y0 / kTile, hs = A.hs;
  constexpr int PX = Shape<G>::PX;
  const int tiles_x = (A.nx + kTile - 1) / kTile, tiles_y = (A.ny + kTile - 1) / kTile;
  const int reach = (A.Dy + kTile - 1) / kTile, nrows = 2 * reach + 1;
  const float inv_w = S.inv_w;
  for (int jb = 0; jb < nrows; jb += 32) {
    // the lanes look up the cluster ranges of 32 tile rows, the patch's own first, then outwards
    int r0 = 0, r1 = 0, rm = 0;
    {
      const int j = jb + lane, kk = (j + 1) >> 1, k = j & 1 ? kk : -kk;
      const int T = T0 + k;
      const int d = PASS == 1 ? kTile * kk + kTile - 1 : max(0, kTile * kk - (kTile - 1));
      if (j < nrows && T >= 0 && T < tiles_y && d <= A.Dy) {
        const int a = A.Dx[d];
        int ta, tb;
        if (PASS == 1) {  // every column of the patch within reach of every column of the tile
          ta = max(0, (X0 + PX - 1 - a + kTile - 1) >> 2);
          tb = min(tiles_x - 1, (X0 + a - (kTile - 1)) >> 2);
        } else {
          ta = max(0, X0 - a) / kTile;
          tb = min(A.nx - 1, X0 + PX - 1 + a) / kTile;
        }
        if (ta <= tb) {
          const int32_t *o = A.coff + (size_t)T * (tiles_x + 1);
          r0 = o[ta];
          r1 = o[tb + 1];
          rm = o[X0 / kTile];
        }
      }
    }
    for (unsigned rows = __ballot_sync(kFull, r1 > r0); rows; rows &= rows - 1) {
      const int jj = __ffs(rows) - 1;
      const int cb = __shfl_sync(kFull, r0, jj), ce = __shfl_sync(kFull, r1, jj);
      const int kk = (jb + jj + 1) >> 1, k = (jb + jj) & 1 ? kk : -kk;
      // In the second sweep from the patch's own columns to the right, then to the left: the nearest
      // segments come first, and those that reach less far than they change nothing (a plane of equal
      // ends would otherwise be approached step by step, with ties at each).
      const int cm = __shfl_sync(kFull, rm, jj), right = ce - cm;
      auto load = [&](int p) {
        if (p >= ce - cb) return make_float4(INFINITY, -INFINITY, 0.f, 0.f);
        return __ldcg(A.cl + (PASS == 1 ? cb + p : p < right ? cm + p : cm - 1 - (p - right)));
      };
      float4 cn[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) cn[i] = load(32 * i + lane);
      __syncwarp();
      if (PASS == 1) {
        const float *src = A.Hp + (kTile * kk + kTile - 1) * hs;
        for (int i = lane; i < hs; i += 32) M.hrow1[i] = src[i];
      } else if (k == 0) {
        for (int r = 0; r < 2 * kTile - 1; ++r) {
          const float *src = A.Hp + abs(r - (kTile - 1)) * hs;
          for (int i = lane; i < hs; i += 32) M.hrow[r * hs + i] = src[i];
        }
      } else {
        const float4 *src = reinterpret_cast<const float4 *>(A.Hp + (kTile * kk - (kTile - 1)) * hs);
        for (int i = lane; i < (2 * kTile - 1) * hs / 4; i += 32) reinterpret_cast<float4 *>(M.hrow)[i] = src[i];
      }
      __syncwarp();
      // second sweep: the nearest rows
      const float *hM = M.hrow + (k == 0 ? (kTile - 1) * hs : 0);
      const int n = ce - cb;
      for (int c0 = 0; c0 < n; c0 += 64) {
        float4 c[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) c[i] = cn[i];
        if (c0 + 64 < n) {
#pragma unroll
          for (int i = 0; i < 2; ++i) cn[i] = load(c0 + 64 + 32 * i + lane);
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          if (c0 + 32 * i >= n) break;
          const int info = __float_as_int(c[i].w), t = (info >> 5) * kTile - X0;
          const bool in = c0 + 32 * i + lane < n;
          if (PASS == 1) {
            const float h = in ? M.hrow1[max(t + kTile - 1, PX - 1 - t)] : -1.f;
            const float lo = c[i].x - h, hi = c[i].y + h;
            if (2.f * h >= S.cthr) {  // every segment of the cluster gives a long interval
              float2 *bin = M.ml + cover_bin_of(lo, inv_w, S.cshift);
              // values are positive: their bit patterns are ordered like them
              if (lo < bin->x) atomicMin(reinterpret_cast<int *>(&bin->x), __float_as_int(lo));
              if (hi > bin->y) atomicMax(reinterpret_cast<int *>(&bin->y), __float_as_int(hi));
            }
          } else {
            const float h = in ? hM[max(0, max(-t - (kTile - 1), t - (PX - 1)))] : 0.f;
            const float lo = c[i].x - h, hi = c[i].y + h;
            const float2 b = component_of(M, S, lo);
            const bool keep = in && !(b.x <= lo && hi <= b.y);
            const unsigned w = __ballot_sync(kFull, keep);
            if (keep)
              M.clist[S.cn + __popc(w & ((1u << lane) - 1u))] = make_int2(__float_as_int(c[i].z), info);
            S.cn += __popc(w);
          }
        }
        if (PASS == 2) {
          const bool last = c0 + 64 >= n;
          if (S.cn > (last ? 0 : 32) || (last && S.qn > 0))
            if (!expand_clusters<G>(A, M, S, k, last)) return false;
        }
      }
    }
  }
  return true;
}

// Components of the cover from its bins, and the entries that come with them.
template <int G>
__device__ __forceinline__ bool cover_entries(const PatchMem &M, PatchState &S, int nbins) {  // nbins: of the cover
  const int lane = S.lane;
  const float E = S.E;
  int m = 0;
  float carry = -INFINITY;
  for (int b0 = 0; b0 < nbins; b0 += 32) {
    const int b = b0 + lane;
    const float2 v = b < nbins ? M.ml[b] : make_float2(INFINITY, -INFINITY);
    const bool full = v.y > -INFINITY;
    if (!__any_sync(kFull, full)) continue;
    float mx = v.y;
    for (int o = 1; o < 32; o <<= 1) {
      const float y = __shfl_up_sync(kFull, mx, o);
      if (lane >= o) mx = fmaxf(mx, y);
    }
    float before = __shfl_up_sync(kFull, mx, 1);  // largest upper end of the earlier bins
    before = fmaxf(carry, lane ? before : -INFINITY);
    const bool start = full && !(v.x <= before - E);
    const unsigned w = __ballot_sync(kFull, start);
    const int c = m + __popc(w & ((1u << lane) - 1u));  // component starting here
    if (start) {
      if (c < kComps) M.bnd[c + 1].x = v.x;
      if (c > 0 && c <= kComps) M.bnd[c].y = before;
    }
    m += __popc(w);
    carry = fmaxf(carry, __shfl_sync(kFull, mx, 31));
  }
  if (lane == 0) {
    if (m > 0 && m <= kComps) M.bnd[m].y = carry;
    M.bnd[0] = make_float2(INFINITY, -INFINITY);
  }
  m = min(m, kComps);  // any part of the cover may be left out
  __syncwarp();
  constexpr int COLS = Shape<G>::COLS;
  if (S.g == 0) M.sv[S.col] = make_float2(-INFINITY, INFINITY);  // entry 0: bins without an entry, never updated
  S.nent = m + 1;
  // Entry k + 1: the bins wholly inside component k. Their intervals attach to
  // the component, so only upper ends matter; the entry starts just short of
  // the component's end, which a segment of every column reaches.
  for (int k = 0; k < m; ++k) {
    const float2 c = M.bnd[k + 1];
    const int bf = (int)ceilf((c.x + 2.f * E) * S.inv_w + 0.5f), bl = (int)floorf((c.y - 2.f * E) * S.inv_w - 0.5f);
    for (int b = max(bf, 0) + lane; b <= min(bl, kBins - 1); b += 32) M.cmap[b] = (unsigned short)(k + 1);
    if (S.g == 0) {
      const int a = COLS * (k + 1) + S.col;
      M.sv[a] = make_float2(-INFINITY, c.y - 3.f * E);
      M.idl[a] = make_int2(-1, 0);
      M.idh[a] = make_int2(-1, 0);
    }
  }
  __syncwarp();
  // bins in which a component starts: segments there may lie in it. bnd holds the components shrunk by
  // the guard band from here on.
  for (int k = 0; k < m; ++k) {
    const float2 c = M.bnd[k + 1], in = make_float2(c.x + E, c.y - E);
    const int b = (int)bin_of(c.x, S.inv_w);
    __syncwarp();
    if (lane == 0) M.bnd[k + 1] = in;
    if (M.cmap[b] == 0) {
      if (lane == 0) M.bnd[S.nent] = in;
      if (!new_entry<G>(M, S, b)) return false;
    }
  }
  S.nbnd = S.nent;
  __syncwarp();
  return true;
}

// Inserts a kept-aside interval into a column's finished union (n intervals);
// returns the new count, or -1 beyond the capacity.
template <int COLS>
__device__ __noinline__ int insert_short(const FastArgs &A, float2 *cv, int2 *cl, int2 *ch, int n, int cap, float E,
                                         float lo, float hi, int k, int da) {
  const int2 il = make_int2(2 * k, da), ih = make_int2(2 * k + 1, da);
  int j = 0;
  while (j < n) {
    const float t = lo - cv[COLS * j].y;
    if (!GUARD(t, E, exact_less(A.H64, A.W, A.zx, ch[COLS * j], true, il, false))) break;
    ++j;
  }
  if (j == n || GUARD(cv[COLS * j].x - hi, E, exact_less(A.H64, A.W, A.zx, ih, true, cl[COLS * j], false))) {
    if (n >= cap) return -1;
    for (int i = n; i > j; --i) {
      cv[COLS * i] = cv[COLS * (i - 1)];
      cl[COLS * i] = cl[COLS * (i - 1)];
      ch[COLS * i] = ch[COLS * (i - 1)];
    }
    cv[COLS * j] = make_float2(lo, hi);
    cl[COLS * j] = il;
    ch[COLS * j] = ih;
    return n + 1;
  }
  if (GUARD(cv[COLS * j].x - lo, E, exact_less(A.H64, A.W, A.zx, il, false, cl[COLS * j], false))) {
    cv[COLS * j].x = lo;
    cl[COLS * j] = il;
  }
  if (GUARD(hi - cv[COLS * j].y, E, exact_less(A.H64, A.W, A.zx, ch[COLS * j], true, ih, true))) {
    cv[COLS * j].y = hi;
    ch[COLS * j] = ih;
    int i = j + 1;  // absorb the intervals that it now reaches
    while (i < n) {
      if (GUARD(cv[COLS * i].x - cv[COLS * j].y, E, exact_less(A.H64, A.W, A.zx, ch[COLS * j], true, cl[COLS * i], false)))
        break;
      if (GUARD(cv[COLS * i].y - cv[COLS * j].y, E, exact_less(A.H64, A.W, A.zx, ch[COLS * j], true, ch[COLS * i], true))) {
        cv[COLS * j].y = cv[COLS * i].y;
        ch[COLS * j] = ch[COLS * i];
      }
      ++i;
    }
    const int gone = i - j - 1;
    if (gone > 0) {
      for (; i < n; ++i) {
        cv[COLS * (i - gone)] = cv[COLS * i];
        cl[COLS * (i - gone)] = cl[COLS * i];
        ch[COLS * (i - gone)] = ch[COLS * i];
      }
      n -= gone;
    }
  }
  return n;
}

// The union of this lane's column, in M.cv / cl / ch: its interval count; -1
// beyond a capacity (of any lane or of the patch); -2 when an end of this
// lane's union has no identity (never for finite inputs).
template <int G>
__device__ __forceinline__ int patch_union(const FastArgs &A, const PatchMem &M, PatchState &S, int nbins) {
  const int lane = S.lane;
  const float E = S.E;
  S.cshift = nbins > kCoverBins ? 1 : 0;
  S.cthr = S.cshift ? 2.f * S.thr : S.thr;
  const int cbins = (nbins + S.cshift) >> S.cshift;
  for (int b = lane; b < cbins; b += 32) M.ml[b] = make_float2(INFINITY, -INFINITY);
  for (int b = lane; b < kBins / 2; b += 32) reinterpret_cast<unsigned *>(M.cmap)[b] = 0u;
  __syncwarp();
  sweep<1, G>(A, M, S);
  __syncwarp();
  if (!cover_entries<G>(M, S, cbins)) return -1;
  if (!sweep<2, G>(A, M, S)) return -1;
  // the entries in bin order (bins inside one component share an entry), listed in the memory of the
  // queue and loaded two ahead
  unsigned short *const list = reinterpret_cast<unsigned short *>(M.ml);
  int ne = 0;
  for (int b0 = 0, last = 0; b0 < nbins; b0 += 32) {
    const int e = M.cmap[b0 + lane];
    int prev = __shfl_up_sync(kFull, e, 1);
    if (lane == 0) prev = last;
    last = __shfl_sync(kFull, e, 31);
    const bool first = e != 0 && e != prev;
    const unsigned w = __ballot_sync(kFull, first);
    if (first) list[ne + __popc(w & ((1u << lane) - 1u))] = (unsigned short)e;
    ne += __popc(w);
  }
  __syncwarp();
  constexpr int COLS = Shape<G>::COLS;
  int2 *const cl = M.cl + S.col, *const ch = M.ch + S.col;
  float2 *const cv = M.cv + S.col;
  if (S.g > 0) ne = 0;  // one lane per column
  int n = 0;
  bool open = false, full = false, bad = false;
  float2 cur = make_float2(0.f, 0.f);
  int2 il = make_int2(-1, 0), ih = make_int2(-1, 0);
  constexpr int kAhead = 3;
  float2 pv[kAhead];
  int2 pl[kAhead], ph[kAhead];
#pragma unroll
  for (int i = 0; i < kAhead; ++i) {
    const int e = COLS * (i < ne ? list[i] : 0) + S.col;
    pv[i] = M.sv[e];
    pl[i] = M.idl[e];
    ph[i] = M.idh[e];
  }
  for (int j0 = 0; j0 < ne; j0 += kAhead) {
#pragma unroll
    for (int i = 0; i < kAhead; ++i) {
      const int j = j0 + i;
      if (j >= ne) break;
      float2 v = pv[i];
      const int2 vl = pl[i], vh = ph[i];
      {
        const int e = COLS * (j + kAhead < ne ? list[j + kAhead] : 0) + S.col;
        pv[i] = M.sv[e];
        pl[i] = M.idl[e];
        ph[i] = M.idh[e];
      }
      if (!(v.y > -INFINITY)) continue;
      v.x -= E;
      v.y += E;
      if (open) {
        const float t = v.x - cur.y;
        if (!GUARD(t, E, vl.x >= 0 && ih.x >= 0 && exact_less(A.H64, A.W, A.zx, ih, true, vl, false))) {
          // overlapping or touching: extend the open interval
          const float tl = cur.x - v.x;
          if (vl.x >= 0 && il.x >= 0 && GUARD(tl, E, exact_less(A.H64, A.W, A.zx, vl, false, il, false))) {
            cur.x = v.x;  // a tie across a bin's edge
            il = vl;
            if (n > 0 && !GUARD(cur.x - cv[COLS * (n - 1)].y, E,
                                exact_less(A.H64, A.W, A.zx, ch[COLS * (n - 1)], true, il, false))) {
              --n;  // it reaches the interval before
              cur.x = cv[COLS * n].x;
              il = cl[COLS * n];
              if (ih.x < 0 || GUARD(cv[COLS * n].y - cur.y, E, exact_less(A.H64, A.W, A.zx, ih, true, ch[COLS * n], true))) {
                cur.y = cv[COLS * n].y;
                ih = ch[COLS * n];
              }
            }
          }
          const float th = v.y - cur.y;
          if (GUARD(th, E, ih.x < 0 || (vh.x >= 0 && exact_less(A.H64, A.W, A.zx, ih, true, vh, true)))) {
            cur.y = v.y;
            ih = vh;
          }
          continue;
        }
        if (n < M.nunion - 1) {
          cv[COLS * n] = cur;
          cl[COLS * n] = il;
          ch[COLS * n] = ih;
          bad |= il.x < 0 || ih.x < 0;
          ++n;
        } else {
          full = true;
        }
      }
      open = true;
      cur = v;
      il = vl;
      ih = vh;
    }
  }
  if (open) {
    if (n < M.nunion - 1) {
      cv[COLS * n] = cur;
      cl[COLS * n] = il;
      ch[COLS * n] = ih;
      bad |= il.x < 0 || ih.x < 0;
      ++n;
    } else {
      full = true;
    }
  }
  // kept-aside segments
  for (int s = 0; s < (S.g == 0 ? S.ns : 0); s += 4) {
    // four at a time, so that their loads overlap
    float lo[4], hi[4];
    int key[4], da[4];
    unsigned need = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float4 c = M.shorts[min(s + i, S.ns - 1)];
      const int at = __float_as_int(c.w);
      const int dx = abs((at & 0xffff) - 1024 - S.lx), dy = abs((at >> 16) - 1024 - S.ly);
      const float h = A.Hp[dy * A.hs + dx];
      lo[i] = c.x - h;
      hi[i] = c.y + h;
      key[i] = __float_as_int(c.z);
      da[i] = dy | (dx << 8);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 v = M.sv[COLS * M.cmap[bin_of(lo[i], S.inv_w)] + S.col];
      // intervals that are long in this column have been merged
      if (s + i < S.ns && hi[i] >= lo[i] && hi[i] - lo[i] < S.thr && (lo[i] < v.x || hi[i] > v.y)) need |= 1u << i;
    }
    if (full || bad) need = 0;
    for (; need; need &= need - 1) {
      const int i = __ffs(need) - 1;
      const float l = i == 0 ? lo[0] : i == 1 ? lo[1] : i == 2 ? lo[2] : lo[3];
      const float u = i == 0 ? hi[0] : i == 1 ? hi[1] : i == 2 ? hi[2] : hi[3];
      const int ks = i == 0 ? key[0] : i == 1 ? key[1] : i == 2 ? key[2] : key[3];
      const int ds = i == 0 ? da[0] : i == 1 ? da[1] : i == 2 ? da[2] : da[3];
      const int r = insert_short<COLS>(A, cv, cl, ch, n, M.nunion - 1, E, l, u, ks, ds);
      if (r < 0) {
        full = true;
        need = 0;
        break;
      }
      n = r;
    }
  }
  if (__any_sync(kFull, full)) return -1;
  return bad ? -2 : n;
}

// Persistent: a warp per block takes patches of the launch's dilations from a
// queue (dilations in the order of vols; each one's patches in bands of 512
// columns, all rows of a band before the next, so that the patches in flight
// share their source rows in L2). BIG: the second tier, over the patches that
// the first one listed, with larger working lists.
template <bool BIG, int G>
__global__ void __launch_bounds__(32, 20) k_patch(const BatchVol *__restrict__ vols, int nitems, PatchQueue Q,
                                                  int hs_max, PatchScratch scratch) {
  constexpr int ne = BIG ? kEntriesBig : kEntries, PX = Shape<G>::PX, COLS = Shape<G>::COLS;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ BatchVol V;
  PatchMem M;
  M.ne = ne;
  M.nunion = BIG ? kUnionBig : kUnion;
  M.nshort = BIG ? kShortBig : kShort;
  const size_t wb = blockIdx.x;
  // shared memory: what lasts for the whole patch, then the bins of the cover, whose memory the queue,
  // the cluster list and the rows of H take over in the second sweep
  unsigned char *p = smem;
  M.bnd = reinterpret_cast<float2 *>(p);
  p += sizeof(float2) * (2 * kComps + 2);
  M.cmap = reinterpret_cast<unsigned short *>(p);
  p += sizeof(unsigned short) * kBins;
  M.hrow1 = reinterpret_cast<float *>(p);
  p += sizeof(float) * hs_max;
  M.ml = reinterpret_cast<float2 *>(p);
  M.hrow = reinterpret_cast<float *>(p);
  p += sizeof(float) * (2 * kTile - 1) * hs_max;
  M.queue = reinterpret_cast<float4 *>(p);
  p += sizeof(float4) * (kQueue + kPad);
  M.clist = reinterpret_cast<int2 *>(p);
  p += sizeof(int2) * kClusters;
  M.qk = reinterpret_cast<int *>(p);
  M.sv = scratch.sv + wb * COLS * ne;
  M.shorts = scratch.shorts + wb * M.nshort;
  M.idl = scratch.ids + wb * 2 * COLS * ne;
  M.idh = M.idl + COLS * ne;
  M.cv = scratch.cv + wb * COLS * M.nunion;
  M.cl = scratch.cids + wb * 2 * COLS * M.nunion;
  M.ch = M.cl + COLS * M.nunion;
  PatchState S;
  S.lane = threadIdx.x;
  S.col = threadIdx.x % COLS;
  S.g = threadIdx.x / COLS;
  S.lx = S.col % PX;
  S.ly = S.col / PX;
  int cur = -1;
  const int todo = BIG ? min(Q.count[1], nitems) : nitems;
  for (;;) {
    int item = 0, listed = 0;  // (of the patch before: its load and the queue's overlap)
    if (S.lane == 0) {
      item = atomicAdd(&Q.count[BIG ? 2 : 0], 1);
      if (!BIG && cur >= 0) listed = *(volatile int *)V.listed;
    }
    item = __shfl_sync(kFull, item, 0);
    if (item >= todo) return;
    if (BIG) item = Q.list[item];
    int v = max(cur, 0);
    if (BIG)
      while (item < vols[v].item0) --v;
    while (item >= vols[v].item1) ++v;
    if (v != cur) {
      __syncwarp();
      for (int i = S.lane; i < (int)(sizeof(BatchVol) / sizeof(int)); i += 32)
        reinterpret_cast<int *>(&V)[i] = reinterpret_cast<const int *>(&vols[v])[i];
      cur = v;
      listed = 0;
      __syncwarp();
    }
    constexpr int kBand = 512 / PX;
    const int nx = V.A.nx, ny = V.A.ny;
    const int tiles_x = (nx + PX - 1) / PX, tiles_y = (ny + kPatchY - 1) / kPatchY;
    const int rel = item - V.item0, band = rel / (kBand * tiles_y), rb = rel - band * kBand * tiles_y;
    const int bw = min(kBand, tiles_x - band * kBand);
    S.X0 = (band * kBand + rb % bw) * PX;
    S.Y0 = (rb / bw) * kPatchY;
    S.nent = 1;
    S.ns = S.qn = S.cn = 0;
    const FastPar *par = V.A.par;
    S.E = par->E;
    S.inv_w = par->inv_w;
    S.thr = par->thr;
    // beyond `most` listed patches the dilation is left undone (one lane looks: the answer may change meanwhile)
    if (BIG && S.lane == 0) listed = *(volatile int *)V.listed;
    const bool undone = __shfl_sync(kFull, listed, 0) > V.most;
    if (BIG && undone) {
      if (S.lane == 0) atomicOr(V.ovf, 8);
      continue;
    }
    const int n = undone ? -1 : patch_union<G>(V.A, M, S, par->nbins);
    const int x = S.X0 + S.lx, y = S.Y0 + S.ly;
    const bool in = S.g == 0 && x < nx && y < ny;
    const bool over = __any_sync(kFull, n == -1);
    if (over && !BIG) {  // the whole patch goes to the next tier
      const int cols = __popc(__ballot_sync(kFull, in));
      if (S.lane == 0) {
        atomicAdd(V.listed, 1);
        if (!undone) Q.list[atomicAdd(&Q.count[1], 1)] = item;
        atomicAdd(&Q.count[3], cols);
      }
      if (in) V.obeg[x + nx * y] = V.oend[x + nx * y] = 0;
    } else if (in) {
      const int c = x + nx * y;
      unsigned dst = 0;
      int m = n;
      if (over || n < 0) {
        V.big_list[atomicAdd(V.big_count, 1)] = c;  // the FP64 tier
        m = 0;
      } else if (!place_union(V, x, y, n, dst)) {
        m = 0;
        dst = 0;
      } else {
        double2 *o = V.oz + dst;
        for (int k = 0; k < n; ++k)
          o[k] = make_double2(exact_val(V.A.H64, V.A.W, V.A.zx, M.cl[COLS * k + S.col], false),
                              exact_val(V.A.H64, V.A.W, V.A.zx, M.ch[COLS * k + S.col], true));
      }
      V.obeg[c] = (int32_t)dst;
      V.oend[c] = (int32_t)(dst + (unsigned)m);
    }
    __syncwarp();
  }
}

// ------------------------------------------------------------ FP64 lists

// Inserts [lo, hi] into the sorted list L of n disjoint closed intervals.
__device__ bool big_insert(double2 *L, int &n, int cap, double lo, double hi) {
  int l = 0, r = n;
  while (l < r) {
    const int m = (l + r) >> 1;
    if (L[m].y >= lo)
      r = m;
    else
      l = m + 1;
  }
  const int i = l;
  if (i == n || L[i].x > hi) {
    if (n >= cap) return false;
    for (int k = n; k > i; --k) L[k] = L[k - 1];
    L[i] = make_double2(lo, hi);
    ++n;
    return true;
  }
  int j = i;
  while (j + 1 < n && L[j + 1].x <= hi) ++j;
  L[i] = make_double2(L[i].x < lo ? L[i].x : lo, L[j].y > hi ? L[j].y : hi);
  if (j > i) {
    const int sh = j - i;
    for (int k = i + 1; k + sh < n; ++k) L[k] = L[k + sh];
    n -= sh;
  }
  return true;
}

// A column's union in a list of `cap` intervals: their count, or -1 beyond it.
// Source columns come ring by ring from the column's own outwards: the nearest
// give the longest intervals, in which most of the others then lie (row by row,
// the list holds far more intervals on the way: scattered segments, 256^2
// columns, 12 of them each over 30000, radius 16: 5.2 s against 1.7).
__device__ __noinline__ int big_union(const FastArgs &A, int x, int y, double2 *L, int cap) {
  // (copies: the list's stores would have the members loaded again after each)
  const int nx = A.nx, ny = A.ny, W = A.W, Dy = A.Dy;
  const int32_t *__restrict__ beg = A.beg, *__restrict__ end = A.end;
  const double2 *__restrict__ z = reinterpret_cast<const double2 *>(A.zd);
  const double *__restrict__ H = A.H64;
  const int *__restrict__ Dx = A.Dx;
  int n = 0;
  bool ok = true;
  auto column = [&](int d, int a) {
    if (d > Dy || a > Dx[d]) return;
    const double h = H[d * W + a];
    for (int s = 0; s < 4; ++s) {
      if (((s & 1) && a == 0) || ((s & 2) && d == 0)) continue;
      const int xs = s & 1 ? x + a : x - a, ys = s & 2 ? y + d : y - d;
      if (xs < 0 || xs >= nx || ys < 0 || ys >= ny) continue;
      const int cs = xs + nx * ys;
      for (int k = beg[cs], e = end[cs]; k < e && ok; ++k) {
        const double2 v = z[k];
        ok = big_insert(L, n, cap, __dsub_rn(v.x, h), __dadd_rn(v.y, h));
      }
    }
  };
  for (int ring = 0; ring < max(Dy + 1, W) && ok; ++ring)
    for (int i = 0; i < 2 * ring + 1 && ok; ++i) column(min(i, ring), min(ring, 2 * ring - i));
  return ok ? n : -1;
}

// ------------------------------------------------------------ small radii

// By how much at most a segment reaches beyond one of the segments of each of
// its four neighbour columns (FP16 bits, rounded up to 12). Where H grows by at
// least as much over the step to that neighbour, the neighbour's candidate holds
// the segment's, in exact arithmetic and so after rounding, and the segment is
// passed over for all columns on that side: by patches on their nearest column's
// growth, which is the least (2048^2, r = 32: 33.0 to 24.7 ms, this kernel
// included; 1024^2 spheres, r = 32: 5.1 to 4.0), by k_direct on each column's
// own. For k_direct (RECORDS) with the ends in FP32 and the column, the segments
// of a row contiguous (CSR inputs are already so: SLOTS false); else the widths
// alone, in the input's order, and the scalars of the dilation from the values'
// range (mm, zeroed before: orders of the largest value and of the largest
// negated value, the blocks that are done, whether values lie beyond); a pass of its own over the
// values took 0.5 ms at 2048^2. A block per row: it loads what it needs of five
// columns, and is bound by the latency of that (0.7 ms at 2048^2).
template <bool SLOTS, bool RECORDS, bool SHIFT>
__global__ void __launch_bounds__(kPrepThreads) k_widths(int nx, int ny, const int32_t *__restrict__ beg,
                                                              const int32_t *__restrict__ end,
                                                              const longlong2 *__restrict__ z, uint4 *__restrict__ rec,
                                                              longlong2 *__restrict__ rz, int32_t *__restrict__ rbeg,
                                                              int32_t *__restrict__ rend, uint2 *__restrict__ wide,
                                                              float R, unsigned long long *mm, FastPar *par,
                                                              const double offset) {
  const double off = SHIFT ? offset : 0.0;
  __shared__ int s_sum[kPrepThreads / 32];
  const int y = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int base = SLOTS ? beg[nx * y] : 0;
  ValueRange range;  // widths alone: the values' range besides
  for (int x0 = 0; x0 < nx; x0 += kPrepThreads) {
    const int x = x0 + threadIdx.x, c = x + nx * y;
    const int k0 = x < nx ? beg[c] : 0, n = x < nx ? end[c] - k0 : 0;
    int out = k0;
    if (SLOTS) {
      int upto = n;
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(kFull, upto, o);
        if (lane >= o) upto += v;
      }
      __syncthreads();
      if (lane == 31) s_sum[warp] = upto;
      __syncthreads();
      int before = 0, all = 0;
      for (int w = 0; w < kPrepThreads / 32; ++w) {
        before += w < warp ? s_sum[w] : 0;
        all += s_sum[w];
      }
      out = base + before + upto - n;
      base += all;
      if (x < nx) {
        rbeg[c] = out;
        rend[c] = out + n;
      }
    }
    if (n <= 0) continue;
    int nb[4], ne[4];
#pragma unroll
    for (int d = 0; d < 4; ++d) {
      const bool ok = d == 0 ? x > 0 : d == 1 ? x + 1 < nx : d == 2 ? y > 0 : y + 1 < ny;
      const int cn = ok ? c + (d == 0 ? -1 : d == 1 ? 1 : d == 2 ? -nx : nx) : c;
      nb[d] = beg[cn];
      ne[d] = ok ? end[cn] : nb[d];
    }
    for (int k = 0; k < n; ++k) {
      const longlong2 v = z[k0 + k];
      if (!RECORDS) {
        range.take(v.x);
        range.take(v.y);
      }
      const float lo = trunc32_bits(v.x, off), hi = trunc32_bits(v.y, off);
      unsigned w[4];
#pragma unroll
      for (int d = 0; d < 4; ++d) {
        float best = INFINITY;
        // of the neighbour's segments the first two that reach this one (any other choice is safe too)
        int j = nb[d];
        longlong2 u = make_longlong2(0, 0);
        for (; j < ne[d]; ++j) {
          u = z[j];
          if (!(trunc32_bits(u.y, off) < lo)) break;
        }
        nb[d] = j;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          if (j + q < ne[d]) {
            if (q) u = z[j + q];
            const float a = trunc32_bits(u.x, off), b = trunc32_bits(u.y, off);
            const float e = 4.76837158203125e-7f * (fabsf(a) + fabsf(b) + fabsf(lo) + fabsf(hi)) + 1e-30f;
            best = fminf(best, fmaxf(fmaxf(a - lo, hi - b), 0.f) + e);
          }
        }
        w[d] = min(0xfffu, (__half_as_ushort(__float2half_ru(best)) + 7u) >> 3);
      }
      if (!RECORDS)
        wide[out + k] = make_uint2(w[0] | w[1] << 12, w[2] | w[3] << 12);
      else
        rec[out + k] = make_uint4(__float_as_uint(lo), __float_as_uint(hi), w[0] | w[1] << 12 | (unsigned)(x & 0xff) << 24,
                                w[2] | w[3] << 12 | (unsigned)(x >> 8) << 24);
      if (SLOTS) rz[out + k] = v;
    }
  }
  if (!RECORDS) range.finish(mm, R, par);
}

// A column beyond k_direct's list: for the caller's last tier, or, with a pool of FP64 lists, here and now.
__device__ __noinline__ void beyond_list(const BatchVol &V, int x, int y) {
  const int c = x + V.A.nx * y, i = atomicAdd(V.big_count, 1);
  int n = 0;
  unsigned dst = 0;
  if (!V.pool) {
    V.big_list[i] = c;
  } else {
    const int slot = atomicAdd(V.pool_used, 1);
    double2 *L = V.pool + (size_t)slot * kPoolCap;
    n = slot < kFewColumns ? big_union(V.A, x, y, L, kPoolCap) : -1;
    if (n < 0 || !place_union(V, x, y, n, dst)) {
      if (n < 0) atomicOr(V.ovf, 8);
      n = 0;
      dst = 0;
    }
    for (int k = 0; k < n; ++k) V.oz[dst + k] = L[k];
  }
  V.obeg[c] = (int32_t)dst;
  V.oend[c] = (int32_t)(dst + (unsigned)n);
}

// Dilations by small radii, one thread per column: few columns are in reach, so
// that the candidates are met one by one, without clusters, cover or bins. A
// candidate that its neighbour's holds (k_widths), or that lies, in FP32
// and by more than its error, inside one of the first kHot intervals found, is
// passed over. What is left each lane takes from a list of its own, so that the
// lanes do not wait for one another's: it is compared with all intervals found,
// extends one that it is certain to meet, in FP64, or else begins another. Ends
// are compared as integers (Key). Intervals that have come to meet are merged at
// the end; more than kList of them are inserted into a sorted list at once.
//
// What bounds it: the ALU pipe (1024^2, 1.5 segments per column, radius 6: 90
// instructions per candidate and warp, the pipe busy 82 % of its cycles), in inputs of many segments the
// latency of the lists in local memory, and in small volumes that of a thread's
// chain. There G = 4 threads share a column, each taking every fourth row, and
// the first one inserts the others' unions into its own: with four threads 64^2
// takes 0.027 instead of 0.051 ms at radius 4, 276^2 0.054 instead of 0.043 and
// 0.146 instead of 0.153 at 2.75 and 6, 512^2 0.23 instead of 0.17 at 4. Hence
// the line at 2^16 columns.
//
// Against patches, packing included (ms; segments per column; radius 4, 6, 8):
//   276^2   1.5   0.10 / 0.21   0.15 / 0.21   0.21 / 0.20
//   1024^2  1.5   0.39 / 1.09   0.68 / 1.36   1.01 / 1.43
//   2048^2  5.1   11.1 / 16.5   21.9 / 21.4   36.0 / 24.4
// A patch's candidates are those of the whole patch's reach, at radius 4 four
// times a column's, and its steps take some ten thousand cycles however few they
// are; but their number grows more slowly. Both take the same between 290 and
// 580 candidates per column: the line of direct_choice is 450. (In FP64
// throughout, without the neighbours' test, 1024^2 took 0.53, 1.1 and 1.9 ms.)
template <int G, bool SHIFT>
__global__ void __launch_bounds__(128, 8) k_direct(const BatchVol *__restrict__ vols, int nv) {
  __shared__ BatchVol V;
  __shared__ bool s_undone;
  extern __shared__ float2 s_tab[];
  int v = 0;
  for (int r = nv - 1; v < r;) {
    const int m = (v + r) >> 1;
    if ((int)blockIdx.x < vols[m].item1) r = m; else v = m + 1;
  }
  for (int i = threadIdx.x; i < (int)(sizeof(BatchVol) / sizeof(int)); i += 128)
    reinterpret_cast<int *>(&V)[i] = reinterpret_cast<const int *>(&vols[v])[i];
  __syncthreads();
  if (threadIdx.x == 0) s_undone = *(volatile int *)V.listed > V.most;
  constexpr int COLS = 32 / G;
  const int nx = V.A.nx, ny = V.A.ny, W = V.A.W, tw = min(W, nx);
  // H in FP32 and its growth inwards, for the distances that occur
  for (int i = threadIdx.x; i < tw * (min(V.A.Dy, ny - 1) + 1); i += 128) {
    const int d = i / tw, a = i - d * tw;
    s_tab[i] = make_float2(V.A.Hp[d * V.A.hs + a], __int_as_float(V.A.Dx[V.A.Dy + 1 + d * W + a]));
  }
  __syncthreads();
  const int blocks_x = (nx + COLS - 1) / COLS, blk = (int)blockIdx.x - V.item0;
  const int lane = threadIdx.x & 31, part = lane / COLS;
  const int x = blk % blocks_x * COLS + lane % COLS, y = blk / blocks_x * 4 + (threadIdx.x >> 5);
  const bool inside = x < nx && y < ny;
  if (s_undone) {  // too many columns listed: the dilation is left undone
    if (inside && part == 0) V.obeg[x + nx * y] = V.oend[x + nx * y] = 0;
    return;
  }
  Key2 A[kDirectCap];
  Key2 found[kList];  // intervals found so far; those that have come to meet are merged at the end
  float2 sure[kHot];  // of the first ones, inside which an FP32 candidate is certain to lie in them
#pragma unroll
  for (int i = 0; i < kHot; ++i) sure[i] = make_float2(INFINITY, -INFINITY);
  float2 *const all = s_tab + tw * (min(V.A.Dy, ny - 1) + 1) + threadIdx.x;  // the same of all, 128 apart
  int n = 0, m = 0;
  const float reach = 2.f * V.A.Hp[0];
  auto insert = [&](Key2 u) {
    if (n < 0) return;
    const int2 at = union_insert_keys(A, n, kDirectCap, u.x, u.y);
    n = at.x < 0 ? -1 : at.y;
  };
  auto inner = [&](Key2 u) {
    const float lo = SHIFT ? trunc32(u.x, V.A.off) : trunc32(u.x), hi = SHIFT ? trunc32(u.y, V.A.off) : trunc32(u.y);
    const float e = 9.5367431640625e-07f * (fabsf(lo) + fabsf(hi) + reach);
    return make_float2(lo + e, hi - e);
  };
  const double2 *z = V.A.rz;
  const uint4 *rec = V.A.rec;
  if (inside) {
    // rows outwards from the column's own one, before them its own segments; the threads of a column take
    // every G-th row, or every G-th step of a grid of one row
    const int rows = 2 * min(V.A.Dy, ny - 1);
    const int row_step = ny > 1 ? G : 1, k_first = ny > 1 ? 0 : kStep * part, k_step = ny > 1 ? kStep : kStep * G;
    for (int row = part == 0 ? -1 : ny > 1 ? part : 0; row <= rows; row += row < 0 ? 1 : row_step) {
      const int ady = (row + 1) >> 1, ys = row & 1 ? y - ady : y + ady;
      const bool own = row < 0;
      if (!own && (ys < 0 || ys >= ny)) continue;
      const int reach_x = own ? 0 : V.A.Dx[ady];
      const int cy = own ? y : ys;
      const float2 *tab = s_tab + (own ? 0 : ady) * tw;
      const bool above = cy < y;
      int k = V.A.rbeg[max(0, x - reach_x) + nx * cy] + (own ? 0 : k_first);
      const int ke = V.A.rend[min(nx - 1, x + reach_x) + nx * cy];
      for (; k < ke; k += own ? kStep : k_step) {
        uint4 v[kStep];
#pragma unroll
        for (int i = 0; i < kStep; ++i) v[i] = rec[min(k + i, ke - 1)];
        unsigned todo = 0;
#pragma unroll
        for (int i = 0; i < kStep; ++i) {
          const int dx = (int)((v[i].z >> 24) | (v[i].w >> 24) << 8) - x;
          const float2 t = tab[abs(dx)];
          const int g = __float_as_int(t.y);
          const int wx = (int)(dx < 0 ? v[i].z >> 12 & 0xfff : v[i].z & 0xfff) << 3;
          const int wy = (int)(above ? v[i].w >> 12 & 0xfff : v[i].w & 0xfff) << 3;
          const float lo = __uint_as_float(v[i].x) - t.x, hi = __uint_as_float(v[i].y) + t.x;
          bool out = wx <= (short)g || wy <= g >> 16 || k + i >= ke;
#pragma unroll
          for (int j = 0; j < kHot; ++j) out |= lo >= sure[j].x && hi <= sure[j].y;
          todo |= out ? 0u : 1u << i;
        }
        // what is not certain to change nothing, in FP64: each lane its own next one
        for (; todo; todo &= todo - 1) {
          const int i = __ffs(todo) - 1;
          const uint4 r = rec[k + i];
          const int a = abs((int)((r.z >> 24) | (r.w >> 24) << 8) - x);
          const float h = tab[a].x;
          const float lo = __uint_as_float(r.x) - h, hi = __uint_as_float(r.y) + h;
          int at = -1;
          bool in = false;
          for (int j = 0; j < m; ++j) {
            const float2 s = all[128 * j];
            in |= lo >= s.x && hi <= s.y;
            if (lo <= s.y && hi >= s.x) at = j;  // certain to meet it
          }
          if (in) continue;
          const double2 u = z[k + i];
          const double d = V.A.H64[(own ? 0 : ady) * W + a];
          Key2 w = make_longlong2(key_of(__dsub_rn(u.x, d)), key_of(__dadd_rn(u.y, d)));
          if (at >= 0) {
            const Key2 q = found[at];
            w = make_longlong2(kmin(w.x, q.x), kmax(w.y, q.y));
          } else if (m < kList) {
            at = m++;
          } else {
            insert(w);
            continue;
          }
          found[at] = w;
          const float2 s = inner(w);
          all[128 * at] = s;
#pragma unroll
          for (int j = 0; j < kHot; ++j)
            if (j == at) sure[j] = s;
        }
      }
    }
  }
#pragma unroll 1
  for (int i = 0; i < m; ++i) insert(found[i]);
  // the other lanes' unions into the first one's
#pragma unroll 1
  for (int p = 1; p < G; ++p) {
    const int from = lane % COLS + p * COLS, m = __shfl_sync(kFull, n, from);
    if (part == 0 && m < 0) n = -1;
    const int most = __reduce_max_sync(kFull, m);
#pragma unroll 1
    for (int i = 0; i < most; ++i) {
      const Key2 u = A[i];
      const Key lo = __shfl_sync(kFull, u.x, from), hi = __shfl_sync(kFull, u.y, from);
      if (part == 0 && n >= 0 && i < m) {
        const int2 at = union_insert_keys(A, n, kDirectCap, lo, hi);
        n = at.x < 0 ? -1 : at.y;
      }
    }
  }
  if (!inside || part != 0) return;
  const int c = x + nx * y;
  unsigned dst = 0;
  if (n < 0) {
    beyond_list(V, x, y);
    return;
  }
  if (!place_union(V, x, y, n, dst)) {
    n = 0;
    dst = 0;
  }
  for (int i = 0; i < n; ++i) V.oz[dst + i] = make_double2(value_of(A[i].x), value_of(A[i].y));
  V.obeg[c] = (int32_t)dst;
  V.oend[c] = (int32_t)(dst + (unsigned)n);
}

// ------------------------------------------------------------ last tiers

// The patches of `list` (items of a launch of one dilation, with G lanes per column) as columns of its over_list.
__global__ void k_patch_columns(const BatchVol *vols, const int *list, const int *count, int px) {
  const BatchVol &V = vols[0];
  const int nx = V.A.nx, ny = V.A.ny, band_most = 512 / px;
  const int tiles_x = (nx + px - 1) / px, tiles_y = (ny + kPatchY - 1) / kPatchY;
  for (int i = blockIdx.x; i < *count; i += gridDim.x) {
    const int item = list[i], band = item / (band_most * tiles_y), rb = item - band * band_most * tiles_y;
    const int bw = min(band_most, tiles_x - band * band_most);
    const int x = (band * band_most + rb % bw) * px + threadIdx.x % px, y = (rb / bw) * kPatchY + threadIdx.x / px;
    const bool in = (int)threadIdx.x < px * kPatchY && x < nx && y < ny;
    if (in) V.over_list[atomicAdd(V.over_count, 1)] = x + nx * y;
  }
}

// The listed columns of every dilation in FP64 (grid-stride), each built in a
// list of `cap` intervals in global scratch and placed like the other tiers; a
// union beyond it sets the overflow flag. Every SM has a block: with 16 in all the
// scattered segments of k_column's comment took 77 ms at radius 2 and 1,300 at 4,
// with one per SM 21 and 178 (two: 20 and 177).
__global__ void __launch_bounds__(kBigThreads) k_big(const BatchVol *vols, int nv, double2 *scratch, int cap) {
  const int tid = blockIdx.x * blockDim.x + threadIdx.x, nth = gridDim.x * blockDim.x;
  double2 *L = scratch + (size_t)tid * cap;
  for (int v = 0; v < nv; ++v) {
    const BatchVol &V = vols[v];
    const FastArgs &A = V.A;
    const int m = *V.big_count;
    for (int i = tid; i < m; i += nth) {
      const int c = V.big_list[i];
      const int x = c % A.nx, y = c / A.nx;
      int n = big_union(A, x, y, L, cap);
      unsigned dst = 0;
      if (n > kUnionLarge) atomicAdd(V.large, 1);
      if (n < 0) {
        atomicOr(V.ovf, 1);
        n = 0;
      } else if (!place_union(V, x, y, n, dst)) {
        n = 0;
        dst = 0;
      }
      for (int k = 0; k < n; ++k) V.oz[dst + k] = L[k];
      V.obeg[c] = (int32_t)dst;
      V.oend[c] = (int32_t)(dst + (unsigned)n);
    }
  }
}

static_assert(sizeof(BatchVol) % sizeof(int) == 0, "BatchVol is copied as ints");

}  // namespace

// ================================================================ host side

namespace {

int sm_count_fast() {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms > 0 ? sms : 148;
}

size_t patch_smem(int hs_max) {
  const size_t kept = sizeof(float2) * (2 * kComps + 2) + sizeof(unsigned short) * kBins + sizeof(float) * hs_max;
  const size_t second = sizeof(float) * (2 * kTile - 1) * hs_max + (sizeof(float4) + sizeof(int)) * (kQueue + kPad) +
                        sizeof(int2) * kClusters;
  return kept + std::max(second, sizeof(float2) * kCoverBins);
}

}  // namespace

int patch_count(const vo_grid &g, int split) {
  const int px = kPatchX / split;
  return ((g.nx + px - 1) / px) * ((g.ny + kPatchY - 1) / kPatchY);
}

// Lanes per column for a launch over the given columns. A launch of few
// patches is bound by the longest one's chain of dependent steps, not by
// throughput: with four lanes per column a warp merges four segments at a
// time into 2 x 4 columns, at the cost of sweeping the same clusters four
// times as often.
int64_t patch_total(const vo_grid *const *grids, int n) {
  int64_t patches = 0;
  for (int i = 0; i < n; ++i) patches += patch_count(*grids[i], 1);
  return patches;
}
int patch_split(const vo_grid *const *grids, int n) {
  const int64_t patches = patch_total(grids, n);
  return patches <= 9 * (int64_t)sm_count_fast() ? kSplit : 1;
}

namespace {
using PatchFn = void (*)(const BatchVol *, int, PatchQueue, int, PatchScratch);
PatchFn patch_fn(bool big, int split) {
  return split == 1 ? (big ? &k_patch<true, 1> : &k_patch<false, 1>)
                    : (big ? &k_patch<true, kSplit> : &k_patch<false, kSplit>);
}
}  // namespace

KernelShape patch_shape(int split) {
  cudaFuncAttributes a{};
  cudaFuncGetAttributes(&a, patch_fn(false, split));
  return KernelShape{split, kUnion, a.numRegs};
}

void patch_launch(bool big, const PatchPlan &P, cudaStream_t st, const BatchVol *vols) {
  patch_fn(big, P.split)<<<P.grid[big], 32, patch_smem(P.hs_max), st>>>(vols, P.nitems, P.Q, P.hs_max, P.scratch[big]);
}

int patch_plan(vo_ctx *ctx, int nitems, int split, int hs_max, PatchPlan &P) {
  P = PatchPlan();
  P.nitems = nitems;
  P.split = split;
  P.hs_max = hs_max;
  int per_sm = 0;
  cudaError_t e =
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, patch_fn(false, split), 32, patch_smem(hs_max));
  if (e != cudaSuccess) return cuda_error(ctx, e, "k_patch");
  P.grid[0] = std::max(1, std::min(nitems, std::max(1, per_sm) * sm_count_fast()));
  P.grid[1] = std::max(1, std::min(nitems, kPatchBigBlocks));
  return VO_OK;
}

namespace {
size_t tier_entries(bool big) { return big ? kEntriesBig : kEntries; }
size_t tier_unions(bool big) { return big ? kUnionBig : kUnion; }
size_t tier_shorts(bool big) { return big ? kShortBig : kShort; }
}  // namespace

size_t patch_scratch_bytes(const PatchPlan &P, bool big) {
  const size_t cols = 32 / P.split;
  return P.grid[big] * (cols * (tier_entries(big) + tier_unions(big)) * (sizeof(float2) + 2 * sizeof(int2)) +
                        tier_shorts(big) * sizeof(float4));
}

void patch_scratch_set(PatchPlan &P, bool big, void *mem) {
  const size_t w = P.grid[big], ne = tier_entries(big), nu = tier_unions(big), cols = 32 / P.split;
  PatchScratch &S = P.scratch[big];
  unsigned char *p = static_cast<unsigned char *>(mem);
  S.shorts = reinterpret_cast<float4 *>(p);
  p += w * tier_shorts(big) * sizeof(float4);
  S.sv = reinterpret_cast<float2 *>(p);
  p += w * cols * ne * sizeof(float2);
  S.ids = reinterpret_cast<int2 *>(p);
  p += w * 2 * cols * ne * sizeof(int2);
  S.cv = reinterpret_cast<float2 *>(p);
  p += w * cols * nu * sizeof(float2);
  S.cids = reinterpret_cast<int2 *>(p);
}

int big_blocks(int64_t columns) {
  return (int)std::max<int64_t>(1, std::min<int64_t>(sm_count_fast(), (columns + kBigThreads - 1) / kBigThreads));
}
size_t big_scratch_elems(int blocks, int cap) { return (size_t)blocks * kBigThreads * cap; }

void big_launch(cudaStream_t st, const BatchVol *vols, int nv, double2 *scratch, int blocks, int cap) {
  k_big<<<blocks, kBigThreads, 0, st>>>(vols, nv, scratch, cap);
}

size_t pack_offsets(const vo_grid &g) {
  return (size_t)((g.ny + kTile - 1) / kTile) * ((g.nx + kTile - 1) / kTile + 1);
}

void fast_prepare(cudaStream_t st, const FastArgs &A, float R, double mean_segs, unsigned long long *mm,
                  const PackOut &out) {
  const double2 *z = reinterpret_cast<const double2 *>(A.zd);
  cudaMemsetAsync(mm, 0, 4 * sizeof(unsigned long long), st);
  // warps per block by the segments of a tile: twice the mean should fit a warp's share of the sort
  const double most = 2.2 * mean_segs * kTile * std::min(kTile, A.ny);
  const int warps = most <= kPackSort / 32 ? 32 : most <= kPackSort / 16 ? 16 : 8;
  auto *pack = warps == 32 ? &k_pack<32> : warps == 16 ? &k_pack<16> : &k_pack<8>;
  (A.off != 0.0 ? &k_widths<false, false, true> : &k_widths<false, false, false>)<<<A.ny, kPrepThreads, 0, st>>>(
      A.nx, A.ny, A.beg, A.end, reinterpret_cast<const longlong2 *>(z), nullptr, nullptr, nullptr, nullptr, out.wide, R, mm,
      out.par, A.off);
  pack<<<(A.ny + kTile - 1) / kTile, 32 * warps, 0, st>>>(A.nx, A.ny, A.beg, A.end, z, out.par, out.zf, out.wide, out.code,
                                                          out.zx, out.cl, out.coff);
}

FastArgs fast_args(const vo_grid &g, const DeviceTables &T, const int32_t *beg, const int32_t *end, const double2 *z,
                   const PackOut &out) {
  const int nx = g.nx, ny = g.ny;
  return FastArgs{nx,  ny,  T.host.W, T.host.Dy, T.host.hs, beg, end, (const double *)z, out.zf, out.code,
                  (const double *)out.zx, out.cl, out.coff, T.Hp, T.H, T.Dx, out.par, out.rec, out.zx ? out.zx : z,
                  out.zx ? out.rbeg : beg, out.zx ? out.rbeg + (size_t)nx * ny : end, value_offset(g)};
}

// Threads per column: the line is explained at k_direct.
static int direct_split(int64_t cols) {
  return cols <= kDirectSplitCols ? kSplit : 1;
}
int direct_blocks(const vo_grid &g, int64_t launch_cols) {
  const int cols = 32 / direct_split(launch_cols);
  return ((g.nx + cols - 1) / cols) * ((g.ny + 3) / 4);
}
void direct_prepare(cudaStream_t st, const FastArgs &A, const PackOut &out) {
  if (A.ny <= 0) return;
  const longlong2 *z = reinterpret_cast<const longlong2 *>(A.zd);
  const bool shift = A.off != 0.0;
  auto *widths = out.zx ? (shift ? &k_widths<true, true, true> : &k_widths<true, true, false>)
                        : (shift ? &k_widths<false, true, true> : &k_widths<false, true, false>);
  widths<<<A.ny, kPrepThreads, 0, st>>>(A.nx, A.ny, A.beg, A.end, z, out.rec, reinterpret_cast<longlong2 *>(out.zx), out.rbeg,
                                        out.zx ? out.rbeg + (size_t)A.nx * A.ny : nullptr, nullptr, 0.f, nullptr, nullptr,
                                        A.off);
}
static size_t direct_table(int nx, int ny, int W, int Dy) {
  return sizeof(float2) * (size_t)std::min(W, nx) * (std::min(Dy, ny - 1) + 1);
}
size_t direct_smem(const FastArgs &A) { return direct_table(A.nx, A.ny, A.W, A.Dy); }
static auto *direct_kernel(int64_t launch_cols, bool shift) {
  return direct_split(launch_cols) == 1 ? (shift ? &k_direct<1, true> : &k_direct<1, false>)
                                        : (shift ? &k_direct<kSplit, true> : &k_direct<kSplit, false>);
}
KernelShape direct_shape(int64_t launch_cols, bool shift) {
  cudaFuncAttributes a{};
  cudaFuncGetAttributes(&a, direct_kernel(launch_cols, shift));
  return KernelShape{direct_split(launch_cols), kDirectCap, a.numRegs};
}
void direct_launch(cudaStream_t st, const BatchVol *vols, int nv, int blocks, int64_t launch_cols, size_t smem, bool shift) {
  direct_kernel(launch_cols, shift)<<<blocks, 128, smem + sizeof(float2) * kList * 128, st>>>(vols, nv);
}

double reach_columns(const vo_grid &g, const DeviceTables &T) {
  double cols = 0;
  for (int d = 0; d <= std::min(T.host.Dy, g.ny - 1); ++d)
    cols += (d ? 2.0 : 1.0) * (1.0 - (double)d / g.ny) * std::min(2 * T.host.Dx[d] + 1, g.nx);
  return cols;
}

bool direct_choice(const vo_grid &g, const DeviceTables &T, double mean_segs) {
  const double cols = reach_columns(g, T);
  // patches are four rows high: of a grid of fewer rows they use as much less
  if (g.nx < 1 || g.ny < 1 || g.nx > 65535 || direct_table(g.nx, g.ny, T.host.W, T.host.Dy) > 31 * 1024) return false;
  return cols * std::max(mean_segs, 1.0) <= kDirectWork * kPatchY / std::min(g.ny, kPatchY);
}

int dilate_fast(vo_ctx *ctx, double R, const vo_volume *in, vo_volume **out, vo_timings *tm) {
  const vo_grid g = in->grid;
  const int nx = g.nx, ny = g.ny, ncols = nx * ny;
  const DeviceTables *T = nullptr;
  int rc = get_tables(ctx, R, std::max(nx, ny), &T);
  if (rc) return rc;
  const double mean_segs = (double)in->nseg / std::max(ncols, 1);
  Engine engine = direct_choice(g, *T, mean_segs) ? Engine::kDirect : Engine::kPatches;
  {
    bool columns = false;
    rc = column_choice(ctx, g, *T, mean_segs, in->offs, in->offs + 1, in->z, [] {}, &columns);
    if (rc) return rc;
    if (columns || (engine == Engine::kPatches && in->nseg > kPatchSegments)) engine = Engine::kColumns;
  }
  int union_slots = column_slots(mean_segs);
  SlotLayout slots = slots_first(ncols, mean_segs);
  std::vector<void *> mem;
  auto take = [&](void **p, size_t bytes) -> int {
    unsigned char *q = nullptr;
    const int r = dalloc(ctx, &q, bytes);
    *p = q;
    if (!r) mem.push_back(q);
    return r;
  };
  auto take_n = [&](auto **p, size_t n) -> int { return *p ? VO_OK : take((void **)p, n * sizeof(**p)); };
  const size_t nseg = (size_t)std::max<int64_t>(in->nseg, 1);
  // misc: range orders (4 x 8 bytes), FastPar at 64, counters at 128 (4 of the queue, FP64-tier columns,
  // spill used, overflow flags, columns for k_column_list, listed patches, large unions), the launch's BatchVol at 256 and
  // its ColumnArgs, then the columns' slots and the FP64 tier's list; all up to the slots is written by one copy
  struct Head {
    unsigned char zeros[256];
    BatchVol V;
    ColumnArgs C;
  } head;
  static_assert(offsetof(Head, V) == 256, "the counters lie before the launch's description");
  constexpr int kCounters = 10;
  const size_t head_bytes = (sizeof(Head) + 255) / 256 * 256;
  unsigned char *misc = nullptr;
  rc = take((void **)&misc, head_bytes + sizeof(int32_t) * 3 * (size_t)ncols);
  BatchVol *dv = nullptr;
  int32_t *obeg = nullptr;
  int *cnt = nullptr;
  PackOut pk;
  if (!rc) {
    dv = reinterpret_cast<BatchVol *>(misc + offsetof(Head, V));
    obeg = reinterpret_cast<int32_t *>(misc + head_bytes);
    pk.par = reinterpret_cast<FastPar *>(misc + 64);
    cnt = reinterpret_cast<int *>(misc + 128);
  }
  PatchPlan P;
  ColumnPrep cp;
  int *list = nullptr, *over_list = nullptr;
  unsigned char *scratch[2] = {nullptr, nullptr};
  double2 *oz = nullptr, *big = nullptr;
  // what an engine needs beside that
  int *const big_list = obeg ? obeg + 2 * (size_t)ncols : nullptr;
  auto memory = [&](Engine e) -> int {
    int r = VO_OK;
    if (e == Engine::kDirect) {
      if (!r) r = take_n(&pk.rec, nseg);
    } else if (e == Engine::kPatches) {
      const vo_grid *const gp = &g;
      const int split = patch_split(&gp, 1);
      if (!r) r = patch_plan(ctx, patch_count(g, split), split, T->host.hs, P);
      if (!r) r = take_n(&pk.zf, nseg);
      if (!r) r = take_n(&pk.code, nseg);
      if (!r) r = take_n(&pk.wide, nseg);
      if (!r) r = take_n(&pk.zx, nseg);
      if (!r) r = take_n(&pk.cl, nseg);
      if (!r) r = take_n(&pk.coff, pack_offsets(g));
      if (!r) r = take_n(&list, (size_t)P.nitems);
      if (!r) r = take_n(&scratch[0], patch_scratch_bytes(P, false));
      if (!r) patch_scratch_set(P, false, scratch[0]);
      P.Q = PatchQueue{cnt, list};
    } else if (!cp.zf) {
      if (!r) r = column_tables(ctx, T);
      if (!r) r = column_alloc(g, nseg, mean_segs, take, cp);
      if (!r) r = take_n(&over_list, (size_t)ncols);
    }
    return r;
  };
  auto prepare_columns = [&]() {
    column_prepare(ctx->stream, head.C, (float)R, T->dom, cp);
    ctx->launches += 3;
  };
  auto last_tier = [&](int64_t columns) -> int {
    const int blocks = big_blocks(columns);
    const int r = take_n(&big, big_scratch_elems(big_blocks(ncols), kBigCap));
    if (r) return r;
    big_launch(ctx->stream, dv, 1, big, blocks, kBigCap);
    ctx->launches += 1;
    return VO_OK;
  };
  auto describe = [&](Engine e) {
    BatchVol &V = head.V;
    V.A = fast_args(g, *T, in->offs, in->offs + 1, in->z, pk);
    V.obeg = obeg;
    V.oend = obeg + ncols;
    V.oz = oz;
    V.cap = slots.cap;
    V.item1 = e == Engine::kDirect ? direct_blocks(g, ncols) : e == Engine::kPatches ? P.nitems : patch_count(g, 1);
    V.spill_base = (unsigned)((int64_t)ncols * slots.cap);
    V.spill_cap = (unsigned)slots.spill;
    V.big_list = big_list;
    V.big_count = cnt + 4;
    V.spill_used = reinterpret_cast<unsigned *>(cnt + 5);
    V.ovf = cnt + 6;
    V.column = reinterpret_cast<const ColumnArgs *>(misc + offsetof(Head, C));
    V.over_list = over_list;
    V.over_count = cnt + 7;
    V.listed = e == Engine::kDirect ? V.big_count : cnt + 8;
    V.most = e == Engine::kDirect ? kFewColumns + ncols / 64 : kFewPatches + P.nitems / 64;
    V.large = cnt + 9;
    if (cp.zf) head.C = column_args(nx, ny, *T, in->offs, in->offs + 1, in->z, cp);
  };
  if (!rc) rc = memory(engine);
  vo_volume *res = nullptr;
  int cols2 = 0;
  for (int attempt = 0; !rc; ++attempt) {
    rc = dalloc(ctx, &oz, (size_t)ncols * slots.cap + (size_t)slots.spill);
    if (rc) break;
    std::memset(&head, 0, sizeof head);
    describe(engine);
    cudaMemcpyAsync(misc, &head, sizeof head, cudaMemcpyHostToDevice, ctx->stream);
    cudaEventRecord(ctx->ev[0], ctx->stream);
    if (engine == Engine::kDirect)
      direct_prepare(ctx->stream, head.V.A, pk);
    else if (engine == Engine::kPatches)
      fast_prepare(ctx->stream, head.V.A, (float)R, mean_segs, reinterpret_cast<unsigned long long *>(misc), pk);
    else
      prepare_columns();
    cudaEventRecord(ctx->ev[1], ctx->stream);
    cudaEventRecord(ctx->ev[4], ctx->stream);
    if (engine == Engine::kDirect)
      direct_launch(ctx->stream, dv, 1, head.V.item1, ncols, direct_smem(head.V.A), head.V.A.off != 0.0);
    else if (engine == Engine::kPatches)
      patch_launch(false, P, ctx->stream, dv);
    else
      column_launch(ctx->stream, dv, 1, head.V.item1, union_slots, head.C);
    cudaEventRecord(ctx->ev[5], ctx->stream);
    ctx->launches += engine == Engine::kDirect ? 2 : engine == Engine::kPatches ? 3 : 1;
    SlotVol sv;
    sv.grid = g;
    sv.cap = slots.cap;
    sv.beg = obeg;
    sv.end = obeg + ncols;
    sv.z = oz;
    int hc[kCounters] = {0};
    rc = slot_to_volume(ctx, sv, &res, cnt, hc, kCounters);
    if (rc) break;
    const int patches = hc[1], fp64 = hc[4], over = hc[7], listed = engine == Engine::kDirect ? fp64 : hc[8];
    if (engine != Engine::kColumns && listed > head.V.most) {  // left undone: all of it by columns, with room for large unions
      vo_volume_free(ctx, res);
      res = nullptr;
      dfree(ctx, oz);
      oz = nullptr;
      engine = Engine::kColumns;
      union_slots = 24;  // few of its columns have so few, and the more lists it keeps the longer they take to outgrow them
      slots_many(ncols, slots);
      rc = memory(engine);
      --attempt;
      continue;
    }
    cols2 = engine == Engine::kPatches ? std::max(hc[3], fp64) : over;
    if (patches + fp64 + over > 0) {  // what the later tiers take
      vo_volume_free(ctx, res);
      res = nullptr;
      const bool many = (engine == Engine::kDirect && fp64 > kFewColumns) || (engine == Engine::kPatches && patches > kFewPatches);
      if (many) {  // by k_column_list
        rc = memory(Engine::kColumns);
        describe(engine);
        BatchVol &V = head.V;
        if (engine == Engine::kDirect) {  // its list becomes that kernel's
          V.over_list = big_list;
          V.over_count = cnt + 4;
          V.big_list = over_list;
          V.big_count = cnt + 7;
        }
        V.listed = cnt + 8;  // no limit from here on
        V.most = 2147483647;
        if (!rc) {
          cudaMemcpyAsync(dv, &head.V, sizeof head.V + sizeof head.C, cudaMemcpyHostToDevice, ctx->stream);
          prepare_columns();
          if (engine == Engine::kPatches) {
            k_patch_columns<<<std::min(patches, 4096), 32, 0, ctx->stream>>>(dv, list, cnt + 1, kPatchX / P.split);
            ctx->launches += 1;
          }
        }
      } else if (patches > 0) {
        rc = take_n(&scratch[1], patch_scratch_bytes(P, true));
        if (!rc) {
          patch_scratch_set(P, true, scratch[1]);
          patch_launch(true, P, ctx->stream, dv);
          ctx->launches += 1;
        }
      }
      if (!rc && (many || over > 0)) {
        column_list_launch(ctx->stream, dv, 1);
        ctx->launches += 1;
      }
      if (!rc) rc = last_tier(many || patches + over > 0 ? ncols : fp64);
      if (!rc) rc = slot_to_volume(ctx, sv, &res, cnt, hc, kCounters);
      if (rc) break;
      if (engine == Engine::kDirect) cols2 = hc[9];
    }
    if (hc[6] & 1) {
      rc = set_error(ctx, VO_EINTERNAL, "a column exceeds the fallback union capacity");
    } else if (hc[6] & 4) {  // the spill region was too small: its counter says what it takes
      vo_volume_free(ctx, res);
      res = nullptr;
      dfree(ctx, oz);
      oz = nullptr;
      if (attempt >= 2 || !slots_next(ncols, (int64_t)(unsigned)hc[5], slots))
        rc = set_error(ctx, VO_ERANGE, "dilation: the result exceeds the slot range");
      continue;
    }
    break;
  }
  if (!rc) {
    ctx->ovf_cols += cols2;
    if (tm) {
      float e0 = 0, e1 = 0;
      cudaEventElapsedTime(&e0, ctx->ev[0], ctx->ev[1]);
      cudaEventElapsedTime(&e1, ctx->ev[4], ctx->ev[5]);
      tm->pass1_ms += e0;
      tm->pass2_ms += e1;
      tm->kernel_ms[0] += e0;
      tm->kernel_ms[2] += e1;
    }
  }
  dfree(ctx, oz);
  for (void *p : mem) dfree(ctx, p);
  if (rc) {
    if (res) vo_volume_free(ctx, res);
    return rc;
  }
  *out = res;
  return VO_OK;
}

}  // namespace vo
