// Mesh -> dexels by vertical ray casting on sm_103a (replaces create_dexels +
// compute_sign, src/vor3d/Dexelize.cpp:166-274).
//
//  1. host: bounding box, spacing and grid exactly as create_dexels
//     (Dexelize.cpp:254-271) and the CompressedVolume constructor
//     (CompressedVolume.cpp:11-23);
//  2. k_raster: every facet visits the columns whose centre lies in its xy
//     bounding box (inclusive, as geogram's AABB box query), makes the
//     SOS-robust inside test and barycentric z of Dexelize.cpp:56-162 and adds
//     the hit, divided by the spacing, to the column's list;
//  3. k_pairs: the lists are sorted and paired into segments.
//
// A facet that visits its columns loads its vertices once and tests only real
// candidates; columns that look for facets test each one against every column
// around it, gather its vertices anew each time, and do all of it twice, to
// count and to fill (256^2 columns, 32768 facets: 0.5 + 0.4 ms). A column's
// first hits go to its slots; only if some column has more are all hits counted
// exactly, and the facets visited once more to put them into lists of that size.
// All FP64 products/sums use explicit round-to-nearest intrinsics so nothing
// is contracted into FMA: results equal the reference's x86 FP64 arithmetic.
#include <algorithm>
#include <cmath>
#include <vector>

#include "vo_internal.cuh"

namespace vo {
namespace {

constexpr int kHitSlots = 16;       // hits per column kept at a fixed place
constexpr int kHitCap = 4096;       // hits per column at most
constexpr int kRasterWarps = 4;       // warps per k_raster block
constexpr long long kWarpCols = 256;  // candidate columns of a facet that its warp visits; with more, all blocks do
constexpr int kLargeThreads = 128, kLargeChunk = 512;  // k_raster_large: threads, columns per block and turn

__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }

// orientation (Dexelize.cpp:56-67)
__device__ int orientation(double x1, double y1, double x2, double y2, double &tsa) {
  tsa = sub(mul(y1, x2), mul(x1, y2));
  if (tsa > 0) return 1;
  if (tsa < 0) return -1;
  if (y2 > y1) return 1;
  if (y2 < y1) return -1;
  if (x1 > x2) return 1;
  if (x1 < x2) return -1;
  return 0;
}

// point_in_triangle_2d (Dexelize.cpp:73-92) + intersect_ray_z (:137-162).
__device__ bool ray_hit(double qx, double qy, const double3 &p1, const double3 &p2, const double3 &p3, double &z) {
  const double x1 = sub(p1.x, qx), x2 = sub(p2.x, qx), x3 = sub(p3.x, qx);
  const double y1 = sub(p1.y, qy), y2 = sub(p2.y, qy), y3 = sub(p3.y, qy);
  double a, b, c;
  const int sa = orientation(x2, y2, x3, y3, a);
  if (sa == 0) return false;
  const int sb = orientation(x3, y3, x1, y1, b);
  if (sb != sa) return false;
  const int sc = orientation(x1, y1, x2, y2, c);
  if (sc != sa) return false;
  const double sum = add(add(a, b), c);
  a = __ddiv_rn(a, sum);
  b = __ddiv_rn(b, sum);
  c = __ddiv_rn(c, sum);
  z = add(add(mul(a, p1.z), mul(b, p2.z)), mul(c, p3.z));
  return true;
}

// orient_2d_inexact (Dexelize.cpp:107-121): only a non-degenerate projected
// triangle is hit.
__device__ bool degenerate(const double3 &p1, const double3 &p2, const double3 &p3) {
  const double a11 = sub(p2.x, p1.x), a12 = sub(p2.y, p1.y);
  const double a21 = sub(p3.x, p1.x), a22 = sub(p3.y, p1.y);
  return sub(mul(a11, a22), mul(a12, a21)) == 0;
}

struct Mesh {
  const double3 *v;
  const int3 *f;
  int nt;
};

struct GridView {
  int nx, ny;
  double ox, oy, h;
};

// dexelCenter (CompressedVolumeBase.cpp:5-11)
__device__ __forceinline__ double center(int i, double origin, double h) { return add(mul(i + 0.5, h), origin); }

struct Facet {
  double3 a, b, c;
  int x0, y0, w, h;  // the columns whose centres lie in its bounding box
  __device__ long long cols() const { return (long long)w * h; }
};

// Cells lo..hi whose centres lie in [l, u]: a superset first, then its ends by
// the exact test (centres never decrease with the index).
__device__ __forceinline__ void cells_within(double l, double u, double origin, double h, int n, int &lo, int &hi) {
  lo = max((int)floor((l - origin) / h - 0.5) - 1, 0);
  hi = min((int)ceil((u - origin) / h - 0.5) + 1, n - 1);
  while (lo <= hi && center(lo, origin, h) < l) ++lo;
  while (lo <= hi && center(hi, origin, h) > u) --hi;
}

__device__ Facet load_facet(const Mesh &m, const GridView &g, int f) {
  Facet t;
  const int3 v = m.f[f];
  t.a = m.v[v.x], t.b = m.v[v.y], t.c = m.v[v.z];
  int x1, y1;
  cells_within(fmin(t.a.x, fmin(t.b.x, t.c.x)), fmax(t.a.x, fmax(t.b.x, t.c.x)), g.ox, g.h, g.nx, t.x0, x1);
  cells_within(fmin(t.a.y, fmin(t.b.y, t.c.y)), fmax(t.a.y, fmax(t.b.y, t.c.y)), g.oy, g.h, g.ny, t.y0, y1);
  t.w = max(x1 - t.x0 + 1, 0), t.h = max(y1 - t.y0 + 1, 0);
  if (degenerate(t.a, t.b, t.c)) t.w = 0;
  return t;
}

// Where hits go: slot i of column c at slots[i * ncols + c], or, with lists of
// exact size, entry i of the column's list.
struct Hits {
  int32_t *cnt;         // hits per column so far
  double *slots;
  int nslots;
  const int32_t *loffs; // null: slots
  double *lists;
};

__device__ void visit(const Facet &t, const GridView &g, int x, int y, const Hits &H) {
  double z;
  if (!ray_hit(center(x, g.ox, g.h), center(y, g.oy, g.h), t.a, t.b, t.c, z)) return;
  const double v = __ddiv_rn(z, g.h);
  const int c = x + g.nx * y, i = atomicAdd(&H.cnt[c], 1);
  if (H.loffs)
    H.lists[H.loffs[c] + i] = v;
  else if (i < H.nslots)
    H.slots[(size_t)i * g.nx * g.ny + c] = v;
}

// A warp loads up to 32 facets and its lanes share out all their candidate
// columns, whichever facet they belong to: one lane per facet would wait for the
// largest. Facets beyond kWarpCols are left to k_raster_large: a mesh of two
// triangles has as many candidates as one of a hundred thousand. (With kWarpCols
// at 64 the blocks there spend their time loading one small facet each: 32768
// facets over 1024^2 columns 2.9 ms against 1.1.) FP64 arithmetic is what bounds
// both kernels: 0.06 ms for 32768 facets over 256^2 columns, 0.68 over 1024^2.
__global__ void __launch_bounds__(32 * kRasterWarps) k_raster(Mesh m, GridView g, Hits H, int per_warp, int *nlarge,
                                                              int2 *large) {
  __shared__ Facet s_facet[kRasterWarps][32];
  __shared__ int s_first[kRasterWarps][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int f = (blockIdx.x * kRasterWarps + warp) * per_warp + lane;
  int cols = 0;
  if (lane < per_warp && f < m.nt) {
    const Facet t = load_facet(m, g, f);
    if (t.cols() > kWarpCols) {
      large[atomicAdd(nlarge, 1)] = make_int2(f, (int)((t.cols() + kLargeChunk - 1) / kLargeChunk));
    } else {
      cols = (int)t.cols();
      s_facet[warp][lane] = t;
    }
  }
  int upto = cols;
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, upto, o);
    if (lane >= o) upto += v;
  }
  s_first[warp][lane] = upto - cols;
  const int total = __shfl_sync(0xffffffffu, upto, 31);
  __syncwarp();
  for (int j = lane; j < total; j += 32) {
    int k = 0;  // the last facet whose first candidate is not after j (it has candidates)
    for (int o = 16; o > 0; o >>= 1)
      if (s_first[warp][k + o] <= j) k += o;
    const Facet &t = s_facet[warp][k];
    const int i = j - s_first[warp][k];
    visit(t, g, t.x0 + i % t.w, t.y0 + i / t.w, H);
  }
}

// The large facets, cut into chunks of columns that the blocks take in turn;
// every block finds its own by counting through the list, 32 entries at once.
__global__ void __launch_bounds__(kLargeThreads) k_raster_large(Mesh m, GridView g, Hits H, const int *nlarge,
                                                                const int2 *large) {
  const int n = *nlarge, lane = threadIdx.x & 31, nb = gridDim.x;
  int turn = blockIdx.x;  // entries to go until this block's next chunk
  for (int i0 = 0; i0 < n; i0 += 32) {
    const int2 e = i0 + lane < n ? large[i0 + lane] : make_int2(0, 0);
    unsigned mine = 0;
    int first = turn;  // at entry i: its first chunk that is this block's
    for (int i = 0; i < 32; ++i) {
      const int chunks = __shfl_sync(0xffffffffu, e.y, i);
      if (lane == i) first = turn;
      if (turn < chunks) {
        mine |= 1u << i;
        turn = (chunks - turn - 1) % nb;
        turn = nb - 1 - turn;
      } else {
        turn -= chunks;
      }
    }
    for (; mine; mine &= mine - 1) {
      const int i = __ffs(mine) - 1;
      const int f = __shfl_sync(0xffffffffu, e.x, i), chunks = __shfl_sync(0xffffffffu, e.y, i);
      const Facet t = load_facet(m, g, f);
      const long long cols = t.cols();
      for (int q = __shfl_sync(0xffffffffu, first, i); q < chunks; q += nb) {
        const long long k1 = min((q + 1LL) * kLargeChunk, cols);
        for (long long k = (long long)q * kLargeChunk + threadIdx.x; k < k1; k += kLargeThreads)
          visit(t, g, t.x0 + (int)(k % t.w), t.y0 + (int)(k / t.w), H);
      }
      __syncwarp();
    }
  }
}

// Segments per column; status words: 1 columns beyond the hits allowed, 2 odd
// columns, 3 columns beyond the slots.
__global__ void k_pair_counts(int ncols, const int32_t *hits, int32_t *counts, int nslots, int *flags) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  const int n = c < ncols ? hits[c] : 0;
  if (c < ncols) counts[c] = n / 2;
  const unsigned odd = __ballot_sync(0xffffffffu, n & 1), more = __ballot_sync(0xffffffffu, n > nslots),
                 over = __ballot_sync(0xffffffffu, n > kHitCap);
  if ((threadIdx.x & 31) == 0) {
    if (over) flags[1] = 1;
    if (odd) atomicAdd(&flags[2], __popc(odd));
    if (more) flags[3] = 1;
  }
}

// Sorts a column's hits (std::sort, Dexelize.cpp:208) and writes them in
// pairs; an unpaired trailing hit is ignored. The kernel moves each hit twice
// and is bound by the latency of few loads per column.
__device__ __forceinline__ void sort_hits(double *v, int n) {
  for (int i = 1; i < n; ++i) {
    const double x = v[i];
    int j = i;
    for (; j > 0 && v[j - 1] > x; --j) v[j] = v[j - 1];
    v[j] = x;
  }
}

__global__ void k_pairs(int ncols, const int32_t *cnt, const double *slots, const int32_t *loffs, double *lists,
                        const int32_t *ooffs, double2 *oz) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncols) return;
  const int n = cnt[c];
  double buf[kHitSlots], *v = buf;
  if (loffs)
    v = lists + loffs[c];
  else
    for (int i = 0; i < n; ++i) buf[i] = slots[(size_t)i * ncols + c];
  sort_hits(v, n);
  for (int i = 0; i + 1 < n; i += 2) oz[ooffs[c] + i / 2] = make_double2(v[i], v[i + 1]);
}

}  // namespace
}  // namespace vo

using namespace vo;

extern "C" int vo_dexelize_odd_columns(vo_ctx *ctx, int64_t *count) {
  if (!ctx || !count) return VO_EINVAL;
  if (ctx->dexel_odd_columns < 0) return set_error(ctx, VO_EINVAL, "no successful vo_dexelize on this context");
  *count = ctx->dexel_odd_columns;
  return VO_OK;
}

extern "C" int vo_dexelize(vo_ctx *ctx, const double *verts, int nv, const int32_t *tris, int nt,
                           double *spacing, int padding, int num_dexels, vo_volume **out) {
  if (!ctx) return VO_EINVAL;
  if (!verts || nv <= 0 || nt < 0 || (nt > 0 && !tris) || !spacing || !out || padding < 0)
    return set_error(ctx, VO_EINVAL, "dexelize: bad arguments");
  for (int64_t i = 0; i < 3 * (int64_t)nt; ++i)
    if (tris[i] < 0 || tris[i] >= nv) return set_error(ctx, VO_EINVAL, "dexelize: vertex index out of range");
  cudaSetDevice(ctx->device);
  ctx->err.clear();
  ctx->dexel_odd_columns = -1;
  *out = nullptr;
  // create_dexels (Dexelize.cpp:254-271)
  double mn[3], mx[3];
  for (int k = 0; k < 3; ++k) mn[k] = mx[k] = verts[k];
  for (int i = 1; i < nv; ++i)
    for (int k = 0; k < 3; ++k) {
      mn[k] = std::min(mn[k], verts[3 * i + k]);
      mx[k] = std::max(mx[k], verts[3 * i + k]);
    }
  const double ext[3] = {mx[0] - mn[0], mx[1] - mn[1], mx[2] - mn[2]};
  if (num_dexels > 0) *spacing = std::max(ext[0], std::max(ext[1], ext[2])) / num_dexels;
  const double h = *spacing;
  if (!(h > 0) || !std::isfinite(h)) return set_error(ctx, VO_EINVAL, "dexelize: spacing must be > 0");
  vo_grid g;
  g.spacing = h;
  g.padding = padding;
  for (int k = 0; k < 3; ++k) {
    g.origin[k] = mn[k] - padding * h;
    g.extent[k] = ext[k];
  }
  const double fnx = std::ceil(ext[0] / h) + 2 * padding, fny = std::ceil(ext[1] / h) + 2 * padding;
  if (fnx * fny > 2e9) return set_error(ctx, VO_ERANGE, "dexelize: grid too large");
  g.nx = (int)fnx;
  g.ny = (int)fny;
  const int ncols = g.nx * g.ny;

  double3 *dv = nullptr;
  int3 *df = nullptr;
  int32_t *cnt = nullptr, *counts = nullptr, *loffs = nullptr;
  int *nlarge = nullptr;
  int2 *large = nullptr;
  double *slots = nullptr, *lists = nullptr;
  vo_volume *res = nullptr;
  long long nhits = 0, total = 0;
  // slots for as many hits per column as fit 1 GB (all of them up to 2896^2 columns)
  const int nslots = (int)std::min<long long>(kHitSlots, (1LL << 30) / (8LL * std::max(ncols, 1)));
  const int cblocks = (ncols + 127) / 128;
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device);
  // facets per warp: 32, or fewer where that would leave an SM fewer than four warps
  int per_warp = 32;
  while (per_warp > 1 && nt / per_warp < 4 * sms) per_warp /= 2;
  const int fblocks = (nt + per_warp * kRasterWarps - 1) / (per_warp * kRasterWarps);
  int rc = dalloc(ctx, &dv, (size_t)nv);
  if (!rc) rc = dalloc(ctx, &df, (size_t)std::max(nt, 1));
  if (!rc) rc = dalloc(ctx, &cnt, (size_t)ncols);
  if (!rc) rc = dalloc(ctx, &counts, (size_t)ncols);
  if (!rc) rc = dalloc(ctx, &nlarge, 1);
  if (!rc) rc = dalloc(ctx, &large, (size_t)nt);
  if (!rc) rc = dalloc(ctx, &slots, (size_t)nslots * ncols);
  Mesh m{dv, df, nt};
  GridView gv{g.nx, g.ny, g.origin[0], g.origin[1], h};
  auto raster = [&](const Hits &H) {
    cudaMemsetAsync(cnt, 0, sizeof(int32_t) * ncols, ctx->stream);
    if (nt == 0 || ncols == 0) return;
    cudaMemsetAsync(nlarge, 0, sizeof(int), ctx->stream);
    k_raster<<<fblocks, 32 * kRasterWarps, 0, ctx->stream>>>(m, gv, H, per_warp, nlarge, large);
    k_raster_large<<<8 * std::max(sms, 1), kLargeThreads, 0, ctx->stream>>>(m, gv, H, nlarge, large);
  };
  int hf[4] = {0, 0, 0, 0};
  if (!rc) {
    cudaMemcpyAsync(dv, verts, sizeof(double) * 3 * (size_t)nv, cudaMemcpyHostToDevice, ctx->stream);
    if (nt) cudaMemcpyAsync(df, tris, sizeof(int32_t) * 3 * (size_t)nt, cudaMemcpyHostToDevice, ctx->stream);
    cudaMemsetAsync(ctx->d_flags, 0, 4 * sizeof(int), ctx->stream);
    raster(Hits{cnt, slots, nslots, nullptr, nullptr});
    if (ncols) k_pair_counts<<<cblocks, 128, 0, ctx->stream>>>(ncols, cnt, counts, nslots, ctx->d_flags);
    rc = volume_alloc(ctx, g, 0, &res);
  }
  if (!rc) rc = scan_counts(ctx, counts, res->offs, ncols, &total, ctx->d_flags, hf, 4);
  if (!rc && hf[1]) rc = set_error(ctx, VO_EINTERNAL, "dexelize: a column has more than 4096 hits");
  if (!rc) {
    res->nseg = total;
    rc = dalloc(ctx, &res->z, (size_t)total);
  }
  if (!rc && hf[3]) {
    rc = dalloc(ctx, &loffs, (size_t)ncols + 1);
    if (!rc) rc = scan_counts(ctx, cnt, loffs, ncols, &nhits);
    if (!rc) rc = dalloc(ctx, &lists, (size_t)nhits);
    if (!rc) raster(Hits{cnt, nullptr, 0, loffs, lists});
  }
  if (!rc) {
    if (ncols) k_pairs<<<cblocks, 128, 0, ctx->stream>>>(ncols, cnt, slots, loffs, lists, res->offs, res->z);
    cudaError_t e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess)
      rc = cuda_error(ctx, e, "dexelize");
    else
      ctx->dexel_odd_columns = hf[2];
  }
  dfree(ctx, dv);
  dfree(ctx, df);
  dfree(ctx, cnt);
  dfree(ctx, counts);
  dfree(ctx, nlarge);
  dfree(ctx, large);
  dfree(ctx, slots);
  dfree(ctx, loffs);
  dfree(ctx, lists);
  if (rc) {
    if (res) vo_volume_free(ctx, res);
    return rc;
  }
  *out = res;
  return VO_OK;
}
