// Exact separable dilation with FP32 arithmetic and an FP64 guard, column by
// column: one thread per output column (a warp per 8 x 4 patch of them) walks the
// (|dx|, |dy|) pairs in decreasing H and merges each source column's dilated
// segments into a small sorted union (FP32 values in shared memory, endpoint
// identities in local memory). Candidates, guard band and results are those of the
// patch kernel (vo_fast.cu): every comparison within the band is decided in FP64
// from the identities, every written end is FP64.
//
// Dominance: a segment that lies in a segment of its column's neighbour one
// lattice step toward the output column, widened by at most the growth of H over
// that step, adds nothing that the neighbour's candidate does not cover. Bit masks
// per column hold that for eleven growths, so that a source column costs one load
// of its record and two of its masks however many of its segments are held.
//
// It is the better kernel in two places, and the one for inputs of more than 2^30
// segments (kPatchSegments).
// - Smooth dense inputs at small radii, where most segments are held
//   (column_choice has the measured line).
// - Unions of many intervals: the patch kernel's bins and the lists of k_direct
//   hold some fifty per column. Columns beyond them (or whole inputs of such
//   columns) come here: unions of up to kUnionCapMid - 1 in a second launch over
//   the listed columns, larger ones in the FP64 tier. Scattered segments, 256^2
//   columns, 12 of 1 dexel each over 3000: 21 ms at radius 2 (131 intervals per
//   column) and 178 at 4, where the patch kernel's second tier and a small FP64
//   tier took 820 and 1,100.
// Issue slots and divergence bound it: lanes wait for the longest candidate list of
// their warp (1024^2 spheres, r = 32: 73 % of the issue slots, 16 of 32 lanes).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include <cuda_fp16.h>

#include "vo_internal.cuh"
#include "vo_range.cuh"

namespace vo {
namespace {

constexpr int kKM = kUnionCapMid;  // union capacity of the second launch
constexpr int kBlockCols = kPatchX * kPatchY;  // columns of a block: one warp
constexpr int kMidThreads = 32;

// Identities of union endpoints, kept in local memory and read only when an
// FP32 comparison falls inside the guard band or the output is written.
template <int KA>
struct UnionIds {
  // (input value index as unsigned bits, d | a << 8) of the lower / upper endpoint
  int2 lo[KA], hi[KA];
};

// The index of a segment's value among all: unsigned, an input has up to 2^31 - 1 segments.
__device__ __forceinline__ int value_index(int k, bool upper) { return (int)(2u * (unsigned)k + (upper ? 1u : 0u)); }
__device__ __forceinline__ double value_at(const double *z, int index) { return z[(unsigned)index]; }
// FP32 copies of a segment's ends.
__device__ __forceinline__ float2 copies_at(const float *zf, int k) { return reinterpret_cast<const float2 *>(zf)[k]; }

__device__ __forceinline__ double exact_val(const ColumnArgs &A, int idx, int da, bool plus) {
  const double h = A.H64[(da & 255) * A.W + (da >> 8)];
  const double z = value_at(A.zd, idx);
  return plus ? __dadd_rn(z, h) : __dsub_rn(z, h);
}

// Exact comparisons, out of line: identities are loaded only here.
// Union endpoint (j, hi?) < candidate endpoint (idx, da, plus)?
template <int KA>
__device__ __noinline__ bool ex_u_lt_c(const ColumnArgs &A, const UnionIds<KA> &U, int j, bool jhi, int idx, int da,
                                       bool plus) {
  const double u = jhi ? exact_val(A, U.hi[j].x, U.hi[j].y, true) : exact_val(A, U.lo[j].x, U.lo[j].y, false);
  return u < exact_val(A, idx, da, plus);
}
// Candidate endpoint < union endpoint?
template <int KA>
__device__ __noinline__ bool ex_c_lt_u(const ColumnArgs &A, const UnionIds<KA> &U, int idx, int da, bool plus, int j,
                                       bool jhi) {
  const double u = jhi ? exact_val(A, U.hi[j].x, U.hi[j].y, true) : exact_val(A, U.lo[j].x, U.lo[j].y, false);
  return exact_val(A, idx, da, plus) < u;
}
// Union endpoint (i, ihi) < union endpoint (j, jhi)?
template <int KA>
__device__ __noinline__ bool ex_u_lt_u(const ColumnArgs &A, const UnionIds<KA> &U, int i, bool ihi, int j, bool jhi) {
  const double a = ihi ? exact_val(A, U.hi[i].x, U.hi[i].y, true) : exact_val(A, U.lo[i].x, U.lo[i].y, false);
  const double b = jhi ? exact_val(A, U.hi[j].x, U.hi[j].y, true) : exact_val(A, U.lo[j].x, U.lo[j].y, false);
  return a < b;
}

// The FP16 in the low (lo != 0) or high half of v.
__device__ __forceinline__ __half half_of(unsigned v, int lo) {
  return __ushort_as_half((unsigned short)(lo ? (v & 0xffffu) : (v >> 16)));
}

// FP32 difference t = y - x decides x < y outside the guard band [-E, E].
#define GUARD(t, E, exact) ((t) > (E) ? true : ((t) < -(E) ? false : (exact)))

// Returns the number of intervals of the union (identities in U), or -1 when
// more than KA - 1 are needed (the last of the KA slots holds the sentinel).
//
// `mask` holds the lanes of the warp running this function together. For each
// (|dx|, |dy|) pair the four source columns' segments form one list per lane;
// every lane of the warp iterates to the warp's longest list with a predicate,
// and the loop body has no early exits, so the lanes reconverge after every
// candidate instead of drifting apart over the source transitions.
template <int KA>
__device__ int fast_column(const ColumnArgs &A, float E, int x, int y, float2 *sv, int stride, UnionIds<KA> &U,
                           unsigned mask) {
  int n = 0;
  bool overflow = false;
#define SV(k) sv[(k) * stride]
  // SV(n) holds a sentinel above every value, so the cursor walk stops at
  // the end of the union without a bounds test; the union holds up to KA - 1
  // intervals.
  const float2 kTop = make_float2(INFINITY, INFINITY);
  SV(0) = kTop;
  // Per pair: its four source columns' records and their segment dominance
  // masks at the pair's levels, loaded when the pair starts (only the pair's
  // own table entry is loaded one pair ahead: holding the source records
  // across the merge loop cost more in register spills than their load
  // latency, which the other resident warps hide).
  // Source S: x + a if S & 1 (its neighbour toward the output is at x - 1,
  // direction "x-" = 0), else x - a ("x+" = 1); likewise y with S & 2
  // ("y-" = 2, "y+" = 3).
  const unsigned ncols = (unsigned)A.nx * (unsigned)A.ny;  // the masks of 2^26 columns have indices below 2^32
  const int mbits = A.mask_bits;
#define MASK(DIR, LV, C)                                                                                \
  ((LV) < kDomLevels ? (mbits == 16 ? (unsigned)static_cast<const unsigned short *>(A.dmask)[((DIR) * kDomLevels + (LV)) * ncols + (unsigned)(C)] \
                                    : static_cast<const unsigned *>(A.dmask)[((DIR) * kDomLevels + (LV)) * ncols + (unsigned)(C)])        \
                     : 0u)
#define LOAD_ONE(OK, XS, YS, S, R, D)                                                                   \
  {                                                                                                     \
    const int c_ = (OK) ? (XS) + A.nx * (YS) : 0;                                                       \
    R = (OK) ? reinterpret_cast<const int2 *>(A.col)[2 * c_] : make_int2(0, 0);                          \
    D = (OK) ? (MASK((S) & 1 ? 0 : 1, lx_, c_) | MASK((S) & 2 ? 2 : 3, ly_, c_)) : 0u;                  \
  }
#define LOAD_SOURCES(PR)                                                                                \
  {                                                                                                     \
    const int ad_ = __float_as_int((PR).x), a_ = ad_ & 0xff, d_ = (ad_ >> 8) & 0xff;                    \
    const int lx_ = (ad_ >> 16) & 0xf, ly_ = (ad_ >> 20) & 0xf;                                         \
    const bool xm = x - a_ >= 0, xp = a_ > 0 && x + a_ < A.nx;                                          \
    const bool ym = y - d_ >= 0, yp = d_ > 0 && y + d_ < A.ny;                                          \
    LOAD_ONE(xm && ym, x - a_, y - d_, 0, c0, d0)                                                       \
    LOAD_ONE(xp && ym, x + a_, y - d_, 1, c1, d1)                                                       \
    LOAD_ONE(xm && yp, x - a_, y + d_, 2, c2, d2)                                                       \
    LOAD_ONE(xp && yp, x + a_, y + d_, 3, c3, d3)                                                       \
  }
  float4 pr = A.prec[0];
  for (int p = 0; p < A.npairs; ++p) {
    if (__all_sync(mask, overflow)) break;
    const float4 pc = pr;
    if (p + 1 < A.npairs) pr = A.prec[p + 1];
    int2 c0, c1, c2, c3;  // (beg, end) of each source column
    unsigned d0, d1, d2, d3;
    LOAD_SOURCES(pc)
    const int ad = __float_as_int(pc.x), a = ad & 0xff, d = (ad >> 8) & 0xff;
    const float h = pc.y;
    const int da = d | (a << 8);
    // growth of H over one step toward the output column (x step, y step),
    // against which the sources' dominance widths are tested
    const float dhx = pc.z, dhy = pc.w;
    // FP16 bounds of the pair's growths (rounded down) for the source tests
    const __half dhx_h = __float2half_rd(dhx), dhy_h = __float2half_rd(dhy);
    // Per source: [kb, ke) and the mask of its kept segments (bit j: segment
    // kb + j); a source of more than mbits segments keeps all (m = 0, dense).
    // A source of up to mbits segments that is dominated whole has an empty kept
    // mask; a source of more segments (no masks) is tested with its column
    // widths.
#define SRC(S, XS, YS, C, DM, KB, KE, M)                                                                \
  {                                                                                                     \
    KB = (C).x;                                                                                         \
    KE = (C).y;                                                                                         \
    const int ns_ = KE - KB;                                                                            \
    if (ns_ > mbits) {                                                                                  \
      const int4 cr_ = A.col[(XS) + A.nx * (YS)];                                                       \
      if (__hle(half_of((unsigned)cr_.z, (S) & 1), dhx_h) || __hle(half_of((unsigned)cr_.w, (S) & 2), dhy_h)) \
        KE = KB;                                                                                        \
    }                                                                                                   \
    M = ns_ <= mbits ? ~(DM) & (ns_ == 32 ? 0xffffffffu : ((1u << ns_) - 1u)) : 0u;                    \
  }
    int kb0, ke0, kb1, ke1, kb2, ke2, kb3, ke3;
    unsigned m0, m1, m2, m3;
    SRC(0, x - a, y - d, c0, d0, kb0, ke0, m0)
    SRC(1, x + a, y - d, c1, d1, kb1, ke1, m1)
    SRC(2, x - a, y + d, c2, d2, kb2, ke2, m2)
    SRC(3, x + a, y + d, c3, d3, kb3, ke3, m3)
#undef SRC
#define KEPT(KB, KE, M) ((KE) - (KB) > mbits ? (KE) - (KB) : __popc(M))
    const int t0 = KEPT(kb0, ke0, m0), t1 = KEPT(kb1, ke1, m1), t2 = KEPT(kb2, ke2, m2), t3 = KEPT(kb3, ke3, m3);
#undef KEPT
    const int total = t0 + t1 + t2 + t3;
    const int iters = __reduce_max_sync(mask, total);
    // Walk state: the sources still to visit that keep candidates (bit s),
    // the current source s, its remaining mask ms (sparse) or next index kc
    // (dense); NEXT yields the next kept candidate (KN, SN), or KN = -1. A
    // source is entered only when it keeps a candidate, so NEXT takes at most
    // one source switch and no loop.
    unsigned srcs = (t0 > 0 ? 1u : 0u) | (t1 > 0 ? 2u : 0u) | (t2 > 0 ? 4u : 0u) | (t3 > 0 ? 8u : 0u);
    int s = -1, kc = 0, kend = 0, kbs = 0;
    unsigned ms = 0;
    bool dense = false;
#define NEXT(KN, SN)                                                                                    \
  {                                                                                                     \
    if ((dense ? kc >= kend : ms == 0u) && srcs) {                                                      \
      s = __ffs(srcs) - 1;                                                                              \
      srcs &= srcs - 1;                                                                                 \
      kbs = s == 0 ? kb0 : s == 1 ? kb1 : s == 2 ? kb2 : kb3;                                           \
      kend = s == 0 ? ke0 : s == 1 ? ke1 : s == 2 ? ke2 : ke3;                                          \
      ms = s == 0 ? m0 : s == 1 ? m1 : s == 2 ? m2 : m3;                                                \
      dense = kend - kbs > mbits;                                                                       \
      kc = kbs;                                                                                         \
    }                                                                                                   \
    KN = -1;                                                                                            \
    if (dense) {                                                                                        \
      if (kc < kend) KN = kc++;                                                                         \
    } else if (ms) {                                                                                    \
      KN = kbs + __ffs(ms) - 1;                                                                         \
      ms &= ms - 1;                                                                                     \
    }                                                                                                   \
    SN = s;                                                                                             \
  }
    int cur = 0, cur_src = -1;
    float2 cv = make_float2(0.f, 0.f);
    int kn, sn;
    NEXT(kn, sn)
    float2 znext = kn >= 0 ? copies_at(A.zf, kn) : make_float2(0.f, 0.f);
    for (int it = 0; it < iters; ++it) {
      if (it < total && !overflow) {
        const int k = kn, src = sn;
        const float2 zf = znext;
        NEXT(kn, sn)
        if (kn >= 0) znext = copies_at(A.zf, kn);
        if (src != cur_src) {  // first candidate of a new source column: restart the cursor
          cur_src = src;
          cur = 0;
          cv = SV(0);
        }
        {
          const float lo = zf.x - h, hi = zf.y + h;
          const int il = value_index(k, false), ih = value_index(k, true);
          // skip union intervals that end strictly below the candidate: U.hi[cur] < lo
          // (the next interval's values are loaded one step ahead)
          if (lo - cv.y > E) {  // two intervals per step: cur < n here, so cur + 1 <= n
            float2 c1 = SV(cur + 1), c2 = SV(min(cur + 2, n));
            for (;;) {
              if (!(lo - c1.y > E)) {
                cur += 1;
                cv = c1;
                break;
              }
              if (!(lo - c2.y > E)) {
                cur += 2;
                cv = c2;
                break;
              }
              cur += 2;
              c1 = SV(cur + 1);
              c2 = SV(min(cur + 2, n));
            }
          }
          while (cur < n && GUARD(lo - cv.y, E, ex_u_lt_c(A, U, cur, true, il, da, false))) {
            ++cur;
            cv = SV(cur);
          }
          // covered: inside U[cur]; else ext_lo / ext_hi: the candidate reaches
          // below / above U[cur] (both decided once, used again to extend it)
          bool covered = false, ext_lo = false, ext_hi = false;
          if (cur < n) {
            if (lo - cv.x > E && cv.y - hi > E) {
              covered = true;  // inside U[cur] by more than the guard band
            } else {
              ext_lo = GUARD(cv.x - lo, E, ex_c_lt_u(A, U, il, da, false, cur, false));
              ext_hi = GUARD(hi - cv.y, E, ex_u_lt_c(A, U, cur, true, ih, da, true));
              covered = !ext_lo && !ext_hi;
            }
          }
          if (!covered) {
            if (cur == n || GUARD(cv.x - hi, E, ex_c_lt_u(A, U, ih, da, true, cur, false))) {
              // disjoint: insert before cur
              if (n >= KA - 1) {
                overflow = true;
              } else {
                for (int j = n; j > cur; --j) {
                  SV(j) = SV(j - 1);
                  U.lo[j] = U.lo[j - 1];
                  U.hi[j] = U.hi[j - 1];
                }
                cv = make_float2(lo, hi);
                SV(cur) = cv;
                U.lo[cur] = make_int2(il, da);
                U.hi[cur] = make_int2(ih, da);
                ++n;
                SV(n) = kTop;
              }
            } else {
              // overlapping or touching U[cur]: extend it
              if (ext_lo) {
                cv.x = lo;
                U.lo[cur] = make_int2(il, da);
              }
              if (ext_hi) {
                cv.y = hi;
                U.hi[cur] = make_int2(ih, da);
                // absorb following intervals that now start at or below the new end
                int j = cur + 1;
                while (j < n) {
                  const float2 nv = SV(j);
                  if (GUARD(nv.x - cv.y, E, ex_u_lt_u(A, U, cur, true, j, false))) break;  // U.hi[cur] < U.lo[j]
                  if (GUARD(nv.y - cv.y, E, ex_u_lt_u(A, U, cur, true, j, true))) {       // U.hi[cur] < U.hi[j]
                    cv.y = nv.y;
                    U.hi[cur] = U.hi[j];
                  }
                  ++j;
                }
                const int gone = j - cur - 1;
                if (gone > 0) {
                  for (int m = cur + 1; m + gone < n; ++m) {
                    SV(m) = SV(m + gone);
                    U.lo[m] = U.lo[m + gone];
                    U.hi[m] = U.hi[m + gone];
                  }
                  n -= gone;
                  SV(n) = kTop;
                }
              }
              SV(cur) = cv;
            }
          }
        }
      }
    }
  }
#undef SV
#undef LOAD_SOURCES
#undef LOAD_ONE
#undef MASK
#undef NEXT
  return overflow ? -1 : n;
}


// Writes the exact FP64 union held by U (n intervals) to out[0..n).
template <int KA>
__device__ __forceinline__ void write_union(const ColumnArgs &A, const UnionIds<KA> &U, int n, double2 *out) {
  for (int k = 0; k < n; ++k)
    out[k] = make_double2(exact_val(A, U.lo[k].x, U.lo[k].y, false), exact_val(A, U.hi[k].x, U.hi[k].y, true));
}

// The n intervals (-1: too many) of column (x, y) to its output slots, or the column to `list`.
template <int KA>
__device__ __forceinline__ void finish_column(const BatchVol &V, const ColumnArgs &A, const UnionIds<KA> &U, int x, int y,
                                              int n, int *list, int *count) {
  const int c = x + A.nx * y;
  unsigned dst = 0;
  if (n < 0) {
    list[atomicAdd(count, 1)] = c;
    n = 0;
  } else if (!place_union(V, x, y, n, dst)) {
    n = 0;
    dst = 0;
  } else {
    write_union(A, U, n, V.oz + dst);
  }
  V.obeg[c] = (int32_t)dst;
  V.oend[c] = (int32_t)(dst + (unsigned)n);
}

// Patches of the launch's dilations, a block (warp) each, in bands of 512 columns,
// all rows of a band before the next: the blocks running together cover a compact
// region, whose source columns stay in L2. At most 64 registers, so that 32 warps
// fit an SM. Unions of more than KA - 1 intervals are listed. SINGLE: the
// launch has one dilation, whose arguments come as the kernel's (constant bank).
template <int KA, bool SINGLE>
__global__ void __launch_bounds__(kBlockCols, 32) k_column(const BatchVol *__restrict__ vols, int nv, const ColumnArgs A1) {
  extern __shared__ float2 sv_dyn[];
  __shared__ BatchVol V;
  __shared__ ColumnArgs s_args;
  int v = 0;
  for (int r = nv - 1; v < r;) {
    const int m = (v + r) >> 1;
    if ((int)blockIdx.x < vols[m].item1) r = m; else v = m + 1;
  }
  for (int i = threadIdx.x; i < (int)(sizeof(BatchVol) / sizeof(int)); i += kBlockCols)
    reinterpret_cast<int *>(&V)[i] = reinterpret_cast<const int *>(&vols[v])[i];
  __syncwarp();
  if (!SINGLE) {
    for (int i = threadIdx.x; i < (int)(sizeof(ColumnArgs) / sizeof(int)); i += kBlockCols)
      reinterpret_cast<int *>(&s_args)[i] = reinterpret_cast<const int *>(V.column)[i];
    __syncwarp();
  }
  const ColumnArgs &A = SINGLE ? A1 : s_args;
  constexpr int kBand = 512 / kPatchX;
  const int tiles_x = (A.nx + kPatchX - 1) / kPatchX, tiles_y = (A.ny + kPatchY - 1) / kPatchY;
  const int item = (int)blockIdx.x - V.item0, band = item / (kBand * tiles_y), rb = item - band * kBand * tiles_y;
  const int bw = min(kBand, tiles_x - band * kBand);
  const int x = (band * kBand + rb % bw) * kPatchX + threadIdx.x % kPatchX;
  const int y = (rb / bw) * kPatchY + threadIdx.x / kPatchX;
  if (x >= A.nx || y >= A.ny) return;
  UnionIds<KA> U;
  const unsigned mask = __activemask();
  const int n = fast_column<KA>(A, A.par->E, x, y, sv_dyn + threadIdx.x, kBlockCols, U, mask);
  finish_column(V, A, U, x, y, n, V.over_list, V.over_count);
}

// The listed columns of every dilation (grid-stride) with kKM slots; larger unions go to the FP64 tier's list.
__global__ void __launch_bounds__(kMidThreads) k_column_list(const BatchVol *__restrict__ vols, int nv) {
  __shared__ float2 sv[kKM * kMidThreads];
  const int nth = gridDim.x * kMidThreads;
  for (int v = 0; v < nv; ++v) {
    const BatchVol &V = vols[v];
    const int m = *V.over_count;
    if (m <= 0) continue;
    const ColumnArgs &A = *V.column;
    const float E = A.par->E;
    for (int i = blockIdx.x * kMidThreads + threadIdx.x; i < m; i += nth) {
      const int c = V.over_list[i], x = c % A.nx, y = c / A.nx;
      UnionIds<kKM> U;
      const unsigned mask = __activemask();
      const int n = fast_column<kKM>(A, E, x, y, sv + threadIdx.x, kMidThreads, U, mask);
      if (n > kUnionLarge) atomicAdd(V.large, 1);
      finish_column(V, A, U, x, y, n, V.big_list, V.big_count);
    }
  }
}

// ---------------------------------------------------------------- preparation

// Visits the columns' segments: with `packed` (CSR) in the order of memory, else column by column.
template <typename Visit>
__device__ __forceinline__ void for_segments(int ncols, const int32_t *beg, const int32_t *end, bool packed, Visit visit) {
  const long long first = (long long)blockIdx.x * blockDim.x + threadIdx.x, step = (long long)gridDim.x * blockDim.x;
  if (packed) {
    const long long e = end[ncols - 1];
    for (long long k = beg[0] + first; k < e; k += step) visit(k);
  } else {
    for (long long c = first; c < ncols; c += step)
      for (long long k = beg[c]; k < end[c]; ++k) visit(k);
  }
}

// The values' range and from it the dilation's scalars (mm and set_par: vo_range.cuh).
__global__ void __launch_bounds__(256) k_column_range(int ncols, const int32_t *__restrict__ beg,
                                                      const int32_t *__restrict__ end, bool packed,
                                                      const longlong2 *__restrict__ z, float R,
                                                      unsigned long long *mm, FastPar *par) {
  ValueRange range;
  for_segments(ncols, beg, end, packed, [&](long long k) {
    const longlong2 v = z[k];
    range.take(v.x);
    range.take(v.y);
  });
  range.finish(mm, R, par);
}

// FP32 copies of the columns' values, relative to the base; those beyond the range (set_par) infinite.
__global__ void __launch_bounds__(256) k_column_values(int ncols, const int32_t *__restrict__ beg,
                                                       const int32_t *__restrict__ end, bool packed,
                                                       const double2 *__restrict__ z, const FastPar *__restrict__ par,
                                                       float2 *__restrict__ zf) {
  const double base = par->base;
  auto in_fp32 = [=](double v) {
    return fabs(v) > kFar ? (v < 0 ? -INFINITY : INFINITY) : __double2float_rn(__dsub_rn(v, base));
  };
  for_segments(ncols, beg, end, packed, [&](long long k) {
    const double2 v = z[k];
    zf[k] = make_float2(in_fp32(v.x), in_fp32(v.y));
  });
}

// Dominance widths, one thread per column. For segment i and direction k
// (neighbour (x-1, y), (x+1, y), (x, y-1), (x, y+1)):
//   w_i = min over the neighbour's segments j of max(z1_j - z1_i, z2_i - z2_j),
// evaluated in FP32 on bounds of the FP64 values with every difference
// rounded up, so w bounds the exact value from above (+inf outside the grid
// or without a neighbour segment). The scan stops after the
// first neighbour segment starting above segment i: every later neighbour
// segment gives a larger value. The column's width per direction is the max
// over its segments (-inf for an empty column), stored as FP16 rounded up in
// the column record col[c] = (beg, end, x- | x+ << 16, y- | y+ << 16).
// (FP32 copies are within half an ulp, and FastPar::q for the base taken off, of
// the FP64 values.)
__global__ void k_dominance(int nx, int ny, const int32_t *__restrict__ beg, const int32_t *__restrict__ end,
                            const float2 *__restrict__ zf, int4 *__restrict__ col, void *__restrict__ dmask,
                            int mask_bits, const DomLevels L, const FastPar *__restrict__ par) {
  const float q = par->q;
  const int ncols = nx * ny;
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncols) return;
  const int x = c % nx, y = c / nx;
  const int k0 = beg[c], k1 = end[c];
  int nb0[4], nb1[4];
  for (int k = 0; k < 4; ++k) {
    const int xn = x + (k == 0 ? -1 : k == 1 ? 1 : 0), yn = y + (k == 2 ? -1 : k == 3 ? 1 : 0);
    const bool in = xn >= 0 && xn < nx && yn >= 0 && yn < ny;
    const int cn = in ? xn + nx * yn : 0;
    nb0[k] = in ? beg[cn] : 0;
    nb1[k] = in ? end[cn] : 0;
  }
  float cmax[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
  unsigned bits[4][kDomLevels];
  for (int k = 0; k < 4; ++k)
    for (int l = 0; l < kDomLevels; ++l) bits[k][l] = 0u;
  const bool masked = k1 - k0 <= mask_bits;
  for (int i = k0; i < k1; ++i) {
    // bounds of the exact values: an FP32 copy is within half an ulp of its
    // FP64 value, so the neighbouring floats enclose it
    const float2 fi = zf[i];
    const float i1 = nextafterf(fi.x, -INFINITY), i2 = nextafterf(fi.y, INFINITY);
    for (int k = 0; k < 4; ++k) {
      float best = INFINITY;
      for (int j = nb0[k]; j < nb1[k]; ++j) {
        const float2 fj = zf[j];
        const float lo = __fsub_ru(nextafterf(fj.x, INFINITY), i1);
        const float hi = __fsub_ru(i2, nextafterf(fj.y, -INFINITY));
        const float m = lo > hi ? lo : hi;
        best = m < best ? m : best;
        if (fj.x > fi.y) break;  // any early stop only leaves the bound larger
      }
      best = __fadd_ru(best, q);
      cmax[k] = best > cmax[k] ? best : cmax[k];
      if (masked)
        for (int l = 0; l < kDomLevels; ++l)
          if (best <= L.t[l]) bits[k][l] |= 1u << (i - k0);
    }
  }
  for (int k = 0; k < 4; ++k)
    for (int l = 0; l < kDomLevels; ++l) {
      const size_t idx = (size_t)(k * kDomLevels + l) * ncols + c;
      if (mask_bits == 16) static_cast<unsigned short *>(dmask)[idx] = (unsigned short)bits[k][l];
      else static_cast<unsigned *>(dmask)[idx] = bits[k][l];
    }
  unsigned h[4];
  for (int k = 0; k < 4; ++k) h[k] = __half_as_ushort(__float2half_ru(cmax[k]));
  col[c] = make_int4(k0, k1, (int)(h[0] | (h[1] << 16)), (int)(h[2] | (h[3] << 16)));
}

// Of kSampleColumns columns spread over the grid the first kSampleSegs segments: how many pairs (segment, neighbour
// column) there are and how many of those segments lie in one of that column widened by kSampleGrowth, block by block
// to page-locked host memory. A thread per column and neighbour: the latency of its loads is what it takes.
constexpr int kSampleColumns = 2048, kSampleThreads = 1024, kSampleBlocks = 4 * kSampleColumns / kSampleThreads;
constexpr int kSampleSegs = 64;
constexpr double kSampleGrowth = 0.45;
static_assert(2 * kSampleBlocks <= kScanExtra, "h_total holds the blocks' counts");
__global__ void __launch_bounds__(kSampleThreads) k_sample_held(int nx, int ny, const int32_t *__restrict__ beg,
                                                                const int32_t *__restrict__ end,
                                                                const double2 *__restrict__ z, int2 *out) {
  __shared__ int s_all, s_held;
  if (threadIdx.x == 0) s_all = s_held = 0;
  __syncthreads();
  const unsigned t = blockIdx.x * kSampleThreads + threadIdx.x, i = t >> 2, d = t & 3;
  const long long ncols = (long long)nx * ny;
  // evenly spread, with a step that shares no period with the rows
  const int c = (int)(((unsigned long long)i * 0x9e3779b97f4a7c15ull >> 32) * ncols >> 32);
  const int x = c % nx, y = c / nx;
  int all = 0, held = 0;
  if (x > 0 && y > 0 && x + 1 < nx && y + 1 < ny) {
    const int cn = c + (d == 0 ? -1 : d == 1 ? 1 : d == 2 ? -nx : nx), e = end[cn];
    const int k0 = beg[c], n = min(end[c] - k0, kSampleSegs);
    all = n;
    int at = beg[cn];
    for (int k = 0; k < n; ++k) {
      const double2 s = z[k0 + k];
      // of the neighbour's segments the first that reaches this one, or the next
      while (at < e && z[at].y < s.x) ++at;
      bool in = false;
      for (int j = 0; j < 2 && at + j < e; ++j) in |= z[at + j].x - s.x <= kSampleGrowth && s.y - z[at + j].y <= kSampleGrowth;
      held += in;
    }
  }
  all = __reduce_add_sync(0xffffffffu, all);
  held = __reduce_add_sync(0xffffffffu, held);
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(&s_all, all);
    atomicAdd(&s_held, held);
  }
  __syncthreads();
  if (threadIdx.x == 0) out[blockIdx.x] = make_int2(s_all, s_held);
}

static_assert(kDomLevels <= 15, "pair records hold a level in 4 bits, 15 meaning none");
static_assert(sizeof(BatchVol) % sizeof(int) == 0 && sizeof(ColumnArgs) % sizeof(int) == 0, "copied as ints");

}  // namespace

// ================================================================ host side

// FP32 lower bound of a - b: the FP64 difference rounded to
// nearest is moved down one ulp when its TwoSum error is negative, then the
// FP32 conversion rounded to nearest is moved down when it lies above.
static float sub_rd_f32(double a, double b) {
  const double c = -b, s = a + c, bb = s - a;
  const double e = (a - (s - bb)) + (c - bb);
  const double sd = e < 0.0 ? std::nextafter(s, -INFINITY) : s;
  float f = (float)sd;
  if ((double)f > sd) f = std::nextafterf(f, -INFINITY);
  return f;
}

// Dominance level thresholds for the tables' radius: t[0] = 0 and t[l] for
// l >= 1 the value at quantile (l - 1/2) / (kDomLevels - 1) of the sorted
// growths of H over one lattice step (x steps for a >= 1, y steps for
// d >= 1), each as the FP32 lower bound the device's pair records hold.
static DomLevels dom_levels(const Tables &t) {
  DomLevels L;
  std::vector<float> g;
  for (int d = 0; d <= t.Dy; ++d)
    for (int a = 0; a <= t.Dx[d]; ++a) {
      const double h = t.H[(size_t)d * t.W + a];
      if (a >= 1) g.push_back(sub_rd_f32(t.H[(size_t)d * t.W + a - 1], h));
      if (d >= 1) g.push_back(sub_rd_f32(t.H[(size_t)(d - 1) * t.W + a], h));
    }
  std::sort(g.begin(), g.end());
  L.t[0] = 0.f;
  for (int l = 1; l < kDomLevels; ++l) {
    float v = 0.f;
    if (!g.empty()) {
      const double q = ((double)l - 0.5) / (double)(kDomLevels - 1);
      v = g[(size_t)std::floor(q * (double)(g.size() - 1) + 0.5)];
    }
    L.t[l] = v > 0.f ? v : 0.f;
  }
  return L;
}

// Pair records: (a | d << 8 | x-step level << 16 | y-step level << 20 as float bits, H in FP32, growth of H
// over an x step and over a y step towards the centre, rounded down), in decreasing H; the level is the largest
// whose threshold is not above the growth.
std::vector<float4> column_pairs(const Tables &h, DomLevels &L) {
  L = dom_levels(h);
  struct Pair {
    int a, d;
    double H;
  };
  std::vector<Pair> pairs;
  for (int d = 0; d <= h.Dy; ++d)
    for (int a = 0; a <= h.Dx[d]; ++a) pairs.push_back({a, d, h.H[(size_t)d * h.W + a]});
  std::stable_sort(pairs.begin(), pairs.end(), [](const Pair &p, const Pair &q) { return p.H > q.H; });
  std::vector<float4> out;
  out.reserve(pairs.size());
  auto level = [&](float g) {
    int lv = 15;
    for (int l = 0; l < kDomLevels; ++l)
      if (L.t[l] <= g) lv = l;
    return lv;
  };
  for (const Pair &p : pairs) {
    const float gx = p.a ? sub_rd_f32(h.H[(size_t)p.d * h.W + p.a - 1], p.H) : -INFINITY;
    const float gy = p.d ? sub_rd_f32(h.H[(size_t)(p.d - 1) * h.W + p.a], p.H) : -INFINITY;
    const int code = p.a | (p.d << 8) | (level(gx) << 16) | (level(gy) << 20);
    float4 r;
    std::memcpy(&r.x, &code, sizeof code);
    r.y = (float)p.H;
    r.z = gx;
    r.w = gy;
    out.push_back(r);
  }
  return out;
}

int column_alloc(const vo_grid &g, size_t entries, double mean_segs, const std::function<int(void **, size_t)> &alloc,
                 ColumnPrep &P) {
  const size_t ncols = (size_t)g.nx * g.ny;
  P.mask_bits = mean_segs <= kMask16MeanSegs ? 16 : 32;
  int rc = alloc((void **)&P.zf, sizeof(float2) * entries);
  if (!rc) rc = alloc((void **)&P.col, sizeof(int4) * ncols);
  if (!rc) rc = alloc(&P.dmask, (size_t)4 * kDomLevels * ncols * (P.mask_bits / 8));
  if (!rc) rc = alloc((void **)&P.par, 64 + 4 * sizeof(unsigned long long));
  P.mm = reinterpret_cast<unsigned long long *>(reinterpret_cast<unsigned char *>(P.par) + 64);
  return rc;
}

ColumnArgs column_args(int nx, int ny, const DeviceTables &T, const int32_t *beg, const int32_t *end, const double2 *z,
                       const ColumnPrep &P) {
  return ColumnArgs{nx, ny, T.host.W, T.npairs, P.mask_bits, 0, beg, end, (const double *)z, (const float *)P.zf, T.H, T.prec,
                    P.par, P.col, P.dmask};
}

void column_prepare(cudaStream_t st, const ColumnArgs &A, float R, const DomLevels &L, const ColumnPrep &P) {
  const int ncols = A.nx * A.ny;
  const double2 *z = reinterpret_cast<const double2 *>(A.zd);
  cudaMemsetAsync(P.mm, 0, 4 * sizeof(unsigned long long), st);
  const bool packed = A.end == A.beg + 1;
  const int blocks = std::max(1, std::min((ncols + 255) / 256, 2048));
  k_column_range<<<blocks, 256, 0, st>>>(ncols, A.beg, A.end, packed, reinterpret_cast<const longlong2 *>(z), R, P.mm, P.par);
  k_column_values<<<blocks, 256, 0, st>>>(ncols, A.beg, A.end, packed, z, P.par, P.zf);
  k_dominance<<<(ncols + 127) / 128, 128, 0, st>>>(A.nx, A.ny, A.beg, A.end, P.zf, P.col, P.dmask, P.mask_bits, L, P.par);
}

// Union slots per column from the input's mean segment count: more keep fewer warps per SM, fewer send
// more columns to the second launch.
int column_slots(double mean_segs) { return mean_segs > 24.0 ? 64 : mean_segs > 10.0 ? 48 : mean_segs > 6.0 ? 32 : 24; }

template <bool SINGLE>
static auto *column_kernel(int slots) {
  return slots == 64 ? &k_column<64, SINGLE>
         : slots == 48 ? &k_column<48, SINGLE> : slots == 32 ? &k_column<32, SINGLE> : &k_column<24, SINGLE>;
}
KernelShape column_shape(int slots, bool single) {
  cudaFuncAttributes a{};
  cudaFuncGetAttributes(&a, single ? column_kernel<true>(slots) : column_kernel<false>(slots));
  return KernelShape{1, slots, a.numRegs};
}
void column_launch(cudaStream_t st, const BatchVol *vols, int nv, int blocks, int slots, const ColumnArgs &A) {
  (nv == 1 ? column_kernel<true>(slots) : column_kernel<false>(slots))<<<blocks, kBlockCols,
                                                                        sizeof(float2) * slots * kBlockCols, st>>>(vols, nv, A);
}

void column_list_launch(cudaStream_t st, const BatchVol *vols, int nv) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  k_column_list<<<16 * std::max(sms, 1), kMidThreads, 0, st>>>(vols, nv);
}

// Against k_direct and the patch kernel, preparation and copy included (ms; segments per column; radius; the better
// of those two, this kernel):
//   spheres     512^2    4.0   r 4   0.52 / 0.53     r 6   0.86 / 0.74     r 8   1.04 / 1.00     r 10  1.02 / 1.30
//               1024^2   2.9         1.13 / 1.08           1.97 / 1.64           2.71 / 2.33           2.83 / 3.20
//               1024^2   5.1         2.01 / 1.75           3.59 / 2.66           4.17 / 3.76           4.20 / 5.01
//               2048^2   6.1         8.89 / 8.00           15.7 / 12.6           18.1 / 17.9           19.5 / 24.6
//               1024^2   9.6         4.27 / 4.01           7.35 / 5.70           6.72 / 7.35
//               1024^2   1.0         0.63 / 0.75           1.04 / 1.21           1.53 / 1.77
//   cylinders   1024^2   4.4         3.75 / 5.56           6.30 / 8.61           6.74 / 10.8
//                        16.2        17.0 / 25.0           21.7 / 31.9           17.9 / 36.6
// Below 2^18 columns four threads share one in k_direct, which is the best there (256^2, 4.1 segments, r = 6: 0.39 /
// 0.48). What tells the inputs apart is how many segments a neighbour column holds when widened by what H grows in
// a step, its median at any of these radii (0.41 to 0.49 dexels; 0.58 at radius 5, where many growths are alike, so that
// the growth is a constant here): 0.64 to 0.66 of them for spheres, with some cylinders among them 0.59 to 0.63, 0.49
// for thin cylinders, none for scattered segments. The line is 0.55. The sample takes 15 to 30 us with the wait for it, so it
// is not taken where there is less to gain: calls of about a millisecond (work over all columns; 512^2 thin cylinders,
// 2.5 segments, r = 6, lie below: 1.05 ms, with a sample 1.13 before it was made shorter), and from radius 7.5 fewer
// than 2^19 columns (513^2 spheres, 3.4 segments, r = 8: 0.85 / 0.88).
constexpr double kHeldShare = 0.55, kColumnWorkFrom = 190, kColumnWorkTo = 1050, kSampleWork = 8e7;
constexpr int64_t kColumnCols = 1 << 18;
constexpr double kColumnSegs = 2.0, kColumnRadiusFrom = 3.5, kColumnRadiusMid = 7.5, kColumnRadiusTo = 9.0;

int column_choice(vo_ctx *ctx, const vo_grid &g, const DeviceTables &T, double mean_segs, const int32_t *beg,
                  const int32_t *end, const double2 *z, const std::function<void()> &ready, bool *columns) {
  *columns = false;
  const double work = reach_columns(g, T) * mean_segs, ncols = (double)g.nx * g.ny;
  if (ncols < kColumnCols || std::min(g.nx, g.ny) < kPatchY || mean_segs < kColumnSegs || T.host.R < kColumnRadiusFrom ||
      T.host.R >= kColumnRadiusTo || work < kColumnWorkFrom || ncols * work < kSampleWork ||
      (T.host.R >= kColumnRadiusMid && (work > kColumnWorkTo || ncols < 2 * kColumnCols)))
    return VO_OK;
  ready();
  int2 *h = reinterpret_cast<int2 *>(ctx->h_total + 1);
  k_sample_held<<<kSampleBlocks, kSampleThreads, 0, ctx->stream>>>(g.nx, g.ny, beg, end, z, h);
  ctx->launches += 1;
  VO_CK(ctx, cudaGetLastError());
  VO_CK(ctx, cudaStreamSynchronize(ctx->stream));
  double all = 0, held = 0;
  for (int i = 0; i < kSampleBlocks; ++i) {
    all += h[i].x;
    held += h[i].y;
  }
  *columns = all > 0 && held >= kHeldShare * all;
  return VO_OK;
}

}  // namespace vo
