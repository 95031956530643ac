// Batch plans: many volumes of uneven grids, radii and operations (including
// the erosion -> dilation chains of opening and closing) executed as one
// CUDA graph, with every dilation of a round in one persistent launch
// (VO_METHOD_FAST only; no reference counterpart beyond calling
// VoronoiMorpho::dilation / erosion once per volume, Voronoi.h:18-29, and the
// chaining of offset3d.cpp:124-133).
//
// Planning (vo_batch_create) walks the operation chains round by round. Every
// device step is recorded as a launch closure; the plan runs the closures
// eagerly only when a later step needs the data (the input features of a
// learned-sized dilation, the capacity of a complement of a dilation result).
// Per dilation:
//   * the kernel: patches, the small-radius kernel or the per-column kernel, as
//     a single dilation chooses it (a sample of the input may be taken);
//   * output slots: with a sizer attached, every 32 x 32 tile of output
//     columns gets the capacity the network predicts for its largest union
//     (plus a margin, at most kUnionCapMid); without one, every column gets
//     kUnionCap slots; either way a spill region takes the columns that need
//     more;
//   * work queue: dilations in decreasing predicted total work (the network's
//     per-tile candidate counts, or the mean cost per column), the patches of
//     each in bands of 512 columns, all rows of a band before the next;
//   * lanes per column of the patch kernel (1 or 4) from the round's size, or
//     from the autotuner below where the size does not decide it (cached per
//     context).
// Then the closures are captured into one graph. vo_batch_run replays it and
// re-runs, through the single-volume path, every volume whose overflow flag
// is set (a union larger than its slot with the spill region exhausted, beyond the
// FP64 lists, or more unions beyond the first kernel's lists than the round's tiers
// take), so results never depend on the predictions. vo_morph_batched, which runs a plan once, runs each
// step once, as it is planned, without a graph (24 mixed volumes: 18.1 ms
// against 26.8 with a capture and a replay; one of 1001^2 columns and 19 segments
// each: 18.9 against 23.1); its stretches of steps are timed one by one.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>
#include <functional>
#include <memory>
#include <vector>

#include "vo_internal.cuh"
#include "vo_slots.h"

using namespace vo;

namespace {

enum StepKind { kDil, kNeg, kNorm, kNegInv };

// Operation chains (Voronoi.cpp:8-17 erosion; offset3d.cpp:124-133 opening/closing).
std::vector<StepKind> steps_of(int op) {
  switch (op) {
    case VO_DILATION:
      return {kDil};
    case VO_EROSION:
      return {kNeg, kNorm, kDil, kNegInv};
    case VO_OPENING:
      return {kNeg, kNorm, kDil, kNegInv, kDil};
    default:
      return {kDil, kNeg, kNorm, kDil, kNegInv};
  }
}

using Launch = std::function<void(cudaStream_t)>;

// Counters of a dilation: spill space used, FP64-tier columns, columns for k_column_list, patches listed, large unions.
constexpr int kDilCounters = 5;
constexpr int kRoundCounters = 5;  // of a round before them: four of the patch queue, lists of the pool taken

struct DilPlan {
  int vol = 0;
  SlotVol in, out;
  const DeviceTables *T = nullptr;
  FastArgs A{};
  PackOut pk;
  unsigned long long *mm = nullptr;
  int *big_list = nullptr;
  int *counters = nullptr;  // kDilCounters of them (zeroed before every replay)
  int32_t *tcap = nullptr, *toff = nullptr;
  int tiles32_x = 0, tiles32 = 0;
  std::vector<float> tile_work;  // predicted candidates per column of each sizing tile
  int spill_base = 0, spill_cap = 0;
  double cost = 0;  // mean candidates per column (no sizer)
  double mean_segs = 0;
  Engine engine = Engine::kPatches;
  ColumnPrep cp;  // kColumns
  ColumnArgs C{};
  int *over_list = nullptr;
  int64_t slot_entries = 0;
};

}  // namespace

struct vo_batch {
  int n = 0;
  std::vector<int> ops;
  std::vector<double> radii;
  std::vector<const vo_volume *> ins;
  std::vector<vo_volume *> normalized;  // owned copies of inputs with inverted pairs rewritten
  std::vector<Launch> rec;             // recorded device steps, in order
  size_t executed = 0;                 // closures already run eagerly
  int kernels = 0;                     // kernel launches per replay
  std::vector<void *> dmem;            // device allocations of the plan
  std::vector<SlotVol> owned;
  std::vector<SlotVol> finals;
  int *d_flags = nullptr;  // [v]: overflow flags of volume v, [n]: complement slot overflow
  double2 *big_scratch = nullptr;  // working lists of the FP64 tier
  unsigned char *scratch[2] = {nullptr, nullptr};  // working memory of the patch kernel's tiers
  size_t scratch_bytes[2] = {0, 0};
  // Per dilation round: its counters (kRoundCounters, then kDilCounters per dilation) and the dilations' spill
  // capacities.
  struct Round {
    const int *counters;
    std::vector<int> caps;
  };
  std::vector<Round> rounds;
  bool once = false;  // a plan for one run: its steps run as they are recorded, with no graph
  std::vector<std::pair<cudaEvent_t, cudaEvent_t>> stretches;  // when they did (run_pending)
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  std::vector<vo_volume *> rerun;
  // Radius tables used by the plan, copied into plan memory: the context's
  // table cache evicts entries, and the graph reads these on every replay.
  std::vector<std::unique_ptr<DeviceTables>> tables;
  vo_batch_stats stats{};
};

namespace {

template <typename T>
int plan_alloc(vo_ctx *ctx, vo_batch *b, T **p, size_t n) {
  int rc = dalloc(ctx, p, n);
  if (!rc) b->dmem.push_back((void *)*p);
  return rc;
}

// Runs the recorded closures not yet run. Of a plan for one run each such stretch is timed: its run reports the
// steps' time on the device, without the planning between them.
void run_pending(vo_ctx *ctx, vo_batch *b) {
  if (b->executed == b->rec.size()) return;
  cudaEvent_t from = nullptr, to = nullptr;
  if (b->once && (cudaEventCreate(&from) != cudaSuccess || cudaEventCreate(&to) != cudaSuccess)) {
    cudaGetLastError();  // a stretch without its time
    if (from) cudaEventDestroy(from);
    from = nullptr;
  }
  if (from) cudaEventRecord(from, ctx->stream);
  for (; b->executed < b->rec.size(); ++b->executed) b->rec[b->executed](ctx->stream);
  if (from) {
    cudaEventRecord(to, ctx->stream);
    b->stretches.push_back({from, to});
  }
}

void record(vo_batch *b, int kernels, Launch f) {
  b->rec.push_back(std::move(f));
  b->kernels += kernels;
}

// Maximum segment count of a slot volume (synchronising).
int max_count(vo_ctx *ctx, const SlotVol &v, int *out) {
  int *d = nullptr;
  int rc = dalloc(ctx, &d, 1);
  if (rc) return rc;
  cudaMemsetAsync(d, 0, sizeof(int), ctx->stream);
  slot_max_count(ctx, v, d);
  int h = 0;
  cudaMemcpyAsync(&h, d, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream);
  dfree(ctx, d);
  VO_CK(ctx, cudaStreamSynchronize(ctx->stream));
  *out = h;
  return VO_OK;
}

// Output slot layout of one dilation: learned per-tile capacities, or fixed.
int size_output(vo_ctx *ctx, vo_batch *b, DilPlan &d, double radius) {
  const vo_grid &g = d.in.grid;
  const int ncols = g.nx * g.ny;
  d.tiles32_x = (g.nx + kSizerTile - 1) / kSizerTile;
  d.tiles32 = d.tiles32_x * ((g.ny + kSizerTile - 1) / kSizerTile);
  int rc = VO_OK;
  int64_t entries = (int64_t)ncols * kUnionCap;
  if (ctx->sizer) {
    float *feats = nullptr, *pred = nullptr;
    int nt = 0;
    rc = dalloc(ctx, &feats, (size_t)d.tiles32 * VO_SIZER_FEATURES);
    if (!rc) rc = dalloc(ctx, &pred, (size_t)d.tiles32 * 4);
    if (!rc) rc = sizer_features_device(ctx, d.in, radius, feats, &nt);
    if (!rc) rc = sizer_predict_device(ctx, ctx->sizer, feats, nt, pred);
    std::vector<float> hp((size_t)d.tiles32 * 4);
    if (!rc) {
      cudaMemcpyAsync(hp.data(), pred, sizeof(float) * hp.size(), cudaMemcpyDeviceToHost, ctx->stream);
      cudaError_t e = cudaStreamSynchronize(ctx->stream);
      if (e != cudaSuccess) rc = cuda_error(ctx, e, "sizer prediction");
    }
    dfree(ctx, feats);
    dfree(ctx, pred);
    if (rc) return rc;
    std::vector<int32_t> cap(d.tiles32), off(d.tiles32);
    d.tile_work.resize(d.tiles32);
    int64_t total = 0;
    for (int t = 0; t < d.tiles32; ++t) {
      const int tx = t % d.tiles32_x, ty = t / d.tiles32_x;
      const int cols = std::min(kSizerTile, g.nx - tx * kSizerTile) * std::min(kSizerTile, g.ny - ty * kSizerTile);
      // predicted max segments per column, with a margin against the error of a log2 estimate
      const double mx = std::exp2((double)hp[(size_t)t * 4]) - 1.0;
      const int c = (int)std::min<double>(kUnionCapMid, std::max(1.0, std::ceil(mx * 1.5 + 2.0)));
      cap[t] = c;
      off[t] = (int32_t)total;
      total += (int64_t)c * cols;
      const double w = std::exp2((double)hp[(size_t)t * 4 + 2]) - 1.0;
      d.tile_work[t] = w >= 0 && w < 1e30 ? (float)w : 0.f;  // a diverged network must not break the sort
    }
    d.spill_base = (int)total;
    d.spill_cap = (int)std::max<int64_t>(4096, total / 4);
    entries = total + d.spill_cap;
    if (entries > 2147483647LL) return set_error(ctx, VO_ERANGE, "batch: slot layout exceeds int32 offsets");
    rc = plan_alloc(ctx, b, &d.tcap, (size_t)d.tiles32);
    if (!rc) rc = plan_alloc(ctx, b, &d.toff, (size_t)d.tiles32);
    if (rc) return rc;
    cudaMemcpyAsync(d.tcap, cap.data(), sizeof(int32_t) * cap.size(), cudaMemcpyHostToDevice, ctx->stream);
    cudaMemcpyAsync(d.toff, off.data(), sizeof(int32_t) * off.size(), cudaMemcpyHostToDevice, ctx->stream);
    VO_CK(ctx, cudaStreamSynchronize(ctx->stream));  // the host vectors go out of scope
  } else {
    // fixed capacity kUnionCap per column, spill space for 1/8 of that
    d.spill_base = (int)std::min<int64_t>(entries, 2147483647LL);
    d.spill_cap = (int)std::max<int64_t>(4096, entries / 8);
    entries += d.spill_cap;
    if (entries > 2147483647LL) return set_error(ctx, VO_ERANGE, "batch: slot layout exceeds int32 offsets");
  }
  d.slot_entries = entries;
  d.out = SlotVol();
  d.out.grid = g;
  d.out.cap = kUnionCap;
  d.out.entries = entries;
  d.out.owns = false;  // plan memory
  rc = plan_alloc(ctx, b, &d.out.beg, (size_t)ncols);
  if (!rc) rc = plan_alloc(ctx, b, &d.out.end, (size_t)ncols);
  if (!rc) rc = plan_alloc(ctx, b, &d.out.z, (size_t)entries);
  return rc;
}

BatchVol batch_vol(const DilPlan &d, int *ovf) {
  BatchVol v;
  std::memset(&v, 0, sizeof v);
  v.A = d.A;
  v.obeg = d.out.beg;
  v.oend = d.out.end;
  v.oz = d.out.z;
  v.tcap = d.tcap;
  v.toff = d.toff;
  v.cap = kUnionCap;
  v.tiles32_x = d.tiles32_x;
  v.spill_base = (unsigned)d.spill_base;
  v.spill_cap = (unsigned)d.spill_cap;
  v.spill_used = reinterpret_cast<unsigned *>(d.counters);
  v.big_list = d.big_list;
  v.big_count = d.counters + 1;
  v.over_list = d.over_list;
  v.over_count = d.counters + 2;
  v.listed = d.engine == Engine::kDirect ? v.big_count : d.counters + 3;
  v.most = d.engine == Engine::kDirect ? kFewColumns : kFewPatches;
  v.large = d.counters + 4;
  v.ovf = ovf;
  return v;
}

// Estimated total work of a dilation (candidates).
double total_work(const DilPlan &d) {
  const vo_grid &g = d.in.grid;
  if (d.tile_work.empty()) return d.cost * g.nx * (double)g.ny;
  double w = 0;
  for (int t = 0; t < d.tiles32; ++t) {
    const int tx = t % d.tiles32_x, ty = t / d.tiles32_x;
    w += (double)d.tile_work[t] * std::min(kSizerTile, g.nx - tx * kSizerTile) *
         std::min(kSizerTile, g.ny - ty * kSizerTile);
  }
  return w;
}

int sm_count() {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms > 0 ? sms : 1;
}

// Autotuner: rounds of kTuneFrom to kTuneTo patches per SM lie where one lane
// per column (throughput) and four (the longest patch's latency) cross, at a
// point that depends on the input (8 dexels: 0.19 against 0.27 ms at 200^2,
// 0.33 against 0.31 ms at 276^2 with four and one). Such a round times both
// once, and the context keeps the choice per shape (one dilation or several,
// log2 of the patches, radius / 8, segments per column, learned or not).
// Smaller and larger rounds follow patch_split.
constexpr int kTuneFrom = 5, kTuneTo = 24;

int tune_split(vo_ctx *ctx, vo_batch *b, const std::vector<DilPlan> &dils, int64_t patches,
               const std::function<int(int, float *)> &time, int *split) {
  double rmax = 0, segs = 0;
  for (const DilPlan &d : dils) {
    rmax = std::max(rmax, b->radii[d.vol]);
    segs = std::max(segs, d.mean_segs);
  }
  const long long key = (dils.size() == 1 ? 1LL << 40 : 0) | ((long long)std::ilogb((double)patches) << 16) |
                        ((long long)(rmax / 8) << 8) | ((long long)std::min(segs / 4, 60.0) << 2) | (ctx->sizer ? 1 : 0);
  for (const auto &kv : ctx->tune_cache)
    if (kv.first == key) {
      *split = kv.second;
      return VO_OK;
    }
  float ms[2] = {0, 0};
  int rc = time(1, &ms[0]);
  if (!rc) rc = time(4, &ms[1]);
  if (rc) return rc;
  b->stats.tune_ms[0] = ms[0];
  b->stats.tune_ms[2] = ms[1];
  *split = ms[1] < ms[0] ? 4 : 1;
  ctx->tune_cache.push_back({key, *split});
  return VO_OK;
}

// Order of a round's dilations in its launches.
int launch_order(Engine e) { return e == Engine::kPatches ? 0 : e == Engine::kColumns ? 1 : 2; }

// The pair records of plan-owned tables (the context's own entry may be evicted).
int plan_column_tables(vo_ctx *ctx, vo_batch *b, const DeviceTables *T) {
  if (T->prec) return VO_OK;
  DeviceTables *own = const_cast<DeviceTables *>(T);
  const std::vector<float4> pairs = column_pairs(T->host, own->dom);
  int rc = plan_alloc(ctx, b, &own->prec, pairs.size());
  if (rc) return rc;
  own->npairs = (int)pairs.size();
  cudaMemcpyAsync(own->prec, pairs.data(), sizeof(float4) * pairs.size(), cudaMemcpyHostToDevice, ctx->stream);
  VO_CK(ctx, cudaStreamSynchronize(ctx->stream));
  return VO_OK;
}

int plan_dilation_round(vo_ctx *ctx, vo_batch *b, std::vector<DilPlan> &dils, bool later_rounds) {
  int rc = VO_OK;
  for (DilPlan &d : dils) {
    const vo_grid &g = d.in.grid;
    const int ncols = g.nx * g.ny;
    const size_t entries = (size_t)std::max<int64_t>(d.in.entries, 1);
    // mean segments per column of the input, exact for CSR inputs, the capacity's half for slots
    d.mean_segs = d.in.owns ? d.in.cap * 0.5 : (double)d.in.entries / std::max(ncols, 1);
    const float R = (float)b->radii[d.vol];
    // candidates per column: lattice points of the disc x mean segments of the input (no sizer)
    d.cost = 3.14159 * (R + 0.5) * (R + 0.5) * (d.mean_segs + 0.5);
    d.engine = (d.in.owns || d.in.end == d.in.beg + 1) && direct_choice(g, *d.T, d.mean_segs) ? Engine::kDirect : Engine::kPatches;
    bool columns = false;
    rc = column_choice(ctx, g, *d.T, d.mean_segs, d.in.beg, d.in.end, d.in.z, [&] { run_pending(ctx, b); }, &columns);
    if (columns || (d.engine == Engine::kPatches && (int64_t)entries > kPatchSegments)) d.engine = Engine::kColumns;
    if (!rc) rc = plan_alloc(ctx, b, &d.big_list, (size_t)ncols);
    if (rc) return rc;
    if (d.engine == Engine::kDirect) {
      rc = plan_alloc(ctx, b, &d.pk.rec, entries);
      if (!rc && d.in.owns) rc = plan_alloc(ctx, b, &d.pk.zx, entries);
      if (!rc && d.in.owns) rc = plan_alloc(ctx, b, &d.pk.rbeg, 2 * (size_t)ncols);
      if (rc) return rc;
      d.A = fast_args(g, *d.T, d.in.beg, d.in.end, d.in.z, d.pk);
      const DilPlan c = d;
      record(b, 1, [c](cudaStream_t st) { direct_prepare(st, c.A, c.pk); });
      continue;
    }
    if (d.engine == Engine::kColumns) {
      rc = plan_column_tables(ctx, b, d.T);
      auto take = [&](void **p, size_t bytes) {
        unsigned char *q = nullptr;
        const int r = plan_alloc(ctx, b, &q, bytes);
        *p = q;
        return r;
      };
      if (!rc) rc = column_alloc(g, entries, d.mean_segs, take, d.cp);
      if (!rc) rc = plan_alloc(ctx, b, &d.over_list, (size_t)ncols);
      if (rc) return rc;
      d.A = fast_args(g, *d.T, d.in.beg, d.in.end, d.in.z, d.pk);
      d.C = column_args(g.nx, g.ny, *d.T, d.in.beg, d.in.end, d.in.z, d.cp);
      const DilPlan c = d;
      record(b, 3, [c, R](cudaStream_t st) { column_prepare(st, c.C, R, c.T->dom, c.cp); });
      continue;
    }
    rc = plan_alloc(ctx, b, &d.pk.zf, entries);
    if (!rc) rc = plan_alloc(ctx, b, &d.pk.code, entries);
    if (!rc) rc = plan_alloc(ctx, b, &d.pk.wide, entries);
    if (!rc) rc = plan_alloc(ctx, b, &d.pk.zx, entries);
    if (!rc) rc = plan_alloc(ctx, b, &d.pk.cl, entries);
    if (!rc) rc = plan_alloc(ctx, b, &d.pk.coff, pack_offsets(g));
    if (!rc) rc = plan_alloc(ctx, b, &d.pk.par, 1);
    if (!rc) rc = plan_alloc(ctx, b, &d.mm, 4);
    if (rc) return rc;
    d.A = fast_args(g, *d.T, d.in.beg, d.in.end, d.in.z, d.pk);
    const DilPlan c = d;
    record(b, 2, [c, R](cudaStream_t st) { fast_prepare(st, c.A, R, c.mean_segs, c.mm, c.pk); });
  }
  if (ctx->sizer) run_pending(ctx, b);  // features need the dilation inputs
  int *counters = nullptr;
  rc = plan_alloc(ctx, b, &counters, kRoundCounters + kDilCounters * dils.size());
  if (rc) return rc;
  for (size_t i = 0; i < dils.size(); ++i) {
    DilPlan &d = dils[i];
    d.counters = counters + kRoundCounters + kDilCounters * i;
    rc = size_output(ctx, b, d, b->radii[d.vol]);
    if (rc) return rc;
    b->stats.slot_bytes += d.slot_entries * (int64_t)sizeof(double2);
  }
  // the queue: dilations in decreasing estimated total work (longest first, for the balance of the
  // persistent grid), each one's patches in the order of the kernel
  std::vector<std::pair<double, int>> order;
  for (size_t i = 0; i < dils.size(); ++i) order.push_back({total_work(dils[i]), (int)i});
  std::stable_sort(order.begin(), order.end(), [](const std::pair<double, int> &x, const std::pair<double, int> &y) {
    return x.first > y.first;
  });
  // those by patches first, then those by columns
  std::stable_sort(order.begin(), order.end(), [&](const std::pair<double, int> &x, const std::pair<double, int> &y) {
    return launch_order(dils[x.second].engine) < launch_order(dils[y.second].engine);
  });
  int np = 0, nc = 0, slots = 0;
  int64_t direct_cols = 0;
  size_t direct_shared = 0;
  bool direct_shift = false;
  for (const DilPlan &d : dils) {
    if (d.engine == Engine::kDirect) {
      direct_cols += (int64_t)d.in.grid.nx * d.in.grid.ny;
      direct_shared = std::max(direct_shared, direct_smem(d.A));
      direct_shift |= d.A.off != 0.0;
    } else if (d.engine == Engine::kColumns) {
      ++nc;
      slots = std::max(slots, column_slots(d.mean_segs));
    } else {
      ++np;
    }
  }
  // FP64 lists: of the last tier's threads, or of k_direct's columns (a union beyond kPoolCap runs the volume again)
  const int nd = (int)dils.size() - np - nc, big_grid = big_blocks(1 << 30);
  const size_t big_elems = std::max(big_scratch_elems(big_grid, kPoolCap), (size_t)kFewColumns * kPoolCap);
  if (!b->big_scratch) rc = plan_alloc(ctx, b, &b->big_scratch, big_elems);
  ColumnArgs *dcolumns = nullptr;
  if (!rc && nc > 0) rc = plan_alloc(ctx, b, &dcolumns, (size_t)nc);
  if (rc) return rc;
  const size_t counter_bytes = sizeof(int) * (kRoundCounters + kDilCounters * dils.size());
  double2 *big_scratch = b->big_scratch;
  // the round's launch with `split` lanes per column
  struct RoundLaunch {
    PatchPlan P;
    BatchVol *dvols = nullptr;  // in the order above
    int column_items = 0, direct_items = 0;
    ColumnArgs column{};  // of the first dilation by columns
  };
  auto prepare = [&](int split, RoundLaunch &L) -> int {
    std::vector<BatchVol> hv;
    std::vector<ColumnArgs> hc;
    int64_t items = 0, column_items = 0;
    int hs = 0;
    for (const auto &o : order) {
      const DilPlan &d = dils[o.second];
      BatchVol v = batch_vol(d, b->d_flags + d.vol);
      if (d.engine == Engine::kDirect) {
        v.item0 = L.direct_items;
        L.direct_items += direct_blocks(d.in.grid, direct_cols);
        v.item1 = L.direct_items;
        v.pool = big_scratch;
        v.pool_used = counters + 4;
      } else if (d.engine == Engine::kColumns) {
        v.item0 = (int)column_items;
        column_items += patch_count(d.in.grid, 1);
        v.item1 = (int)column_items;
        v.column = dcolumns + hc.size();
        hc.push_back(d.C);
      } else {
        v.item0 = (int)items;
        items += patch_count(d.in.grid, split);
        v.item1 = (int)items;
        hs = std::max(hs, d.T->host.hs);
      }
      if (items > 2147483647LL || column_items > 2147483647LL) return set_error(ctx, VO_ERANGE, "batch: too many columns");
      hv.push_back(v);
    }
    L.column_items = (int)column_items;
    if (nc > 0) L.column = hc[0];
    int r = plan_alloc(ctx, b, &L.dvols, hv.size());
    int *list = nullptr;
    if (!r && np > 0) r = patch_plan(ctx, (int)items, split, hs, L.P);
    if (!r && np > 0) r = plan_alloc(ctx, b, &list, (size_t)items);
    // the rounds run one after the other: they share the largest working memory of each tier
    for (int t = 0; t < 2 && !r && np > 0; ++t) {
      const size_t bytes = patch_scratch_bytes(L.P, t);
      if (bytes > b->scratch_bytes[t]) {
        r = plan_alloc(ctx, b, &b->scratch[t], bytes);
        b->scratch_bytes[t] = bytes;
      }
      if (!r) patch_scratch_set(L.P, t, b->scratch[t]);
    }
    if (r) return r;
    L.P.Q = PatchQueue{counters, list};
    cudaMemcpyAsync(L.dvols, hv.data(), sizeof(BatchVol) * hv.size(), cudaMemcpyHostToDevice, ctx->stream);
    if (nc > 0) cudaMemcpyAsync(dcolumns, hc.data(), sizeof(ColumnArgs) * hc.size(), cudaMemcpyHostToDevice, ctx->stream);
    VO_CK(ctx, cudaStreamSynchronize(ctx->stream));
    return VO_OK;
  };
  auto launch = [=](const RoundLaunch &L, cudaStream_t st) {
    cudaMemsetAsync(counters, 0, counter_bytes, st);
    if (np > 0) {
      patch_launch(false, L.P, st, L.dvols);
      patch_launch(true, L.P, st, L.dvols);
    }
    if (nc > 0) {
      column_launch(st, L.dvols + np, nc, L.column_items, slots, L.column);
      column_list_launch(st, L.dvols + np, nc);
    }
    if (np + nc > 0) big_launch(st, L.dvols, np + nc, big_scratch, big_grid, kPoolCap);
    if (nd > 0) direct_launch(st, L.dvols + np + nc, nd, L.direct_items, direct_cols, direct_shared, direct_shift);
  };
  std::vector<const vo_grid *> grids;
  for (const DilPlan &d : dils)
    if (d.engine == Engine::kPatches) grids.push_back(&d.in.grid);
  int split = patch_split(grids.data(), (int)grids.size());
  RoundLaunch L;
  const int64_t patches = patch_total(grids.data(), (int)grids.size());
  const int sms = sm_count();
  if (np == 0 || patches < kTuneFrom * sms || patches > kTuneTo * sms) {
    rc = prepare(split, L);
  } else {
    rc = tune_split(ctx, b, dils, patches, [&](int sp, float *ms) -> int {
      RoundLaunch T;
      int r = prepare(sp, T);
      if (r) return r;
      run_pending(ctx, b);  // tuning reads the dilation inputs; its outputs are written again by the real launch
      for (int k = 0; k < 2; ++k) {  // the first run warms caches and clocks
        cudaEventRecord(ctx->ev[2], ctx->stream);
        launch(T, ctx->stream);
        cudaEventRecord(ctx->ev[3], ctx->stream);
      }
      cudaError_t e = cudaStreamSynchronize(ctx->stream);
      if (e != cudaSuccess) return cuda_error(ctx, e, "autotune");
      cudaEventElapsedTime(ms, ctx->ev[2], ctx->ev[3]);
      return VO_OK;
    }, &split);
    if (!rc) rc = prepare(split, L);
  }
  if (rc) return rc;
  record(b, (np > 0 ? 2 : 0) + (nc > 0 ? 2 : 0) + (np + nc > 0 ? 1 : 0) + (nd > 0 ? 1 : 0), [launch, L](cudaStream_t st) { launch(L, st); });
  b->rounds.push_back({counters, {}});
  for (const DilPlan &d : dils) b->rounds.back().caps.push_back(d.spill_cap);
  if (!b->once) {
    const KernelShape s = np > 0 ? patch_shape(split) : nc > 0 ? column_shape(slots, nc == 1) : direct_shape(direct_cols, direct_shift);
    b->stats.tile_rows = s.lanes;
    b->stats.union_cap = s.slots;
    b->stats.persistent = np > 0 ? 1 : 0;
    b->stats.regs = s.regs;
  }
  b->stats.tiles += L.P.nitems + L.column_items + L.direct_items;
  if (later_rounds) run_pending(ctx, b);
  return VO_OK;
}

void plan_free(vo_ctx *ctx, vo_batch *b) {
  for (const auto &s : b->stretches) {
    cudaEventDestroy(s.first);
    cudaEventDestroy(s.second);
  }
  if (b->exec) cudaGraphExecDestroy(b->exec);
  if (b->graph) cudaGraphDestroy(b->graph);
  for (SlotVol &s : b->owned) slot_free(ctx, s);
  for (void *p : b->dmem) dfree(ctx, p);
  for (vo_volume *v : b->normalized)
    if (v) vo_volume_free(ctx, v);
  for (vo_volume *v : b->rerun)
    if (v) vo_volume_free(ctx, v);
  cudaStreamSynchronize(ctx->stream);
  delete b;
}

// Plan-owned copy of the tables of radius R (H, Hp and Dx on the device, the
// host tables), shared by the plan's volumes of the same radius. The cached
// context entry is copied before any other table lookup can evict it.
int plan_tables(vo_ctx *ctx, vo_batch *b, double R, int kmax, const DeviceTables **out) {
  for (const auto &t : b->tables)
    if (t->R == R && t->kmax >= kmax) {
      *out = t.get();
      return VO_OK;
    }
  const DeviceTables *T = nullptr;
  int rc = get_tables(ctx, R, kmax, &T);
  if (rc) return rc;
  std::unique_ptr<DeviceTables> own(new (std::nothrow) DeviceTables());
  if (!own) return set_error(ctx, VO_ENOMEM, "host allocation");
  own->R = T->R;
  own->kmax = T->kmax;
  own->host = T->host;
  const size_t nh = T->host.H.size(), np = T->host.Hp.size(), nd = T->host.Dx.size();
  rc = plan_alloc(ctx, b, &own->H, nh);
  if (!rc) rc = plan_alloc(ctx, b, &own->Hp, np);
  if (!rc) rc = plan_alloc(ctx, b, &own->Dx, nd);
  if (rc) return rc;
  cudaMemcpyAsync(own->H, T->H, sizeof(double) * nh, cudaMemcpyDeviceToDevice, ctx->stream);
  cudaMemcpyAsync(own->Hp, T->Hp, sizeof(float) * np, cudaMemcpyDeviceToDevice, ctx->stream);
  cudaMemcpyAsync(own->Dx, T->Dx, sizeof(int) * nd, cudaMemcpyDeviceToDevice, ctx->stream);
  VO_CK(ctx, cudaStreamSynchronize(ctx->stream));
  *out = own.get();
  b->tables.push_back(std::move(own));
  return VO_OK;
}

int plan_build(vo_ctx *ctx, vo_batch *b) {
  const int n = b->n;
  int rc = plan_alloc(ctx, b, &b->d_flags, (size_t)n + 1);
  if (rc) return rc;
  int *flags = b->d_flags;
  record(b, 0, [flags, n](cudaStream_t st) { cudaMemsetAsync(flags, 0, sizeof(int) * (n + 1), st); });
  std::vector<std::vector<StepKind>> chain(n);
  std::vector<SlotVol> cur(n);
  std::vector<const DeviceTables *> tabs(n);
  for (int v = 0; v < n; ++v) {
    chain[v] = steps_of(b->ops[v]);
    const vo_volume *in = b->ins[v];
    if (chain[v][0] == kDil) {  // inverted pairs in a dilation input are rewritten first
      rc = normalize_inverted(ctx, in, &b->normalized[v]);
      if (rc) return rc;
      if (b->normalized[v]) in = b->normalized[v];
    }
    cur[v] = slot_view(in, 0);
    rc = max_count(ctx, cur[v], &cur[v].cap);
    if (!rc) rc = plan_tables(ctx, b, b->radii[v], std::max(in->grid.nx, in->grid.ny) + 2, &tabs[v]);
    if (rc) return rc;
  }
  std::vector<size_t> next(n, 0);
  for (;;) {
    std::vector<DilPlan> dils;
    bool any = false;
    for (int v = 0; v < n; ++v) {
      if (next[v] >= chain[v].size()) continue;
      any = true;
      const StepKind k = chain[v][next[v]++];
      const SlotVol in = cur[v];
      SlotVol out;
      int *ovf = b->d_flags + n;
      if (k == kDil) {
        DilPlan d;
        d.vol = v;
        d.in = in;
        d.T = tabs[v];
        dils.push_back(d);
        continue;
      }
      // complement steps: slot outputs sized from the input's largest column
      if (k == kNeg) {
        vo_grid g2 = in.grid;
        g2.nx += 2;
        g2.ny += 2;
        rc = slot_alloc(ctx, g2, in.cap + 1, out);
        if (!rc) record(b, 1, [in, out, ovf](cudaStream_t st) { slot_negate_launch(st, in, out, ovf); });
      } else if (k == kNorm) {
        rc = slot_alloc(ctx, in.grid, in.cap + 2, out);
        if (!rc) record(b, 1, [in, out, ovf](cudaStream_t st) { slot_normalize_launch(st, in, out, ovf); });
      } else {
        const vo_grid g = b->ins[v]->grid;
        rc = slot_alloc(ctx, g, in.cap + 1, out);
        if (!rc) record(b, 1, [in, g, out, ovf](cudaStream_t st) { slot_negate_inv_launch(st, in, g, out, ovf); });
      }
      if (rc) return rc;
      b->owned.push_back(out);
      cur[v] = out;
    }
    if (!any) break;
    if (dils.empty()) continue;
    bool later = false;
    for (const DilPlan &d : dils) later |= next[d.vol] < chain[d.vol].size();
    rc = plan_dilation_round(ctx, b, dils, later);
    if (rc) return rc;
    for (DilPlan &d : dils) {
      cur[d.vol] = d.out;
      // a complement of this result needs its largest column (the data exists: the round ran)
      if (next[d.vol] < chain[d.vol].size()) {
        rc = max_count(ctx, d.out, &cur[d.vol].cap);
        if (rc) return rc;
      }
    }
  }
  b->finals = cur;
  b->stats.learned = ctx->sizer ? 1 : 0;
  b->stats.graph_kernels = b->kernels;
  if (b->once) {
    run_pending(ctx, b);
    VO_CK(ctx, cudaGetLastError());
    return VO_OK;
  }
  // ---- capture every recorded step into one graph
  VO_CK(ctx, cudaStreamSynchronize(ctx->stream));
  VO_CK(ctx, cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal));
  for (Launch &f : b->rec) f(ctx->stream);
  cudaError_t e = cudaStreamEndCapture(ctx->stream, &b->graph);
  if (e != cudaSuccess) return cuda_error(ctx, e, "graph capture");
  e = cudaGraphInstantiate(&b->exec, b->graph, 0);
  if (e != cudaSuccess) return cuda_error(ctx, e, "graph instantiate");
  size_t nodes = 0;
  cudaGraphGetNodes(b->graph, nullptr, &nodes);
  b->stats.graph_nodes = (int)nodes;
  return VO_OK;
}

// Single-volume re-run of volume v (any union size).
int rerun_volume(vo_ctx *ctx, vo_batch *b, int v, vo_volume **out) {
  vo_timings t;
  std::memset(&t, 0, sizeof t);
  const vo_volume *in = b->ins[v];
  const double r = b->radii[v];
  switch (b->ops[v]) {
    case VO_DILATION:
      return dilate(ctx, VO_METHOD_FAST, r, in, out, &t);
    case VO_EROSION:
      return erode(ctx, VO_METHOD_FAST, r, in, out, &t);
    default: {
      vo_volume *tmp = nullptr;
      const bool open = b->ops[v] == VO_OPENING;
      int rc = open ? erode(ctx, VO_METHOD_FAST, r, in, &tmp, &t) : dilate(ctx, VO_METHOD_FAST, r, in, &tmp, &t);
      if (!rc) rc = open ? dilate(ctx, VO_METHOD_FAST, r, tmp, out, &t) : erode(ctx, VO_METHOD_FAST, r, tmp, out, &t);
      if (tmp) vo_volume_free(ctx, tmp);
      return rc;
    }
  }
}

int volume_copy(vo_ctx *ctx, const vo_volume *src, vo_volume **out) {
  vo_volume *v = nullptr;
  int rc = volume_alloc(ctx, src->grid, src->nseg, &v);
  if (rc) return rc;
  const size_t ncols = (size_t)src->grid.nx * src->grid.ny;
  cudaMemcpyAsync(v->offs, src->offs, sizeof(int32_t) * (ncols + 1), cudaMemcpyDeviceToDevice, ctx->stream);
  if (src->nseg > 0)
    cudaMemcpyAsync(v->z, src->z, sizeof(double2) * src->nseg, cudaMemcpyDeviceToDevice, ctx->stream);
  v->inverted = src->inverted;
  *out = v;
  return VO_OK;
}

bool valid_batch(int n, const int *ops, const double *radii, int method, const vo_volume *const *ins) {
  if (n < 0 || (n > 0 && (!ops || !radii || !ins))) return false;
  if (method != VO_METHOD_FAST) return false;
  for (int i = 0; i < n; ++i)
    if (!ins[i] || ops[i] < VO_DILATION || ops[i] > VO_CLOSING || !(radii[i] >= 0) || radii[i] > 255) return false;
  return true;
}

int create(vo_ctx *ctx, int n, const int *ops, const double *radii, int method, const vo_volume *const *ins,
           bool once, vo_batch **out) {
  if (!ctx || !out) return VO_EINVAL;
  *out = nullptr;
  if (!valid_batch(n, ops, radii, method, ins))
    return set_error(ctx, VO_EINVAL, "batch: bad volume, op, radius or method (VO_METHOD_FAST only)");
  cudaSetDevice(ctx->device);
  for (int i = 0; i < n; ++i) vol_wait(ctx, ins[i]);  // before any capture: the plan then reads them in order
  ctx->err.clear();
  const auto t0 = std::chrono::steady_clock::now();
  vo_batch *b = new vo_batch();
  b->n = n;
  b->once = once;
  b->ops.assign(ops, ops + n);
  b->radii.assign(radii, radii + n);
  b->ins.assign(ins, ins + n);
  b->normalized.assign(n, nullptr);
  b->rerun.assign(n, nullptr);
  std::memset(&b->stats, 0, sizeof b->stats);
  const int rc = plan_build(ctx, b);
  if (rc) {
    cudaStreamSynchronize(ctx->stream);
    cudaGetLastError();
    plan_free(ctx, b);
    return rc;
  }
  b->stats.plan_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
  *out = b;
  return VO_OK;
}

}  // namespace

extern "C" {

int vo_batch_create(vo_ctx *ctx, int n, const int *ops, const double *radii, int method,
                    const vo_volume *const *ins, vo_batch **out) {
  return create(ctx, n, ops, radii, method, ins, false, out);
}

int vo_batch_run(vo_ctx *ctx, vo_batch *b, vo_timings *tm) {
  if (!ctx || !b) return VO_EINVAL;
  cudaSetDevice(ctx->device);
  const auto t0 = std::chrono::steady_clock::now();
  for (vo_volume *&v : b->rerun)
    if (v) {
      vo_volume_free(ctx, v);
      v = nullptr;
    }
  const int n = b->n;
  std::vector<int> flags(n + 1, 0);
  std::vector<std::vector<int>> counters;
  if (!b->once) {
    cudaEventRecord(ctx->ev[0], ctx->stream);
    VO_CK(ctx, cudaGraphLaunch(b->exec, ctx->stream));
    cudaEventRecord(ctx->ev[1], ctx->stream);
  }
  cudaMemcpyAsync(flags.data(), b->d_flags, sizeof(int) * (n + 1), cudaMemcpyDeviceToHost, ctx->stream);
  for (const vo_batch::Round &r : b->rounds) {
    counters.emplace_back(kRoundCounters + kDilCounters * r.caps.size());
    cudaMemcpyAsync(counters.back().data(), r.counters, sizeof(int) * counters.back().size(), cudaMemcpyDeviceToHost,
                    ctx->stream);
  }
  VO_CK(ctx, cudaStreamSynchronize(ctx->stream));
  float graph_ms = 0;
  if (!b->once) cudaEventElapsedTime(&graph_ms, ctx->ev[0], ctx->ev[1]);
  for (const auto &s : b->stretches) {
    float ms = 0;
    if (cudaEventElapsedTime(&ms, s.first, s.second) == cudaSuccess) graph_ms += ms;
  }
  // spill use of every dilation (the largest fraction and its round)
  b->stats.spill_peak = 0;
  b->stats.spill_peak_round = -1;
  for (size_t r = 0; r < b->rounds.size(); ++r)
    for (size_t i = 0; i < b->rounds[r].caps.size(); ++i) {
      const int cap = b->rounds[r].caps[i];
      const double f = cap > 0 ? (double)counters[r][kRoundCounters + kDilCounters * i] / cap : 0.0;
      if (f > b->stats.spill_peak) {
        b->stats.spill_peak = f;
        b->stats.spill_peak_round = (int)r;
      }
    }
  int reruns = 0;
  const int launches0 = ctx->launches;
  b->stats.rerun_first = -1;
  b->stats.rerun_cause = 0;
  for (int v = 0; v < n; ++v) {
    if (!flags[v] && !flags[n]) continue;
    if (reruns == 0) {
      b->stats.rerun_first = v;
      b->stats.rerun_cause = flags[v] | (flags[n] ? 2 : 0);
    }
    ++reruns;
    const int rc = rerun_volume(ctx, b, v, &b->rerun[v]);
    if (rc) return rc;
  }
  b->stats.reruns = reruns;
  if (tm) {
    std::memset(tm, 0, sizeof *tm);
    tm->total_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    tm->pass2_ms = graph_ms;
    tm->kernel_ms[3] = graph_ms;
    for (int v = 0; v < n; ++v) tm->in_segments += b->ins[v]->nseg;
    tm->kernel_launches = b->kernels + (ctx->launches - launches0);
    tm->overflow_columns = reruns;
  }
  return VO_OK;
}

int vo_batch_outputs(vo_ctx *ctx, vo_batch *b, vo_volume **outs) {
  if (!ctx || !b || (b->n > 0 && !outs)) return VO_EINVAL;
  cudaSetDevice(ctx->device);
  int rc = VO_OK;
  for (int v = 0; v < b->n; ++v) outs[v] = nullptr;
  for (int v = 0; v < b->n && !rc; ++v)
    rc = b->rerun[v] ? volume_copy(ctx, b->rerun[v], &outs[v]) : slot_to_volume(ctx, b->finals[v], &outs[v]);
  if (!rc) {
    cudaError_t e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) rc = cuda_error(ctx, e, "batch outputs");
  }
  if (rc)
    for (int v = 0; v < b->n; ++v)
      if (outs[v]) {
        vo_volume_free(ctx, outs[v]);
        outs[v] = nullptr;
      }
  return rc;
}

int vo_batch_stats_get(vo_ctx *ctx, const vo_batch *b, vo_batch_stats *s) {
  if (!ctx || !b || !s) return VO_EINVAL;
  *s = b->stats;
  return VO_OK;
}

void vo_batch_destroy(vo_ctx *ctx, vo_batch *b) {
  if (!ctx || !b) return;
  cudaSetDevice(ctx->device);
  plan_free(ctx, b);
}

}  // extern "C"

namespace vo {

int morph_batched_fast(vo_ctx *ctx, int n, const int *ops, const double *radii, const vo_volume *const *ins,
                       vo_volume **outs, vo_timings *tm) {
  const auto t0 = std::chrono::steady_clock::now();
  vo_batch *b = nullptr;
  // a replay would run the steps that the plan had to run for a later step's sizes a second time
  int rc = create(ctx, n, ops, radii, VO_METHOD_FAST, ins, true, &b);
  if (rc) return rc;
  rc = vo_batch_run(ctx, b, tm);
  if (!rc) rc = vo_batch_outputs(ctx, b, outs);
  if (!rc && tm) {
    tm->total_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    for (int v = 0; v < n; ++v) tm->out_segments += outs[v]->nseg;
  }
  vo_batch_destroy(ctx, b);
  return rc;
}

}  // namespace vo
