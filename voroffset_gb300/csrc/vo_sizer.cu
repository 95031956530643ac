// Learned sizing for batched dilation (no reference counterpart).
//
// A small MLP predicts, for every 32 x 32 tile of output columns, the largest
// and the mean output segment count per column and the mean number of
// candidate intervals per column (the work), from statistics of the input
// columns (occupancy, mean / max segment count, a histogram of the gaps
// between consecutive segments in 8 log2 bins, coverage, the radius). The
// batched executor uses the predictions to size each tile's output slots and
// to order its work queue, which removes the exact count pass; any column that
// outgrows its predicted slot is detected exactly and its volume re-runs
// through the plain path, so results never depend on the prediction.
//
// Network: 16 inputs -> 64 ReLU -> 64 ReLU -> 4 outputs (3 used), weights in
// BF16 for inference, FP32 master copies, FP32 accumulation everywhere;
// trained on the GPU with the kernels below (squared error on log2 targets,
// under-prediction of the max count weighted 4x; Adam). Layout of the flat parameter vector: W1[16][64], b1[64],
// W2[64][64], b2[64], W3[64][4], b3[4] (row-major, [in][out]).
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "vo_internal.cuh"

namespace vo {
namespace {

constexpr int NF = VO_SIZER_FEATURES, NH = 64, NO = 4, NUSED = VO_SIZER_OUTPUTS;
constexpr int OFF_W1 = 0, OFF_B1 = OFF_W1 + NF * NH, OFF_W2 = OFF_B1 + NH, OFF_B2 = OFF_W2 + NH * NH,
              OFF_W3 = OFF_B2 + NH, OFF_B3 = OFF_W3 + NH * NO, NPARAM = OFF_B3 + NO;
constexpr int kTile = kSizerTile;

// ---------------------------------------------------------------- features

// One block per 32 x 32 tile of columns: occupancy, mean / max count, gap
// histogram (log2 bins: < 1, < 2, ..., < 64, >= 64 dexels), coverage.
__global__ void k_tile_stats(int nx, int ny, const int32_t *__restrict__ beg, const int32_t *__restrict__ end,
                             const double2 *__restrict__ z, float *stats) {
  __shared__ float s_occ, s_sum, s_len, s_hist[8];
  __shared__ int s_max;
  const int tiles_x = (nx + kTile - 1) / kTile;
  const int t = blockIdx.x;
  const int x0 = (t % tiles_x) * kTile, y0 = (t / tiles_x) * kTile;
  if (threadIdx.x == 0) {
    s_occ = s_sum = s_len = 0;
    s_max = 0;
    for (int b = 0; b < 8; ++b) s_hist[b] = 0;
  }
  __syncthreads();
  float occ = 0, sum = 0, len = 0, hist[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  int mx = 0;
  for (int i = threadIdx.x; i < kTile * kTile; i += blockDim.x) {
    const int x = x0 + i % kTile, y = y0 + i / kTile;
    if (x >= nx || y >= ny) continue;
    const int c = x + nx * y;
    const int k0 = beg[c], k1 = end[c], n = k1 - k0;
    occ += n > 0;
    sum += n;
    mx = max(mx, n);
    for (int k = k0; k < k1; ++k) {
      const double2 s = z[k];
      len += (float)(s.y - s.x);
      if (k > k0) {
        const float gap = (float)(s.x - z[k - 1].y);
        int b = gap < 1.f ? 0 : min(7, 1 + (int)floorf(log2f(gap)));
        hist[b] += 1;
      }
    }
  }
  atomicAdd(&s_occ, occ);
  atomicAdd(&s_sum, sum);
  atomicAdd(&s_len, len);
  atomicMax(&s_max, mx);
  for (int b = 0; b < 8; ++b) atomicAdd(&s_hist[b], hist[b]);
  __syncthreads();
  if (threadIdx.x == 0) {
    const int w = min(kTile, nx - x0), h = min(kTile, ny - y0);
    const float cols = (float)(w * h);
    float *f = stats + (size_t)t * NF;
    f[0] = s_occ / cols;
    f[1] = s_sum / cols;
    f[2] = (float)s_max;
    float gaps = 0;
    for (int b = 0; b < 8; ++b) gaps += s_hist[b];
    for (int b = 0; b < 8; ++b) f[3 + b] = gaps > 0 ? s_hist[b] / gaps : 0.f;
    f[11] = s_len / cols / 64.f;
  }
}

// Final features: log-scaled counts, the 3 x 3 tile neighbourhood mean count
// (the dilation reaches across tiles) and the radius terms.
__global__ void k_tile_features(int tiles_x, int tiles_y, float radius, float npairs, const float *stats,
                                float *feats) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= tiles_x * tiles_y) return;
  const int tx = t % tiles_x, ty = t / tiles_x;
  const float *s = stats + (size_t)t * NF;
  float nb = 0;
  int cnt = 0;
  for (int dy = -1; dy <= 1; ++dy)
    for (int dx = -1; dx <= 1; ++dx) {
      const int ux = tx + dx, uy = ty + dy;
      if (ux < 0 || uy < 0 || ux >= tiles_x || uy >= tiles_y) continue;
      nb += stats[(size_t)(ux + tiles_x * uy) * NF + 1];
      ++cnt;
    }
  float *f = feats + (size_t)t * NF;
  f[0] = s[0];
  f[1] = log2f(1.f + s[1]);
  f[2] = log2f(1.f + s[2]);
  for (int b = 0; b < 8; ++b) f[3 + b] = s[3 + b];
  f[11] = s[11];
  f[12] = log2f(1.f + nb / (float)max(cnt, 1));
  f[13] = radius / 64.f;
  f[14] = log2f(1.f + npairs) / 12.f;
  f[15] = 1.f;
}

// Per column: output count (from a result) and candidate count (sum over the
// alive (|dx|, |dy|) pairs of the source columns' segment counts).
__global__ void k_tile_targets(int nx, int ny, const int32_t *__restrict__ ibeg, const int32_t *__restrict__ iend,
                               const int32_t *__restrict__ ooffs, const int2 *__restrict__ pairs, int npairs,
                               float *targets) {
  __shared__ float s_mean, s_work;
  __shared__ int s_max;
  const int tiles_x = (nx + kTile - 1) / kTile;
  const int t = blockIdx.x;
  const int x0 = (t % tiles_x) * kTile, y0 = (t / tiles_x) * kTile;
  if (threadIdx.x == 0) {
    s_mean = s_work = 0;
    s_max = 0;
  }
  __syncthreads();
  float mean = 0, work = 0;
  int mx = 0;
  for (int i = threadIdx.x; i < kTile * kTile; i += blockDim.x) {
    const int x = x0 + i % kTile, y = y0 + i / kTile;
    if (x >= nx || y >= ny) continue;
    const int c = x + nx * y;
    const int n = ooffs[c + 1] - ooffs[c];
    mean += n;
    mx = max(mx, n);
    int wk = 0;
    for (int p = 0; p < npairs; ++p) {
      const int a = pairs[p].x, d = pairs[p].y;
      for (int s = 0; s < 4; ++s) {
        if (((s & 1) && a == 0) || ((s & 2) && d == 0)) continue;
        const int xs = (s & 1) ? x + a : x - a, ys = (s & 2) ? y + d : y - d;
        if (xs < 0 || xs >= nx || ys < 0 || ys >= ny) continue;
        const int cs = xs + nx * ys;
        wk += iend[cs] - ibeg[cs];
      }
    }
    work += (float)wk;
  }
  atomicAdd(&s_mean, mean);
  atomicAdd(&s_work, work);
  atomicMax(&s_max, mx);
  __syncthreads();
  if (threadIdx.x == 0) {
    const int w = min(kTile, nx - x0), h = min(kTile, ny - y0);
    const float cols = (float)(w * h);
    float *o = targets + (size_t)t * NUSED;
    o[0] = log2f(1.f + (float)s_max);
    o[1] = log2f(1.f + s_mean / cols);
    o[2] = log2f(1.f + s_work / cols);
  }
}

// ---------------------------------------------------------------- network

// Pairs of FP32 values in a 64-bit register: one instruction rounds both
// products (or sums) as two scalar ones would. The product is a fused
// multiply-add with -0, which is exact; -0 is a kernel argument, since the
// assembler turned a packed product (or one with a -0 it could see) and the
// packed addition after it into one fused operation, whose rounding differs.
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pair(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 unpair(f32x2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b, f32x2 neg0) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(neg0));
  return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// acc[0..8) += x * w[0..8), each product rounded before its addition
__device__ __forceinline__ void axpy8(f32x2 (&acc)[4], float x, const float *w, f32x2 neg0) {
  const ulonglong2 w0 = *reinterpret_cast<const ulonglong2 *>(w), w1 = *reinterpret_cast<const ulonglong2 *>(w + 4);
  const f32x2 xx = pair(x, x);
  acc[0] = add2(acc[0], mul2(xx, w0.x, neg0));
  acc[1] = add2(acc[1], mul2(xx, w0.y, neg0));
  acc[2] = add2(acc[2], mul2(xx, w1.x, neg0));
  acc[3] = add2(acc[3], mul2(xx, w1.y, neg0));
}

constexpr f32x2 kNegZeros = 0x8000000080000000ull;
constexpr float kUnderWeight = 4.f;
constexpr int kMlpThreads = 128;

// Forward pass and, with TRAIN, the backward pass through the activations, one
// sample per thread. Weights are BF16, staged in shared memory as FP32;
// accumulation is FP32 in the order of the inputs, eight outputs at a time.
// What bounds it is the shared-memory path that hands the weights to the lanes
// (128 bytes a cycle): one read per product took 92 + 125 us for 65,536
// samples, two 16-byte reads per eight products take 68 us (two samples per
// thread, which would halve the reads, spill: 73 us).
// TRAIN: dz2 = (dout W3^T) * [h2 > 0], dz1 = (dz2 W2^T) * [h1 > 0], with
// dout = 2 w (out - target) / (n * NUSED) on the used outputs. The loss is the
// weighted squared error with w = kUnderWeight where the max-count output is
// below its target (slots sized too small cost spills and re-runs, too large
// only memory), else 1. Activations and their gradients are stored by unit,
// ld samples apart, so that neighbouring threads store side by side.
template <bool TRAIN>
__global__ void __launch_bounds__(kMlpThreads, 4) k_mlp(const float *__restrict__ X, int n, int ld,
                                                     const __nv_bfloat16 *__restrict__ w, float *__restrict__ out,
                                                     const float *__restrict__ tgt, float *__restrict__ h1s,
                                                     float *__restrict__ h2s, float *__restrict__ dout,
                                                     float *__restrict__ dz2, float *__restrict__ dz1, float *loss,
                                                     f32x2 neg0) {
  __shared__ __align__(16) float sw[NPARAM];
  __shared__ __align__(16) float swt[TRAIN ? NH * NH : 4];  // W2 transposed
  for (int i = threadIdx.x; i < NPARAM; i += kMlpThreads) sw[i] = __bfloat162float(w[i]);
  if (TRAIN)
    for (int i = threadIdx.x; i < NH * NH; i += kMlpThreads)
      swt[(i % NH) * NH + i / NH] = __bfloat162float(w[OFF_W2 + i]);
  __syncthreads();
  const int s = blockIdx.x * kMlpThreads + threadIdx.x;
  float l = 0;
  if (s < n) {
    float h1[NH], o[NO];
    {
      float x[NF];
#pragma unroll
      for (int i = 0; i < NF; i += 4) {
        const float4 v = *reinterpret_cast<const float4 *>(X + (size_t)s * NF + i);
        x[i] = v.x, x[i + 1] = v.y, x[i + 2] = v.z, x[i + 3] = v.w;
      }
#pragma unroll
      for (int j = 0; j < NH; j += 8) {
        f32x2 acc[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[q] = *reinterpret_cast<const f32x2 *>(sw + OFF_B1 + j + 2 * q);
#pragma unroll
        for (int i = 0; i < NF; ++i) axpy8(acc, x[i], sw + OFF_W1 + i * NH + j, neg0);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float2 v = unpair(acc[q]);
          h1[j + 2 * q] = fmaxf(v.x, 0.f);
          h1[j + 2 * q + 1] = fmaxf(v.y, 0.f);
        }
      }
    }
    unsigned long long on1 = 0, on2 = 0;  // units with a positive activation
    if (TRAIN) {
#pragma unroll
      for (int j = 0; j < NH; ++j) {
        h1s[(size_t)j * ld + s] = h1[j];
        on1 |= h1[j] > 0.f ? 1ull << j : 0ull;
      }
    }
    for (int k = 0; k < NO; ++k) o[k] = sw[OFF_B3 + k];
    for (int j = 0; j < NH; j += 8) {
      f32x2 acc[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[q] = *reinterpret_cast<const f32x2 *>(sw + OFF_B2 + j + 2 * q);
#pragma unroll
      for (int i = 0; i < NH; ++i) axpy8(acc, h1[i], sw + OFF_W2 + i * NH + j, neg0);
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const float2 v = unpair(acc[q / 2]);
        const float h = fmaxf(q & 1 ? v.y : v.x, 0.f);
        if (TRAIN) {
          h2s[(size_t)(j + q) * ld + s] = h;
          on2 |= h > 0.f ? 1ull << (j + q) : 0ull;
        }
#pragma unroll
        for (int k = 0; k < NO; ++k) o[k] += h * sw[OFF_W3 + (j + q) * NO + k];
      }
    }
    *reinterpret_cast<float4 *>(out + (size_t)s * NO) = make_float4(o[0], o[1], o[2], o[3]);
    if (TRAIN) {
      float go[NO];
#pragma unroll
      for (int k = 0; k < NO; ++k) {
        const float e = k < NUSED ? o[k] - tgt[(size_t)s * NUSED + k] : 0.f;
        const float wgt = (k == 0 && e < 0.f) ? kUnderWeight : 1.f;
        l += wgt * e * e;
        go[k] = 2.f * wgt * e / (float)(n * NUSED);
        dout[(size_t)k * ld + s] = go[k];
      }
      float g2[NH];
#pragma unroll
      for (int j = 0; j < NH; ++j) {
        float a = 0;
#pragma unroll
        for (int k = 0; k < NO; ++k) a += go[k] * sw[OFF_W3 + j * NO + k];
        g2[j] = on2 >> j & 1 ? a : 0.f;
        dz2[(size_t)j * ld + s] = g2[j];
      }
      for (int i = 0; i < NH; i += 8) {
        f32x2 acc[4] = {0, 0, 0, 0};
#pragma unroll
        for (int j = 0; j < NH; ++j) axpy8(acc, g2[j], swt + j * NH + i, neg0);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const float2 v = unpair(acc[q / 2]);
          dz1[(size_t)(i + q) * ld + s] = on1 >> (i + q) & 1 ? (q & 1 ? v.y : v.x) : 0.f;
        }
      }
    }
  }
  if (TRAIN) {
    for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(loss, l / (float)(n * NUSED));
  }
}

// Features by unit, ld samples apart (once per training run).
__global__ void k_transpose(const float *__restrict__ X, int n, int ld, float *__restrict__ XT) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s < n)
    for (int i = 0; i < NF; ++i) XT[(size_t)i * ld + s] = X[(size_t)s * NF + i];
}

// Weight gradients as reductions over the samples, dW[i][j] = sum_s A[s][i] *
// G[s][j] and db[j] = sum_s G[s][j]: a block per chunk of kGradChunk samples
// sums every parameter of its part in the order of the samples (deterministic),
// and k_grad_step adds the chunks in order. blockIdx.y 0, 1: the halves of W2,
// 2 x 4 parameters per thread from tiles of kGradTile samples in shared
// memory, so that six 16-byte reads feed 32 products (one thread per parameter
// read both factors from memory: 532 us for 65,536 samples; now 53 us); 2: the
// other parameters.
constexpr int kGradChunk = 512, kGradThreads = 256, kGradTile = 32, kGradPitch = kGradTile + 4;

// ROWS rows of kGradTile samples: fetched into registers while the tile before
// is summed (101 us when each was waited for), then stored.
// row(r) is row r's samples; past the last sample come zeros.
template <int ROWS>
struct GradTile {
  static constexpr int N = (ROWS * (kGradTile / 4) + kGradThreads - 1) / kGradThreads;
  float4 v[N];
  template <typename Row>
  __device__ __forceinline__ void fetch(const Row &row, int s0, int n) {
#pragma unroll
    for (int q = 0; q < N; ++q) {
      const int i = threadIdx.x + q * kGradThreads, r = i / (kGradTile / 4), c = 4 * (i % (kGradTile / 4));
      // rows hold a multiple of four samples: the read stays inside the array
      v[q] = r < ROWS && s0 + c < n ? *reinterpret_cast<const float4 *>(row(r) + s0 + c)
                                    : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
  __device__ __forceinline__ void store(float *dst) const {
#pragma unroll
    for (int q = 0; q < N; ++q) {
      const int i = threadIdx.x + q * kGradThreads, r = i / (kGradTile / 4), c = 4 * (i % (kGradTile / 4));
      if (r < ROWS) *reinterpret_cast<float4 *>(dst + r * kGradPitch + c) = v[q];
    }
  }
};

__global__ void __launch_bounds__(kGradThreads) k_mlp_wgrad(const float *__restrict__ XT, const float *__restrict__ h1s,
                                                            const float *__restrict__ h2s,
                                                            const float *__restrict__ dout,
                                                            const float *__restrict__ dz2,
                                                            const float *__restrict__ dz1, int n, int ld,
                                                            float *__restrict__ part) {
  constexpr int kRest = NF + 3 * NH + NO;
  __shared__ __align__(16) float tile[kRest * kGradPitch];
  const int tid = threadIdx.x;
  const int c0 = blockIdx.x * kGradChunk, c1 = min(n, c0 + kGradChunk);
  float *p = part + (size_t)blockIdx.x * NPARAM;
  const int ti = tid % 16, tj = tid / 16;
  if (blockIdx.y < 2) {
    // parameters (i0 + ti + 16 a, tj + 16 b): the rows of a warp lie next to each other, in different banks
    const int i0 = blockIdx.y * (NH / 2);
    const float *ta = tile, *tb = tile + (NH / 2) * kGradPitch;
    auto row = [&](int r) { return r < NH / 2 ? h1s + (size_t)(i0 + r) * ld : dz2 + (size_t)(r - NH / 2) * ld; };
    GradTile<NH / 2 + NH> next;
    next.fetch(row, c0, n);
    float acc[2][4] = {};
    for (int s0 = c0; s0 < c1; s0 += kGradTile) {
      __syncthreads();
      next.store(tile);
      __syncthreads();
      if (s0 + kGradTile < c1) next.fetch(row, s0 + kGradTile, n);
      const int cnt = min(kGradTile, c1 - s0);
      int t = 0;
      for (; t + 4 <= cnt; t += 4) {
        float4 A[2], G[4];
#pragma unroll
        for (int a = 0; a < 2; ++a) A[a] = *reinterpret_cast<const float4 *>(ta + (ti + 16 * a) * kGradPitch + t);
#pragma unroll
        for (int b = 0; b < 4; ++b) G[b] = *reinterpret_cast<const float4 *>(tb + (tj + 16 * b) * kGradPitch + t);
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
          for (int b = 0; b < 4; ++b) {
            acc[a][b] += A[a].x * G[b].x;
            acc[a][b] += A[a].y * G[b].y;
            acc[a][b] += A[a].z * G[b].z;
            acc[a][b] += A[a].w * G[b].w;
          }
      }
      for (; t < cnt; ++t)
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
          for (int b = 0; b < 4; ++b)
            acc[a][b] += ta[(ti + 16 * a) * kGradPitch + t] * tb[(tj + 16 * b) * kGradPitch + t];
    }
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) p[OFF_W2 + (i0 + ti + 16 * a) * NH + tj + 16 * b] = acc[a][b];
    return;
  }
  // rows: X, dz1, h2, dz2, dout
  const float *tx = tile, *tz1 = tx + NF * kGradPitch, *th2 = tz1 + NH * kGradPitch, *tz2 = th2 + NH * kGradPitch,
              *to = tz2 + NH * kGradPitch;
  auto row = [&](int r) {
    return r < NF ? XT + (size_t)r * ld
           : r < NF + NH ? dz1 + (size_t)(r - NF) * ld
           : r < NF + 2 * NH ? h2s + (size_t)(r - NF - NH) * ld
           : r < NF + 3 * NH ? dz2 + (size_t)(r - NF - 2 * NH) * ld : dout + (size_t)(r - NF - 3 * NH) * ld;
  };
  GradTile<kRest> next;
  next.fetch(row, c0, n);
  // W1: (ti, tj + 16 b); W3: one parameter per thread; biases: one per thread of the first 132
  float w1[4] = {}, w3 = 0.f, bias = 0.f;
  const float *rx = tx + ti * kGradPitch, *rh = th2 + (tid / NO) * kGradPitch, *ro = to + (tid % NO) * kGradPitch;
  const float *rb = tid < NH ? tz1 + tid * kGradPitch
                    : tid < 2 * NH ? tz2 + (tid - NH) * kGradPitch
                    : tid < 2 * NH + NO ? to + (tid - 2 * NH) * kGradPitch : to;
  for (int s0 = c0; s0 < c1; s0 += kGradTile) {
    __syncthreads();
    next.store(tile);
    __syncthreads();
    if (s0 + kGradTile < c1) next.fetch(row, s0 + kGradTile, n);
    const int cnt = min(kGradTile, c1 - s0);
    int t = 0;
    for (; t + 4 <= cnt; t += 4) {
      const float4 x = *reinterpret_cast<const float4 *>(rx + t), h = *reinterpret_cast<const float4 *>(rh + t),
                   o = *reinterpret_cast<const float4 *>(ro + t), g = *reinterpret_cast<const float4 *>(rb + t);
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const float4 z = *reinterpret_cast<const float4 *>(tz1 + (tj + 16 * b) * kGradPitch + t);
        w1[b] += x.x * z.x;
        w1[b] += x.y * z.y;
        w1[b] += x.z * z.z;
        w1[b] += x.w * z.w;
      }
      w3 += h.x * o.x;
      w3 += h.y * o.y;
      w3 += h.z * o.z;
      w3 += h.w * o.w;
      bias += g.x;
      bias += g.y;
      bias += g.z;
      bias += g.w;
    }
    for (; t < cnt; ++t) {
#pragma unroll
      for (int b = 0; b < 4; ++b) w1[b] += rx[t] * tz1[(tj + 16 * b) * kGradPitch + t];
      w3 += rh[t] * ro[t];
      bias += rb[t];
    }
  }
#pragma unroll
  for (int b = 0; b < 4; ++b) p[OFF_W1 + ti * NH + tj + 16 * b] = w1[b];
  p[OFF_W3 + tid] = w3;
  if (tid < NH) p[OFF_B1 + tid] = bias;
  else if (tid < 2 * NH) p[OFF_B2 + tid - NH] = bias;
  else if (tid < 2 * NH + NO) p[OFF_B3 + tid - 2 * NH] = bias;
}
static_assert(kGradThreads == NH * NO && kGradThreads >= 2 * NH + NO && NF == 16 && NH == 64, "layout of k_mlp_wgrad");

// Adds the chunks in order and, with `step`, takes the Adam step.
__global__ void k_grad_step(const float *__restrict__ part, int nchunks, float *__restrict__ grad,
                            float *__restrict__ wm, float *__restrict__ m, float *__restrict__ v,
                            __nv_bfloat16 *__restrict__ wb, bool step, float lr, float b1, float b2, float c1,
                            float c2) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= NPARAM) return;
  float acc = 0;
  int c = 0;
  for (; c + 16 <= nchunks; c += 16) {
    float t[16];
#pragma unroll
    for (int q = 0; q < 16; ++q) t[q] = part[(size_t)(c + q) * NPARAM + p];
#pragma unroll
    for (int q = 0; q < 16; ++q) acc += t[q];
  }
  for (; c < nchunks; ++c) acc += part[(size_t)c * NPARAM + p];
  grad[p] = acc;
  if (!step) return;
  m[p] = b1 * m[p] + (1.f - b1) * acc;
  v[p] = b2 * v[p] + (1.f - b2) * acc * acc;
  const float mh = m[p] / c1, vh = v[p] / c2;
  wm[p] -= lr * mh / (sqrtf(vh) + 1e-8f);
  wb[p] = __float2bfloat16_rn(wm[p]);
}

__global__ void k_to_bf16(const float *__restrict__ wm, __nv_bfloat16 *__restrict__ wb) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p < NPARAM) wb[p] = __float2bfloat16_rn(wm[p]);
}

}  // namespace
}  // namespace vo

struct vo_sizer {
  float *wm = nullptr;        // FP32 master parameters
  __nv_bfloat16 *wb = nullptr;  // BF16 parameters used by the forward pass
  float *m = nullptr, *v = nullptr, *grad = nullptr;
  int step = 0;
};

using namespace vo;

namespace {

struct Work {
  float *X = nullptr, *XT = nullptr, *T = nullptr, *out = nullptr, *h1 = nullptr, *h2 = nullptr, *dout = nullptr,
        *dz2 = nullptr, *dz1 = nullptr, *loss = nullptr, *part = nullptr;
  int ld = 0;  // samples per unit row: n rounded up to 4
};

int nchunks(int n) { return (n + kGradChunk - 1) / kGradChunk; }

int work_alloc(vo_ctx *ctx, int n, bool train, Work &w) {
  w.ld = (n + 3) & ~3;
  const size_t ld = (size_t)w.ld;
  int rc = dalloc(ctx, &w.X, (size_t)n * NF);
  if (!rc) rc = dalloc(ctx, &w.out, (size_t)n * NO);
  if (train) {
    if (!rc) rc = dalloc(ctx, &w.XT, ld * NF);
    if (!rc) rc = dalloc(ctx, &w.T, (size_t)n * NUSED);
    if (!rc) rc = dalloc(ctx, &w.h1, ld * NH);
    if (!rc) rc = dalloc(ctx, &w.h2, ld * NH);
    if (!rc) rc = dalloc(ctx, &w.dout, ld * NO);
    if (!rc) rc = dalloc(ctx, &w.dz2, ld * NH);
    if (!rc) rc = dalloc(ctx, &w.dz1, ld * NH);
    if (!rc) rc = dalloc(ctx, &w.loss, 1);
    if (!rc) rc = dalloc(ctx, &w.part, (size_t)nchunks(n) * NPARAM);
  }
  return rc;
}

void work_free(vo_ctx *ctx, Work &w) {
  for (float *p : {w.X, w.XT, w.T, w.out, w.h1, w.h2, w.dout, w.dz2, w.dz1, w.loss, w.part}) dfree(ctx, p);
  w = Work();
}

void forward_launch(vo_ctx *ctx, const float *X, int n, const __nv_bfloat16 *wb, float *out) {
  k_mlp<false><<<(n + kMlpThreads - 1) / kMlpThreads, kMlpThreads, 0, ctx->stream>>>(
      X, n, 0, wb, out, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, kNegZeros);
  ctx->launches += 1;
}

// One forward + backward pass over the n samples in w: gradients in s->grad
// and, with `step`, an Adam step (s->step counts it).
void grad_pass(vo_ctx *ctx, vo_sizer *s, int n, Work &w, bool step, float lr) {
  cudaMemsetAsync(w.loss, 0, sizeof(float), ctx->stream);
  k_mlp<true><<<(n + kMlpThreads - 1) / kMlpThreads, kMlpThreads, 0, ctx->stream>>>(
      w.X, n, w.ld, s->wb, w.out, w.T, w.h1, w.h2, w.dout, w.dz2, w.dz1, w.loss, kNegZeros);
  k_mlp_wgrad<<<dim3(nchunks(n), 3), kGradThreads, 0, ctx->stream>>>(w.XT, w.h1, w.h2, w.dout, w.dz2, w.dz1, n, w.ld,
                                                                     w.part);
  const float b1 = 0.9f, b2 = 0.999f;
  const float t = (float)(s->step + 1);
  k_grad_step<<<(NPARAM + 63) / 64, 64, 0, ctx->stream>>>(w.part, nchunks(n), s->grad, s->wm, s->m, s->v, s->wb, step,
                                                          lr, b1, b2, 1.f - std::pow(b1, t), 1.f - std::pow(b2, t));
  if (step) ++s->step;
  ctx->launches += 3;
}

std::vector<int2> alive_pairs(const Tables &h) {
  std::vector<int2> pairs;
  for (int d = 0; d <= h.Dy; ++d)
    for (int a = 0; a <= h.Dx[d]; ++a) pairs.push_back(make_int2(a, d));
  return pairs;
}

}  // namespace

namespace vo {

// Features of the 32 x 32 tiles of a slot view into a device array (n tiles).
int sizer_features_device(vo_ctx *ctx, const SlotVol &in, double radius, float *feats, int *ntiles) {
  const vo_grid &g = in.grid;
  const int tx = (g.nx + kTile - 1) / kTile, ty = (g.ny + kTile - 1) / kTile;
  *ntiles = tx * ty;
  const DeviceTables *T = nullptr;
  int rc = get_tables(ctx, radius, std::max(g.nx, g.ny) + 2, &T);
  if (rc) return rc;
  float *stats = nullptr;
  rc = dalloc(ctx, &stats, (size_t)tx * ty * NF);
  if (rc) return rc;
  const float npairs = (float)alive_pairs(T->host).size();
  k_tile_stats<<<tx * ty, 256, 0, ctx->stream>>>(g.nx, g.ny, in.beg, in.end, in.z, stats);
  k_tile_features<<<(tx * ty + 127) / 128, 128, 0, ctx->stream>>>(tx, ty, (float)radius, npairs, stats, feats);
  ctx->launches += 2;
  dfree(ctx, stats);
  return VO_OK;
}

// Predictions (n x VO_SIZER_OUTPUTS-padded-to-4) for device features.
int sizer_predict_device(vo_ctx *ctx, const vo_sizer *s, const float *feats, int n, float *out4) {
  if (n <= 0) return VO_OK;
  forward_launch(ctx, feats, n, s->wb, out4);
  return VO_OK;
}

}  // namespace vo

extern "C" {

int vo_sizer_create(vo_ctx *ctx, uint64_t seed, vo_sizer **out) {
  if (!ctx || !out) return VO_EINVAL;
  *out = nullptr;
  vo_sizer *s = new vo_sizer();
  int rc = dalloc(ctx, &s->wm, NPARAM);
  if (!rc) rc = dalloc(ctx, &s->wb, NPARAM);
  if (!rc) rc = dalloc(ctx, &s->m, NPARAM);
  if (!rc) rc = dalloc(ctx, &s->v, NPARAM);
  if (!rc) rc = dalloc(ctx, &s->grad, NPARAM);
  if (rc) {
    vo_sizer_destroy(ctx, s);
    return rc;
  }
  // He-uniform initialisation from a splitmix64 stream, biases zero.
  std::vector<float> w(NPARAM, 0.f);
  uint64_t st = seed;
  auto uni = [&]() {
    uint64_t z = (st += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    return (double)(z >> 11) * (1.0 / 9007199254740992.0);
  };
  auto fill = [&](int off, int fan_in, int cnt) {
    const double lim = std::sqrt(6.0 / fan_in);
    for (int i = 0; i < cnt; ++i) w[off + i] = (float)((2 * uni() - 1) * lim);
  };
  fill(OFF_W1, NF, NF * NH);
  fill(OFF_W2, NH, NH * NH);
  fill(OFF_W3, NH, NH * NO);
  rc = vo_sizer_set_params(ctx, s, w.data(), NPARAM);
  if (rc) {
    vo_sizer_destroy(ctx, s);
    return rc;
  }
  *out = s;
  return VO_OK;
}

void vo_sizer_destroy(vo_ctx *ctx, vo_sizer *s) {
  if (!ctx || !s) return;
  if (ctx->sizer == s) ctx->sizer = nullptr;
  dfree(ctx, s->wm);
  dfree(ctx, s->wb);
  dfree(ctx, s->m);
  dfree(ctx, s->v);
  dfree(ctx, s->grad);
  cudaStreamSynchronize(ctx->stream);
  delete s;
}

int vo_sizer_num_params(void) { return NPARAM; }

int vo_sizer_set_params(vo_ctx *ctx, vo_sizer *s, const float *params, int count) {
  if (!ctx || !s || !params || count != NPARAM) return VO_EINVAL;
  VO_CK(ctx, cudaMemcpyAsync(s->wm, params, sizeof(float) * NPARAM, cudaMemcpyHostToDevice, ctx->stream));
  cudaMemsetAsync(s->m, 0, sizeof(float) * NPARAM, ctx->stream);
  cudaMemsetAsync(s->v, 0, sizeof(float) * NPARAM, ctx->stream);
  k_to_bf16<<<(NPARAM + 127) / 128, 128, 0, ctx->stream>>>(s->wm, s->wb);
  s->step = 0;
  VO_CK(ctx, cudaStreamSynchronize(ctx->stream));
  return VO_OK;
}

int vo_sizer_get_params(vo_ctx *ctx, const vo_sizer *s, float *params, int count) {
  if (!ctx || !s || !params || count != NPARAM) return VO_EINVAL;
  VO_CK(ctx, cudaMemcpyAsync(params, s->wm, sizeof(float) * NPARAM, cudaMemcpyDeviceToHost, ctx->stream));
  VO_CK(ctx, cudaStreamSynchronize(ctx->stream));
  return VO_OK;
}

int vo_sizer_tile_features(vo_ctx *ctx, const vo_volume *v, double radius, float *feats, int *ntiles) {
  if (!ctx || !v || !ntiles) return VO_EINVAL;
  vol_wait(ctx, v);
  const int tx = (v->grid.nx + kTile - 1) / kTile, ty = (v->grid.ny + kTile - 1) / kTile;
  if (!feats) {
    *ntiles = tx * ty;
    return VO_OK;
  }
  float *d = nullptr;
  int rc = dalloc(ctx, &d, (size_t)tx * ty * NF);
  if (rc) return rc;
  int n = 0;
  rc = sizer_features_device(ctx, slot_view(v, 0), radius, d, &n);
  if (!rc) cudaMemcpyAsync(feats, d, sizeof(float) * n * NF, cudaMemcpyDeviceToHost, ctx->stream);
  dfree(ctx, d);
  if (rc) return rc;
  VO_CK(ctx, cudaStreamSynchronize(ctx->stream));
  *ntiles = n;
  return VO_OK;
}

int vo_sizer_tile_targets(vo_ctx *ctx, const vo_volume *in, const vo_volume *result, double radius, float *targets,
                          int *ntiles) {
  if (!ctx || !in || !result || !targets || !ntiles) return VO_EINVAL;
  if (in->grid.nx != result->grid.nx || in->grid.ny != result->grid.ny) return VO_EINVAL;
  vol_wait(ctx, in);
  vol_wait(ctx, result);
  const int nx = in->grid.nx, ny = in->grid.ny;
  const int tx = (nx + kTile - 1) / kTile, ty = (ny + kTile - 1) / kTile;
  const DeviceTables *T = nullptr;
  int rc = get_tables(ctx, radius, std::max(nx, ny) + 2, &T);
  if (rc) return rc;
  const std::vector<int2> pairs = alive_pairs(T->host);
  int2 *dp = nullptr;
  float *dt = nullptr;
  rc = dalloc(ctx, &dp, pairs.size());
  if (!rc) rc = dalloc(ctx, &dt, (size_t)tx * ty * NUSED);
  if (!rc) {
    cudaMemcpyAsync(dp, pairs.data(), sizeof(int2) * pairs.size(), cudaMemcpyHostToDevice, ctx->stream);
    k_tile_targets<<<tx * ty, 256, 0, ctx->stream>>>(nx, ny, in->offs, in->offs + 1, result->offs, dp,
                                                     (int)pairs.size(), dt);
    cudaMemcpyAsync(targets, dt, sizeof(float) * tx * ty * NUSED, cudaMemcpyDeviceToHost, ctx->stream);
  }
  dfree(ctx, dp);
  dfree(ctx, dt);
  if (rc) return rc;
  VO_CK(ctx, cudaStreamSynchronize(ctx->stream));
  *ntiles = tx * ty;
  return VO_OK;
}

int vo_sizer_forward(vo_ctx *ctx, const vo_sizer *s, const float *feats, int n, float *pred) {
  if (!ctx || !s || !feats || !pred || n < 0) return VO_EINVAL;
  if (n == 0) return VO_OK;
  Work w;
  int rc = work_alloc(ctx, n, false, w);
  if (!rc) {
    cudaMemcpyAsync(w.X, feats, sizeof(float) * n * NF, cudaMemcpyHostToDevice, ctx->stream);
    forward_launch(ctx, w.X, n, s->wb, w.out);
    std::vector<float> o((size_t)n * NO);
    cudaMemcpyAsync(o.data(), w.out, sizeof(float) * n * NO, cudaMemcpyDeviceToHost, ctx->stream);
    cudaError_t e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) rc = cuda_error(ctx, e, "sizer forward");
    for (int i = 0; i < n && !rc; ++i)
      for (int k = 0; k < NUSED; ++k) pred[(size_t)i * NUSED + k] = o[(size_t)i * NO + k];
  }
  work_free(ctx, w);
  return rc;
}

int vo_sizer_gradients(vo_ctx *ctx, vo_sizer *s, const float *feats, const float *targets, int n, float *grads,
                       float *loss) {
  if (!ctx || !s || !feats || !targets || !grads || n <= 0) return VO_EINVAL;
  Work w;
  int rc = work_alloc(ctx, n, true, w);
  if (!rc) {
    cudaMemcpyAsync(w.X, feats, sizeof(float) * n * NF, cudaMemcpyHostToDevice, ctx->stream);
    cudaMemcpyAsync(w.T, targets, sizeof(float) * n * NUSED, cudaMemcpyHostToDevice, ctx->stream);
    k_transpose<<<(n + 127) / 128, 128, 0, ctx->stream>>>(w.X, n, w.ld, w.XT);
    grad_pass(ctx, s, n, w, false, 0.f);
    cudaMemcpyAsync(grads, s->grad, sizeof(float) * NPARAM, cudaMemcpyDeviceToHost, ctx->stream);
    float l = 0;
    cudaMemcpyAsync(&l, w.loss, sizeof(float), cudaMemcpyDeviceToHost, ctx->stream);
    cudaError_t e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) rc = cuda_error(ctx, e, "sizer gradients");
    if (loss) *loss = l;
  }
  work_free(ctx, w);
  return rc;
}

int vo_sizer_train(vo_ctx *ctx, vo_sizer *s, const float *feats, const float *targets, int n, int steps, float lr,
                   float *final_loss) {
  if (!ctx || !s || !feats || !targets || n <= 0 || steps < 0) return VO_EINVAL;
  Work w;
  int rc = work_alloc(ctx, n, true, w);
  float l = 0;
  if (!rc) {
    cudaMemcpyAsync(w.X, feats, sizeof(float) * n * NF, cudaMemcpyHostToDevice, ctx->stream);
    cudaMemcpyAsync(w.T, targets, sizeof(float) * n * NUSED, cudaMemcpyHostToDevice, ctx->stream);
    k_transpose<<<(n + 127) / 128, 128, 0, ctx->stream>>>(w.X, n, w.ld, w.XT);
    for (int it = 0; it < steps; ++it) grad_pass(ctx, s, n, w, true, lr);
    // loss of the final parameters
    grad_pass(ctx, s, n, w, false, 0.f);
    cudaMemcpyAsync(&l, w.loss, sizeof(float), cudaMemcpyDeviceToHost, ctx->stream);
    cudaError_t e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) rc = cuda_error(ctx, e, "sizer train");
  }
  work_free(ctx, w);
  if (final_loss) *final_loss = l;
  return rc;
}

int vo_set_sizer(vo_ctx *ctx, vo_sizer *s) {
  if (!ctx) return VO_EINVAL;
  ctx->sizer = s;
  return VO_OK;
}

}  // extern "C"
