// The value range of a dilation's input and the scalars of its FP32 arithmetic
// that follow from it, for the kernels that form them on the way.
#pragma once
#include "vo_internal.cuh"

namespace vo {

constexpr double kFar = 1e30;  // magnitudes beyond this stand outside the range
constexpr int kBins = 1024;    // bins of the patch kernel's lower ends (a power of two: bin_of masks its indexes)

// Doubles as unsigned integers of the same order (zero: below every one).
__device__ __forceinline__ unsigned long long order_of(double v) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v);
  return b >> 63 ? ~b : b | 0x8000000000000000ull;
}
__device__ __forceinline__ double order_value(unsigned long long o) {
  return __longlong_as_double((long long)(o >> 63 ? o & 0x7fffffffffffffffull : ~o));
}

// The scalars of a dilation from the orders of the largest value and of the
// largest negated value (0: there is none) of magnitude up to kFar, and from
// whether there are others below (bit 0) and above (bit 1): infinite ones, for
// which no base and no bin width would do. Those keep their order towards every
// candidate of the others when they stand in FP32 at the nearest places where
// even their own candidates of any H lie beyond all of those: 2 R and more away.
// What is decided in FP64 uses their own values.
// Guard band: with U bounding the magnitude of every FP32 value (relative to
// the base), each candidate endpoint is within 1.5 ulp32(U) of its FP64 value
// (rounding of z, of H and of the sum) and a difference of two adds one more
// ulp32(U): at most 4 ulp32(U) = 2^-21 U. E = 2^-20 U leaves a factor of two;
// the rounding of the FP64 endpoints themselves is below 2^-50 times the
// largest magnitude.
static __device__ void set_par(unsigned long long a, unsigned long long b, unsigned far, float R, FastPar *par) {
  const double zmax = a ? order_value(a) : 0.0, zmin = b ? -order_value(b) : 0.0;
  FastPar p;
  // above the rounding of what follows, and of two values less the base
  const double q = 1.8e-15 * fmax(fabs(zmax), fabs(zmin));
  p.q = (float)q;
  p.base = floor(far & 1 ? zmin - 2.0 * (R + 3.0 + q) : zmin - R - 3.0);
  p.lo = far & 1 ? R + 2.f : 0.f;
  p.hi = far & 2 ? (float)(zmax - p.base + 2.0 * (R + 3.0 + q)) : INFINITY;
  const float U = far & 2 ? p.hi + R + 3.f : (float)(zmax - p.base + R + 3.0);
  p.E = U * 9.5367431640625e-07f + (float)(fmax(fabs(zmax), fabs(zmin)) * 8.8817841970012523e-16);
  // bin width: the power of two at or above a quarter of the radius, wide
  // enough for the range and far above the guard band
  const float w0 = fmaxf(fmaxf(U / (float)(kBins - 8), 0.25f * R), fmaxf(64.f * p.E, 1e-20f));
  int e;
  const float m = frexpf(fminf(w0, 1e30f), &e);
  if (m == 0.5f) --e;
  const float w = ldexpf(1.f, e);
  p.inv_w = ldexpf(1.f, -e);
  p.thr = w + 4.f * p.E;
  p.nbins = (int)fminf((float)kBins, U * p.inv_w + 3.f);
  *par = p;
}

// The range of the values that a block's threads take: ordinary numbers by their keys, NaN left out, those
// beyond kFar noted as such. mm, zeroed before: orders of the largest value and of the largest negated value,
// the blocks that are done, whether values lie beyond. The last block to finish sets par.
struct ValueRange {
  Key top = kKeyMin, bottom = kKeyMax;
  unsigned far = 0;
  __device__ __forceinline__ void take(Key bits) {
    const Key size = bits & 0x7fffffffffffffffll, key = bits ^ (bits < 0 ? 0x7fffffffffffffffll : 0);
    if (size > 0x46293e5939a08ceall) {  // the bits of kFar
      if (size <= 0x7ff0000000000000ll) far |= bits < 0 ? 1u : 2u;
      return;
    }
    top = kmax(top, key);
    bottom = kmin(bottom, key);
  }
  __device__ __forceinline__ void finish(unsigned long long *mm, float R, FastPar *par) {
    for (int o = 16; o > 0; o >>= 1) {
      top = kmax(top, __shfl_xor_sync(0xffffffffu, top, o));
      bottom = kmin(bottom, __shfl_xor_sync(0xffffffffu, bottom, o));
    }
    far = __reduce_or_sync(0xffffffffu, far);
    if ((threadIdx.x & 31) == 0) {
      if (top >= bottom) {
        atomicMax(&mm[0], order_of(value_of(top)));
        atomicMax(&mm[1], order_of(-value_of(bottom)));
      }
      if (far) atomicOr(&mm[3], (unsigned long long)far);
    }
    __syncthreads();
    if (threadIdx.x) return;
    __threadfence();
    if (atomicAdd(&mm[2], 1ull) + 1 != gridDim.x) return;
    __threadfence();
    set_par(atomicMax(&mm[0], 0ull), atomicMax(&mm[1], 0ull), (unsigned)atomicOr(&mm[3], 0ull), R, par);
  }
};

}  // namespace vo
