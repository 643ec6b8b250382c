// Deterministic block and grid reductions used by the solver kernels: each
// block reduces its threads in a fixed tree, writes one partial per block,
// and the last block to arrive (atomic ticket) sums the partials in a fixed
// order.  Same grid, same inputs -> bitwise the same result.
#pragma once

#include <cstdint>

namespace elx {

constexpr int kThreads = 256;

template <class T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
  return v;
}

// A sum in integer form: value = m 2^e with |m| < 2^58.  GB300 runs an FP64
// instruction of a warp in 64 clocks per SM quarter, however few lanes are
// active, and each of the five dependent adds of a shuffle tree waits for the
// one before (109 clocks a level with its shuffles).  The sum of a warp's 32
// values in integers -- aligned to the largest exponent, added as three limbs
// by redux.sync -- leaves the FP64 pipe to the products, and is off by at
// most 32 units of 2^-58 of the largest value: one rounding of an FP64 add.
struct FixSum {
  int64_t m;
  int32_t e;
};
constexpr int32_t kFixBad = 1 << 20;  // exponent of a sum with an infinity or NaN

__device__ __forceinline__ FixSum fix_of(double v) {
  const int64_t b = __double_as_longlong(v);
  const int ex = (int)((uint64_t)b >> 52) & 0x7ff;
  int64_t m = b & 0xfffffffffffffll;
  if (ex) m |= 0x10000000000000ll;
  FixSum f;
  f.m = (b < 0 ? -m : m) << 5;
  f.e = ex == 0x7ff ? kFixBad : m ? max(ex, 1) - 1080 : -4096;
  return f;
}

__device__ __forceinline__ FixSum fix_of(float v) {
  const uint32_t b = __float_as_uint(v);
  const int ex = (int)(b >> 23) & 0xff;
  int64_t m = b & 0x7fffffu;
  if (ex) m |= 0x800000;
  m <<= 34;
  FixSum f;
  f.m = (int32_t)b < 0 ? -m : m;
  f.e = ex == 0xff ? kFixBad : m ? max(ex, 1) - 184 : -4096;
  return f;
}

// The sum over the 32 lanes, in every lane.
__device__ __forceinline__ FixSum warp_sum(FixSum f) {
  const int e = __reduce_max_sync(0xffffffffu, f.e);
  const int64_t m = f.m >> min(e - f.e, 63);
  const uint32_t lo = __reduce_add_sync(0xffffffffu, (uint32_t)m & 0x7ffffffu);
  const uint32_t mid = __reduce_add_sync(0xffffffffu, (uint32_t)(m >> 27) & 0x7ffffffu);
  const int32_t hi = __reduce_add_sync(0xffffffffu, (int32_t)(m >> 54));
  const int64_t t = ((int64_t)hi << 54) + ((int64_t)mid << 27) + (int64_t)lo;
  // back to 58 bits (leading zeros of |t| to 6), so that no stage loses bits
  const int sh = 6 - __clzll(t < 0 ? -t : t);
  FixSum r;
  r.m = sh > 0 ? t >> sh : t << -sh;
  r.e = t ? e + sh : -4096;
  return r;
}

__device__ __forceinline__ double fix_value(FixSum f) {
  if (f.e >= kFixBad) return __longlong_as_double(0x7ff8000000000000ll);
  if (f.m == 0) return 0.0;
  // 58 bits rounded to 53; the carry of a rounding up runs into the exponent
  const uint64_t a = (uint64_t)(f.m < 0 ? -f.m : f.m) + 16 >> 5;
  const int ex = f.e + 1080;
  if (ex >= 1 && ex <= 2045 && a >> 52) {
    const uint64_t b = ((uint64_t)ex << 52) + (a - 0x10000000000000ull);
    return __longlong_as_double((int64_t)(f.m < 0 ? b | 1ull << 63 : b));
  }
  // near the ends of the range: 2^e in two normal factors
  const int e1 = max(f.e, -1000), e2 = max(f.e - e1, -200);
  double v = (double)f.m * __longlong_as_double((int64_t)(min(e1, 1023) + 1023) << 52);
  if (e2) v *= __longlong_as_double((int64_t)(e2 + 1023) << 52);
  return v;
}

// Block-wide sum of NV values (fixed order); result valid in thread 0.
template <int NV>
__device__ __forceinline__ void block_sum(double (&v)[NV]) {
  __shared__ double sh[NV][kThreads / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int i = 0; i < NV; i++) {
    v[i] = warp_sum(v[i]);
    if (lane == 0) sh[i][w] = v[i];
  }
  __syncthreads();
  if (w == 0) {
#pragma unroll
    for (int i = 0; i < NV; i++) {
      double t = lane < kThreads / 32 ? sh[i][lane] : 0.0;
      v[i] = warp_sum(t);
    }
  }
}

// Block-wide sum of NV per-thread values of type T (float in the FP32
// kernels): the warp stage adds in T, the per-warp sums are widened to double
// and added in a fixed order.  Keeps the FP32 kernels off the (narrow) FP64
// pipe except for a handful of additions per block.  Result in thread 0.
template <int NV, class T>
__device__ __forceinline__ void block_sum_widen(const T (&v)[NV], double (&out)[NV]) {
  __shared__ double sh[NV][kThreads / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int i = 0; i < NV; i++) {
    const T s = warp_sum(v[i]);
    if (lane == 0) sh[i][w] = (double)s;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < NV; i++) out[i] = 0.0;
  if (w == 0) {
#pragma unroll
    for (int i = 0; i < NV; i++) {
      double t = lane < kThreads / 32 ? sh[i][lane] : 0.0;
      out[i] = warp_sum(t);
    }
  }
}

// Writes this block's NV partials and returns true in thread 0 of the last
// block to arrive, after which that thread may read every block's partials.
template <int NV>
__device__ __forceinline__ bool publish_partials(const double (&v)[NV], double *partials,
                                                 unsigned int *counter) {
  __shared__ bool last;
  if (threadIdx.x == 0) {
#pragma unroll
    for (int i = 0; i < NV; i++) partials[(size_t)i * gridDim.x + blockIdx.x] = v[i];
    __threadfence();
    const unsigned int ticket = atomicAdd(counter, 1u);
    last = ticket == gridDim.x - 1;
  }
  __syncthreads();
  return last;
}

// In the last block: every thread sums a strided slice of the partials, then
// a fixed tree; thread 0 gets the totals and resets the counter.
template <int NV>
__device__ __forceinline__ void gather_partials(double (&tot)[NV], const double *partials,
                                                unsigned int *counter) {
  __threadfence();
#pragma unroll
  for (int i = 0; i < NV; i++) {
    double s = 0.0;
    // L2 loads (__ldcg: the partials were written by other blocks, ordered by
    // the fence + ticket); several in flight per thread
#pragma unroll 4
    for (int b = threadIdx.x; b < (int)gridDim.x; b += kThreads)
      s += __ldcg(partials + (size_t)i * gridDim.x + b);
    tot[i] = s;
  }
  block_sum<NV>(tot);
  if (threadIdx.x == 0) *counter = 0u;
}


}  // namespace elx
