// Deterministic block and grid reductions used by the solver kernels: each
// block adds its threads' values in integers, writes one partial per block,
// and the last block to arrive (atomic ticket) sums the partials in a fixed
// order.  Same grid, same inputs -> bitwise the same result.
#pragma once

#include <cstdint>

namespace elx {

constexpr int kThreads = 256;

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
// Exponent of a sum with an infinity or NaN: m then counts the +infinities
// (from bit 0), -infinities (bit 20) and NaNs (bit 40) among its terms.
constexpr int32_t kFixBad = 1 << 20;

__device__ __forceinline__ int64_t fix_class(bool nan, bool neg) {
  return nan ? 1ll << 40 : neg ? 1ll << 20 : 1ll;
}

// m of a term in a sum with exponent e, k bits lower.
__device__ __forceinline__ int64_t fix_align(FixSum f, int e, int k) {
  if (e >= kFixBad) return f.e >= kFixBad ? f.m : 0;
  return f.m >> min(e - f.e + k, 63);
}

__device__ __forceinline__ FixSum fix_of(double v) {
  const int64_t b = __double_as_longlong(v);
  const int ex = (int)((uint64_t)b >> 52) & 0x7ff;
  int64_t m = b & 0xfffffffffffffll;
  FixSum f;
  if (ex == 0x7ff) {
    f.m = fix_class(m != 0, b < 0);
    f.e = kFixBad;
    return f;
  }
  if (ex) m |= 0x10000000000000ll;
  f.m = (b < 0 ? -m : m) << 5;
  f.e = m ? max(ex, 1) - 1080 : -4096;
  return f;
}

__device__ __forceinline__ FixSum fix_of(float v) {
  const uint32_t b = __float_as_uint(v);
  const int ex = (int)(b >> 23) & 0xff;
  int64_t m = b & 0x7fffffu;
  FixSum f;
  if (ex == 0xff) {
    f.m = fix_class(m != 0, (int32_t)b < 0);
    f.e = kFixBad;
    return f;
  }
  if (ex) m |= 0x800000;
  m <<= 34;
  f.m = (int32_t)b < 0 ? -m : m;
  f.e = m ? max(ex, 1) - 184 : -4096;
  return f;
}

// The sum over the 32 lanes, in every lane.
__device__ __forceinline__ FixSum warp_sum(FixSum f) {
  const int e = __reduce_max_sync(0xffffffffu, f.e);
  const int64_t m = fix_align(f, e, 0);
  const uint32_t lo = __reduce_add_sync(0xffffffffu, (uint32_t)m & 0x7ffffffu);
  const uint32_t mid = __reduce_add_sync(0xffffffffu, (uint32_t)(m >> 27) & 0x7ffffffu);
  const int32_t hi = __reduce_add_sync(0xffffffffu, (int32_t)(m >> 54));
  const int64_t t = ((int64_t)hi << 54) + ((int64_t)mid << 27) + (int64_t)lo;
  // back to 58 bits (leading zeros of |t| to 6), so that no stage loses bits
  const int sh = 6 - __clzll(t < 0 ? -t : t);
  FixSum r;
  if (e >= kFixBad) {
    r.m = t;
    r.e = kFixBad;
    return r;
  }
  r.m = sh > 0 ? t >> sh : t << -sh;
  r.e = t ? e + sh : -4096;
  return r;
}

__device__ __forceinline__ double fix_value(FixSum f) {
  if (f.e >= kFixBad) {
    const bool pos = f.m & 0xfffff, neg = f.m >> 20 & 0xfffff;
    return __longlong_as_double(f.m >> 40 || (pos && neg) ? 0x7ff8000000000000ll
                                : neg ? (int64_t)0xfff0000000000000ull : 0x7ff0000000000000ll);
  }
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

// Block-wide sum of NV per-thread values (double or float; kThreads threads);
// result valid in thread 0.  In integers (FixSum): as FP64 shuffle trees the
// two stages were 45 FP64 warp instructions a block, 12 us of 95 in a product
// of 64 rows per block, and 1,200 clocks at the end of every fused dot.
template <int NV, class T>
__device__ __forceinline__ void block_sum_widen(const T (&v)[NV], double (&out)[NV]) {
  __shared__ FixSum sh[NV][kThreads / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int i = 0; i < NV; i++) {
    const FixSum s = warp_sum(fix_of(v[i]));
    if (lane == 0) sh[i][w] = s;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < NV; i++) out[i] = 0.0;
  if (w == 0) {
#pragma unroll
    for (int i = 0; i < NV; i++) {
      FixSum t;
      t.m = 0;
      t.e = -4096;
      if (lane < kThreads / 32) t = sh[i][lane];
      out[i] = fix_value(warp_sum(t));
    }
  }
}

template <int NV>
__device__ __forceinline__ void block_sum(double (&v)[NV]) {
  double out[NV];
  block_sum_widen<NV>(v, out);
#pragma unroll
  for (int i = 0; i < NV; i++) v[i] = out[i];
}

// Writes this block's NV partials and returns true in thread 0 of the last
// block to arrive, after which that thread may read every block's partials.
// The ticket counts to the grid's size and gather_partials sets it back; with
// MOD (at least the grid's size) a launch adds MOD to it whatever its grid (block
// 0 the difference beforehand), and the last to arrive completes a multiple:
// nobody sets it back, and launches that overlapped leave it as any others do.
template <int NV, unsigned int MOD = 0>
__device__ __forceinline__ bool publish_partials(const double (&v)[NV], double *partials,
                                                 unsigned int *counter) {
  __shared__ bool last;
  if (threadIdx.x == 0) {
#pragma unroll
    for (int i = 0; i < NV; i++) partials[(size_t)i * gridDim.x + blockIdx.x] = v[i];
    __threadfence();
    if (MOD && blockIdx.x == 0) atomicAdd(counter, MOD - gridDim.x);
    const unsigned int ticket = atomicAdd(counter, 1u);
    last = MOD ? ticket % (MOD ? MOD : 1u) == MOD - 1 : ticket == gridDim.x - 1;
  }
  __syncthreads();
  return last;
}

// In the last block: every thread sums a strided slice of the partials, then
// a fixed tree; thread 0 gets the totals and resets the counter (without MOD).
template <int NV, unsigned int MOD = 0>
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
  if (MOD == 0 && threadIdx.x == 0) *counter = 0u;
}


}  // namespace elx
