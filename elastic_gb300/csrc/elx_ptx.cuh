// Thin inline-PTX wrappers for the asynchronous copy machinery of sm_100+:
// mbarriers, 1-D bulk copies (cp.async.bulk, the TMA engine's non-tensor
// form), per-thread cp.async gathers and streaming loads.  Every wait is bounded: a wait that
// gives up records an error code in a device word instead of spinning
// forever, and the host turns it into ELX_ERR_TIMEOUT.
#pragma once

#include <cstdint>

namespace elx {
namespace ptx {

__device__ __forceinline__ uint32_t smem_addr(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count)
               : "memory");
}

// Makes barrier initialisation visible to the async proxy (the bulk-copy unit).
__device__ __forceinline__ void fence_barrier_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// Orders this thread's generic-proxy shared-memory accesses before later
// async-proxy (bulk copy) accesses of the same memory.
__device__ __forceinline__ void fence_proxy_async() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)),
               "r"(bytes)
               : "memory");
}

// 1-D bulk copy global -> shared, completing `bytes` on the barrier.
// dst and src 16-byte aligned, bytes a multiple of 16.
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes,
                                         uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
          "r"(smem_addr(dst)),
      "l"(src), "r"(bytes), "r"(smem_addr(bar))
      : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_addr(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// The GPU's nanosecond clock.
__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Waits for the barrier phase `parity` for at most limit_ns nanoseconds (each
// try_wait may itself suspend for a while, so the bound is on the clock, with
// an iteration cap behind it).  On timeout it stores `code` into *err and
// returns false.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t *bar, uint32_t parity, int32_t *err,
                                                  int32_t code,
                                                  uint64_t limit_ns = 1000000000ull) {
  const uint64_t t0 = global_ns();
  for (uint32_t it = 0; it < (1u << 24); it++) {
    if (mbar_try_wait(bar, parity)) return true;
    if (global_ns() - t0 > limit_ns) break;
    if (it > 64) __nanosleep(64);
  }
  atomicExch(err, code);
  return false;
}

// Per-thread asynchronous 4- or 8-byte copy global -> shared (a gather).
template <int BYTES>
__device__ __forceinline__ void cp_async(void *dst, const void *src) {
  static_assert(BYTES == 4 || BYTES == 8, "cp.async size");
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_addr(dst)), "l"(src),
               "n"(BYTES)
               : "memory");
}

__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;" ::: "memory");
}

template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

__device__ __forceinline__ void named_barrier(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// The hardware barrier over a cluster's threads (whole warps); memory written
// before the arrival is visible after the wait.
__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}

__device__ __forceinline__ void cluster_wait() {
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// 16 bytes to the place of `p` (this block's shared memory) in block `rank`.
__device__ __forceinline__ void store_cluster(void *p, int rank, int64_t a, int64_t b) {
  asm volatile(
      "{\n\t.reg .u32 t;\n\tmapa.shared::cluster.u32 t, %0, %1;\n\t"
      "st.shared::cluster.v2.b64 [t], {%2, %3};\n\t}" ::"r"(smem_addr(p)),
      "r"(rank), "l"(a), "l"(b)
      : "memory");
}

// Streaming loads of read-only data that is used once (matrix values and
// indices): not kept in L1, and issued in program order (volatile), so that a
// group of them is in flight before the first use.
__device__ __forceinline__ float4 ld_stream4(const float *p) {
  float4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "l"(p));
  return v;
}

__device__ __forceinline__ double2 ld_stream2(const double *p) {
  double2 v;
  asm volatile("ld.global.nc.L1::no_allocate.v2.f64 {%0, %1}, [%2];"
               : "=d"(v.x), "=d"(v.y)
               : "l"(p));
  return v;
}

__device__ __forceinline__ double ld_stream(const double *p) {
  double v;
  asm volatile("ld.global.nc.L1::no_allocate.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}

__device__ __forceinline__ float ld_stream(const float *p) {
  float v;
  asm volatile("ld.global.nc.L1::no_allocate.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}

__device__ __forceinline__ int16_t ld_stream(const int16_t *p) {
  int16_t v;
  asm volatile("ld.global.nc.L1::no_allocate.s16 %0, [%1];" : "=h"(v) : "l"(p));
  return v;
}

__device__ __forceinline__ int32_t ld_stream(const int32_t *p) {
  int32_t v;
  asm volatile("ld.global.nc.L1::no_allocate.s32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}

// Read-only loads issued in program order (volatile) but cached as usual:
// for data that lanes of a warp share (the same block read by the lane
// group of a row) and that should be in flight as a group.
__device__ __forceinline__ float ld_nc_ordered(const float *p) {
  float v;
  asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}

__device__ __forceinline__ double ld_nc_ordered(const double *p) {
  double v;
  asm volatile("ld.global.nc.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}

__device__ __forceinline__ int32_t ld_nc_ordered(const int32_t *p) {
  int32_t v;
  asm volatile("ld.global.nc.s32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}

}  // namespace ptx
}  // namespace elx
