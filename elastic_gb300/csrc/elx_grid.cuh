// Grid-wide sums and barriers inside one cooperative launch (persist.cu).
//
// A sum over the blocks is one integer atomic per digit: every block adds its
// partial, cut into five 32-bit digits of a 160-bit window, to five words in
// L2, and polls them until all blocks have added (each word counts its
// additions in its upper bits).  Integer adds commute, so the total is the same
// whatever the order, and every block reads the same total one L2 round trip
// after the slowest block arrives: 1,500 clocks on 152 blocks, where slots
// written by every block and polled by all take 2,800 to 4,200 and a last
// block that adds the partials a fence, an atomic and two more round trips.
// The words are never reset: a total is their difference from the last one.
//
// The window reaches 120 bits below the sum's reference (the last residual's
// norm), and takes partials up to 30 above (two bits are left for the carries of
// the sum and its sign).  A partial above that, an infinity or a NaN marks the
// sum, and all blocks repeat it through slots, each with its own exponent.
#pragma once

#include <cstdint>

#include "elx_krylov.h"
#include "elx_ptx.cuh"
#include "elx_reduce.cuh"

namespace elx {

constexpr int kGridMaxBlocks = 160;
constexpr uint64_t kGridWaitNs = 1000000000ull;  // bound of every grid wait
constexpr int kDigits = 5;
constexpr int kClusterBlocks = 16;  // the most that a cluster has

// Shared by the blocks of a launch; zeroed before each launch.
struct alignas(128) GridWords {
  unsigned long long digit[32];  // kDigits for each sum
};
struct alignas(16) GridSlot {
  int64_t m;
  uint64_t tag;  // epoch << 24 | exponent + 4096
};
struct GridSync {
  GridWords sum[2];  // (p, q) and (r, z)
  GridWords arrive;  // digit[0]: arrivals at the barrier
  GridSlot slot[kGridCols][kGridMaxBlocks];
};

namespace grid {

__device__ __forceinline__ unsigned long long load_relaxed(const unsigned long long *p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void red_add(unsigned long long *p, unsigned long long v) {
  asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

__device__ __forceinline__ void store_slot(GridSlot *s, int64_t m, uint64_t tag) {
  asm volatile(
      "{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\t"
      "st.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(s),
      "l"(m), "l"(tag)
      : "memory");
}

__device__ __forceinline__ GridSlot load_slot(const GridSlot *s) {
  GridSlot r;
  asm volatile(
      "{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\t"
      "mov.b128 {%0, %1}, t;\n\t}"
      : "=l"(r.m), "=l"(r.tag)
      : "l"(s)
      : "memory");
  return r;
}

__device__ __forceinline__ void fence() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

__device__ __forceinline__ FixSum fix_shfl(FixSum f, int lane) {
  FixSum r;
  r.m = __shfl_sync(0xffffffffu, f.m, lane);
  r.e = __shfl_sync(0xffffffffu, f.e, lane);
  return r;
}

// Counts polls and bounds them by the GPU's clock.
struct Bound {
  uint64_t t0 = 0;
  uint32_t it = 0;
  __device__ __forceinline__ bool over() {
    if (++it & 1023u) return false;
    const uint64_t now = ptx::global_ns();
    if (!t0) t0 = now;
    return now - t0 > kGridWaitNs;
  }
};

// The blocks that work together: all of a launch, or some.
struct Team {
  int me, n;
  // With `stall` (ELX_GRID_STALL_TEST) a team's last block does not take part,
  // and the others' waits run out.
  __device__ __forceinline__ bool missing(int stall) const {
    return stall && n > 1 && me == n - 1;
  }
};

// The blocks' sums through a slot of each block (value, exponent and epoch in
// one 16-byte store); one warp, lane c holds sum c.
template <int NC>
__device__ __forceinline__ bool slot_sum(Team t, GridSlot (*slots)[kGridMaxBlocks], FixSum &f,
                                         uint64_t epoch) {
  constexpr int K = kGridMaxBlocks / 32;
  const int lane = threadIdx.x & 31;
  if (lane < NC)
    store_slot(slots[lane] + t.me, f.m,
               epoch << 24 | (uint64_t)(uint32_t)(f.e + 4096));
  bool ok = true;
  Bound bound;
  for (int c = 0; c < NC; c++) {
    FixSum v[K];
#pragma unroll
    for (int k = 0; k < K; k++) {
      v[k].m = 0;
      v[k].e = -4096;
      const int b = lane + 32 * k;
      while (b < t.n && ok) {
        const GridSlot g = load_slot(slots[c] + b);
        if (g.tag >> 24 == epoch) {
          v[k].m = g.m;
          v[k].e = (int32_t)(g.tag & 0xffffffu) - 4096;
          break;
        }
        ok = !bound.over();
      }
    }
    int e = v[0].e;
#pragma unroll
    for (int k = 1; k < K; k++) e = max(e, v[k].e);
    FixSum q;
    q.m = 0;
#pragma unroll
    for (int k = 0; k < K; k++) q.m += fix_align(v[k], e, 3);
    q.e = e >= kFixBad ? e : e + 3;
    q = warp_sum(q);
    if (lane == c) f = q;
  }
  return __all_sync(0xffffffffu, ok);
}

// Exponent of a window's lowest bit for sums near |ref|.
__device__ __forceinline__ int window_of(double ref) {
  const int ex = (int)((uint64_t)__double_as_longlong(ref) >> 52) & 0x7ff;
  return ex - 1023 - 120;
}

constexpr unsigned long long kOne = 1ull << 48, kBias = 1ull << 33, kMark = 1ull << 56;

// Adds this block's f to the digits (one warp; lane c holds sum c and `lo`,
// the exponent of its lowest digit).
template <int NC>
__device__ __forceinline__ void digit_add(GridWords *words, FixSum f, int lo) {
  static_assert(NC * kDigits <= 32, "one lane per digit");
  const int lane = threadIdx.x & 31;
  const int col = min(lane / kDigits, NC - 1), k0 = lane - col * kDigits;
  const FixSum g = fix_shfl(f, col);
  const int glo = __shfl_sync(0xffffffffu, lo, col);
  if (lane >= NC * kDigits) return;
  uint64_t a = g.m < 0 ? -g.m : g.m;
  int s = g.e - glo;  // place of a's lowest bit in the window
  unsigned long long add = kOne + kBias;
  if (g.m != 0) {
    if (s > 32 * kDigits - 68) {  // 58 bits and 8 of 152 addends
      add += kMark;
    } else {
      if (s < 0) {
        a >>= min(-s, 63);
        s = 0;
      }
      const int off = 32 * k0 - s;
      const uint64_t d =
          (off >= 64 || off <= -32 ? 0 : off >= 0 ? a >> off : a << -off) & 0xffffffffull;
      add += g.m < 0 ? -d : d;
    }
  }
  red_add(words->digit + lane, add);
}

// Waits for the n blocks' additions and replaces f by the sums (the same warp).
// `seen`: this lane's word after the last sum.  False in every lane when the
// bound ran out.
template <int NC>
__device__ __forceinline__ bool digit_read(Team t, GridSlot (*slots)[kGridMaxBlocks],
                                           GridWords *words, FixSum &f, int lo,
                                           unsigned long long &seen, uint64_t epoch) {
  const int lane = threadIdx.x & 31, n = t.n;
  unsigned long long w = 0;
  bool ok = true;
  if (lane < NC * kDigits) {
    Bound bound;
    for (;;) {
      w = load_relaxed(words->digit + lane);
      if (((w - seen) >> 48 & 0xff) == (unsigned)n) break;
      if (bound.over()) {
        ok = false;
        break;
      }
    }
  }
  if (!__all_sync(0xffffffffu, ok)) return false;
  const unsigned long long diff = w - seen;
  seen = w;
  if (__any_sync(0xffffffffu, diff >> 56 != 0)) return slot_sum<NC>(t, slots, f, epoch);
  const int64_t d = (int64_t)(diff & (kOne - 1)) - (int64_t)n * (int64_t)kBias;
  // lane c: its sum's digits, carried upwards (32 bits each, the top one signed)
  int64_t c[kDigits];
  const int base = min(lane, NC - 1) * kDigits;
#pragma unroll
  for (int k = 0; k < kDigits; k++) c[k] = __shfl_sync(0xffffffffu, d, base + k);
#pragma unroll
  for (int k = 1; k < kDigits; k++) c[k] += c[k - 1] >> 32;
  const bool neg = c[kDigits - 1] < 0;
  uint32_t u[kDigits];
  uint32_t carry = neg ? 1 : 0;  // |total|: two's complement
#pragma unroll
  for (int k = 0; k < kDigits; k++) {
    const uint32_t x = neg ? ~(uint32_t)c[k] : (uint32_t)c[k];
    u[k] = x + carry;
    carry = carry && u[k] == 0;
  }
  // the 64 highest bits from the top digit that is not zero
  uint64_t hi = 0;
  int at = 0;
#pragma unroll
  for (int k = kDigits - 1; k >= 0; k--)
    if (hi == 0 && u[k]) {
      const uint32_t below = k > 0 ? u[k - 1] : 0, below2 = k > 1 ? u[k - 2] : 0;
      const int z = __clz(u[k]);
      hi = ((uint64_t)u[k] << 32 | below) << z | (z ? below2 >> (32 - z) : 0);
      at = 32 * (k - 1) - z;
    }
  f.m = (int64_t)(hi >> 6);  // 58 bits
  if (neg) f.m = -f.m;
  f.e = hi ? lo + at + 6 : -4096;
  return true;
}

template <int T, int NC>
struct Scratch {
  FixSum part[NC][T / 32];
  int32_t ok;
};

// The sums of v[c] over the team's blocks, each near |ref[c]| (shared memory;
// nullptr: of any size).  `then(total)` runs in lane c of warp 0 with sum c
// (FP64 arithmetic on the totals costs the pipe once instead of once per
// warp) and leaves what the block needs in shared memory; `meanwhile()` runs
// in the other warps while warp 0 waits: work that does not need the totals.
// T: threads of the block (a multiple of 32, at most 1024).  False in every
// thread when a wait ran out (the caller returns).
template <int T, int NC, class V, class F, class H>
__device__ __forceinline__ bool sum(Team team, const V (&v)[NC], GridSync *gs, int which,
                                    const double *ref, unsigned long long &seen, uint64_t epoch, Scratch<T, NC> &sh,
                                    F then, H meanwhile) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int c = 0; c < NC; c++) {
    const FixSum s = warp_sum(fix_of(v[c]));
    if (lane == 0) sh.part[c][w] = s;
  }
  __syncthreads();
  if (w == 0) {
    FixSum mine;
    mine.m = 0;
    mine.e = -4096;
#pragma unroll
    for (int c = 0; c < NC; c++) {
      FixSum t;
      t.m = 0;
      t.e = -4096;
      if (lane < T / 32) t = sh.part[c][lane];
      t = warp_sum(t);
      if (lane == c) mine = t;
    }
    bool ok;
    if (ref) {
      const int lo = window_of(ref[lane < NC ? lane : 0]);
      digit_add<NC>(&gs->sum[which], mine, lo);
      ok = digit_read<NC>(team, gs->slot, &gs->sum[which], mine, lo, seen, epoch);
    } else {
      ok = slot_sum<NC>(team, gs->slot, mine, epoch);
    }
    if (lane < NC) then(fix_value(mine));
    if (lane == 0) sh.ok = ok;
  } else {
    meanwhile();
  }
  __syncthreads();
  return sh.ok != 0;
}

// The same for the blocks of one cluster: every block writes its partials into
// all blocks' shared memory, and the hardware's cluster barrier stands for the
// polls.  `slots` alternate with `which`; between two uses of one lies another
// barrier, which a block reaches after reading the first.
template <int NC>
struct Cluster {
  int me, n;
  FixSum (*slots)[NC][kClusterBlocks];  // [2], shared memory
};

template <int T, int NC, class V, class F, class H>
__device__ __forceinline__ bool sum(Cluster<NC> team, const V (&v)[NC], GridSync *, int which,
                                    const double *, unsigned long long &, uint64_t,
                                    Scratch<T, NC> &sh, F then, H meanwhile) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int c = 0; c < NC; c++) {
    const FixSum s = warp_sum(fix_of(v[c]));
    if (lane == 0) sh.part[c][w] = s;
  }
  __syncthreads();
  if (w == 0) {
    FixSum mine;
    mine.m = 0;
    mine.e = -4096;
#pragma unroll
    for (int c = 0; c < NC; c++) {
      FixSum t;
      t.m = 0;
      t.e = -4096;
      if (lane < T / 32) t = sh.part[c][lane];
      t = warp_sum(t);  // in every lane: one for each block
      if (lane < team.n) ptx::store_cluster(&team.slots[which][c][team.me], lane, t.m, t.e);
    }
    __syncwarp();
    ptx::cluster_arrive();
    ptx::cluster_wait();
#pragma unroll
    for (int c = 0; c < NC; c++) {
      FixSum t;
      t.m = 0;
      t.e = -4096;
      if (lane < team.n) t = team.slots[which][c][lane];
      t = warp_sum(t);
      if (lane == c) mine = t;
    }
    if (lane < NC) then(fix_value(mine));
  } else {
    ptx::cluster_arrive();
    meanwhile();
    __syncwarp();
    ptx::cluster_wait();
  }
  __syncthreads();
  return true;
}

// Makes the blocks' global stores visible to one another.  The fences on both
// sides order the data (and drop stale L1 lines).  `count`: barriers passed
// in this launch, this one included.
template <int T, int NC>
__device__ __forceinline__ bool barrier(Team team, GridSync *gs, uint32_t count,
                                        Scratch<T, NC> &sh) {
  __syncthreads();
  if (threadIdx.x == 0) {
    fence();
    unsigned long long *p = gs->arrive.digit;
    red_add(p, 1);
    const unsigned long long want = (unsigned long long)count * team.n;
    bool ok = true;
    Bound bound;
    while (ok && load_relaxed(p) < want) ok = !bound.over();
    fence();
    sh.ok = ok;
  }
  __syncthreads();
  return sh.ok != 0;
}

template <int T, int NC>
__device__ __forceinline__ bool barrier(Cluster<NC>, GridSync *, uint32_t, Scratch<T, NC> &) {
  __syncwarp();
  ptx::cluster_arrive();
  ptx::cluster_wait();
  return true;
}

}  // namespace grid
}  // namespace elx
