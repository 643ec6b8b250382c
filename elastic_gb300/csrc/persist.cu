// Jacobi PCG in one cooperative launch (pcg, mef/src/Iters.f:252-524).
//
// An iteration of krylov.cu is three launches whose last blocks add the
// partial dots: on 152 SMs the launches, the reductions and their FP64
// divisions take 15 us however small the system (16.2 us an iteration at 2,176
// equations, 19.8 at 90,902).  Here one block per SM stays resident and owns a
// run of slices of the sliced matrix, cut so that every block has the same
// number of slot groups.  Its rows of x, r, M and p stay in shared memory for
// the whole launch (in L2 when they do not fit); p is also written to global
// memory, where the other blocks gather it.  An iteration is the same
// recurrence with three waits on the other blocks (elx_grid.cuh): the two
// dots and the new p.  Arithmetic that does not need a dot runs in the other
// warps while the first waits for it: x, the slices cut between warps, the
// stopping test.  Per iteration, launches -> here: 16.2 -> 7.0 us (2,176
// equations, QUAD4), 19.8 -> 10.3 (90,902, TRIA3), 33.1 -> 11.2 (26,460,
// HEXA8), 72.2 -> 60.3 (345,744, HEXA8), 142 -> 130 (811,200, HEXA8: the
// FP64 pipe's floor is 110).
//
// Inside a block every warp takes the same number of slot groups (the FP64
// pipe is charged per warp instruction; one group in flight measured faster
// than two, 130 against 134 us at 811,200 equations); a slice cut between
// warps is summed by its first warp and the heads of the following ones, in
// warp order, so results do not depend on timing.
#include <algorithm>

#include "elx_context.h"
#include "elx_grid.cuh"
#include "elx_sell.cuh"

namespace elx {
namespace {

constexpr int kPT = 512;  // threads of a block
constexpr int kPW = kPT / 32;

struct PersistArgs {
  int nb, n;
  const int32_t *sell_ptr, *sell_col;
  const double *sval;
  const int32_t *cta;  // (grid + 1): first slice of each block
  const double *m;
  double *x, *r, *p;
  PcgScalars *sc;
  GridSync *gs;
  int32_t *err;
  int rows;  // rows of the largest block
  int slices;  // slices of the largest block
};

// Shared memory: the block's rows of q (and of x, r, M, p), the warps' heads,
// the reduction scratch and the slice tables.
template <int B, bool SMEM>
size_t persist_smem(int rows, int slices) {
  return sizeof(double) * ((size_t)rows * (SMEM ? 5 : 1) + (size_t)kPW * kSliceRows * B) +
         sizeof(int32_t) * ((size_t)(slices + 1) + (kPW + 1) + kPW);
}

template <int B, bool SMEM>
__global__ void __launch_bounds__(kPT, 1)
pcg_persist_kernel(PersistArgs a, int steps) {
  constexpr int BB = B * B, R = kSliceRows, RB = R * B;
  extern __shared__ __align__(16) unsigned char smem[];
  double *sq = reinterpret_cast<double *>(smem);
  double *sx = sq + a.rows, *sr = sx + (SMEM ? a.rows : 0), *sm = sr + (SMEM ? a.rows : 0);
  double *sp = sm + (SMEM ? a.rows : 0), *shead = sp + (SMEM ? a.rows : 0);
  __shared__ grid::Scratch<kPT> sred;
  __shared__ int32_t sstop, sncut, scut[kPW];
  __shared__ double sd;
  int32_t *sptr = reinterpret_cast<int32_t *>(shead + kPW * RB);  // group pointers of the slices
  int32_t *sga = sptr + a.slices + 1, *swsl = sga + kPW + 1;  // warps' first groups and slices
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  PcgScalars *sc = a.sc;
  if (sc->done) return;
  const int s0 = a.cta[blockIdx.x], s1 = a.cta[blockIdx.x + 1], ns = s1 - s0;
  const int row0 = s0 * RB, nrows = min(a.n, s1 * RB) - row0;
  double d = sc->d, pq = 0.0;  // thread 0 keeps them up to date
  double alpha = 0.0, beta = 0.0;
  const double conv = sc->conv;
  const int maxit = sc->maxit;
  int iters = sc->iters;
  uint64_t epoch = 0;
  if (tid == 0) {
    sstop = 0;
    sd = d;
  }
  for (int i = tid; i <= ns; i += kPT) sptr[i] = a.sell_ptr[s0 + i];
  if (SMEM)
    for (int i = tid; i < nrows; i += kPT) {
      sx[i] = a.x[row0 + i];
      sr[i] = a.r[row0 + i];
      sm[i] = a.m[row0 + i];
      sp[i] = a.p[row0 + i];
    }
  __syncthreads();
  if (tid <= kPW) {
    // two groups per warp at least, warps in fours (one per SM quarter)
    const int total = sptr[ns] - sptr[0], wn = min(kPW, max(4, total / 2 & ~3));
    const int g = sptr[0] + (int)((int64_t)total * min(tid, wn) / wn);
    sga[tid] = g;
    if (tid < kPW) {
      int lo = 0, hi = ns - 1;  // the slice of group g
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (sptr[mid] <= g) lo = mid; else hi = mid - 1;
      }
      swsl[tid] = lo;
    }
  }
  __syncthreads();
  // the slices cut between warps, with the heads that belong to each
  if (tid == 0) {
    int n = 0;
    for (int k = 1; k < kPW; k++) {
      const int sl = swsl[k];
      if (sga[k] == sptr[sl] || sga[k + 1] == sga[k]) continue;
      if (n && (scut[n - 1] & 0xffff) == sl)
        scut[n - 1] += 1 << 24;  // one more head
      else
        scut[n++] = sl | k << 16 | 1 << 24;
    }
    sncut = n;
  }
  __syncthreads();
  unsigned long long seen_pq = 0, seen_rz = 0;  // warp 0: this lane's digits so far
  for (int step = 0; step < steps; step++) {
    epoch += 2;  // of the slots, one for each sum
    // q = K p over the warp's groups, and their share of (p, q)
    double v = 0.0;
    {
      int g = sga[w], sl = swsl[w];
      const int gend = sga[w + 1];
      while (g < gend) {
        const int ge = min(sptr[sl + 1], gend);
        double *dst = g == sptr[sl] ? sq + sl * RB : shead + w * RB;
        double acc[B];
#pragma unroll
        for (int b = 0; b < B; b++) acc[b] = 0.0;
        for (; g < ge; g++) {
          double bv[BB], xv[B];
          const int J = sell_ld<true>(a.sell_col + (size_t)g * R + lane);
          sell_load<double, B, true>(a.sval + (size_t)g * BB * R, lane, bv);
#pragma unroll
          for (int b = 0; b < B; b++) xv[b] = a.p[J * B + b];
#pragma unroll
          for (int c = 0; c < B; c++)
#pragma unroll
            for (int b = 0; b < B; b++) acc[c] += bv[c * B + b] * xv[b];
        }
        const int i = sl * RB + lane * B;
        if (i < nrows)
#pragma unroll
          for (int b = 0; b < B; b++) {
            dst[lane * B + b] = acc[b];
            v += (SMEM ? sp[i + b] : a.p[row0 + i + b]) * acc[b];
          }
        sl++;
      }
    }
    // alpha = d / (p, q); meanwhile the slices cut between warps are put together
    if (!grid::sum<kPT>(v, a.gs, 0, sd, seen_pq, epoch, sred, alpha,
                        [&](double t) {
                          pq = t;
                          return t != 0.0 ? d / t : 0.0;  // p = 0: no step
                        },
                        [&] {
                          for (int q = tid - 32; q < sncut * RB; q += kPT - 32) {
                            const int c = scut[q / RB], i = q % RB;
                            const int sl = c & 0xffff, k0 = c >> 16 & 0xff, n = c >> 24;
                            double t = sq[sl * RB + i];
                            for (int k = 0; k < n; k++) t += shead[(k0 + k) * RB + i];
                            sq[sl * RB + i] = t;
                          }
                        })) {
      if (tid == 0) atomicExch(a.err, 2);
      return;
    }
    // r -= alpha q and (r, M r); meanwhile x += alpha p
    v = 0.0;
    for (int i = tid; i < nrows; i += kPT) {
      const double ri = (SMEM ? sr[i] : a.r[row0 + i]) - alpha * sq[i];
      const double zi = ri * (SMEM ? sm[i] : a.m[row0 + i]);
      if (SMEM) sr[i] = ri; else a.r[row0 + i] = ri;
      sq[i] = zi;
      v += ri * zi;
    }
    if (!grid::sum<kPT>(v, a.gs, 1, sd, seen_rz, epoch + 1, sred, beta,
                        [&](double t) {
                          const double q = t / d;
                          d = t;
                          sd = t;
                          return q;
                        },
                        [&] {
                          for (int i = tid - 32; i < nrows; i += kPT - 32) {
                            if (SMEM) sx[i] += alpha * sp[i];
                            else a.x[row0 + i] += alpha * a.p[row0 + i];
                          }
                        })) {
      if (tid == 0) atomicExch(a.err, 2);
      return;
    }
    iters++;
    // p = M r + beta p, the stopping test in one warp beside it
    if (tid == kPT - 32)
      sstop = sqrt(fabs(sd)) < conv ? 1 : iters >= maxit || !(sd == sd) ? 2 : 0;
    for (int i = tid; i < nrows; i += kPT) {
      const double pi = sq[i] + beta * (SMEM ? sp[i] : a.p[row0 + i]);
      if (SMEM) sp[i] = pi;
      a.p[row0 + i] = pi;
    }
    if (!grid::barrier<kPT>(a.gs, step + 1, sred)) {
      if (tid == 0) atomicExch(a.err, 2);
      return;
    }
    if (sstop) break;
  }
  if (SMEM)
    for (int i = tid; i < nrows; i += kPT) {
      a.x[row0 + i] = sx[i];
      a.r[row0 + i] = sr[i];
    }
  if (blockIdx.x == 0 && tid == 0) {
    sc->d = d;
    sc->alpha = alpha;
    sc->beta = beta;
    sc->pq = pq;
    sc->iters = iters;
    sc->status = sstop == 2 ? ELX_ERR_NO_CONVERGENCE : ELX_OK;
    sc->done = sstop != 0;
  }
}

template <int B>
void launch(const PersistArgs &a, int grid, bool in_smem, int steps, cudaStream_t st) {
  const void *f = in_smem ? (const void *)pcg_persist_kernel<B, true>
                          : (const void *)pcg_persist_kernel<B, false>;
  const size_t bytes = in_smem ? persist_smem<B, true>(a.rows, a.slices)
                               : persist_smem<B, false>(a.rows, a.slices);
  ELX_CUDA(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  PersistArgs arg = a;
  void *args[] = {&arg, &steps};
  ELX_CUDA(cudaLaunchCooperativeKernel(f, dim3(grid), dim3(kPT), args, bytes, st));
}

}  // namespace

// Cuts the slices into one run per block with equal numbers of slot groups.
std::vector<int32_t> persist_cuts(const Structure &s, int grid) {
  std::vector<int32_t> t(grid + 1, 0);
  const int64_t total = s.sell_ptr[s.nslices];
  int sl = 0;
  for (int c = 0; c < grid; c++) {
    t[c] = sl;
    const int64_t target = total * (c + 1) / grid;
    const int last = s.nslices - (grid - 1 - c);  // leave a slice for each later block
    sl = std::min(sl + 1, last);
    while (sl < last && s.sell_ptr[sl] + (s.sell_ptr[sl + 1] - s.sell_ptr[sl]) / 2 < target) sl++;
  }
  t[grid] = s.nslices;
  return t;
}

}  // namespace elx

namespace elx_api {

// Plans the cooperative PCG of the context's matrix (once per structure).
// False: krylov.cu's launches are used.
bool ensure_persist(elx_ctx *c) {
  if (c->persist_grid != 0) return c->persist_grid > 0;
  c->persist_grid = -1;
  const elx::Structure &s = c->s;
  if (!c->use_blocks || s.nslices < 1) return false;
  const int grid = std::min({elx::sm_count(), elx::kGridMaxBlocks, s.nslices});
  const std::vector<int32_t> cuts = elx::persist_cuts(s, grid);
  int slices = 0;
  for (int k = 0; k < grid; k++) slices = std::max(slices, cuts[k + 1] - cuts[k]);
  const int rows = slices * elx::kSliceRows * s.bsize;
  int limit = 0;
  ELX_CUDA(cudaDeviceGetAttribute(&limit, cudaDevAttrMaxSharedMemoryPerBlockOptin, c->device));
  const bool b3 = s.bsize == 3;
  const size_t need1 = b3 ? elx::persist_smem<3, true>(rows, slices)
                          : elx::persist_smem<2, true>(rows, slices);
  const size_t need0 = b3 ? elx::persist_smem<3, false>(rows, slices)
                          : elx::persist_smem<2, false>(rows, slices);
  if (need0 > (size_t)limit) return false;
  c->persist_smem = need1 <= (size_t)limit;
  try {
    c->upload(c->persist_cta, cuts.data(), cuts.size());
    c->alloc(c->persist_sync, sizeof(elx::GridSync));
  } catch (const Error &e) {
    if (e.code != ELX_ERR_OOM) throw;
    c->release(c->persist_cta);
    return false;  // a memory budget without room for the slots
  }
  c->sync();
  c->persist_rows = rows;
  c->persist_slices = slices;
  c->persist_grid = grid;
  return true;
}

// Up to `steps` PCG iterations in one launch.
void persist_steps(elx_ctx *c, int steps) {
  elx::PersistArgs a;
  a.nb = c->s.nb;
  a.n = c->s.nb * c->s.bsize;
  a.sell_ptr = c->sell_ptr.as<int32_t>();
  a.sell_col = c->sell_col.as<int32_t>();
  a.sval = c->sell_val64.as<double>();
  a.cta = c->persist_cta.as<int32_t>();
  a.m = c->m.as<double>();
  a.x = c->xs.as<double>();
  a.r = c->r.as<double>();
  a.p = c->p.as<double>();
  a.sc = c->scal.as<elx::PcgScalars>();
  a.gs = c->persist_sync.as<elx::GridSync>();
  ELX_CUDA(cudaMemsetAsync(a.gs, 0, sizeof(elx::GridSync), c->stream));
  a.err = c->flags.as<int32_t>() + 2;
  a.rows = c->persist_rows;
  a.slices = c->persist_slices;
  if (c->s.bsize == 3)
    elx::launch<3>(a, c->persist_grid, c->persist_smem, steps, c->stream);
  else
    elx::launch<2>(a, c->persist_grid, c->persist_smem, steps, c->stream);
  c->launches += 1;
}

}  // namespace elx_api
