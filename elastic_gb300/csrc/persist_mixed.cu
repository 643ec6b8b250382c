// The mixed-precision PCG in one cooperative launch: the iteration of
// krylov.cu's rel_* kernels (FP32 CG with reliable updates: FP64 solution,
// residual replacements and stopping test) on the grid waits of persist.cu.
//
// The launches cost here what they cost there: at 345,744 TETRA4 equations an
// iteration was 9.0 us of product, 6.8 of update (5 of it the last block's
// reduction), 2.0 of direction and 1.0 of replacement kernels that return at
// once.  A block keeps its rows of x_lo, r, p, q and M in shared memory; a
// replacement, one iteration in some hundred, runs between two waits of its
// own.  Per iteration, launches -> here: 21 -> 12 us (345,744 TETRA4
// equations, the FP32 copy stays in L2), 60 -> 53 us (771,120 HEXA8, 45 of
// them the matrix from HBM at 0.8 of its measured rate).
//
// The FP32 product streams the matrix: kMT threads with kMU slot groups each
// in flight (768 x 3 measured faster than 1024 x 2, 768 x 2 and 512 x 4: HBM
// latency times bandwidth is 45 KB an SM, and gathers of p come on top).
#include <algorithm>

#include "elx_context.h"
#include "elx_grid.cuh"
#include "elx_sell.cuh"

namespace elx {
namespace {

constexpr int kMT = 768;  // threads of a block
constexpr int kMW = kMT / 32;
constexpr int kMU = 3;  // slot groups in flight

struct MixedArgs {
  int n;
  const int32_t *sell_ptr, *sell_col;
  const int16_t *col16;
  const float *sval32;
  const double *sval64;
  const int32_t *cta;
  const double *b, *m;
  const float *m32;
  double *xhi;
  float *xlo, *r, *p;
  PcgScalars *sc;
  GridSync *gs;
  int32_t *err;
  int rows, slices, stall;
};

template <int B>
size_t mixed_smem(int rows, int slices) {
  return sizeof(float) * ((size_t)rows * 5 + (size_t)kMW * kSliceRows * B) +
         sizeof(int32_t) * ((size_t)(slices + 1) + (kMW + 1) + kMW);
}

template <int B, bool LD, bool D16>
__global__ void __launch_bounds__(kMT, 1) mixed_persist_kernel(MixedArgs a, int replace_every, int steps) {
  constexpr int BB = B * B, R = kSliceRows, RB = R * B, U = kMU;
  extern __shared__ __align__(16) unsigned char smem[];
  float *sq = reinterpret_cast<float *>(smem);
  float *sx = sq + a.rows, *sr = sx + a.rows, *sp = sr + a.rows, *sm = sp + a.rows;
  float *shead = sm + a.rows;
  __shared__ grid::Scratch<kMT, 1> sred;
  __shared__ PcgScalars S;  // lane 0 of warp 0 and one thread of the last warp write it
  __shared__ double sd[1];
  __shared__ float salpha, sbeta;
  __shared__ int32_t sncut, scut[kMW];
  int32_t *sptr = reinterpret_cast<int32_t *>(shead + kMW * RB);
  int32_t *sga = sptr + a.slices + 1, *swsl = sga + kMW + 1;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const grid::Team team{(int)blockIdx.x, (int)gridDim.x};
  if (team.missing(a.stall)) return;
  // block 0 writes the scalars after the last wait
  if (a.sc->done) return;
  const int s0 = a.cta[blockIdx.x], s1 = a.cta[blockIdx.x + 1], ns = s1 - s0;
  const int row0 = s0 * RB, nrows = min(a.n, s1 * RB) - row0;
  for (int i = tid; i <= ns; i += kMT) sptr[i] = a.sell_ptr[s0 + i];
  if (tid == 0) {
    S = *a.sc;
    sd[0] = S.d;
  }
  for (int i = tid; i < nrows; i += kMT) {
    sx[i] = a.xlo[row0 + i];
    sr[i] = a.r[row0 + i];
    sp[i] = a.p[row0 + i];
    sm[i] = a.m32[row0 + i];
  }
  __syncthreads();
  if (tid <= kMW) {
    const int total = sptr[ns] - sptr[0], wn = min(kMW, max(4, total / 2 & ~3));
    const int g = sptr[0] + (int)((int64_t)total * min(tid, wn) / wn);
    sga[tid] = g;
    if (tid < kMW) {
      int lo = 0, hi = ns - 1;
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (sptr[mid] <= g) lo = mid; else hi = mid - 1;
      }
      swsl[tid] = lo;
    }
  }
  __syncthreads();
  if (tid == 0) {
    int n = 0;
    for (int k = 1; k < kMW; k++) {
      const int sl = swsl[k];
      if (sga[k] == sptr[sl] || sga[k + 1] == sga[k]) continue;
      if (n && (scut[n - 1] & 0xffff) == sl)
        scut[n - 1] += 1 << 24;
      else
        scut[n++] = sl | k << 16 | 1 << 24;
    }
    sncut = n;
  }
  __syncthreads();
  unsigned long long seen_pq = 0, seen_rz = 0;
  uint64_t epoch = 0;
  uint32_t barriers = 0;
#define ELX_GIVE_UP                          \
  do {                                       \
    if (tid == 0) atomicExch(a.err, 2);      \
    return;                                  \
  } while (0)
  for (int step = 0; step < steps && !S.done; step++) {
    epoch += 3;
    // q = K p (FP32) over the warp's groups, and their share of (p, q)
    float v[1] = {0.0f};
    {
      int g = sga[w], sl = swsl[w];
      const int gend = sga[w + 1];
      while (g < gend) {
        const int ge = min(sptr[sl + 1], gend);
        float *dst = g == sptr[sl] ? sq + sl * RB : shead + w * RB;
        float acc[B];
#pragma unroll
        for (int b = 0; b < B; b++) acc[b] = 0.0f;
        for (; g < ge; g += U) {
          const int nu = min(U, ge - g);
          int J[U];
          float bv[U][BB];
#pragma unroll
          for (int u = 0; u < U; u++)
            if (u < nu) J[u] = sell_column<D16, LD>(a.sell_col, a.col16, s0 + sl, g + u, lane);
#pragma unroll
          for (int u = 0; u < U; u++)
            if (u < nu) sell_load<float, B, LD>(a.sval32 + (size_t)(g + u) * BB * R, lane, bv[u]);
#pragma unroll
          for (int u = 0; u < U; u++)
            if (u < nu) {
              float xv[B];
#pragma unroll
              for (int b = 0; b < B; b++) xv[b] = a.p[J[u] * B + b];
#pragma unroll
              for (int c = 0; c < B; c++)
#pragma unroll
                for (int b = 0; b < B; b++) acc[c] += bv[u][c * B + b] * xv[b];
            }
        }
        g = ge;
        const int i = sl * RB + lane * B;
        if (i < nrows)
#pragma unroll
          for (int b = 0; b < B; b++) {
            dst[lane * B + b] = acc[b];
            v[0] += sp[i + b] * acc[b];
          }
        sl++;
      }
    }
    if (!grid::sum<kMT, 1>(team, v, a.gs, 0, sd, seen_pq, epoch, sred,
                           [&](double t) {
                             S.pq = t;
                             S.alpha = t != 0.0 ? sd[0] / t : 0.0;
                             salpha = (float)S.alpha;
                           },
                           [&] {
                             for (int q = tid - 32; q < sncut * RB; q += kMT - 32) {
                               const int c = scut[q / RB], i = q % RB;
                               const int sl = c & 0xffff, k0 = c >> 16 & 0xff, n = c >> 24;
                               float t = sq[sl * RB + i];
                               for (int k = 0; k < n; k++) t += shead[(k0 + k) * RB + i];
                               sq[sl * RB + i] = t;
                             }
                           }))
      ELX_GIVE_UP;
    // r -= alpha q and (r, M r), z = M r in q's place; meanwhile x_lo += alpha p
    v[0] = 0.0f;
    {
      const float al = salpha;
      for (int i = tid; i < nrows; i += kMT) {
        const float ri = sr[i] - al * sq[i], zi = ri * sm[i];
        sr[i] = ri;
        sq[i] = zi;
        v[0] += ri * zi;
      }
    }
    if (!grid::sum<kMT, 1>(team, v, a.gs, 1, sd, seen_rz, epoch + 1, sred,
                           [&](double t) {
                             // an FP32 residual of exactly zero: beta = 0, and
                             // the next replacement point takes over
                             S.beta = sd[0] != 0.0 ? t / sd[0] : 0.0;
                             sbeta = (float)S.beta;
                             sd[0] = t;
                           },
                           [&] {
                             const float al = salpha;
                             for (int i = tid - 32; i < nrows; i += kMT - 32) sx[i] += al * sp[i];
                           }))
      ELX_GIVE_UP;
    // the replacement and stopping flags of rel_update_kernel, beside the new p
    if (tid == kMT - 32) {
      const double t = sd[0];
      const int it = S.iters + 1;
      S.iters = it;
      if (!(t == t) || isinf(t)) {
        S.done = 1;
        S.status = ELX_ERR_NO_CONVERGENCE;
        S.failed = 1;
      } else {
        const double rn = sqrt(fabs(t));
        if (rn < S.delta * S.rmax || rn < S.conv || it >= S.maxit ||
            it - S.last_rep >= kMixedCheckEvery || rn > kMixedDiverge * S.rmax)
          S.update = 1;
      }
    }
    {
      const float be = sbeta;
      for (int i = tid; i < nrows; i += kMT) {
        const float pi = sq[i] + be * sp[i];
        sp[i] = pi;
        a.p[row0 + i] = pi;
      }
    }
    if (!grid::barrier<kMT, 1>(team, a.gs, ++barriers, sred)) ELX_GIVE_UP;
    if (S.done || !S.update || S.iters % replace_every) continue;
    // replacement (rel_accumulate, FP64 product, rel_residual): x_hi += x_lo,
    // r = b - K x_hi in FP64
    for (int i = tid; i < nrows; i += kMT) {
      a.xhi[row0 + i] += (double)sx[i];
      sx[i] = 0.0f;
    }
    if (!grid::barrier<kMT, 1>(team, a.gs, ++barriers, sred)) ELX_GIVE_UP;
    double vd[1] = {0.0};
    for (int sl = w; sl < ns; sl += kMW) {
      double acc[B];
#pragma unroll
      for (int b = 0; b < B; b++) acc[b] = 0.0;
      for (int g = sptr[sl]; g < sptr[sl + 1]; g++) {
        double bv[BB];
        const int J = sell_column<D16, true>(a.sell_col, a.col16, s0 + sl, g, lane);
        sell_load<double, B, true>(a.sval64 + (size_t)g * BB * R, lane, bv);
#pragma unroll
        for (int b = 0; b < B; b++) {
          const double xb = a.xhi[J * B + b];
#pragma unroll
          for (int c = 0; c < B; c++) acc[c] += bv[c * B + b] * xb;
        }
      }
      const int i = sl * RB + lane * B;
      if (i < nrows)
#pragma unroll
        for (int b = 0; b < B; b++) {
          const double ri = a.b[row0 + i + b] - acc[b];
          sr[i + b] = (float)ri;
          vd[0] += ri * (ri * a.m[row0 + i + b]);
        }
    }
    if (!grid::sum<kMT, 1>(team, vd, a.gs, 1, sd, seen_rz, epoch + 2, sred,
                           [&](double t) {
                             const double rt = sqrt(fabs(t));
                             S.update = 0;
                             S.nupdates += 1;
                             S.last_rep = S.iters;
                             if (rt < S.conv) {
                               S.done = 1;
                             } else if (!(t == t) || rt > kMixedDiverge * S.best) {
                               S.done = 1;
                               S.status = ELX_ERR_NO_CONVERGENCE;
                               S.failed = 1;
                             } else if (S.iters >= S.maxit) {
                               S.done = 1;
                               S.status = ELX_ERR_NO_CONVERGENCE;
                             } else {
                               S.stall = rt < 0.5 * S.best ? 0 : S.stall + 1;
                               S.best = fmin(S.best, rt);
                               if (S.stall >= kMixedStall) {
                                 S.done = 1;
                                 S.status = ELX_ERR_NO_CONVERGENCE;
                                 S.failed = 1;
                               }
                               sd[0] = t;
                               S.rmax = rt;
                             }
                           },
                           [] {}))
      ELX_GIVE_UP;
  }
#undef ELX_GIVE_UP
  for (int i = tid; i < nrows; i += kMT) {
    a.xlo[row0 + i] = sx[i];
    a.r[row0 + i] = sr[i];
  }
  if (blockIdx.x == 0 && tid == 0) {
    S.d = sd[0];
    *a.sc = S;
  }
}

template <int B, bool LD, bool D16>
void launch_mixed(const MixedArgs &a, int grid, int replace_every, int steps, cudaStream_t st) {
  const void *f = (const void *)mixed_persist_kernel<B, LD, D16>;
  const size_t bytes = mixed_smem<B>(a.rows, a.slices);
  ELX_CUDA(allow_shared(f));
  MixedArgs arg = a;
  void *args[] = {&arg, &replace_every, &steps};
  ELX_CUDA(cudaLaunchCooperativeKernel(f, dim3(grid), dim3(kMT), args, bytes, st));
}

}  // namespace
}  // namespace elx

namespace elx_api {

// Whether the mixed PCG of the context's matrix runs in cooperative launches.
bool mixed_persist(elx_ctx *c) {
  if (!c->use_blocks || !ensure_persist(c)) return false;
  int limit = 0;
  ELX_CUDA(cudaDeviceGetAttribute(&limit, cudaDevAttrMaxSharedMemoryPerBlockOptin, c->device));
  const size_t need = c->s.bsize == 3 ? elx::mixed_smem<3>(c->persist_rows, c->persist_slices)
                                      : elx::mixed_smem<2>(c->persist_rows, c->persist_slices);
  return need + 2048 <= (size_t)limit;
}

// Up to `steps` iterations from the scalars in c->scal, in one launch.
void mixed_persist_steps(elx_ctx *c, int replace_every, int steps) {
  elx::MixedArgs a;
  a.n = c->s.nb * c->s.bsize;
  a.sell_ptr = c->sell_ptr.as<int32_t>();
  a.sell_col = c->sell_col.as<int32_t>();
  a.col16 = static_cast<const int16_t *>(c->sell_d16.p);
  a.sval32 = c->sell_val.as<float>();
  a.sval64 = c->sell_val64.as<double>();
  a.cta = c->persist_cta.as<int32_t>();
  a.b = c->b.as<double>();
  a.m = c->m.as<double>();
  a.m32 = c->m32.as<float>();
  a.xhi = c->xs.as<double>();
  a.xlo = c->x32.as<float>();
  a.r = c->r32.as<float>();
  a.p = c->p32.as<float>();
  a.sc = c->scal.as<elx::PcgScalars>();
  a.gs = c->persist_sync.as<elx::GridSync>();
  a.err = c->flags.as<int32_t>() + 2;
  a.rows = c->persist_rows;
  a.slices = c->persist_slices;
  a.stall = elx::grid_stall();
  ELX_CUDA(cudaMemsetAsync(a.gs, 0, sizeof(elx::GridSync), c->stream));
  const int g = c->persist_grid;
  if (c->s.bsize == 3) {
    if (a.col16)
      c->sell_stream ? elx::launch_mixed<3, true, true>(a, g, replace_every, steps, c->stream)
                     : elx::launch_mixed<3, false, true>(a, g, replace_every, steps, c->stream);
    else
      c->sell_stream ? elx::launch_mixed<3, true, false>(a, g, replace_every, steps, c->stream)
                     : elx::launch_mixed<3, false, false>(a, g, replace_every, steps, c->stream);
  } else {
    c->sell_stream ? elx::launch_mixed<2, true, false>(a, g, replace_every, steps, c->stream)
                   : elx::launch_mixed<2, false, false>(a, g, replace_every, steps, c->stream);
  }
  c->launches += 1;
}

}  // namespace elx_api
