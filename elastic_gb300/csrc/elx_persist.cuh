// The cooperative PCG's block (persist.cu has the design and the figures), for
// the kernels that run it: a solve on the whole GPU (persist.cu) and the solve
// server's pack, a team of blocks for each load case (server.cu).
#pragma once

#include "elx_grid.cuh"
#include "elx_krylov.h"
#include "elx_sell.cuh"

namespace elx {

struct PersistArgs {
  int n;    // rows of the sliced matrix: nb B
  int neq;  // equations
  const int32_t *sell_ptr, *sell_col;
  const double *sval;
  const int32_t *cta;  // (grid + 1): first slice of each block
  const int32_t *eq;   // (n) equation of each row, -1: none (nullptr: the row)
  const double *m;     // (neq)
  const double *b;     // (neq, NC)
  double *x;           // (neq, NC): the solution, when a launch ends the solve
  double *sx, *sr, *p;  // (n, NC) by rows: x and r between launches, p
  PersistCol *cols;
  GridSync *gs;
  int32_t *err;
  double tol;
  int maxit;
  int rows, slices;  // of the largest block
  int stall = 0;     // grid::Team::missing
};

// Shared memory: the block's rows of q (and of x, r, p, M), the warps' heads
// and the slice tables.
template <int T, int B, int NC, bool SMEM>
size_t persist_smem(int rows, int slices) {
  constexpr int kPW = T / 32;
  return sizeof(double) * ((size_t)rows * ((SMEM ? 4 : 1) * NC + (SMEM ? 1 : 0)) +
                           (size_t)kPW * kSliceRows * B * NC) +
         sizeof(int32_t) * ((size_t)(slices + 1) + (kPW + 1) + kPW);
}

// Block `team.me` of a solve's blocks (T threads; grid::Team or grid::Cluster):
// up to `steps` iterations, the first of a solve with `start`.  `epoch` is above that of any earlier use
// of a.gs's slots; a.gs's words are zero.
template <int T, int B, int NC, bool SMEM, class Blocks>
__device__ __forceinline__ void persist_pcg(const PersistArgs &a, const Blocks team,
                                            const int start, const int steps, uint64_t epoch) {
  constexpr int kPT = T, kPW = T / 32;
  constexpr int BB = B * B, R = kSliceRows, RB = R * B, RBC = RB * NC;
  extern __shared__ __align__(16) unsigned char smem[];
  double *sq = reinterpret_cast<double *>(smem);
  double *sx = sq + (size_t)a.rows * NC, *sr = sx + (SMEM ? a.rows * NC : 0);
  double *sp = sr + (SMEM ? a.rows * NC : 0), *sm = sp + (SMEM ? a.rows * NC : 0);
  double *shead = sm + (SMEM ? a.rows : 0);
  __shared__ grid::Scratch<kPT, NC> sred;
  __shared__ double sd[NC], salpha[NC], sbeta[NC], sconv[NC];
  __shared__ int32_t siters[NC], son[NC], snext[NC], sstat[NC], sleft;
  __shared__ int32_t sncut, scut[kPW];
  int32_t *sptr = reinterpret_cast<int32_t *>(shead + kPW * RBC);  // group pointers of the slices
  int32_t *sga = sptr + a.slices + 1, *swsl = sga + kPW + 1;  // warps' first groups and slices
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  // every block reads the columns' states before the first wait, and block 0
  // writes them after the last
  int left = start;
  if (!start)
    for (int c = 0; c < NC; c++) left |= !a.cols[c].done;
  if (!left) return;
  const int s0 = a.cta[team.me], s1 = a.cta[team.me + 1], ns = s1 - s0;
  const int row0 = s0 * RB, nrows = min(a.n, s1 * RB) - row0, ne = nrows * NC;
  double *gx = a.sx + (size_t)row0 * NC, *gr = a.sr + (size_t)row0 * NC;
  double *gp = a.p + (size_t)row0 * NC;
  const double *gm = a.m + row0;  // only without an equation map
  for (int i = tid; i <= ns; i += kPT) sptr[i] = a.sell_ptr[s0 + i];
  if (tid < NC) {
    sleft = 1;
    siters[tid] = start ? 0 : a.cols[tid].iters;
    sstat[tid] = start ? ELX_OK : a.cols[tid].status;
    son[tid] = snext[tid] = start ? 1 : !a.cols[tid].done;
    sd[tid] = start ? 0.0 : a.cols[tid].d;
    sconv[tid] = start ? 0.0 : a.cols[tid].conv;
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
  // M by rows; without shared memory for it, through the map each time
  auto m_of = [&](int row) -> double {
    if (SMEM) return sm[row];
    if (!a.eq) return gm[row];
    const int q = a.eq[row0 + row];
    return q < 0 ? 0.0 : a.m[q];
  };
  if (SMEM)
    for (int i = tid; i < nrows; i += kPT) {
      const int q = a.eq ? a.eq[row0 + i] : row0 + i;
      sm[i] = q < 0 ? 0.0 : a.m[q];
    }
  unsigned long long seen_pq = 0, seen_rz = 0;  // warp 0: this lane's digits so far
  uint32_t barriers = 0;
  if (SMEM && !start)
    for (int i = tid; i < ne; i += kPT) {
      sx[i] = gx[i];
      sr[i] = gr[i];
      sp[i] = gp[i];
    }
  __syncthreads();
  if (start) {
    // x = 0, r = b, p = M b, d = (b, M b), conv = tol sqrt|d| (Iters.f:343-360)
    double v[NC];
#pragma unroll
    for (int c = 0; c < NC; c++) v[c] = 0.0;
    for (int i = tid; i < nrows; i += kPT) {
      const int q = a.eq ? a.eq[row0 + i] : row0 + i;
      const double mi = m_of(i);
#pragma unroll
      for (int c = 0; c < NC; c++) {
        const double bi = q < 0 ? 0.0 : a.b[(size_t)c * a.neq + q], zi = bi * mi;
        const int e = i * NC + c;
        (SMEM ? sx : gx)[e] = 0.0;
        (SMEM ? sr : gr)[e] = bi;
        if (SMEM) sp[e] = zi;
        gp[e] = zi;
        v[c] += bi * zi;
      }
    }
    epoch++;
    if (!grid::sum<kPT, NC>(team, v, a.gs, 0, nullptr, seen_pq, epoch, sred,
                            [&](double t) {
                              sd[lane] = t;
                              sconv[lane] = a.tol * sqrt(fabs(t));
                              // b = 0: x = 0 is exact
                              const int on = t != 0.0 && a.maxit > 0;
                              son[lane] = snext[lane] = on;
                              if (a.maxit <= 0 && t != 0.0) sstat[lane] = ELX_ERR_NO_CONVERGENCE;
                            },
                            [] {})) {
      if (tid == 0) atomicExch(a.err, 2);
      return;
    }
    if (!grid::barrier<kPT, NC>(team, a.gs, ++barriers, sred)) {
      if (tid == 0) atomicExch(a.err, 2);
      return;
    }
    if (tid == 0) {
      int k = 0;
      for (int c = 0; c < NC; c++) k += son[c];
      sleft = k;
    }
    __syncthreads();
  }
  // Columns are loaded a group ahead: the gathers of p, one L2 round trip, then
  // follow each other without a second one for their column (us an iteration,
  // before and after: 10.3 / 9.9 at 90,902 equations of TRIA3, 128.3 / 126.7 at
  // 811,200 of HEXA8).  Values or p a group ahead as well: 10.1, and 126.1 to
  // 128.3.
  const int first = sga[w] < sga[w + 1] ? sell_ld<true>(a.sell_col + (size_t)sga[w] * R + lane) : 0;
  for (int step = 0; step < steps && sleft; step++) {
    epoch += 2;  // of the slots, one for each sum
    // q = K p over the warp's groups, and their share of (p, q)
    double v[NC];
#pragma unroll
    for (int c = 0; c < NC; c++) v[c] = 0.0;
    {
      int g = sga[w], sl = swsl[w], next = first;
      const int gend = sga[w + 1];
      while (g < gend) {
        const int ge = min(sptr[sl + 1], gend);
        double *dst = g == sptr[sl] ? sq + sl * RBC : shead + w * RBC;
        double acc[B][NC];
#pragma unroll
        for (int b = 0; b < B; b++)
#pragma unroll
          for (int c = 0; c < NC; c++) acc[b][c] = 0.0;
        for (; g < ge; g++) {
          double bv[BB];
          const int J = next;
          if (g + 1 < gend) next = sell_ld<true>(a.sell_col + (size_t)(g + 1) * R + lane);
          sell_load<double, B, true>(a.sval + (size_t)g * BB * R, lane, bv);
          const double *px = a.p + (size_t)J * (B * NC);
#pragma unroll
          for (int b = 0; b < B; b++) {
            double xv[NC];
#pragma unroll
            for (int c = 0; c < NC; c++) xv[c] = px[b * NC + c];
#pragma unroll
            for (int k = 0; k < B; k++)
#pragma unroll
              for (int c = 0; c < NC; c++) acc[k][c] += bv[k * B + b] * xv[c];
          }
        }
        const int i = sl * RB + lane * B;
        if (i < nrows)
#pragma unroll
          for (int b = 0; b < B; b++)
#pragma unroll
            for (int c = 0; c < NC; c++) {
              const int e = b * NC + c;
              dst[lane * (B * NC) + e] = acc[b][c];
              v[c] += (SMEM ? sp : gp)[i * NC + e] * acc[b][c];
            }
        sl++;
      }
    }
    // alpha = d / (p, q); meanwhile the slices cut between warps are put together
    if (!grid::sum<kPT, NC>(team, v, a.gs, 0, sd, seen_pq, epoch, sred,
                            [&](double t) {
                              // p = 0: no step; a stopped column stays as it is
                              salpha[lane] = son[lane] && t != 0.0 ? sd[lane] / t : 0.0;
                            },
                            [&] {
                              for (int q = tid - 32; q < sncut * RBC; q += kPT - 32) {
                                const int c = scut[q / RBC], i = q % RBC;
                                const int sl = c & 0xffff, k0 = c >> 16 & 0xff, n = c >> 24;
                                double t = sq[sl * RBC + i];
                                for (int k = 0; k < n; k++) t += shead[(k0 + k) * RBC + i];
                                sq[sl * RBC + i] = t;
                              }
                            })) {
      if (tid == 0) atomicExch(a.err, 2);
      return;
    }
    // r -= alpha q and (r, M r), z = M r in q's place; meanwhile x += alpha p
#pragma unroll
    for (int c = 0; c < NC; c++) v[c] = 0.0;
    for (int i = tid; i < nrows; i += kPT) {
      const double mi = m_of(i);
#pragma unroll
      for (int c = 0; c < NC; c++) {
        const int e = i * NC + c;
        const double ri = NC > 1 && !son[c] ? (SMEM ? sr : gr)[e]
                                            : (SMEM ? sr : gr)[e] - salpha[c] * sq[e];
        const double zi = ri * mi;
        (SMEM ? sr : gr)[e] = ri;
        sq[e] = zi;
        v[c] += ri * zi;
      }
    }
    if (!grid::sum<kPT, NC>(team, v, a.gs, 1, sd, seen_rz, epoch + 1, sred,
                            [&](double t) {
                              if (son[lane]) {
                                sbeta[lane] = t / sd[lane];
                                sd[lane] = t;
                              }
                            },
                            [&] {
                              for (int e = tid - 32; e < ne; e += kPT - 32) {
                                const int c = e % NC;
                                if (NC > 1 && !son[c]) continue;
                                (SMEM ? sx : gx)[e] += salpha[c] * (SMEM ? sp : gp)[e];
                              }
                            })) {
      if (tid == 0) atomicExch(a.err, 2);
      return;
    }
    // p = M r + beta p; the stopping test beside it in the last warp
    if (w == kPW - 1) {
      int on = 0;
      if (lane < NC && son[lane]) {
        const double d = sd[lane];
        const int it = ++siters[lane];
        on = 1;
        if (sqrt(fabs(d)) < sconv[lane]) {
          on = 0;
        } else if (it >= a.maxit || !(d == d)) {
          on = 0;
          sstat[lane] = ELX_ERR_NO_CONVERGENCE;
        }
      }
      if (lane < NC) snext[lane] = on;
      const unsigned any = __ballot_sync(0xffffffffu, on);
      if (lane == 0) sleft = any != 0;
    }
    for (int e = tid; e < ne; e += kPT) {
      const int c = e % NC;
      if (NC > 1 && !son[c]) continue;
      const double pi = sq[e] + sbeta[c] * (SMEM ? sp : gp)[e];
      if (SMEM) sp[e] = pi;
      gp[e] = pi;
    }
    if (!grid::barrier<kPT, NC>(team, a.gs, ++barriers, sred)) {
      if (tid == 0) atomicExch(a.err, 2);
      return;
    }
    if (tid < NC) son[tid] = snext[tid];  // read again after the next sum's first wait
    if (NC > 1) __syncthreads();
  }
  const bool all = !sleft;
  for (int i = tid; i < nrows; i += kPT) {
    const int q = a.eq ? a.eq[row0 + i] : row0 + i;
#pragma unroll
    for (int c = 0; c < NC; c++) {
      const int e = i * NC + c;
      const double xi = (SMEM ? sx : gx)[e];
      if (all && q >= 0) a.x[(size_t)c * a.neq + q] = xi;
      if (SMEM && !all) {
        gx[e] = xi;
        gr[e] = sr[e];
      }
    }
  }
  if (team.me == 0 && tid < NC) {
    PersistCol &o = a.cols[tid];
    o.d = sd[tid];
    o.conv = sconv[tid];
    o.iters = siters[tid];
    o.status = sstat[tid];
    o.done = !snext[tid];
    o.started = 1;
  }
}

}  // namespace elx
