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
// Up to kGridCols load cases go through one launch: they share the matrix
// reads and the waits, and five of them are not padded to a block of eight
// (5 cases of 66,820 QUAD4 equations: 119 ms as launches of width 8, 55 ms
// here).  A matrix with partly fixed nodes is padded to whole node blocks
// (structure.cpp:build_padded) with a map from rows to equations, read at the
// start and the end of a solve: the same kernel in place of the scalar gather
// (205,556 equations with rollers: 68 against 38 us an iteration).
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
};

// Shared memory: the block's rows of q (and of x, r, p, M), the warps' heads
// and the slice tables.
template <int B, int NC, bool SMEM>
size_t persist_smem(int rows, int slices) {
  return sizeof(double) * ((size_t)rows * ((SMEM ? 4 : 1) * NC + (SMEM ? 1 : 0)) +
                           (size_t)kPW * kSliceRows * B * NC) +
         sizeof(int32_t) * ((size_t)(slices + 1) + (kPW + 1) + kPW);
}

template <int B, int NC, bool SMEM>
__global__ void __launch_bounds__(kPT, 1)
pcg_persist_kernel(PersistArgs a, int start, int steps) {
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
  const grid::Team team{(int)blockIdx.x, (int)gridDim.x};
  // every block reads the columns' states before the first wait, and block 0
  // writes them after the last
  int left = start;
  if (!start)
    for (int c = 0; c < NC; c++) left |= !a.cols[c].done;
  if (!left) return;
  const int s0 = a.cta[blockIdx.x], s1 = a.cta[blockIdx.x + 1], ns = s1 - s0;
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
  uint64_t epoch = 0;
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
  for (int step = 0; step < steps && sleft; step++) {
    epoch += 2;  // of the slots, one for each sum
    // q = K p over the warp's groups, and their share of (p, q)
    double v[NC];
#pragma unroll
    for (int c = 0; c < NC; c++) v[c] = 0.0;
    {
      int g = sga[w], sl = swsl[w];
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
          const int J = sell_ld<true>(a.sell_col + (size_t)g * R + lane);
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
  if (blockIdx.x == 0 && tid < NC) {
    PersistCol &o = a.cols[tid];
    o.d = sd[tid];
    o.conv = sconv[tid];
    o.iters = siters[tid];
    o.status = sstat[tid];
    o.done = !snext[tid];
  }
}

template <int B, int NC>
size_t smem_of(bool in_smem, int rows, int slices) {
  return in_smem ? persist_smem<B, NC, true>(rows, slices)
                 : persist_smem<B, NC, false>(rows, slices);
}

template <int B, int NC>
void launch(const PersistArgs &a, int grid, bool in_smem, int start, int steps, cudaStream_t st) {
  const void *f = in_smem ? (const void *)pcg_persist_kernel<B, NC, true>
                          : (const void *)pcg_persist_kernel<B, NC, false>;
  const size_t bytes = smem_of<B, NC>(in_smem, a.rows, a.slices);
  ELX_CUDA(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  PersistArgs arg = a;
  void *args[] = {&arg, &start, &steps};
  ELX_CUDA(cudaLaunchCooperativeKernel(f, dim3(grid), dim3(kPT), args, bytes, st));
}

#define ELX_NC_DISPATCH(nc, call)                             \
  switch (nc) {                                               \
    case 1: call(1); break;                                   \
    case 2: call(2); break;                                   \
    case 3: call(3); break;                                   \
    case 4: call(4); break;                                   \
    case 5: call(5); break;                                   \
    case 6: call(6); break;                                   \
    default: throw Error{ELX_ERR_ARG, "too many columns"};    \
  }

size_t smem_bytes(int B, int nc, bool in_smem, int rows, int slices) {
  size_t r = 0;
#define CALL(NC) r = B == 3 ? smem_of<3, NC>(in_smem, rows, slices) : smem_of<2, NC>(in_smem, rows, slices)
  ELX_NC_DISPATCH(nc, CALL)
#undef CALL
  return r;
}

}  // namespace

// Cuts the slices into one run per block with equal numbers of slot groups.
std::vector<int32_t> persist_cuts(const std::vector<int32_t> &sell_ptr, int grid) {
  const int nslices = (int)sell_ptr.size() - 1;
  std::vector<int32_t> t(grid + 1, 0);
  const int64_t total = sell_ptr[nslices];
  int sl = 0;
  for (int c = 0; c < grid; c++) {
    t[c] = sl;
    const int64_t target = total * (c + 1) / grid;
    const int last = nslices - (grid - 1 - c);  // leave a slice for each later block
    sl = std::min(sl + 1, last);
    while (sl < last && sell_ptr[sl] + (sell_ptr[sl + 1] - sell_ptr[sl]) / 2 < target) sl++;
  }
  t[grid] = nslices;
  return t;
}

}  // namespace elx

namespace elx_api {

// Rows of the sliced matrix the cooperative PCG works on (the equations, or
// more with partly fixed nodes).
int persist_rows(const elx_ctx *c) {
  return c->use_blocks ? c->s.nb * c->s.bsize : c->s.p_nb * c->s.p_bsize;
}

// Plans the cooperative PCG of the context's matrix (once per structure).
// False: krylov.cu's launches are used.
bool ensure_persist(elx_ctx *c) {
  const elx::Structure &s = c->s;
  const bool padded = !c->use_blocks;
  if (c->persist_grid < 0 || (padded && !(c->want_blocks && s.padded))) return false;
  if (c->persist_grid == 0) {
    c->persist_grid = -1;
    const std::vector<int32_t> &ptr = padded ? s.p_ptr : s.sell_ptr;
    const int nslices = (int)ptr.size() - 1, B = padded ? s.p_bsize : s.bsize;
    const int grid = std::min({elx::sm_count(), elx::kGridMaxBlocks, nslices});
    const std::vector<int32_t> cuts = elx::persist_cuts(ptr, grid);
    int slices = 0;
    for (int k = 0; k < grid; k++) slices = std::max(slices, cuts[k + 1] - cuts[k]);
    const int rows = slices * elx::kSliceRows * B;
    int limit = 0;
    ELX_CUDA(cudaDeviceGetAttribute(&limit, cudaDevAttrMaxSharedMemoryPerBlockOptin, c->device));
    limit -= 2048;  // the kernel's static arrays
    for (int nc = 1; nc <= elx::kGridCols; nc++)
      c->persist_mode[nc] = elx::smem_bytes(B, nc, true, rows, slices) <= (size_t)limit    ? 2
                            : elx::smem_bytes(B, nc, false, rows, slices) <= (size_t)limit ? 1
                                                                                           : 0;
    if (!c->persist_mode[1]) return false;
    try {
      c->upload(c->persist_cta, cuts.data(), cuts.size());
      c->alloc(c->persist_sync, sizeof(elx::GridSync) + sizeof(elx::PersistCol) * elx::kGridCols);
      c->alloc(c->persist_vec, 3 * 8 * (size_t)persist_rows(c));
      if (padded) {
        c->upload(c->p_ptr, s.p_ptr.data(), s.p_ptr.size());
        c->upload(c->p_col, s.p_col.data(), s.p_col.size());
        c->upload(c->p_off, s.p_off.data(), s.p_off.size());
        c->upload(c->p_eq, s.p_eq.data(), s.p_eq.size());
        c->alloc(c->p_val, s.p_col.size() * B * B * 8 + 64);
      }
    } catch (const Error &e) {
      if (e.code != ELX_ERR_OOM) throw;
      // a memory budget without room for it
      for (DBuf *d : {&c->persist_cta, &c->persist_sync, &c->persist_vec, &c->p_ptr, &c->p_col,
                      &c->p_off, &c->p_eq, &c->p_val})
        c->release(*d);
      return false;
    }
    c->sync();
    c->persist_rows = rows;
    c->persist_slices = slices;
    c->persist_grid = grid;
  }
  if (padded && !c->have_padded) {
    elx::launch_fill_padded64(c->csrc_dev(), s.p_bsize, s.p_nb, (int)s.p_ptr.size() - 1,
                              c->p_ptr.as<int32_t>(), c->p_col.as<int32_t>(),
                              c->p_off.as<int32_t>(), c->p_eq.as<int32_t>(),
                              c->p_val.as<double>(), c->stream);
    c->launches += 1;
    c->have_padded = true;
  }
  return true;
}

// Columns that a launch can take together, at most `want` (0: none).
int persist_columns(elx_ctx *c, int want) {
  if (!ensure_persist(c)) return 0;
  int nc = std::min(want, elx::kGridCols);
  while (nc > 0 && !c->persist_mode[nc]) nc--;
  return nc;
}

// PCG of nc columns b -> x (device, neq x nc), at most `steps` iterations a
// launch, two launches in flight; `work` holds 3 n nc doubles.  The columns'
// results into out.
void persist_solve(elx_ctx *c, int nc, double tol, int maxit, const double *b, double *x,
                   double *work, int steps, elx::PersistCol *out) {
  elx::PersistArgs a;
  const size_t n = (size_t)persist_rows(c);
  const bool padded = !c->use_blocks;
  const int B = padded ? c->s.p_bsize : c->s.bsize;
  a.n = (int)n;
  a.neq = c->s.neq;
  a.sell_ptr = (padded ? c->p_ptr : c->sell_ptr).as<int32_t>();
  a.sell_col = (padded ? c->p_col : c->sell_col).as<int32_t>();
  a.sval = (padded ? c->p_val : c->sell_val64).as<double>();
  a.cta = c->persist_cta.as<int32_t>();
  a.eq = padded ? c->p_eq.as<int32_t>() : nullptr;
  a.m = c->m.as<double>();
  a.b = b;
  a.x = x;
  a.sx = work;
  a.sr = work + n * nc;
  a.p = work + 2 * n * nc;
  a.gs = c->persist_sync.as<elx::GridSync>();
  a.cols = reinterpret_cast<elx::PersistCol *>(a.gs + 1);
  a.err = c->flags.as<int32_t>() + 2;
  a.tol = tol;
  a.maxit = maxit;
  a.rows = c->persist_rows;
  a.slices = c->persist_slices;
  const bool in_smem = c->persist_mode[nc] == 2;
  const int max_launches = maxit / steps + 2;
  int launched = 0, checked = 0;
  auto go = [&] {
    const int slot = launched & 1, start = launched == 0;
    ELX_CUDA(cudaMemsetAsync(a.gs, 0, sizeof(elx::GridSync), c->stream));
#define CALL(NC)                                                                     \
  if (B == 3)                                                                        \
    elx::launch<3, NC>(a, c->persist_grid, in_smem, start, steps, c->stream);        \
  else                                                                               \
    elx::launch<2, NC>(a, c->persist_grid, in_smem, start, steps, c->stream)
    ELX_NC_DISPATCH(nc, CALL)
#undef CALL
    c->launches += 1;
    ELX_CUDA(cudaMemcpyAsync(c->h_cols + slot * elx::kGridCols, a.cols,
                             sizeof(elx::PersistCol) * nc, cudaMemcpyDeviceToHost, c->stream));
    ELX_CUDA(cudaEventRecord(c->ev[slot], c->stream));
    launched++;
  };
  // a server's block solve asks the gate before each launch and polls it
  auto gate = [&](int enter) {
    if (c->batch_gate) c->batch_gate(c->batch_gate_user, enter);
  };
  struct Leave {  // also when a launch or a poll throws
    decltype(gate) &g;
    bool in = false;
    ~Leave() {
      if (in) g(0);
    }
  } leave{gate};
  gate(1);
  leave.in = true;
  go();
  for (;;) {
    if (launched < max_launches && !c->batch_gate) go();
    const elx::PersistCol *h = c->h_cols + (checked & 1) * elx::kGridCols;
    ELX_CUDA(cudaEventSynchronize(c->ev[checked & 1]));
    checked++;
    bool all = true;
    for (int k = 0; k < nc; k++) all = all && h[k].done;
    if (all || checked >= max_launches) {
      std::copy(h, h + nc, out);
      break;
    }
    if (c->batch_gate) {
      leave.in = false;
      gate(0);
      gate(1);
      leave.in = true;
      go();
    }
  }
  c->sync();
}

}  // namespace elx_api
