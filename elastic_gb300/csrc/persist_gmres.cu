// One GMRES(k) restart cycle (gmres, mef/src/Iters.f:528-808) in one
// cooperative launch, on the blocks and grid sums of persist.cu.
//
// krylov_ns.cu launches one kernel per Gram-Schmidt projection, each with a
// last-block reduction: 1,275 of 5.3 us in a cycle of GMRES(50), whatever the
// size.  Modified Gram-Schmidt has a grid wait per projection too, so the
// vectors are orthogonalised here by classical Gram-Schmidt twice ("twice is
// enough", Giraud, Langou, Rozloznik and van den Eshof 2005: orthogonal to
// rounding, where MGS loses it with the condition of the basis): all dots of a
// step with the basis at once, two waits a step instead of i.  In exact
// arithmetic both give the same basis and Hessenberg matrix.  A warp takes
// every 16th basis vector: it adds its block's dot to that vector's digits and
// waits for the total itself.  The rotations of a step run in one warp of every
// block while the norm is summed, so nothing is broadcast.
// GMRES(50) at 113,832 HEXA8 equations: 20.0 ms for two cycles as launches,
// 7.5 ms here (the product 14 us a step at the FP64 pipe, the four passes over
// the basis 18).
#include <algorithm>

#include "elx_context.h"
#include "elx_grid.cuh"
#include "elx_sell.cuh"

namespace elx {
namespace {

constexpr int kGT = 512;
constexpr int kGW = kGT / 32;

// Shared words of one basis vector's dots, in the first and second pass.
struct GmresDot {
  GridWords words;
  GridSlot slot[1][kGridMaxBlocks];
};

struct GmresArgs {
  int n, neq, k;
  const int32_t *sell_ptr, *sell_col;
  const double *sval;
  const int32_t *cta, *eq;
  const double *b, *m;
  double *x;   // (neq)
  double *xr;  // (n) x by rows
  double *g;   // (k + 1, n) the basis by rows
  GmresState *gs;
  GridSync *sync;
  GmresDot *dots;  // (2, k)
  int32_t *err;
  int rows, slices, stall;
};

// Shared memory: w and M by rows, the warps' heads, the Hessenberg columns and
// the small vectors, the dots' words seen so far, the slice tables.
template <int B>
size_t gmres_smem(int rows, int slices, int k) {
  return sizeof(double) * ((size_t)2 * rows + (size_t)kGW * kSliceRows * B +
                           (size_t)(k + 1) * k + 6 * (size_t)(k + 2)) +
         sizeof(unsigned long long) * 2 * kDigits * (size_t)k +
         sizeof(int32_t) * ((size_t)(slices + 1) + (kGW + 1) + kGW);
}

template <int B>
__global__ void __launch_bounds__(kGT, 1) gmres_persist_kernel(GmresArgs a) {
  constexpr int BB = B * B, R = kSliceRows, RB = R * B;
  extern __shared__ __align__(16) unsigned char smem[];
  const int K = a.k;
  double *sw = reinterpret_cast<double *>(smem), *sm = sw + a.rows, *shead = sm + a.rows;
  double *sH = shead + kGW * RB;  // H(i, j) at (j - 1)(K + 1) + i - 1
  double *sc = sH + (size_t)(K + 1) * K, *ss = sc + K + 2, *se = ss + K + 2, *sy = se + K + 2;
  double *sh1 = sy + K + 2, *sh2 = sh1 + K + 2;
  unsigned long long *sseen = reinterpret_cast<unsigned long long *>(sh2 + K + 2);
  int32_t *sptr = reinterpret_cast<int32_t *>(sseen + 2 * kDigits * K);
  int32_t *sga = sptr + a.slices + 1, *swsl = sga + kGW + 1;
  __shared__ grid::Scratch<kGT, 1> sred;
  __shared__ double snorm;
  __shared__ int32_t sncut, scut[kGW], srun, sbad;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const grid::Team team{(int)blockIdx.x, (int)gridDim.x};
  if (team.missing(a.stall)) return;
  if (!a.gs->live) return;  // block 0 writes the state after the last wait
  const double econv = a.gs->econv;
  const int s0 = a.cta[blockIdx.x], s1 = a.cta[blockIdx.x + 1], ns = s1 - s0;
  const int row0 = s0 * RB, nrows = min(a.n, s1 * RB) - row0;
  auto H = [&](int i, int j) -> double & { return sH[(size_t)(j - 1) * (K + 1) + i - 1]; };
  auto col = [&](int j) { return a.g + (size_t)(j - 1) * a.n; };
  auto eq_of = [&](int i) { return a.eq ? a.eq[row0 + i] : row0 + i; };
  for (int i = tid; i <= ns; i += kGT) sptr[i] = a.sell_ptr[s0 + i];
  for (int i = tid; i < 2 * kDigits * K; i += kGT) sseen[i] = 0;
  for (int i = tid; i < nrows; i += kGT) {
    const int q = eq_of(i);
    sm[i] = q < 0 ? 0.0 : a.m[q];
  }
  if (tid == 0) sbad = 0;
  __syncthreads();
  if (tid <= kGW) {
    const int total = sptr[ns] - sptr[0], wn = min(kGW, max(4, total / 2 & ~3));
    const int g = sptr[0] + (int)((int64_t)total * min(tid, wn) / wn);
    sga[tid] = g;
    if (tid < kGW) {
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
    for (int k = 1; k < kGW; k++) {
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
  // columns a group ahead, as in persist_pcg (two cycles of 50 steps at 105,840
  // equations: 7.43 / 7.30 ms before and after)
  const int first = sga[w] < sga[w + 1] ? sell_ld<true>(a.sell_col + (size_t)sga[w] * R + lane) : 0;
  // sw = K v over the block's rows
  auto product = [&](const double *v) {
    int g = sga[w], sl = swsl[w], next = first;
    const int gend = sga[w + 1];
    while (g < gend) {
      const int ge = min(sptr[sl + 1], gend);
      double *dst = g == sptr[sl] ? sw + sl * RB : shead + w * RB;
      double acc[B];
#pragma unroll
      for (int b = 0; b < B; b++) acc[b] = 0.0;
      for (; g < ge; g++) {
        double bv[BB];
        const int J = next;
        if (g + 1 < gend) next = sell_ld<true>(a.sell_col + (size_t)(g + 1) * R + lane);
        sell_load<double, B, true>(a.sval + (size_t)g * BB * R, lane, bv);
#pragma unroll
        for (int b = 0; b < B; b++) {
          const double xb = v[J * B + b];
#pragma unroll
          for (int c = 0; c < B; c++) acc[c] += bv[c * B + b] * xb;
        }
      }
      if (sl * RB + lane * B < nrows)
#pragma unroll
        for (int b = 0; b < B; b++) dst[lane * B + b] = acc[b];
      sl++;
    }
    __syncthreads();
    for (int q = tid; q < sncut * RB; q += kGT) {
      const int c = scut[q / RB], i = q % RB;
      const int s = c & 0xffff, k0 = c >> 16 & 0xff, n = c >> 24;
      double t = sw[s * RB + i];
      for (int k = 0; k < n; k++) t += shead[(k0 + k) * RB + i];
      sw[s * RB + i] = t;
    }
    __syncthreads();
  };
  // h[j] = (w, g_j), j = 1..i, over all blocks: warp w takes j = w + 1, w + 17, ...
  auto project = [&](int pass, int i, double *h) {
    for (int j = w + 1; j <= i; j += kGW) {
      const double *g = col(j) + row0;
      double v = 0.0;
#pragma unroll 4
      for (int q = lane; q < nrows; q += 32) v += sw[q] * g[q];
      const FixSum f = warp_sum(fix_of(v));
      grid::digit_add<1>(&a.dots[(size_t)pass * K + j - 1].words, f, -120);
      // kept for the slots, where a digit window cannot hold the sum
      if (lane == 0) h[j] = fix_value(f);
    }
    for (int j = w + 1; j <= i; j += kGW) {
      GmresDot &d = a.dots[(size_t)pass * K + j - 1];
      unsigned long long *ps = sseen + ((size_t)pass * K + j - 1) * kDigits;
      unsigned long long seen = lane < kDigits ? ps[lane] : 0;
      __syncwarp();
      FixSum f = fix_of(h[j]);
      const bool ok = grid::digit_read<1>(team, d.slot, &d.words, f, -120, seen, i);
      if (lane < kDigits) ps[lane] = seen;
      if (lane == 0) {
        h[j] = fix_value(f);
        if (!ok) sbad = 1;
      }
      __syncwarp();
    }
    __syncthreads();
  };
  // w -= sum_j h[j] g_j
  auto subtract = [&](int i, const double *h) {
    for (int q = tid; q < nrows; q += kGT) {
      const double *g = a.g + row0 + q;
      double t0 = sw[q], t1 = 0.0;
      int j = 0;
#pragma unroll 2
      for (; j + 1 < i; j += 2) {
        t0 -= h[j + 1] * g[(size_t)j * a.n];
        t1 += h[j + 2] * g[(size_t)(j + 1) * a.n];
      }
      if (j < i) t0 -= h[j + 1] * g[(size_t)j * a.n];
      sw[q] = t0 - t1;
    }
    __syncthreads();
  };
  uint64_t epoch = 0;
  uint32_t barriers = 0;
  unsigned long long none = 0;
  // snorm = ||w||; meanwhile: `beside` in the other warps
  auto norm = [&](auto beside) {
    double v[1] = {0.0};
    for (int q = tid; q < nrows; q += kGT) v[0] += sw[q] * sw[q];
    epoch++;
    return grid::sum<kGT, 1>(team, v, a.sync, 0, nullptr, none, epoch, sred,
                             [&](double t) { snorm = sqrt(t); }, beside);
  };
#define ELX_GIVE_UP                          \
  do {                                       \
    if (tid == 0) atomicExch(a.err, 2);      \
    return;                                  \
  } while (0)
  // restart (Iters.f:627-646): g_1 = M (b - K x) / ||.||, e(1) = ||.||
  product(a.xr);
  for (int i = tid; i < nrows; i += kGT) {
    const int q = eq_of(i);
    sw[i] = ((q < 0 ? 0.0 : a.b[q]) - sw[i]) * sm[i];
  }
  __syncthreads();
  if (!norm([] {})) ELX_GIVE_UP;
  if (tid == 0) se[1] = snorm;
  for (int q = tid; q < nrows; q += kGT) a.g[row0 + q] = sw[q] / snorm;
  if (!grid::barrier<kGT, 1>(team, a.sync, ++barriers, sred)) ELX_GIVE_UP;
  int ni = 0;
  for (int i = 1; i <= K; i++) {
    product(col(i));
    for (int q = tid; q < nrows; q += kGT) sw[q] *= sm[q];
    __syncthreads();
    project(0, i, sh1);
    if (sbad) ELX_GIVE_UP;
    subtract(i, sh1);
    project(1, i, sh2);
    if (sbad) ELX_GIVE_UP;
    subtract(i, sh2);
    // the norm of w; beside it the stored rotations applied to column i
    // (Iters.f:681-690)
    if (!norm([&] {
          if (w != 1) return;
          for (int j = 1 + lane; j <= i; j += 32) H(j, i) = sh1[j] + sh2[j];
          __syncwarp();
          if (lane == 0) {
            double h = H(1, i);
            for (int j = 1; j <= i - 1; j++) {
              const double h1 = H(j + 1, i);
              H(j, i) = sc[j] * h + ss[j] * h1;
              h = -ss[j] * h + sc[j] * h1;
            }
            H(i, i) = h;
          }
        }))
      ELX_GIVE_UP;
    ni = i;
    // the new rotation and the residual estimate (Iters.f:691-704) in one warp
    // beside the new basis vector
    if (tid == kGT - 32) {
      const double hi = H(i, i), hn = snorm, rr = sqrt(hi * hi + hn * hn);
      sc[i] = hi / rr;
      ss[i] = hn / rr;
      H(i, i) = rr;
      se[i + 1] = -ss[i] * se[i];
      se[i] = sc[i] * se[i];
      srun = !(fabs(se[i + 1]) <= econv || i == K);
    }
    {
      double *g = col(i + 1) + row0;
      for (int q = tid; q < nrows; q += kGT) g[q] = sw[q] / snorm;
    }
    if (!grid::barrier<kGT, 1>(team, a.sync, ++barriers, sred)) ELX_GIVE_UP;
    if (!srun) break;
  }
#undef ELX_GIVE_UP
  // back-substitution H y = e by columns (Iters.f:710-717), one warp
  if (w == 0) {
    for (int j = 1 + lane; j <= ni; j += 32) sy[j] = se[j];
    __syncwarp();
    for (int j = ni; j >= 1; j--) {
      const double yj = sy[j] / H(j, j);
      __syncwarp();
      if (lane == 0) sy[j] = yj;
      for (int i = 1 + lane; i < j; i += 32) sy[i] -= H(i, j) * yj;
      __syncwarp();
    }
  }
  __syncthreads();
  // x += sum_j y(j) g_j (Iters.f:721-725)
  for (int q = tid; q < nrows; q += kGT) {
    const double *g = a.g + row0 + q;
    double t = a.xr[row0 + q];
#pragma unroll 4
    for (int j = 0; j < ni; j++) t += sy[j + 1] * g[(size_t)j * a.n];
    a.xr[row0 + q] = t;
    const int e = eq_of(q);
    if (e >= 0) a.x[e] = t;
  }
  if (blockIdx.x == 0 && tid == 0) {
    GmresState &S = *a.gs;
    S.ni = ni;
    S.nit += ni;
    S.cycles += 1;
    S.run = 0;
    S.conv_flag = fabs(se[ni + 1]) <= econv;
    if (S.conv_flag) {
      S.live = 0;
      S.done = 1;
    } else if (S.cycles >= S.maxit) {
      S.live = 0;
      S.done = 1;
      S.status = ELX_ERR_NO_CONVERGENCE;
    }
  }
}

}  // namespace
}  // namespace elx

namespace elx_api {

// Whether a resident cycle of GMRES(k) costs less than its launches.  It saves
// the launches of k (k + 1) / 2 projections and reads the basis four times a
// step where they read it twice, which weighs more the larger the matrix and
// the shorter the cycle; with k = 1 it saves three launches and pays its own
// start.  Launches / resident, us a cycle: QUAD4 of 9,728 equations k = 1 50 / 52,
// k = 2 74 / 68; TRIA3 of 401,000 k = 3 191 / 206, 6 399 / 371; QUAD4 of 701,400
// k = 8 803 / 816, 12 1,381 / 1,271; TRIA3 of 1,261,800 k = 24 6,219 / 6,356, 32
// 10,109 / 9,851; HEXA8 of 9,450 k = 1 78 / 55; of 285,660 k = 1 164 / 155; of
// 669,780 k = 8 1,449 / 1,482, 12 2,304 / 2,260; of 1,299,600 k = 24 9,931 /
// 12,043.  With partly fixed nodes the launches' product is the scalar gather:
// TRIA3 of 1,261,600 k = 1 359 / 240, HEXA8 of 9,450 k = 1 49 / 57, 2 76 / 68.
static bool gmres_cycle_pays(const elx_ctx *c, int k) {
  const double n = c->s.neq;
  if (!c->use_blocks) return k > 1 || n > 1.5e5;
  return k >= (c->s.bsize == 3 ? 0.5 + n * n / 5e10 : 2.0 + n * n / 6e10);
}

// Plans the cooperative cycle of GMRES(k) (its basis by rows of the sliced
// matrix); false: krylov_ns.cu's launches are used.
bool ensure_gmres_persist(elx_ctx *c, int k) {
  if (!gmres_cycle_pays(c, k) || !ensure_persist(c)) return false;
  int limit = 0;
  ELX_CUDA(cudaDeviceGetAttribute(&limit, cudaDevAttrMaxSharedMemoryPerBlockOptin, c->device));
  const int B = c->use_blocks ? c->s.bsize : c->s.p_bsize;
  const size_t need = B == 3 ? elx::gmres_smem<3>(c->persist_rows, c->persist_slices, k)
                             : elx::gmres_smem<2>(c->persist_rows, c->persist_slices, k);
  return need + 2048 <= (size_t)limit;
}

size_t gmres_persist_bytes(int k) { return sizeof(elx::GmresDot) * 2 * (size_t)k; }

// One restart cycle; `basis` (k + 1, rows), `xr` (rows) x by rows, `dots` of
// gmres_persist_bytes(k).
void gmres_persist_cycle(elx_ctx *c, int k, double *basis, double *xr, void *dots) {
  elx::GmresArgs a;
  const bool padded = !c->use_blocks;
  const int B = padded ? c->s.p_bsize : c->s.bsize;
  a.n = persist_rows(c);
  a.neq = c->s.neq;
  a.k = k;
  a.sell_ptr = (padded ? c->p_ptr : c->sell_ptr).as<int32_t>();
  a.sell_col = (padded ? c->p_col : c->sell_col).as<int32_t>();
  a.sval = (padded ? c->p_val : c->sell_val64).as<double>();
  a.cta = c->persist_cta.as<int32_t>();
  a.eq = padded ? c->p_eq.as<int32_t>() : nullptr;
  a.b = c->b.as<double>();
  a.m = c->m.as<double>();
  a.x = c->xs.as<double>();
  a.xr = xr;
  a.g = basis;
  a.gs = c->gstate.as<elx::GmresState>();
  a.sync = c->persist_sync.as<elx::GridSync>();
  a.dots = static_cast<elx::GmresDot *>(dots);
  a.err = c->flags.as<int32_t>() + 2;
  a.rows = c->persist_rows;
  a.slices = c->persist_slices;
  a.stall = elx::grid_stall();
  ELX_CUDA(cudaMemsetAsync(a.sync, 0, sizeof(elx::GridSync), c->stream));
  ELX_CUDA(cudaMemsetAsync(dots, 0, gmres_persist_bytes(k), c->stream));
  const void *f = B == 3 ? (const void *)elx::gmres_persist_kernel<3>
                         : (const void *)elx::gmres_persist_kernel<2>;
  const size_t bytes = B == 3 ? elx::gmres_smem<3>(a.rows, a.slices, k)
                              : elx::gmres_smem<2>(a.rows, a.slices, k);
  ELX_CUDA(elx::allow_shared(f));
  void *args[] = {&a};
  ELX_CUDA(cudaLaunchCooperativeKernel(f, dim3(c->persist_grid), dim3(elx::kGT), args, bytes,
                                       c->stream));
  c->launches += 1;
}

}  // namespace elx_api
