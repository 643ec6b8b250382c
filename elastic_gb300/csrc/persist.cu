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
// equations, QUAD4), 19.8 -> 9.9 (90,902, TRIA3), 33.1 -> 11.2 (26,460,
// HEXA8), 72.2 -> 60.3 (345,744, HEXA8), 142 -> 127 (811,200, HEXA8: the
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
// A small matrix and one load case run as one cluster of up to 16 blocks:
// the sums go through the blocks' shared memory and the hardware's cluster
// barrier takes the place of the polls in L2 (2,176 equations: 7.4 -> 5.4 us an
// iteration; 512 threads a block measured as good as 256, 128 slower).
//
// Inside a block every warp takes the same number of slot groups (the FP64
// pipe is charged per warp instruction; one group in flight measured faster
// than two, 130 against 134 us at 811,200 equations); a slice cut between
// warps is summed by its first warp and the heads of the following ones, in
// warp order, so results do not depend on timing.
#include <algorithm>
#include <cstddef>
#include <cstdlib>

#include "elx_context.h"
#include "elx_persist.cuh"

namespace elx {
namespace {

constexpr int kPT = 512;  // threads of a block
// Clocks that an iteration's waits are shorter in a cluster than in a grid
// (net of its longer vector passes).  Either side of the line, clocks that
// the products are longer and us an iteration as grid / cluster: 1,200 (3,720
// TRIA3 equations) 6.84 / 5.47, 1,700 (2,187, HEXA8) 9.24 / 8.92, then 3,100
// (8,160, TRIA3) 7.07 / 7.23, 3,500 (7,140, QUAD4) 7.23 / 7.34, 3,900 (3,000,
// HEXA8) 9.21 / 9.28.  With two columns nothing is left at 2,176 equations
// (8.9 / 8.7).
constexpr double kClusterGain = 2800;

template <int B, int NC, bool SMEM>
__global__ void __launch_bounds__(kPT, 1)
pcg_persist_kernel(PersistArgs a, int start, int steps) {
  const grid::Team team{(int)blockIdx.x, (int)gridDim.x};
  if (team.missing(a.stall)) return;
  persist_pcg<kPT, B, NC, SMEM>(a, team, start, steps, 0);
}

// The same by one cluster: grid::Cluster's sums and barrier.
template <int B>
__global__ void __launch_bounds__(kPT, 1)
pcg_cluster_kernel(PersistArgs a, int start, int steps) {
  __shared__ __align__(16) FixSum slots[2][1][kClusterBlocks];
  ptx::cluster_arrive();  // the other blocks' shared memory is there
  ptx::cluster_wait();
  persist_pcg<kPT, B, 1, true>(a, grid::Cluster<1>{(int)blockIdx.x, (int)gridDim.x, slots}, start,
                               steps, 0);
}

template <int B, int NC>
size_t smem_of(bool in_smem, int rows, int slices) {
  return in_smem ? persist_smem<kPT, B, NC, true>(rows, slices)
                 : persist_smem<kPT, B, NC, false>(rows, slices);
}

template <int B, int NC>
void launch(const PersistArgs &a, int grid, bool in_smem, int start, int steps, cudaStream_t st) {
  const void *f = in_smem ? (const void *)pcg_persist_kernel<B, NC, true>
                          : (const void *)pcg_persist_kernel<B, NC, false>;
  const size_t bytes = smem_of<B, NC>(in_smem, a.rows, a.slices);
  ELX_CUDA(allow_shared(f));
  PersistArgs arg = a;
  void *args[] = {&arg, &start, &steps};
  ELX_CUDA(cudaLaunchCooperativeKernel(f, dim3(grid), dim3(kPT), args, bytes, st));
}

// `n` blocks as one cluster: the launch, or with `fit` whether the GPU takes
// it (*fit > 0).
template <int B>
cudaError_t cluster_call(const PersistArgs &a, int n, int start, int steps, cudaStream_t st,
                         int *fit) {
  auto f = pcg_cluster_kernel<B>;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(n);
  cfg.blockDim = dim3(kPT);
  cfg.dynamicSmemBytes = persist_smem<kPT, B, 1, true>(a.rows, a.slices);
  cfg.stream = st;
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = n;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  cudaError_t e = allow_shared(f);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e != cudaSuccess) return e;
  return fit ? cudaOccupancyMaxActiveClusters(fit, f, &cfg)
             : cudaLaunchKernelEx(&cfg, f, a, start, steps);
}

cudaError_t cluster_call(int B, const PersistArgs &a, int n, int start, int steps,
                         cudaStream_t st, int *fit) {
  return B == 3 ? cluster_call<3>(a, n, start, steps, st, fit)
                : cluster_call<2>(a, n, start, steps, st, fit);
}

// A block of it has an SM to itself, as the resident kernels' blocks have.
__global__ void residency_kernel() {}

// Whether `grid` blocks of one per SM can run at the same time: not in a process
// that has a part of the GPU's SMs, which the occupancy calls do not know of.
bool resident_together(int grid, cudaStream_t st) {
  cudaFuncAttributes at;
  ELX_CUDA(allow_shared(residency_kernel));
  ELX_CUDA(cudaFuncGetAttributes(&at, residency_kernel));
  const cudaError_t e =
      cudaLaunchCooperativeKernel((const void *)residency_kernel, dim3(grid), dim3(kPT), nullptr,
                                  at.maxDynamicSharedSizeBytes, st);
  if (e == cudaSuccess) return true;
  cudaGetLastError();
  ELX_REQUIRE(e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorNotSupported, ELX_ERR_CUDA,
              cudaGetErrorString(e));
  return false;
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

int grid_stall() {
  const char *env = getenv("ELX_GRID_STALL_TEST");
  return env && atoi(env) == 1 ? 1 : 0;
}

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
    const char *env = getenv("ELX_RESIDENT_BLOCKS");
    const int want = env ? std::max(1, atoi(env)) : elx::sm_count();
    const int grid = std::min({want, elx::kGridMaxBlocks, nslices});
    if (!elx::resident_together(grid, c->stream)) return false;
    std::vector<int32_t> cuts = elx::persist_cuts(ptr, grid);
    const int cl = std::min(elx::kClusterBlocks, nslices);
    const std::vector<int32_t> ccuts = elx::persist_cuts(ptr, cl);
    int slices = 0;
    for (int k = 0; k < grid; k++) slices = std::max(slices, cuts[k + 1] - cuts[k]);
    const int rows = slices * elx::kSliceRows * B;
    int limit = 0;
    ELX_CUDA(cudaDeviceGetAttribute(&limit, cudaDevAttrMaxSharedMemoryPerBlockOptin, c->device));
    limit -= 2048;  // the kernel's static arrays
    // ELX_RESIDENT_MODE=1: the vectors in L2 whatever fits shared memory, 0: the
    // launches
    const char *mode_env = getenv("ELX_RESIDENT_MODE");
    const int most = mode_env ? atoi(mode_env) : 2;
    for (int nc = 1; nc <= elx::kGridCols; nc++) {
      const int mode = elx::smem_bytes(B, nc, true, rows, slices) <= (size_t)limit    ? 2
                       : elx::smem_bytes(B, nc, false, rows, slices) <= (size_t)limit ? 1
                                                                                      : 0;
      c->persist_mode[nc] = std::min(mode, most);
    }
    if (!c->persist_mode[1]) return false;
    // one cluster in place of the grid, for a small matrix
    cuts.insert(cuts.end(), ccuts.begin(), ccuts.end());
    elx::PersistArgs ca = {};
    for (int k = 0; k < cl; k++) ca.slices = std::max(ca.slices, ccuts[k + 1] - ccuts[k]);
    ca.rows = ca.slices * elx::kSliceRows * B;
    // by how many clocks its blocks' products are longer: 16 of an SM's FP64
    // pipe for each entry of a group
    const double longer = ptr[nslices] * (1.0 / cl - 1.0 / grid) * 16 * B * B;
    int fit = 0;
    if (longer <= elx::kClusterGain && most == 2 &&
        elx::smem_bytes(B, 1, true, ca.rows, ca.slices) <= (size_t)limit &&
        elx::cluster_call(B, ca, cl, 0, 0, c->stream, &fit) != cudaSuccess) {
      cudaGetLastError();  // no such cluster on this device
      fit = 0;
    }
    try {
      c->upload(c->persist_cta, cuts.data(), cuts.size());
      c->alloc(c->persist_sync, sizeof(elx::GridSync) + sizeof(elx::PersistState));
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
      c->drop_persist(-1);  // a memory budget without room for it
      return false;
    }
    c->sync();
    c->persist_rows = rows;
    c->persist_slices = slices;
    c->persist_grid = grid;
    c->cluster_grid = fit > 0 ? cl : 0;
    c->cluster_rows = ca.rows;
    c->cluster_slices = ca.slices;
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

// Makes the plan's vectors `bytes` long.  False: the memory budget has no room
// for that; one column's are there again (alloc gives the old ones back first),
// or there is no plan any more.
bool persist_vectors(elx_ctx *c, size_t bytes) {
  if (c->persist_vec.bytes >= bytes) return true;
  for (size_t n : {bytes, 3 * 8 * (size_t)persist_rows(c)}) {
    try {
      c->alloc(c->persist_vec, n);
      return n == bytes;
    } catch (const Error &e) {
      if (e.code != ELX_ERR_OOM) throw;
    }
  }
  c->drop_persist(-1);
  return false;
}

elx::PersistState *persist_state(const elx_ctx *c) {
  return reinterpret_cast<elx::PersistState *>(c->persist_sync.as<elx::GridSync>() + 1);
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
  elx::PersistState *state = persist_state(c);
  a.cols = state->col;
  a.err = &state->err;
  a.stall = elx::grid_stall();
  a.tol = tol;
  a.maxit = maxit;
  a.rows = c->persist_rows;
  a.slices = c->persist_slices;
  const bool cluster = nc == 1 && c->cluster_grid;
  if (cluster) {
    a.cta += c->persist_grid + 1;
    a.rows = c->cluster_rows;
    a.slices = c->cluster_slices;
  }
  const bool in_smem = c->persist_mode[nc] == 2;
  const int max_launches = maxit / steps + 2;
  int launched = 0, checked = 0;
  auto go = [&] {
    const int slot = launched & 1, start = launched == 0;
    if (cluster) {
      ELX_CUDA(elx::cluster_call(B, a, c->cluster_grid, start, steps, c->stream, nullptr));
    } else {
      // a solve's first launch finds no states and no error of an earlier one
      ELX_CUDA(cudaMemsetAsync(a.gs, 0,
                               sizeof(elx::GridSync) + (start ? offsetof(elx::PersistState, diag) : 0),
                               c->stream));
#define CALL(NC)                                                                     \
  if (B == 3)                                                                        \
    elx::launch<3, NC>(a, c->persist_grid, in_smem, start, steps, c->stream);        \
  else                                                                               \
    elx::launch<2, NC>(a, c->persist_grid, in_smem, start, steps, c->stream)
      ELX_NC_DISPATCH(nc, CALL)
#undef CALL
    }
    c->launches += 1;
    ELX_CUDA(cudaMemcpyAsync(c->h_state + slot, state, offsetof(elx::PersistState, diag),
                             cudaMemcpyDeviceToHost, c->stream));
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
    const elx::PersistState &hs = c->h_state[checked & 1];
    const elx::PersistCol *h = hs.col;
    ELX_CUDA(cudaEventSynchronize(c->ev[checked & 1]));
    checked++;
    if (hs.err && !cluster) {  // the states were not written; a cluster has no such waits
      c->sync();
      throw Error{ELX_ERR_TIMEOUT, kResidentWait};
    }
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
