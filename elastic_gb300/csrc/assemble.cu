// Element stiffness integration and CSRC assembly on the GPU:
// pform_mec(isw=2, lhs=.true., rhs=.true.) of mef/src/Pform.f:1-254 with the
// element routines of Elmlib02.f (elmt02..07_mec, isw=2) and the CSR
// scatter of Assbly.f:66-146.
//
// One thread per element.  Elements are processed colour by colour (no two
// elements of a colour share a node), so every read-modify-write of ad, al
// and b is race free without atomics, and the summation order of each entry
// is fixed by the colour order: results are deterministic.
//
// Scatter without search: the reference finds the column of each entry by a
// linear search of the row (Assbly.f:124-128).  Here a node's free equations
// are consecutive and the blocks of two nodes are disjoint, so inside the
// rows of the higher node the lower node's columns form one contiguous run at
// an offset that is the same for every dof row; the host precomputes that
// offset per element and node pair (the slot map).  A node's own lower
// columns are the last entries of its rows.
//
// Stiffness blocks.  For the isotropic 3-D law of elmt06/07_mec the 3x3 block
// of nodes (i, j) at one integration point is
//   wt1 * ( b * g_i g_j^T + c * g_j g_i^T + c * (g_i . g_j) I ),
// using b + 2c = 1 with a, b, c of Elmlib02.f:1697-1705.  Summed over the
// points it only needs M_ij = sum_gp wt1 g_i g_j^T, so each block costs 9
// FMAs per point instead of the ~36 operations of the reference's expanded
// form (Elmlib02.f:1747-1772).  The 2-D laws use the same M_ij with
// d11, d12, d22, d33 (Elmlib02.f:781-795).  Rounding differs from the
// reference's operand order by a few ulps; the assembled values agree to
// well below 1e-13 relative.
#include <cstdlib>
#include <mutex>
#include <type_traits>

#include "elx_internal.h"

namespace elx {
namespace {

// Gauss-Legendre 2-point abscissa (Elmlib.f:2987), weights 1 (Elmlib.f:3018).
__device__ __constant__ double kPg2[2] = {-.577350269189626e0, .577350269189626e0};

struct Law {
  double d11, d12, d22, d33;  // 2-D constitutive terms
  double a, b, c;             // 3-D factors of elmt06/07_mec
  double thic;                // QUAD4 plane-stress thickness
};

// Constitutive constants of the element routines (Elmlib02.f:179-186 plane
// strain, 469-476 plane stress, 1331-1338 / 1697-1705 3-D).
__device__ Law make_law(int iel, const double *e) {
  Law L{};
  const double ym = e[0], ps = e[1];
  if (iel == TRIA3_STRESS || iel == QUAD4_STRESS) {
    const double a1 = 1.0 - ps, a2 = 1.0 - ps * ps;
    const double a = ym / a2, b = ps, c = 0.5 * a1;
    L.d11 = a; L.d12 = a * b; L.d22 = a; L.d33 = a * c;
    L.thic = e[2] == 0.0 ? 1.0 : e[2];
  } else {
    const double a1 = 1.0 - ps, a2 = 1.0 - 2.0 * ps, a3 = 1.0 + ps;
    const double a = (ym * a1) / (a3 * a2), b = ps / a1, c = 0.5 * (a2 / a1);
    L.d11 = a; L.d12 = a * b; L.d22 = a; L.d33 = a * c;
    L.a = a; L.b = b; L.c = c;
    L.thic = 1.0;
  }
  return L;
}

// Everything one thread needs to scatter blocks of its element.
template <int NEN, int NDF>
struct Elem {
  int eq[NEN][NDF];  // 0-based equation or -1
  int first[NEN];    // smallest equation of the node, -1 if none free
  double u[NEN][NDF];
  double p[NEN][NDF];  // p = K_e u_e (lku_m, Elmlib.f:336-368)
};

// Pair index of local nodes lo < hi in the host's slot-map order (pairs
// enumerated lo-major over the mesh's nen nodes per element).
__device__ __forceinline__ int pair_index(int nen, int lo, int hi) {
  return lo * (nen - 1) - (lo * (lo - 1)) / 2 + (hi - lo - 1);
}

// The matrix entries an element adds to: their places and present values, all
// loaded before the geometry is computed and stored at the end.  One thread
// per element has few others to hide behind (20,000 threads a colour on the
// 48^3 TETRA4 mesh), and a read-modify-write at a time waited for L2 once per
// entry: 94 us a colour there, 40 here; QUAD4 64 x 16: 62 us, 28 here; TRIA3 301
// x 150: 26 us, 13 here.
template <int NEN, int NDF>
struct Entries {
  static constexpr int NP = NEN * (NEN - 1) / 2;
  int base[NP][NDF];  // row starts plus the run's offset, less its first column
  bool on[NP], rows_a[NP];
  double old[NP][NDF][NDF], dold[NEN][NDF][NDF];
  int dend[NEN][NDF];

  // pair (a, b), b < a: the rows of the higher node, the columns of the lower
  static __device__ __forceinline__ constexpr int at(int a, int b) { return a * (a - 1) / 2 + b; }

  __device__ __forceinline__ void load(const Elem<NEN, NDF> &E, const CsrcDev &k,
                                       const MeshDev &m, int t) {
#pragma unroll
    for (int a = 1; a < NEN; a++)
#pragma unroll
      for (int b = 0; b < a; b++) {
        const int q = at(a, b), fa = E.first[a], fb = E.first[b];
        on[q] = fa >= 0 && fb >= 0;
        rows_a[q] = fa > fb;
        const int off = m.slot[(size_t)pair_index(m.nen, b, a) * m.numel + t] -
                        (rows_a[q] ? fb : fa);
#pragma unroll
        for (int r = 0; r < NDF; r++) {
          const int row = rows_a[q] ? E.eq[a][r] : E.eq[b][r];
          base[q][r] = on[q] && row >= 0 ? k.ia[row] + off : 0;
        }
      }
#pragma unroll
    for (int a = 0; a < NEN; a++)
#pragma unroll
      for (int r = 0; r < NDF; r++) {
        const int row = E.eq[a][r];
        dend[a][r] = row >= 0 ? k.ia[row + 1] : 0;
        dold[a][r][r] = row >= 0 ? k.ad[row] : 0.0;
      }
#pragma unroll
    for (int a = 1; a < NEN; a++)
#pragma unroll
      for (int b = 0; b < a; b++) {
        const int q = at(a, b);
#pragma unroll
        for (int r = 0; r < NDF; r++)
#pragma unroll
          for (int c = 0; c < NDF; c++) {
            const int row = rows_a[q] ? E.eq[a][r] : E.eq[b][r];
            const int col = rows_a[q] ? E.eq[b][c] : E.eq[a][c];
            old[q][r][c] = on[q] && row >= 0 && col >= 0 ? k.al[base[q][r] + col] : 0.0;
          }
      }
    // a node's own lower columns are the last entries of its rows (column c of
    // row r at ia[r + 1] - (r - c))
#pragma unroll
    for (int a = 0; a < NEN; a++)
#pragma unroll
      for (int r = 0; r < NDF; r++)
#pragma unroll
        for (int c = 0; c < r; c++) {
          const int row = E.eq[a][r], col = E.eq[a][c];
          dold[a][r][c] = row >= 0 && col >= 0 ? k.al[dend[a][r] - (row - col)] : 0.0;
        }
  }
};

// Adds the block K_ab (rows = dofs of local node a, columns = dofs of b) of a
// node pair b < a to al, and both directions of K u to p.
template <int NEN, int NDF>
__device__ __forceinline__ void scatter_pair(Elem<NEN, NDF> &E, const Entries<NEN, NDF> &N,
                                             const CsrcDev &k, int a, int b,
                                             const double (&K)[NDF][NDF], bool with_u) {
  if (with_u) {
#pragma unroll
    for (int r = 0; r < NDF; r++)
#pragma unroll
      for (int c = 0; c < NDF; c++) {
        E.p[a][r] += K[r][c] * E.u[b][c];
        E.p[b][c] += K[r][c] * E.u[a][r];
      }
  }
  const int q = Entries<NEN, NDF>::at(a, b);
  if (!N.on[q]) return;
#pragma unroll
  for (int r = 0; r < NDF; r++)
#pragma unroll
    for (int c = 0; c < NDF; c++) {
      const int row = N.rows_a[q] ? E.eq[a][r] : E.eq[b][r];
      const int col = N.rows_a[q] ? E.eq[b][c] : E.eq[a][c];
      if (row >= 0 && col >= 0)
        k.al[N.base[q][r] + col] = N.old[q][r][c] + (N.rows_a[q] ? K[r][c] : K[c][r]);
    }
}

// Diagonal block of node a: ad and the node's own lower entries.
template <int NEN, int NDF>
__device__ __forceinline__ void scatter_diag(Elem<NEN, NDF> &E, const Entries<NEN, NDF> &N,
                                             const CsrcDev &k, int a,
                                             const double (&K)[NDF][NDF], bool with_u) {
  if (with_u) {
#pragma unroll
    for (int r = 0; r < NDF; r++)
#pragma unroll
      for (int c = 0; c < NDF; c++) E.p[a][r] += K[r][c] * E.u[a][c];
  }
#pragma unroll
  for (int r = 0; r < NDF; r++) {
    const int row = E.eq[a][r];
    if (row < 0) continue;
    k.ad[row] = N.dold[a][r][r] + K[r][r];
#pragma unroll
    for (int c = 0; c < r; c++) {
      const int col = E.eq[a][c];
      if (col >= 0) k.al[N.dend[a][r] - (row - col)] = N.dold[a][r][c] + K[r][c];
    }
  }
}

// Returns whether the element has a non-zero displacement (one without adds
// nothing to b; the first solvm pass has u = 0 away from prescribed values).
template <int NEN, int NDF>
__device__ __forceinline__ bool load_elem(Elem<NEN, NDF> &E, const MeshDev &m, int t,
                                          const int (&node)[NEN], const double *u) {
  bool nz = false;
#pragma unroll
  for (int a = 0; a < NEN; a++) {
    int f = -1;
#pragma unroll
    for (int d = NDF - 1; d >= 0; d--) {
      const int q = m.eq[(size_t)node[a] * NDF + d];
      E.eq[a][d] = q;
      if (q >= 0) f = q;
      E.u[a][d] = u ? u[(size_t)node[a] * NDF + d] : 0.0;
      E.p[a][d] = 0.0;
      nz = nz || E.u[a][d] != 0.0;
    }
    E.first[a] = f;
  }
  return nz;
}

// b(k) = b(k) - p(i) for free dofs (Assbly.f:118).
template <int NEN, int NDF>
__device__ __forceinline__ void finish_rhs(const Elem<NEN, NDF> &E, double *b) {
  if (b == nullptr) return;
#pragma unroll
  for (int a = 0; a < NEN; a++)
#pragma unroll
    for (int d = 0; d < NDF; d++)
      if (E.eq[a][d] >= 0) b[E.eq[a][d]] -= E.p[a][d];
}

__device__ __forceinline__ void mark_bad(int32_t *bad, int elnum) { atomicMin(bad, elnum); }

// 2-D block from M = sum wt g_i g_j^T (rows x, y).
__device__ __forceinline__ void block2d(const Law &L, const double (&M)[2][2],
                                        double (&K)[2][2]) {
  K[0][0] = L.d11 * M[0][0] + L.d33 * M[1][1];
  K[0][1] = L.d12 * M[0][1] + L.d33 * M[1][0];
  K[1][0] = L.d12 * M[1][0] + L.d33 * M[0][1];
  K[1][1] = L.d22 * M[1][1] + L.d33 * M[0][0];
}

// 3-D block from M = sum wt1 g_i g_j^T: b M + c M^T + c tr(M) I.
__device__ __forceinline__ void block3d(const Law &L, const double (&M)[3][3],
                                        double (&K)[3][3]) {
  const double tr = L.c * (M[0][0] + M[1][1] + M[2][2]);
#pragma unroll
  for (int r = 0; r < 3; r++)
#pragma unroll
    for (int c = 0; c < 3; c++) K[r][c] = L.b * M[r][c] + L.c * M[c][r] + (r == c ? tr : 0.0);
}

// ---------------------------------------------------------------- TRIA3
// elmt02_mec / elmt03_mec (Elmlib02.f:50-627): constant-strain triangle,
// wt1 = det/2; the plane-stress thickness is not applied to K (as there).
__global__ void __launch_bounds__(64) tria3_kernel(MeshDev m, CsrcDev k, int begin, int end, int iel,
                             const double *__restrict__ u, double *__restrict__ b,
                             int32_t *bad) {
  const int t = begin + blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= end) return;
  int node[3];
#pragma unroll
  for (int a = 0; a < 3; a++) node[a] = m.conn[(size_t)a * m.numel + t];
  Elem<3, 2> E;
  const bool with_u = load_elem<3, 2>(E, m, t, node, u);
  Entries<3, 2> N;
  N.load(E, k, m, t);
  double xl[3][2];
#pragma unroll
  for (int a = 0; a < 3; a++) {
    xl[a][0] = m.x[(size_t)node[a] * m.ndm + 0];
    xl[a][1] = m.x[(size_t)node[a] * m.ndm + 1];
  }
  const double xj11 = xl[0][0] - xl[2][0], xj12 = xl[0][1] - xl[2][1];
  const double xj21 = xl[1][0] - xl[2][0], xj22 = xl[1][1] - xl[2][1];
  const double det = xj11 * xj22 - xj12 * xj21;
  if (det <= 0.0) { mark_bad(bad, m.elnum[t]); return; }
  const double xji11 = xj22 / det, xji12 = -xj12 / det;
  const double xji21 = -xj21 / det, xji22 = xj11 / det;
  const double g[3][2] = {{xji11, xji21}, {xji12, xji22},
                          {-xji11 - xji12, -xji21 - xji22}};
  const Law L = make_law(iel, m.e + (size_t)m.mat[t] * m.prop);
  const double wt1 = 0.5 * det;
#pragma unroll
  for (int a = 0; a < 3; a++)
#pragma unroll
    for (int bb = 0; bb <= a; bb++) {
      double M[2][2], K[2][2];
#pragma unroll
      for (int r = 0; r < 2; r++)
#pragma unroll
        for (int c = 0; c < 2; c++) M[r][c] = wt1 * g[a][r] * g[bb][c];
      block2d(L, M, K);
      if (a == bb) scatter_diag<3, 2>(E, N, k, a, K, with_u);
      else scatter_pair<3, 2>(E, N, k, a, bb, K, with_u);
    }
  if (with_u) finish_rhs<3, 2>(E, b);
}

// ---------------------------------------------------------------- QUAD4
// elmt04_mec / elmt05_mec (Elmlib02.f:629-1230): 2x2 Gauss with sfquad4_m
// (Elmlib.f:815-886) and jacob2d_m (Elmlib.f:1769-1852).
__global__ void __launch_bounds__(64) quad4_kernel(MeshDev m, CsrcDev k, int begin, int end, int iel,
                             const double *__restrict__ u, double *__restrict__ b,
                             int32_t *bad) {
  const int t = begin + blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= end) return;
  int node[4];
#pragma unroll
  for (int a = 0; a < 4; a++) node[a] = m.conn[(size_t)a * m.numel + t];
  Elem<4, 2> E;
  const bool with_u = load_elem<4, 2>(E, m, t, node, u);
  Entries<4, 2> N;
  N.load(E, k, m, t);
  double xl[4][2];
#pragma unroll
  for (int a = 0; a < 4; a++) {
    xl[a][0] = m.x[(size_t)node[a] * m.ndm + 0];
    xl[a][1] = m.x[(size_t)node[a] * m.ndm + 1];
  }
  const Law L = make_law(iel, m.e + (size_t)m.mat[t] * m.prop);
  double g[4][4][2];  // [gp][node][x,y]
  double wt[4];
#pragma unroll
  for (int ly = 0; ly < 2; ly++)
#pragma unroll
    for (int lx = 0; lx < 2; lx++) {
      const int gp = ly * 2 + lx;
      const double r = kPg2[lx], s = kPg2[ly];
      const double opr = 1.0 + r, ops = 1.0 + s, omr = 1.0 - r, oms = 1.0 - s;
      const double hr[4] = {ops * 0.25, -(ops * 0.25), -(oms * 0.25), oms * 0.25};
      const double hs[4] = {opr * 0.25, omr * 0.25, -(omr * 0.25), -(opr * 0.25)};
      double j11 = 0, j12 = 0, j21 = 0, j22 = 0;
#pragma unroll
      for (int a = 0; a < 4; a++) {
        j11 += hr[a] * xl[a][0];
        j12 += hr[a] * xl[a][1];
        j21 += hs[a] * xl[a][0];
        j22 += hs[a] * xl[a][1];
      }
      const double det = j11 * j22 - j21 * j12;
      if (det <= 1.e-14) { mark_bad(bad, m.elnum[t]); return; }
      const double i11 = j22 / det, i12 = -j12 / det, i21 = -j21 / det, i22 = j11 / det;
#pragma unroll
      for (int a = 0; a < 4; a++) {
        g[gp][a][0] = i11 * hr[a] + i12 * hs[a];
        g[gp][a][1] = i21 * hr[a] + i22 * hs[a];
      }
      wt[gp] = det * L.thic;  // wg(lx)*wg(ly) = 1
    }
#pragma unroll
  for (int a = 0; a < 4; a++)
#pragma unroll
    for (int bb = 0; bb <= a; bb++) {
      double M[2][2] = {{0, 0}, {0, 0}}, K[2][2];
#pragma unroll
      for (int gp = 0; gp < 4; gp++) {
        const double s0 = wt[gp] * g[gp][a][0], s1 = wt[gp] * g[gp][a][1];
        M[0][0] += s0 * g[gp][bb][0];
        M[0][1] += s0 * g[gp][bb][1];
        M[1][0] += s1 * g[gp][bb][0];
        M[1][1] += s1 * g[gp][bb][1];
      }
      block2d(L, M, K);
      if (a == bb) scatter_diag<4, 2>(E, N, k, a, K, with_u);
      else scatter_pair<4, 2>(E, N, k, a, bb, K, with_u);
    }
  if (with_u) finish_rhs<4, 2>(E, b);
}

// --------------------------------------------------------------- TETRA4
// elmt06_mec (Elmlib02.f:1232-1573) with jtetra4 (Elmlib.f:2636-2713):
// constant strain, wt1 = a * det * div6 with the literal div6.
__global__ void __launch_bounds__(64) tetra4_kernel(MeshDev m, CsrcDev k, int begin, int end,
                              const double *__restrict__ u, double *__restrict__ b,
                              int32_t *bad) {
  const int t = begin + blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= end) return;
  int node[4];
#pragma unroll
  for (int a = 0; a < 4; a++) node[a] = m.conn[(size_t)a * m.numel + t];
  Elem<4, 3> E;
  const bool with_u = load_elem<4, 3>(E, m, t, node, u);
  Entries<4, 3> N;
  N.load(E, k, m, t);
  double xl[4][3];
#pragma unroll
  for (int a = 0; a < 4; a++)
#pragma unroll
    for (int d = 0; d < 3; d++) xl[a][d] = m.x[(size_t)node[a] * 3 + d];
  double xj[3][3];
#pragma unroll
  for (int r = 0; r < 3; r++)
#pragma unroll
    for (int d = 0; d < 3; d++) xj[r][d] = xl[r][d] - xl[3][d];
  const double det = xj[0][0] * xj[1][1] * xj[2][2] + xj[0][1] * xj[1][2] * xj[2][0] +
                     xj[0][2] * xj[1][0] * xj[2][1] - xj[2][0] * xj[1][1] * xj[0][2] -
                     xj[0][1] * xj[1][0] * xj[2][2] - xj[0][0] * xj[2][1] * xj[1][2];
  if (det <= 1.e-14) { mark_bad(bad, m.elnum[t]); return; }
  const double deti = 1.0 / det;
  double g[4][3];
  g[0][0] = (xj[1][1] * xj[2][2] - xj[1][2] * xj[2][1]) * deti;
  g[1][0] = (xj[0][2] * xj[2][1] - xj[0][1] * xj[2][2]) * deti;
  g[2][0] = (xj[0][1] * xj[1][2] - xj[0][2] * xj[1][1]) * deti;
  g[0][1] = (xj[1][2] * xj[2][0] - xj[1][0] * xj[2][2]) * deti;
  g[1][1] = (xj[0][0] * xj[2][2] - xj[0][2] * xj[2][0]) * deti;
  g[2][1] = (xj[0][2] * xj[1][0] - xj[0][0] * xj[1][2]) * deti;
  g[0][2] = (xj[1][0] * xj[2][1] - xj[1][1] * xj[2][0]) * deti;
  g[1][2] = (xj[0][1] * xj[2][0] - xj[0][0] * xj[2][1]) * deti;
  g[2][2] = (xj[0][0] * xj[1][1] - xj[0][1] * xj[1][0]) * deti;
#pragma unroll
  for (int d = 0; d < 3; d++) g[3][d] = -g[0][d] - g[1][d] - g[2][d];
  const Law L = make_law(TETRA4, m.e + (size_t)m.mat[t] * m.prop);
  const double div6 = 0.166666666666667e+00;
  const double wt1 = L.a * det * div6;
#pragma unroll
  for (int a = 0; a < 4; a++)
#pragma unroll
    for (int bb = 0; bb <= a; bb++) {
      double M[3][3], K[3][3];
#pragma unroll
      for (int r = 0; r < 3; r++)
#pragma unroll
        for (int c = 0; c < 3; c++) M[r][c] = wt1 * g[a][r] * g[bb][c];
      block3d(L, M, K);
      if (a == bb) scatter_diag<4, 3>(E, N, k, a, K, with_u);
      else scatter_pair<4, 3>(E, N, k, a, bb, K, with_u);
    }
  if (with_u) finish_rhs<4, 3>(E, b);
}

// ---------------------------------------------------------------- HEXA8
// elmt07_mec (Elmlib02.f:1577-2023): 2x2x2 Gauss with sfhexa8_m
// (Elmlib.f:1151-1258) and jacob3d_m (Elmlib.f:1942-2036).  The shape
// function gradients of the 8 points are kept in shared memory, one column
// per thread ([gp][node][xyz][thread]) so that accesses are bank-conflict free.
// (one entry at a time: 36 pairs are too many to load ahead)
// Adds the block K_ab (rows = dofs of local node a, columns = dofs of b) of a
// node pair a != b into al, and both directions of K u into p.
template <int NEN, int NDF>
__device__ __forceinline__ void scatter_pair_rmw(Elem<NEN, NDF> &E, const CsrcDev &k,
                                             const MeshDev &m, int t, int a, int b,
                                             const double (&K)[NDF][NDF], bool with_u) {
  if (with_u) {
#pragma unroll
    for (int r = 0; r < NDF; r++)
#pragma unroll
      for (int c = 0; c < NDF; c++) {
        E.p[a][r] += K[r][c] * E.u[b][c];
        E.p[b][c] += K[r][c] * E.u[a][r];
      }
  }
  const int fa = E.first[a], fb = E.first[b];
  if (fa < 0 || fb < 0) return;
  const int lo = a < b ? a : b, hi = a < b ? b : a;
  const int off = m.slot[(size_t)pair_index(m.nen, lo, hi) * m.numel + t];
  if (fa > fb) {  // rows of a, columns of b
#pragma unroll
    for (int r = 0; r < NDF; r++) {
      const int row = E.eq[a][r];
      if (row < 0) continue;
      const int base = k.ia[row] + off - fb;
#pragma unroll
      for (int c = 0; c < NDF; c++)
        if (E.eq[b][c] >= 0) k.al[base + E.eq[b][c]] += K[r][c];
    }
  } else {  // rows of b, columns of a: entry (b c, a r) = K_ab[r][c]
#pragma unroll
    for (int c = 0; c < NDF; c++) {
      const int row = E.eq[b][c];
      if (row < 0) continue;
      const int base = k.ia[row] + off - fa;
#pragma unroll
      for (int r = 0; r < NDF; r++)
        if (E.eq[a][r] >= 0) k.al[base + E.eq[a][r]] += K[r][c];
    }
  }
}

// Diagonal block of node a: ad and the node's own lower entries, which are
// the last entries of each of its rows (column c of row r at ia[r+1]-(r-c)).
template <int NEN, int NDF>
__device__ __forceinline__ void scatter_diag_rmw(Elem<NEN, NDF> &E, const CsrcDev &k, int a,
                                             const double (&K)[NDF][NDF], bool with_u) {
  if (with_u) {
#pragma unroll
    for (int r = 0; r < NDF; r++)
#pragma unroll
      for (int c = 0; c < NDF; c++) E.p[a][r] += K[r][c] * E.u[a][c];
  }
#pragma unroll
  for (int r = 0; r < NDF; r++) {
    const int row = E.eq[a][r];
    if (row < 0) continue;
    k.ad[row] += K[r][r];
    const int end = k.ia[row + 1];
#pragma unroll
    for (int c = 0; c < r; c++) {
      const int col = E.eq[a][c];
      if (col >= 0) k.al[end - (row - col)] += K[r][c];
    }
  }
}

constexpr int kHexThreads = 64;
constexpr size_t kHexSmem = sizeof(double) * 8 * 8 * 3 * kHexThreads;

__global__ void __launch_bounds__(kHexThreads)
hexa8_kernel(MeshDev m, CsrcDev k, int begin, int end, const double *__restrict__ u,
             double *__restrict__ b, int32_t *bad) {
  extern __shared__ double sg[];
  const int tid = threadIdx.x;
  const int t = begin + blockIdx.x * kHexThreads + tid;
  if (t >= end) return;
#define SG(gp, a, d) sg[(((gp) * 8 + (a)) * 3 + (d)) * kHexThreads + tid]
  int node[8];
#pragma unroll
  for (int a = 0; a < 8; a++) node[a] = m.conn[(size_t)a * m.numel + t];
  double xl[8][3];
#pragma unroll
  for (int a = 0; a < 8; a++)
#pragma unroll
    for (int d = 0; d < 3; d++) xl[a][d] = m.x[(size_t)node[a] * 3 + d];
  const Law L = make_law(HEXA8, m.e + (size_t)m.mat[t] * m.prop);
  double wt[8];
  // natural-coordinate signs of the nodes (Elmlib.f:1177-1184)
  const double rn[8] = {1, -1, -1, 1, 1, -1, -1, 1};
  const double sn[8] = {1, 1, -1, -1, 1, 1, -1, -1};
  const double tn[8] = {1, 1, 1, 1, -1, -1, -1, -1};
  for (int lz = 0; lz < 2; lz++)
    for (int ly = 0; ly < 2; ly++)
      for (int lx = 0; lx < 2; lx++) {
        const int gp = (lz * 2 + ly) * 2 + lx;
        const double r = kPg2[lx], s = kPg2[ly], tt = kPg2[lz];
        double hr[8], hs[8], ht[8];
#pragma unroll
        for (int a = 0; a < 8; a++) {
          const double fr = 1.0 + rn[a] * r, fs = 1.0 + sn[a] * s, ft = 1.0 + tn[a] * tt;
          hr[a] = rn[a] * (fs * ft * 0.125);
          hs[a] = sn[a] * (fr * ft * 0.125);
          ht[a] = tn[a] * (fr * fs * 0.125);
        }
        double xj[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
#pragma unroll
        for (int a = 0; a < 8; a++)
#pragma unroll
          for (int d = 0; d < 3; d++) {
            xj[0][d] += hr[a] * xl[a][d];
            xj[1][d] += hs[a] * xl[a][d];
            xj[2][d] += ht[a] * xl[a][d];
          }
        const double det = xj[0][0] * xj[1][1] * xj[2][2] + xj[0][1] * xj[1][2] * xj[2][0] +
                           xj[0][2] * xj[1][0] * xj[2][1] - xj[2][0] * xj[1][1] * xj[0][2] -
                           xj[1][0] * xj[0][1] * xj[2][2] - xj[0][0] * xj[2][1] * xj[1][2];
        if (det <= 1.e-14) { mark_bad(bad, m.elnum[t]); return; }
        double ji[3][3];
        ji[0][0] = (xj[1][1] * xj[2][2] - xj[1][2] * xj[2][1]) / det;
        ji[1][0] = -(xj[1][0] * xj[2][2] - xj[1][2] * xj[2][0]) / det;
        ji[2][0] = (xj[1][0] * xj[2][1] - xj[1][1] * xj[2][0]) / det;
        ji[0][1] = -(xj[0][1] * xj[2][2] - xj[0][2] * xj[2][1]) / det;
        ji[1][1] = (xj[0][0] * xj[2][2] - xj[0][2] * xj[2][0]) / det;
        ji[2][1] = -(xj[0][0] * xj[2][1] - xj[0][1] * xj[2][0]) / det;
        ji[0][2] = (xj[0][1] * xj[1][2] - xj[0][2] * xj[1][1]) / det;
        ji[1][2] = -(xj[0][0] * xj[1][2] - xj[0][2] * xj[1][0]) / det;
        ji[2][2] = (xj[0][0] * xj[1][1] - xj[0][1] * xj[1][0]) / det;
#pragma unroll
        for (int a = 0; a < 8; a++)
#pragma unroll
          for (int d = 0; d < 3; d++)
            SG(gp, a, d) = ji[d][0] * hr[a] + ji[d][1] * hs[a] + ji[d][2] * ht[a];
        wt[gp] = det * L.a;  // wg^3 = 1
      }
  Elem<8, 3> E;
  const bool with_u = load_elem<8, 3>(E, m, t, node, u);
  for (int a = 0; a < 8; a++) {
    double sa[8][3];
#pragma unroll
    for (int gp = 0; gp < 8; gp++)
#pragma unroll
      for (int d = 0; d < 3; d++) sa[gp][d] = wt[gp] * SG(gp, a, d);
    for (int bb = 0; bb <= a; bb++) {
      double M[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}}, K[3][3];
#pragma unroll
      for (int gp = 0; gp < 8; gp++) {
        const double g0 = SG(gp, bb, 0), g1 = SG(gp, bb, 1), g2 = SG(gp, bb, 2);
#pragma unroll
        for (int r = 0; r < 3; r++) {
          M[r][0] += sa[gp][r] * g0;
          M[r][1] += sa[gp][r] * g1;
          M[r][2] += sa[gp][r] * g2;
        }
      }
      block3d(L, M, K);
      if (a == bb) scatter_diag_rmw<8, 3>(E, k, a, K, with_u);
      else scatter_pair_rmw<8, 3>(E, k, m, t, a, bb, K, with_u);
    }
  }
  if (with_u) finish_rhs<8, 3>(E, b);
#undef SG
}

// HEXA8 with a team of 4 threads per element.  One thread per element
// (hexa8_kernel, ELX_HEX_TEAM=0) left each colour's launch with 32,768 long
// serial threads on the 64^3 cube: 8.45 ms per assembly, latency bound.  The
// FP64 pipe bounds a team (an instruction of a warp costs the same however few
// of its lanes work), so its lanes are filled and its operations counted:
//
//   * Each lane forms two of the 8 integration points.  With G = a c the shear
//     modulus and s = b / c, the block of nodes (i, j) at a point is
//       G det (s g_i g_j^T + g_j g_i^T + (g_i . g_j) I),
//     so one array of gradients scaled by sqrt(G det) serves both sides: the
//     adjugate of the Jacobian times sqrt(G / det), one root and one quotient
//     a point.
//   * The 36 node pairs are nine a lane with no lane idle: lane l takes nodes
//     a = 2l and 2l + 1 with b = a .. a + 3 (mod 8), and the pair (l, l + 4).
//     A block is 72 FMAs (48 on the diagonal) and 11 more operations.
//   * K u needs no sums over the team at the end: for a given step the part of
//     node b belongs to the same neighbour lane in every team, which gets it
//     by a shuffle.
//   * The entries a pair adds to are loaded before its FMAs and stored after
//     them (a read-modify-write at a time waits for L2 nine times a pair).
//
// 64^3 elements: 2.49 ms with u = 0 (8 threads per element, blocks in pair order
// with a read-modify-write at a time and a shuffle tree for K u: 3.76), 61 x 66 x
// 58 with K u 2.65 (4.20).
constexpr int kTeamThreads = 64;
constexpr int kTeamElems = kTeamThreads / 4;
constexpr int kTeamStride = 8 * 8 * 3 + 5;  // doubles of an element, odd: spreads the banks

// Natural derivatives (d/dr, d/ds, d/dt) of the 8 shape functions at the 8
// points (sfhexa8_m, Elmlib.f:1151-1258; point g = lx + 2 ly + 4 lz), the
// same for every element: filled once from the host with the kernel's own
// expressions (exact: the node signs are +-1 and 0.125 a power of two).
__device__ __constant__ double kHexDh[8][3][8];

__global__ void __launch_bounds__(kTeamThreads, 6)
hexa8_team_kernel(MeshDev m, CsrcDev k, int begin, int end, const double *__restrict__ u,
                  double *__restrict__ b, int32_t *bad) {
  __shared__ double sg[kTeamElems * kTeamStride];  // [element][point][node][d], scaled
  __shared__ double sdh[8 * 24];
  __shared__ double su[kTeamElems][8][3];
  __shared__ int seq[kTeamElems][8][3];
  __shared__ int sfirst[kTeamElems][8];
  const int le = threadIdx.x >> 2, lane = threadIdx.x & 3;
  const int t = begin + blockIdx.x * kTeamElems + le;
  const bool active = t < end;
  const int te = active ? t : begin;  // inactive teams read a valid element, write nothing
  for (int i = threadIdx.x; i < 8 * 24; i += kTeamThreads) sdh[i] = (&kHexDh[0][0][0])[i];
  double *ge = sg + le * kTeamStride;
  // a c and b / c of Elmlib02.f:1697-1705
  const double *em = m.e + (size_t)m.mat[te] * m.prop;
  const double G = 0.5 * em[0] / (1.0 + em[1]), sig = 2.0 * em[1] / (1.0 - 2.0 * em[1]);
  const bool neg = G < 0.0;
  __syncthreads();
  {
    double xl[8][3];
#pragma unroll
    for (int a = 0; a < 8; a++) {
      const int no = m.conn[(size_t)a * m.numel + te];
#pragma unroll
      for (int d = 0; d < 3; d++) xl[a][d] = m.x[(size_t)no * 3 + d];
    }
#pragma unroll 1
    for (int half = 0; half < 2; half++) {
      const int gp = lane + 4 * half;
      const double *h = sdh + gp * 24;
      double xj[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
#pragma unroll
      for (int a = 0; a < 8; a++)
#pragma unroll
        for (int r = 0; r < 3; r++)
#pragma unroll
          for (int d = 0; d < 3; d++) xj[r][d] += h[r * 8 + a] * xl[a][d];
      double ad[3][3];  // adjugate
      ad[0][0] = xj[1][1] * xj[2][2] - xj[1][2] * xj[2][1];
      ad[1][0] = -(xj[1][0] * xj[2][2] - xj[1][2] * xj[2][0]);
      ad[2][0] = xj[1][0] * xj[2][1] - xj[1][1] * xj[2][0];
      ad[0][1] = -(xj[0][1] * xj[2][2] - xj[0][2] * xj[2][1]);
      ad[1][1] = xj[0][0] * xj[2][2] - xj[0][2] * xj[2][0];
      ad[2][1] = -(xj[0][0] * xj[2][1] - xj[0][1] * xj[2][0]);
      ad[0][2] = xj[0][1] * xj[1][2] - xj[0][2] * xj[1][1];
      ad[1][2] = -(xj[0][0] * xj[1][2] - xj[0][2] * xj[1][0]);
      ad[2][2] = xj[0][0] * xj[1][1] - xj[0][1] * xj[1][0];
      const double det = xj[0][0] * xj[1][1] * xj[2][2] + xj[0][1] * xj[1][2] * xj[2][0] +
                         xj[0][2] * xj[1][0] * xj[2][1] - xj[2][0] * xj[1][1] * xj[0][2] -
                         xj[1][0] * xj[0][1] * xj[2][2] - xj[0][0] * xj[2][1] * xj[1][2];
      if (active && det <= 1.e-14) mark_bad(bad, m.elnum[t]);
      const double f = sqrt(fabs(G) / det);  // wg^3 = 1
#pragma unroll
      for (int r = 0; r < 3; r++)
#pragma unroll
        for (int d = 0; d < 3; d++) ad[r][d] *= f;
#pragma unroll
      for (int a = 0; a < 8; a++)
#pragma unroll
        for (int d = 0; d < 3; d++)
          ge[gp * 24 + a * 3 + d] =
              ad[d][0] * h[a] + ad[d][1] * h[8 + a] + ad[d][2] * h[16 + a];
    }
  }
  // nodes lane and lane + 4: equations, the smallest of them, displacements
  bool nz = false;
#pragma unroll
  for (int half = 0; half < 2; half++) {
    const int a = lane + 4 * half;
    const int no = m.conn[(size_t)a * m.numel + te];
    int f = -1;
#pragma unroll
    for (int d = 2; d >= 0; d--) {
      const int q = m.eq[(size_t)no * 3 + d];
      seq[le][a][d] = q;
      if (q >= 0) f = q;
      const double ud = u ? u[(size_t)no * 3 + d] : 0.0;
      su[le][a][d] = ud;
      nz = nz || ud != 0.0;
    }
    sfirst[le][a] = f;
  }
  __syncwarp();
  // K u only where the element has a non-zero displacement (an element with
  // u = 0 adds nothing to b; the first solvm pass has u = 0 away from
  // prescribed values): decided per team
  const unsigned team_mask = 0xfu << (threadIdx.x & 28);
  const bool with_u = u != nullptr && (__ballot_sync(0xffffffffu, nz) & team_mask) != 0u;
  const bool any_u = __any_sync(0xffffffffu, with_u);
  double p[2][3] = {{0, 0, 0}, {0, 0, 0}};  // K u of nodes 2 lane, 2 lane + 1
  // one pair: its block K (rows a, columns c), added to the CSRC arrays
  auto pair = [&](int a, int c, double (&K)[3][3], auto is_diag) {
    const int *qa = seq[le][a], *qc = seq[le][c];
    const int fa = sfirst[le][a], fc = sfirst[le][c];
    constexpr bool diag = decltype(is_diag)::value;
    const bool lower = fa > fc;  // rows of a; else rows of c, entry (c d, a r) = K[r][d]
    const bool on = active && fa >= 0 && fc >= 0;
    // where the entries go, and what is there
    int base[3];
    double old[3][3];
    if (on && !diag) {
      const int lo = min(a, c), hi = max(a, c);
      const int off = m.slot[(size_t)pair_index(m.nen, lo, hi) * m.numel + t] - (lower ? fc : fa);
#pragma unroll
      for (int r = 0; r < 3; r++) {
        const int row = lower ? qa[r] : qc[r];
        base[r] = row >= 0 ? k.ia[row] + off : 0;
      }
#pragma unroll
      for (int r = 0; r < 3; r++)
#pragma unroll
        for (int d = 0; d < 3; d++) {
          const int row = lower ? qa[r] : qc[r], cl = lower ? qc[d] : qa[d];
          old[r][d] = row >= 0 && cl >= 0 ? k.al[base[r] + cl] : 0.0;
        }
    } else if (on) {
#pragma unroll
      for (int r = 0; r < 3; r++) {
        const int row = qa[r];
        base[r] = row >= 0 ? k.ia[row + 1] : 0;
        old[r][r] = row >= 0 ? k.ad[row] : 0.0;
#pragma unroll
        for (int d = 0; d < r; d++)
          old[r][d] = row >= 0 && qa[d] >= 0 ? k.al[base[r] - (row - qa[d])] : 0.0;
      }
    }
    double M[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
    const double *pa = ge + a * 3, *pc = ge + c * 3;
#pragma unroll
    for (int gp = 0; gp < 8; gp++) {
      const double s0 = pa[gp * 24], s1 = pa[gp * 24 + 1], s2 = pa[gp * 24 + 2];
      const double g0 = pc[gp * 24], g1 = pc[gp * 24 + 1], g2 = pc[gp * 24 + 2];
      M[0][0] += s0 * g0; M[0][1] += s0 * g1; M[0][2] += s0 * g2;
      if (!diag) M[1][0] += s1 * g0;
      M[1][1] += s1 * g1; M[1][2] += s1 * g2;
      if (!diag) { M[2][0] += s2 * g0; M[2][1] += s2 * g1; }
      M[2][2] += s2 * g2;
    }
    if (diag) {
      M[1][0] = M[0][1];
      M[2][0] = M[0][2];
      M[2][1] = M[1][2];
    }
    const double tr = M[0][0] + M[1][1] + M[2][2];
#pragma unroll
    for (int r = 0; r < 3; r++)
#pragma unroll
      for (int d = 0; d < 3; d++)
        K[r][d] = r == d ? (sig + 1.0) * M[r][r] + tr : sig * M[r][d] + M[d][r];
    if (neg)
#pragma unroll
      for (int r = 0; r < 3; r++)
#pragma unroll
        for (int d = 0; d < 3; d++) K[r][d] = -K[r][d];
    if (on && !diag) {
#pragma unroll
      for (int r = 0; r < 3; r++)
#pragma unroll
        for (int d = 0; d < 3; d++) {
          const int row = lower ? qa[r] : qc[r], cl = lower ? qc[d] : qa[d];
          if (row >= 0 && cl >= 0) k.al[base[r] + cl] = old[r][d] + (lower ? K[r][d] : K[d][r]);
        }
    } else if (on) {
#pragma unroll
      for (int r = 0; r < 3; r++) {
        const int row = qa[r];
        if (row < 0) continue;
        k.ad[row] = old[r][r] + K[r][r];
#pragma unroll
        for (int d = 0; d < r; d++)
          if (qa[d] >= 0) k.al[base[r] - (row - qa[d])] = old[r][d] + K[r][d];
      }
    }
  };
  // K u_c (for node a) and K^T u_a (for node c)
  auto products = [&](int a, int c, const double (&K)[3][3], double (&pa)[3], double (&pc)[3]) {
#pragma unroll
    for (int r = 0; r < 3; r++) {
      pa[r] = K[r][0] * su[le][c][0] + K[r][1] * su[le][c][1] + K[r][2] * su[le][c][2];
      pc[r] = K[0][r] * su[le][a][0] + K[1][r] * su[le][a][1] + K[2][r] * su[le][a][2];
    }
  };
#pragma unroll
  for (int s = 0; s < 2; s++)
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int a = 2 * lane + s, c = (a + q) & 7;
      double K[3][3];
      if (q == 0) pair(a, a, K, std::true_type()); else pair(a, c, K, std::false_type());
      if (any_u) {
        double pa[3], pc[3];
        products(a, c, K, pa, pc);
#pragma unroll
        for (int r = 0; r < 3; r++) {
          p[s][r] += pa[r];
          // node c is node (s + q) & 1 of the lane (s + q) >> 1 further on
          if (q > 0)
            p[(s + q) & 1][r] +=
                __shfl_sync(0xffffffffu, pc[r], (lane - ((s + q) >> 1)) & 3, 4);
        }
      }
    }
  {
    double K[3][3];
    pair(lane, lane + 4, K, std::false_type());
    if (any_u) {
      double pa[3], pc[3];
      products(lane, lane + 4, K, pa, pc);
#pragma unroll
      for (int s = 0; s < 2; s++)
#pragma unroll
        for (int r = 0; r < 3; r++) {
          // node 2 lane + s: node a of lane 2 lane + s, or node c of that - 4
          const int from = (2 * lane + s) & 3;
          const double va = __shfl_sync(0xffffffffu, pa[r], from, 4);
          const double vc = __shfl_sync(0xffffffffu, pc[r], from, 4);
          p[s][r] += lane < 2 ? va : vc;
        }
    }
  }
  if (!with_u || b == nullptr || !active) return;
#pragma unroll
  for (int s = 0; s < 2; s++)
#pragma unroll
    for (int r = 0; r < 3; r++) {
      const int q = seq[le][2 * lane + s][r];
      if (q >= 0) b[q] -= p[s][r];
    }
}

// kHexDh for the current device, once per device.
void fill_hex_table(cudaStream_t st) {
  static std::mutex mu;
  static bool done[64] = {};
  int dev = 0;
  ELX_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(mu);
  if (dev < 0 || dev >= 64 || done[dev]) return;
  static const double rn[8] = {1, -1, -1, 1, 1, -1, -1, 1};
  static const double sn[8] = {1, 1, -1, -1, 1, 1, -1, -1};
  static const double tn[8] = {1, 1, 1, 1, -1, -1, -1, -1};
  static const double pg[2] = {-.577350269189626e0, .577350269189626e0};
  static double h[8][3][8];
  for (int g = 0; g < 8; g++) {
    const double r = pg[g & 1], s = pg[(g >> 1) & 1], t = pg[g >> 2];
    for (int a = 0; a < 8; a++) {
      const double fr = 1.0 + rn[a] * r, fs = 1.0 + sn[a] * s, ft = 1.0 + tn[a] * t;
      h[g][0][a] = rn[a] * (fs * ft * 0.125);
      h[g][1][a] = sn[a] * (fr * ft * 0.125);
      h[g][2][a] = tn[a] * (fr * fs * 0.125);
    }
  }
  ELX_CUDA(cudaMemcpyToSymbolAsync(kHexDh, h, sizeof(h), 0, cudaMemcpyHostToDevice, st));
  ELX_CUDA(cudaStreamSynchronize(st));
  done[dev] = true;
}

}  // namespace

void launch_assembly(const MeshDev &m, const CsrcDev &k, const Segment &seg,
                     const double *u, double *b, int32_t *bad, cudaStream_t st) {
  const int n = seg.end - seg.begin;
  if (n <= 0) return;
  switch (seg.iel) {
    case TRIA3_STRAIN:
    case TRIA3_STRESS:
      tria3_kernel<<<(n + 63) / 64, 64, 0, st>>>(m, k, seg.begin, seg.end, seg.iel, u, b, bad);
      break;
    case QUAD4_STRAIN:
    case QUAD4_STRESS:
      quad4_kernel<<<(n + 63) / 64, 64, 0, st>>>(m, k, seg.begin, seg.end, seg.iel, u, b, bad);
      break;
    case TETRA4:
      tetra4_kernel<<<(n + 63) / 64, 64, 0, st>>>(m, k, seg.begin, seg.end, u, b, bad);
      break;
    case HEXA8: {
      static const bool team = !getenv("ELX_HEX_TEAM") || atoi(getenv("ELX_HEX_TEAM")) != 0;
      if (team) {
        fill_hex_table(st);
        hexa8_team_kernel<<<(n + kTeamElems - 1) / kTeamElems, kTeamThreads, 0, st>>>(
            m, k, seg.begin, seg.end, u, b, bad);
      } else {
        ELX_CUDA(cudaFuncSetAttribute(hexa8_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)kHexSmem));
        hexa8_kernel<<<(n + kHexThreads - 1) / kHexThreads, kHexThreads, kHexSmem, st>>>(
            m, k, seg.begin, seg.end, u, b, bad);
      }
      break;
    }
    default:
      throw Error{ELX_ERR_BAD_ELEMENT, "unsupported element type"};
  }
  ELX_CUDA(cudaGetLastError());
}

}  // namespace elx
