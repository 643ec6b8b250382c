"""Timed cases of the solve path, each a pass through the package's public entry points.

The kinds of pass (``case["kind"]``):

  solve    a solvm step on a meshed model whose structure is kept: the matrix and
           right-hand side are assembled, the system is solved, the nodal
           displacements are updated
  block    several load cases of one assembled matrix, device arrays in and out
  gmres    GMRES restart cycles on one assembled matrix
  recover  the residual b0 - K u and the nodal stresses of a displacement field
  product  y = K x and (x, y) on a caller's own CSRC device arrays
  serve    a burst of requests (new meshes) through the solve server

Models are structured boxes with seeded materials, loads and (jittered)
interior coordinates, in the sizes of the benchmark configurations and tests,
solved to the package's default tolerance.
"""
import dataclasses
import functools
import math

import numpy as np
import torch

import elastic_gb300 as E
from elastic_gb300 import meshgen as M

TYPES = {"tria3": M.TRIA3_STRESS, "quad4": M.QUAD4_STRESS, "quad4_strain": M.QUAD4_STRAIN}
PREC = {"fp64": E.PREC_FP64, "mixed": E.PREC_MIXED}


def listed():
    return [
        # the 64 x 16 cantilever of the tests and of the smallest benchmark
        # configuration: 2,176 equations, where launches and latency count
        {"name": "solve quad4 64x16", "kind": "solve", "mesh": "quad4", "nx": 64, "ny": 16, "nz": 0,
         "bc": "clamp", "jitter": 0.0, "each": False, "precision": "fp64", "tol": 1e-11},
        # an ordinary plane model, odd sizes: 90,902 equations, many cheap iterations
        {"name": "solve tria3 301x150", "kind": "solve", "mesh": "tria3", "nx": 301, "ny": 150, "nz": 0,
         "bc": "clamp", "jitter": 0.0, "each": False, "precision": "fp64", "tol": 1e-11},
        # the benchmark's model: 811,200 equations
        {"name": "solve hexa8 64^3", "kind": "solve", "mesh": "hexa8", "nx": 64, "ny": 64, "nz": 64,
         "bc": "clamp", "jitter": 0.0, "each": False, "precision": "fp64", "tol": 1e-11},
        # the same size in mixed precision, on a distorted mesh of odd sides
        {"name": "solve hexa8 67x59x63 mixed", "kind": "solve", "mesh": "hexa8", "nx": 67, "ny": 59, "nz": 63,
         "bc": "clamp", "jitter": 0.15, "each": False, "precision": "mixed", "tol": 1e-11},
        # the benchmark's distorted tetrahedra with a material per element
        {"name": "solve tetra4 48^3 mixed", "kind": "solve", "mesh": "tetra4", "nx": 48, "ny": 48, "nz": 48,
         "bc": "clamp", "jitter": 0.2, "each": True, "precision": "mixed", "tol": 1e-11},
        # an octant with symmetry planes (rollers): nodes only partly fixed
        {"name": "solve hexa8 41x37x43 rollers", "kind": "solve", "mesh": "hexa8", "nx": 41, "ny": 37, "nz": 43,
         "bc": "rollers", "jitter": 0.0, "each": False, "precision": "fp64", "tol": 1e-11},
        # the benchmark's plate with 16 load cases: the largest
        {"name": "block hexa8 96x96x48 w16 mixed", "kind": "block", "mesh": "hexa8", "nx": 96, "ny": 96, "nz": 48,
         "bc": "clamp", "jitter": 0.0, "each": False, "precision": "mixed", "tol": 1e-11, "nrhs": 16},
        # load cases of a plane model in full precision, as the server solves large plane requests
        {"name": "block quad4 257x129 w5 fp64", "kind": "block", "mesh": "quad4_strain", "nx": 257, "ny": 129,
         "nz": 0, "bc": "clamp", "jitter": 0.0, "each": False, "precision": "fp64", "tol": 1e-11, "nrhs": 5},
        # two GMRES(50) cycles, the default restart length
        {"name": "gmres hexa8 33x35x31 k50", "kind": "gmres", "mesh": "hexa8", "nx": 33, "ny": 35, "nz": 31,
         "bc": "clamp", "jitter": 0.1, "each": False, "ngram": 50, "cycles": 2},
        # residual and stresses of a deformed state, the element loops of every load step
        {"name": "recover hexa8 61x66x58", "kind": "recover", "mesh": "hexa8", "nx": 61, "ny": 66, "nz": 58,
         "bc": "clamp", "jitter": 0.15, "each": False},
        # one product and dot on caller-owned arrays
        {"name": "product hexa8 47x49x45", "kind": "product", "mesh": "hexa8", "nx": 47, "ny": 49, "nz": 45,
         "bc": "clamp", "jitter": 0.1, "each": False},
        # a burst of mixed requests from new meshes to displacements, host preparation included
        {"name": "serve 12 requests", "kind": "serve", "stream": 7, "requests": 12, "dof_min": 2000.0,
         "dof_max": 120000.0, "tol": 1e-11},
    ]


def draw(rng):
    """One more case of the ranges above."""
    def logu(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    kind = rng.choice(["solve", "solve", "solve", "solve", "block", "gmres", "recover", "product", "serve"])
    if kind == "serve":
        return {"kind": kind, "stream": rng.randint(0, 1 << 20), "requests": rng.randint(2, 16), "dof_min": 2000.0,
                "dof_max": round(logu(2e4, 1.2e5)), "tol": 1e-11}
    mesh = rng.choice(["tria3", "quad4", "quad4_strain", "tetra4", "hexa8", "hexa8"])
    c = {"kind": kind, "mesh": mesh, "bc": "clamp", "jitter": 0.0, "each": False}
    if mesh in TYPES:
        dof = logu(1.5e3, 1.2e5 if kind == "solve" else 8e4)
        side = math.sqrt(dof / 2)
        s = rng.uniform(0.6, 2.0)
        c.update(nx=max(3, round(side * s)), ny=max(3, round(side / s)), nz=0)
    else:
        dof = logu(1.5e3, {"solve": 8e5, "block": 3e5, "gmres": 2.5e5, "recover": 7e5, "product": 3.3e5}[kind])
        side = (dof / 3) ** (1 / 3)
        a, b = rng.uniform(0.75, 1.3), rng.uniform(0.75, 1.3)
        c.update(nx=max(3, round(side * a)), ny=max(3, round(side * b)), nz=max(3, round(side / (a * b))))
        c["jitter"] = rng.choice([0.0, 0.1, 0.2 if mesh == "tetra4" else 0.15])
        c["each"] = mesh == "tetra4" and rng.random() < 0.5
    if kind == "solve":
        c["precision"] = "mixed" if mesh not in TYPES and rng.random() < 0.4 else "fp64"
        c["bc"] = rng.choice(["clamp", "clamp", "rollers"])
        c["tol"] = 1e-11
    elif kind == "block":
        c["precision"] = "mixed" if mesh not in TYPES and rng.random() < 0.6 else "fp64"
        c["nrhs"] = rng.randint(2, 16 if c["precision"] == "mixed" else 8)
        c["tol"] = 1e-11
    elif kind == "gmres":
        c["ngram"] = rng.choice([10, 30, 50])
        c["cycles"] = rng.randint(1, 2)
    return c


# ------------------------------------------------------------------- models


@functools.lru_cache(maxsize=2)
def _base(mesh, nx, ny, nz):
    """The undistorted box: connectivity and coordinates, the same for every seed."""
    if mesh in TYPES:
        return M.box2d(nx, ny, 2.0 * nx / (nx + ny), 2.0 * ny / (nx + ny), etype=TYPES[mesh])
    h = 1.0 / (nx * ny * nz) ** (1 / 3)
    box = M.box_hexa8 if mesh == "hexa8" else M.box_tetra4
    return box(nx, ny, nz, nx * h, ny * h, nz * h, pressure=0.0)


def model(case, seed):
    """The mesh of one case: materials, jitter and the nodal forces of one load case from the seed."""
    rng = np.random.default_rng(seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    m = _base(case["mesh"], nx, ny, nz)
    x, ix, e, ie = m.x, m.ix, m.e.copy(), m.ie
    hi = x.max(axis=0)
    if case["jitter"] > 0:
        h = hi / np.array([nx, ny, nz][: m.ndm])
        inner = np.all((x > 0.5 * h) & (x < hi - 0.5 * h), axis=1)
        x0 = x
        x = x0 + np.where(inner[:, None], rng.uniform(-1, 1, x0.shape) * case["jitter"] * h, 0.0)
        if m.nen == 4 and m.ndm == 3:  # a few tetrahedra turn over: their nodes go back
            for _ in range(20):
                det = M.element_dets(dataclasses.replace(m, x=x))
                bad = np.unique(ix[det < 0.01 * h.prod(), :4]) - 1
                if not bad.size:
                    break
                x[bad] = 0.5 * (x[bad] + x0[bad])
    if case["each"]:
        n = m.numel
        e = np.zeros((n, M.PROP))
        e[:, 0], e[:, 1] = np.exp(rng.standard_normal(n)), rng.uniform(0.25, 0.45, n)
        ie = np.full(n, m.ie[0], np.int32)
        ix = ix.copy()
        ix[:, -1] = np.arange(1, n + 1)
    else:
        e[:, 0], e[:, 1] = rng.uniform(0.5, 2.0), rng.uniform(0.25, 0.4)
    idm = np.zeros_like(m.id)
    if case["bc"] == "rollers":
        for d in range(m.ndm):
            idm[x[:, d] == 0.0, d] = 1
    else:
        idm[x[:, 0 if m.ndm == 2 else 2] == 0.0] = 1
    far = x[:, 0 if m.ndm == 2 else 2] == hi[0 if m.ndm == 2 else 2]
    f = np.zeros(x.shape)
    f[far] = rng.standard_normal((int(far.sum()), m.ndf))
    f[idm == 1] = 0.0
    return dataclasses.replace(m, x=x, ix=ix, e=e, ie=ie, id=idm, f=f), rng, far


def context(mesh):
    ctx = E.Context()
    ctx.set_mesh(mesh)
    ctx.build_structure()
    return ctx


def load_cases(case, mesh, rng, far):
    F = np.zeros((case["nrhs"],) + mesh.f.shape)
    for k in range(case["nrhs"]):
        F[k][far] = rng.standard_normal((int(far.sum()), mesh.ndf))
        F[k][mesh.id == 1] = 0.0
    return F


def requests(case, seed):
    """Requests as the benchmark draws them, at most 4 load cases each: the meshes and the number
    of load cases from the case's stream, the materials and forces from the seed."""
    stream, rng = np.random.default_rng(case["stream"]), np.random.default_rng(seed)
    out = []
    for _ in range(case["requests"]):
        m, F = M.serving_request(stream, case["dof_min"], case["dof_max"], max_rhs=4)
        e = m.e.copy()
        e[:, 0], e[:, 1] = rng.uniform(0.5, 2.0), rng.uniform(0.2, 0.45)
        out.append((dataclasses.replace(m, e=e), np.where(F != 0.0, rng.standard_normal(F.shape), 0.0)))
    return out


# ------------------------------------------------------------------- passes


def prepare(case, seed):
    if case["kind"] == "serve":
        return {"case": case, "server": E.Server(), "requests": requests(case, seed)}
    mesh, rng, far = model(case, seed)
    ctx = context(mesh)
    s = {"case": case, "ctx": ctx}
    if case["kind"] == "recover":
        s["u"] = 1e-3 * rng.standard_normal(mesh.f.shape)
        s["b0"], _ = E.pload(mesh, ctx.structure().id)
        return s
    ids = ctx.structure().id
    s["b0"], s["u0"] = E.pload(mesh, ids)
    if case["kind"] == "block":
        F = load_cases(case, mesh, rng, far)
        ctx.assemble(s["u0"], s["b0"])
        free = ids > 0
        B = np.zeros((case["nrhs"], s["b0"].size))
        for k in range(case["nrhs"]):
            B[k][ids[free] - 1] = F[k][free]
        s["B"] = torch.from_numpy(B).cuda()
        s["X"] = torch.empty_like(s["B"])
    elif case["kind"] == "gmres":
        s["b"] = ctx.assemble(s["u0"], s["b0"])
    elif case["kind"] == "product":
        _, ad, al = ctx.assemble(s["u0"], s["b0"], want_matrix=True)
        st = ctx.structure()
        ctx.close()
        del s["ctx"]
        ia, ja = torch.from_numpy(st.ia).cuda(), torch.from_numpy(st.ja).cuda()
        rows = torch.repeat_interleave(torch.arange(1, st.neq + 1, dtype=torch.int32, device="cuda"),
                                       (ia[1:] - ia[:-1]).long())
        order = torch.argsort(ja, stable=True)
        count = torch.bincount(ja.long() - 1, minlength=st.neq)
        iat = torch.cat([torch.ones(1, dtype=torch.int64, device="cuda"), 1 + count.cumsum(0)]).int()
        al = torch.from_numpy(al).cuda()
        s.update(neq=st.neq, ia=ia, ja=ja, ad=torch.from_numpy(ad).cuda(), al=al, iat=iat,
                 jat=rows[order].contiguous(), alt=al[order].contiguous(),
                 x=torch.from_numpy(rng.standard_normal(st.neq)).cuda(),
                 y=torch.empty(st.neq, dtype=torch.float64, device="cuda"),
                 xy=torch.empty(1, dtype=torch.float64, device="cuda"), lib=E.load())
    return s


def run(s):
    c = s["case"]
    if c["kind"] == "solve":
        ctx = s["ctx"]
        b = ctx.assemble(s["u0"], s["b0"])
        x, _ = ctx.solve(b, precision=PREC[c["precision"]], tol=c["tol"], maxit=20000)
        return {"u": ctx.update(x, s["u0"])}
    if c["kind"] == "block":
        s["ctx"].solve_block_device(s["B"].data_ptr(), s["X"].data_ptr(), c["nrhs"],
                                    precision=PREC[c["precision"]], tol=c["tol"], maxit=20000)
        return {"x": s["X"]}
    if c["kind"] == "gmres":
        x, _ = s["ctx"].solve(s["b"], solver=E.SOLVER_GMRES, tol=1e-14, maxit=c["cycles"],
                              ngram=c["ngram"], raise_on_error=False)
        return {"x": x}
    if c["kind"] == "recover":
        return {"b": s["ctx"].assemble(s["u"], s["b0"]), "stress": s["ctx"].stress(s["u"])}
    if c["kind"] == "product":
        p = [s[k].data_ptr() for k in ("ia", "ja", "ad", "al", "iat", "jat", "alt", "x", "y", "xy")]
        st = s["lib"].elx_spmv_dot_noalloc(s["neq"], *p, torch.cuda.current_stream().cuda_stream)
        if st != E.OK:
            raise E.ElasticError(st, "elx_spmv_dot_noalloc")
        return {"y": s["y"], "xy": s["xy"]}
    tickets = [s["server"].submit(mesh, F, tol=c["tol"]) for mesh, F in s["requests"]]
    out = {}
    for k, t in enumerate(tickets):
        U, _, _, status = s["server"].wait(t)
        if status != E.OK:
            raise E.ElasticError(status, "request failed")
        out["u%02d" % k] = U
    return out


def work(case):
    """Bytes and operations of one pass that the path cannot do without.

    Solvers: the matrix (lower entries once, 8 bytes and a 4-byte column; half
    the value bytes in mixed precision) and the vectors of each iteration, two
    operations per entry of the full matrix; the iteration count is that of a
    conjugate gradient on such a box, about `per_side` iterations per element
    along the long side."""
    if case["kind"] == "serve":
        # requests are log-uniform in size: their mean work, at 2.5 load cases each
        lo, hi, n = case["dof_min"], case["dof_max"], 8
        b = f = 0.0
        for k in range(n):
            dof = math.exp(math.log(lo) + (k + 0.5) / n * math.log(hi / lo))
            for mesh, ndf in (("tria3", 2), ("hexa8", 3)):
                side = (dof / ndf) ** (1 / ndf)
                w = _pcg_work(mesh, dof, side * (1.4 if ndf == 2 else 1.0), 8, 2.5)
                b, f = b + w[0] / (2 * n), f + w[1] / (2 * n)
        return {"bytes": case["requests"] * b, "flops": case["requests"] * f}
    ndf = 2 if case["mesh"] in TYPES else 3
    nodes = (case["nx"] + 1) * (case["ny"] + 1) * (case["nz"] + 1)
    neq = ndf * nodes
    nad = neq * _row(case["mesh"])
    if case["kind"] == "product":
        return {"bytes": 12 * nad + 28 * neq, "flops": 4 * nad + 2 * neq}
    if case["kind"] == "recover":
        nel = case["nx"] * case["ny"] * max(1, case["nz"]) * {"tria3": 2, "tetra4": 6}.get(case["mesh"], 1)
        return {"bytes": 8 * (nad + 10 * neq) + 36 * nel, "flops": nel * {"hexa8": 1.1e4, "tetra4": 900}.get(case["mesh"], 600)}
    if case["kind"] == "gmres":
        its = case["ngram"] * case["cycles"]
        return {"bytes": its * (12 * nad + 28 * neq + 16 * neq * case["ngram"] / 2),
                "flops": its * (4 * nad + 2 * neq + 4 * neq * case["ngram"] / 2)}
    vs = 4 if case.get("precision") == "mixed" else 8
    b, f = _pcg_work(case["mesh"], neq, max(case["nx"], case["ny"], case["nz"]), vs, case.get("nrhs", 1))
    return {"bytes": b, "flops": f}


def _row(mesh):
    """Strict-lower entries per equation of a structured box."""
    return {"tria3": 6.5, "quad4": 8.5, "quad4_strain": 8.5, "tetra4": 21.3, "hexa8": 38.8}[mesh]


def _pcg_work(mesh, neq, side, vs, nrhs):
    its = side * {"tria3": 7.0, "quad4": 7.0, "quad4_strain": 7.0, "tetra4": 12.0, "hexa8": 7.5}[mesh] + 40
    nad = neq * _row(mesh)
    return (its * ((vs + 4) * nad + 4 * neq + nrhs * 13 * vs * neq), its * nrhs * (4 * nad + 14 * neq))


# ------------------------------------------------------- the same in 64 bits


def _points(nen, ndm, nodal):
    """Natural derivatives (point, axis, node) at the Gauss points, or at the nodes."""
    if nen == ndm + 1:  # simplex: constant
        d = np.zeros((1, ndm, nen))
        for k in range(ndm):
            d[0, k, k], d[0, k, nen - 1] = 1.0, -1.0
        return torch.from_numpy(np.repeat(d, nen, 0) if nodal else d).cuda()
    if ndm == 2:
        sign = np.array([(1, 1), (-1, 1), (-1, -1), (1, -1)], float)
    else:
        sign = 2.0 * M.HEX_LOCAL - 1.0
    pts = sign if nodal else sign / math.sqrt(3.0)
    d = np.empty((len(pts), ndm, nen))
    for g, p in enumerate(pts):
        f = 1.0 + sign * p
        for k in range(ndm):
            d[g, k] = sign[:, k] * np.prod(np.delete(f, k, axis=1), axis=1) / 2 ** ndm
    return torch.from_numpy(d).cuda()


def _law(mesh):
    """The constitutive matrix per element, (numel, ns, ns): xx yy xy, or xx yy zz xy yz xz."""
    mat = torch.from_numpy(mesh.ix[:, -1].astype(np.int64) - 1).cuda()
    ym, nu = (torch.from_numpy(mesh.e[:, k].copy()).cuda()[mat] for k in (0, 1))
    stress = int(mesh.ie[0]) in (M.TRIA3_STRESS, M.QUAD4_STRESS)
    if stress:
        a, b, c = ym / (1 - nu * nu), nu, 0.5 * (1 - nu)
    else:
        a = ym * (1 - nu) / ((1 + nu) * (1 - 2 * nu))
        b, c = nu / (1 - nu), 0.5 * (1 - 2 * nu) / (1 - nu)
    nd = mesh.ndm
    ns = 3 if nd == 2 else 6
    D = torch.zeros(mesh.numel, ns, ns, dtype=torch.float64, device="cuda")
    for i in range(nd):
        for j in range(nd):
            D[:, i, j] = a if i == j else a * b
    for i in range(nd, ns):
        D[:, i, i] = a * c
    return D, nu, stress


def _strain(mesh, d):
    """Strain operator (numel, ns, nen ndf) and determinant at one point with derivatives d (axis, node)."""
    nd, nen = mesh.ndm, mesh.nen
    conn = torch.from_numpy(mesh.ix[:, :nen].astype(np.int64) - 1).cuda()
    xe = torch.from_numpy(mesh.x).cuda()[conn]
    J = torch.einsum("ka,ead->ekd", d, xe)
    g = torch.linalg.solve(J, d.expand(mesh.numel, -1, -1))
    B = torch.zeros(mesh.numel, 3 if nd == 2 else 6, nen, nd, dtype=torch.float64, device="cuda")
    for k in range(nd):
        B[:, k, :, k] = g[:, k]
    for r, (i, j) in enumerate([(0, 1)] if nd == 2 else [(0, 1), (1, 2), (0, 2)]):
        B[:, nd + r, :, i], B[:, nd + r, :, j] = g[:, j], g[:, i]
    return B.reshape(mesh.numel, -1, nen * nd), torch.linalg.det(J)


def _stiffness(mesh):
    D, _, stress = _law(mesh)
    simplex = mesh.nen == mesh.ndm + 1
    K = 0
    for d in _points(mesh.nen, mesh.ndm, False):
        B, det = _strain(mesh, d)
        w = det * (1 / math.factorial(mesh.ndm) if simplex else 1.0)
        if stress and not simplex:  # thickness 0 stands for 1
            t = torch.from_numpy(mesh.e[:, 2].copy()).cuda()[torch.from_numpy(mesh.ix[:, -1].astype(np.int64) - 1).cuda()]
            w = w * torch.where(t == 0, 1.0, t)
        K = K + torch.einsum("esi,est,etj->eij", B, D * w[:, None, None], B)
    return K


def _matrix(mesh, free_only=True):
    """The assembled matrix (CSR) on the free dofs (or all), and the dofs' places."""
    nd, nen = mesh.ndf, mesh.nen
    free = torch.from_numpy((mesh.id == 0).reshape(-1)).cuda()
    if not free_only:
        free = torch.ones_like(free)
    place = torch.where(free, torch.cumsum(free.long(), 0) - 1, -1)
    dof = (torch.from_numpy(mesh.ix[:, :nen].astype(np.int64) - 1).cuda()[:, :, None] * nd
           + torch.arange(nd, device="cuda")).reshape(mesh.numel, -1)
    p = place[dof]
    r = p[:, :, None].expand(-1, -1, nen * nd).reshape(-1)
    c = p[:, None, :].expand(-1, nen * nd, -1).reshape(-1)
    keep = (r >= 0) & (c >= 0)
    n = int(free.sum())
    K = torch.sparse_coo_tensor(torch.stack([r[keep], c[keep]]), _stiffness(mesh).reshape(-1)[keep], (n, n))
    return K.coalesce().to_sparse_csr(), free


def _solve(mesh, F):
    """Displacements (nrhs, nnode, ndf) under the nodal forces F, to rounding."""
    K, free = _matrix(mesh)
    b = torch.from_numpy(np.ascontiguousarray(F.reshape(F.shape[0], -1).T)).cuda()[free]
    crow, col, val = K.crow_indices(), K.col_indices(), K.values()
    row = torch.repeat_interleave(torch.arange(b.shape[0], device="cuda"), crow[1:] - crow[:-1])
    m = (1.0 / val[row == col])[:, None]
    x, r = torch.zeros_like(b), b.clone()
    z = m * r
    p, d = z.clone(), (r * z).sum(0)
    stop = 1e-28 * d
    for it in range(40000):
        q = K @ p
        a = d / (p * q).sum(0)
        x += a * p
        r -= a * q
        z = m * r
        d1 = (r * z).sum(0)
        p = z + (d1 / d) * p
        d = d1
        if it % 25 == 0 and bool((d <= stop).all()):
            break
        d = torch.where(d == 0, 1e-300, d)
    u = torch.zeros(F.shape[0], mesh.id.size, dtype=torch.float64, device="cuda")
    u[:, free] = x.T
    return u.reshape(F.shape)


def _gmres(K, b, m, k, cycles):
    """`cycles` restart cycles of left-preconditioned GMRES(k), the basis orthogonalised twice."""
    x = torch.zeros_like(b)
    for _ in range(cycles):
        r = m * (b - K @ x)
        beta = r.norm()
        V = torch.zeros(k + 1, b.numel(), dtype=torch.float64, device="cuda")
        H = torch.zeros(k + 1, k, dtype=torch.float64, device="cuda")
        V[0] = r / beta
        for j in range(k):
            w = m * (K @ V[j])
            for _ in range(2):
                h = V[: j + 1] @ w
                w = w - h @ V[: j + 1]
                H[: j + 1, j] += h
            H[j + 1, j] = w.norm()
            V[j + 1] = w / H[j + 1, j]
        e = torch.zeros(k + 1, 1, dtype=torch.float64, device="cuda")
        e[0] = beta
        x = x + torch.linalg.lstsq(H, e).solution[:, 0] @ V[:k]
    return x


def _stresses(mesh, u):
    D, nu, stress = _law(mesh)
    nd, nen = mesh.ndm, mesh.nen
    conn = torch.from_numpy(mesh.ix[:, :nen].astype(np.int64) - 1).cuda()
    ue = u[conn].reshape(mesh.numel, -1, 1)
    t = torch.zeros(mesh.nnode, 4 if nd == 2 else 6, dtype=torch.float64, device="cuda")
    for a, d in enumerate(_points(nen, nd, True)):
        B, _ = _strain(mesh, d)
        s = (D @ (B @ ue))[:, :, 0]
        if nd == 2:
            zz = torch.zeros_like(nu) if stress else nu * (s[:, 0] + s[:, 1])
            s = torch.stack([s[:, 0], s[:, 1], zz, s[:, 2]], 1)
        t.index_add_(0, conn[:, a], s)
    n = torch.bincount(conn.reshape(-1), minlength=mesh.nnode)
    return t / n[:, None]


def exact(case, seed):
    if case["kind"] == "serve":
        return {"u%02d" % k: _solve(mesh, F) for k, (mesh, F) in enumerate(requests(case, seed))}
    mesh, rng, far = model(case, seed)
    if case["kind"] == "solve":
        return {"u": _solve(mesh, mesh.f[None])[0]}
    # the other kinds return vectors in the order of the equation numbers
    ids = torch.from_numpy(E.host_structure(mesh).id.astype(np.int64).reshape(-1)).cuda()

    def equations(v):
        out = torch.empty(int(ids.max()), dtype=torch.float64, device="cuda")
        out[ids[ids > 0] - 1] = v
        return out

    if case["kind"] == "block":
        u = _solve(mesh, load_cases(case, mesh, rng, far)).reshape(case["nrhs"], -1)
        return {"x": torch.stack([equations(v[ids > 0]) for v in u])}
    if case["kind"] == "recover":
        u = torch.from_numpy(1e-3 * rng.standard_normal(mesh.f.shape)).cuda()
        K, _ = _matrix(mesh, free_only=False)
        b = torch.from_numpy(mesh.f.reshape(-1)).cuda() - K @ u.reshape(-1)
        return {"b": equations(b[ids > 0]), "stress": _stresses(mesh, u)}
    K, free = _matrix(mesh)
    if case["kind"] == "product":
        x = torch.from_numpy(rng.standard_normal(int(ids.max()))).cuda()
        y = equations(K @ x[ids[ids > 0] - 1])
        return {"y": y, "xy": torch.dot(x, y).reshape(1)}
    crow, col = K.crow_indices(), K.col_indices()
    row = torch.repeat_interleave(torch.arange(crow.numel() - 1, device="cuda"), crow[1:] - crow[:-1])
    m = 1.0 / K.values()[row == col]
    b = torch.from_numpy(mesh.f.reshape(-1)).cuda()[free]
    return {"x": equations(_gmres(K, b, m, case["ngram"], case["cycles"]))}
