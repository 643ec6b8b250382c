"""The resident PCG with its vectors in L2 (large matrices; here small ones by
ELX_RESIDENT_MODE=1) does the arithmetic of the one with its vectors in shared
memory: the same bits, for one to six columns, partly fixed nodes, several
launches a solve and solves that stop at maxit.  And the launches of one
iteration each on node blocks (ELX_RESIDENT_MODE=0: matrices that fit neither,
contexts without memory for the plan) against the oracle."""
import numpy as np
import pytest

import elastic_gb300 as E
import oracle as O
from elastic_gb300 import meshgen as M
from helpers import rel_inf, rollers

pytestmark = pytest.mark.gpu

# above the cluster's sizes; block rows: 152 slices, 153, more with partly fixed nodes
MESHES = {
    "quad4": lambda: M.box2d(64, 75, etype=M.QUAD4_STRESS),
    "tria3": lambda: M.box2d(72, 67, etype=M.TRIA3_STRAIN),
    "tetra4": lambda: M.box_tetra4(14, 15, 13, jitter=0.2),
    "hexa8": lambda: M.box_hexa8(13, 14, 15, jitter=0.1),
    "hexa8 rollers": lambda: rollers(rollers(M.box_hexa8(14, 13, 15), 0), 1),
    "tria3 rollers": lambda: rollers(M.box2d(90, 71, etype=M.TRIA3_STRESS), 1),
}


def _context(monkeypatch, mesh, mode):
    if mode is None:
        monkeypatch.delenv("ELX_RESIDENT_MODE", raising=False)
    else:
        monkeypatch.setenv("ELX_RESIDENT_MODE", str(mode))
    mesh.f = np.random.default_rng(3).standard_normal(mesh.f.shape) * (mesh.id == 0)
    ctx = E.Context(device=0)
    ctx.set_mesh(mesh)
    ctx.build_structure(True)
    b0, u0 = E.pload(mesh, ctx.structure().id)
    return ctx, ctx.assemble(u0, b0)


@pytest.mark.parametrize("name", sorted(MESHES))
def test_vectors_in_l2_give_the_same_bits(built_lib, monkeypatch, name):
    out = []
    for mode in (None, 1):
        ctx, b = _context(monkeypatch, MESHES[name](), mode)
        with ctx:
            r = []
            for maxit in (20000, 1, 7, 511, 512, 513):
                n0 = ctx.kernel_launches
                x, i = ctx.solve(b, tol=1e-13, maxit=maxit, raise_on_error=False)
                r.append((x, i["iters"], i["status"], i["norm_r"], ctx.kernel_launches - n0))
            out.append(r)
    assert out[0][0][2] == 0
    for a, c in zip(*out):
        assert np.array_equal(a[0], c[0]) and a[1:] == c[1:]


def test_several_launches_from_l2(built_lib, monkeypatch):
    out = []
    for mode in (None, 1):
        ctx, b = _context(monkeypatch, M.box2d(160, 40, etype=M.TRIA3_STRESS), mode)
        with ctx:
            x, i = ctx.solve(b, tol=1e-11, maxit=20000)
            assert i["iters"] > 1024
            out.append((x, i["iters"]))
    assert np.array_equal(out[0][0], out[1][0]) and out[0][1] == out[1][1]


@pytest.mark.parametrize("name", ["quad4", "tetra4"])
@pytest.mark.parametrize("nrhs", [2, 3, 4, 5, 6])
def test_columns_in_l2_give_the_same_bits(built_lib, monkeypatch, name, nrhs):
    out = []
    for mode in (None, 1):
        ctx, b = _context(monkeypatch, MESHES[name](), mode)
        with ctx:
            B = np.random.default_rng(nrhs).standard_normal((b.size, nrhs))
            B[:, 1] = 0.0  # done at once; the last stops long before the others
            if nrhs > 2:
                B[:, -1] = ctx.spmv(ctx.spmv(ctx.spmv(B[:, -1])))
            out.append([ctx.solve_block(B, precision=E.PREC_FP64, tol=1e-11, maxit=m,
                                        raise_on_error=False) for m in (20000, 60)])
    for (X, i), (Y, j) in zip(*out):
        assert np.array_equal(X, Y)
        for p, q in zip(i, j):
            assert all(p[k] == q[k] for k in ("iters", "status", "norm_r", "xkx", "conv"))


@pytest.mark.parametrize("name", sorted(MESHES))
def test_launches_on_node_blocks(built_lib, monkeypatch, name):
    mesh = MESHES[name]()
    ctx, b = _context(monkeypatch, mesh, 0)
    with ctx:
        s = O.structure(mesh, True)
        b0, u0 = O.loads(mesh, s)
        ad, al, b_o = O.assemble(mesh, s, u0, b0)
        x_o, i_o = O.pcg(s, ad, al, b_o, tol=1e-12, maxit=20000)
        n0 = ctx.kernel_launches
        x, i = ctx.solve(b, tol=1e-12, maxit=20000)
        assert ctx.kernel_launches - n0 > 3 * i["iters"]
        assert rel_inf(x_o, x) <= 1e-10 and abs(i["iters"] - i_o["iters"]) <= 2
        x, i = ctx.solve(b, precision=E.PREC_MIXED, tol=1e-10, maxit=20000)
        assert i["status"] == 0 and rel_inf(x_o, x) <= 1e-6
        if "rollers" not in name:
            X, infos = ctx.solve_block(np.outer(b, [1.0, 2.0, 4.0]), precision=E.PREC_FP64,
                                       tol=1e-12, maxit=20000)
            for k in range(3):
                assert rel_inf(x_o, X[:, k] / 2.0 ** k) <= 1e-10
        g_o, _ = O.gmres(s, ad, al, b_o, k=17, tol=1e-14, maxit=1)
        x, _ = ctx.solve(b, solver=E.SOLVER_GMRES, ngram=17, tol=1e-14, maxit=1,
                         raise_on_error=False)
        assert rel_inf(g_o, x) <= 1e-9
