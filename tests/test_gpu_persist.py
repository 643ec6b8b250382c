"""The FP64 PCG in one cooperative launch (persist.cu) where it can go wrong:
one slice of block rows, a last slice that is not full, as many slices as
blocks and one more, partly fixed nodes (padded to whole blocks), blocks of
one to six columns, some of them stopped long before the others, several
launches per solve, loads at the ends of the
exponent range (the digit window of the grid sums follows the residual), a
matrix and a load whose norms differ by many orders, and a load with a NaN.

Bars: the solver tests' (displacements within 1e-10 of the oracle, iterations
within 2); a load scaled by a power of two gives the same iterates scaled
exactly."""
import threading

import numpy as np
import pytest

import elastic_gb300 as E
import oracle as O
from elastic_gb300 import meshgen as M
from helpers import rel_inf, rollers

pytestmark = pytest.mark.gpu

# block rows: 24 (one slice), 32 = one full slice, 33, 152 * 32 and 153 * 32 of QUAD4
CASES = {
    "hexa8 one slice": lambda: M.box_hexa8(2, 3, 2),
    "quad4 full slice": lambda: M.box2d(4, 7, etype=M.QUAD4_STRESS),
    "quad4 two slices": lambda: M.box2d(3, 10, etype=M.QUAD4_STRAIN),
    "quad4 152 slices": lambda: M.box2d(64, 75, etype=M.QUAD4_STRESS),
    "tria3 153 slices": lambda: M.box2d(72, 67, etype=M.TRIA3_STRAIN),
    "tetra4": lambda: M.box_tetra4(9, 8, 7, jitter=0.2, lognormal_E=True, nu_range=(0.25, 0.45)),
    # partly fixed nodes: one, two and three dofs free, on lower and upper neighbours
    "hexa8 rollers": lambda: rollers(rollers(M.box_hexa8(7, 5, 6), 0), 1),
    "tetra4 rollers": lambda: rollers(M.box_tetra4(5, 6, 4, jitter=0.15), 1),
    "quad4 rollers": lambda: rollers(M.box2d(23, 17, etype=M.QUAD4_STRAIN), 1),
    "tria3 rollers": lambda: rollers(M.box2d(90, 71, etype=M.TRIA3_STRESS), 1),
}


def _system(ctx, mesh, seed=3):
    mesh.f = np.random.default_rng(seed).standard_normal(mesh.f.shape) * (mesh.id == 0)
    ctx.set_mesh(mesh)
    ctx.build_structure(True)
    s = O.structure(mesh, True)
    b0, u0 = O.loads(mesh, s)
    ad, al, b = O.assemble(mesh, s, u0, b0)
    ctx.assemble(u0, b0)
    return s, ad, al, b


@pytest.mark.parametrize("name", sorted(CASES))
def test_matches_oracle(gpu_ctx, name):
    s, ad, al, b = _system(gpu_ctx, CASES[name]())
    x_o, i_o = O.pcg(s, ad, al, b, tol=1e-12, maxit=20000)
    x, i = gpu_ctx.solve(b, tol=1e-12, maxit=20000)
    assert rel_inf(x_o, x) <= 1e-10
    assert abs(i["iters"] - i_o["iters"]) <= 2
    x2, i2 = gpu_ctx.solve(b, tol=1e-12, maxit=20000)
    assert np.array_equal(x, x2) and i["iters"] == i2["iters"]


@pytest.mark.parametrize("e", [-400, -60, 60, 400])
def test_scaled_load_scales_exactly(gpu_ctx, e):
    _, _, _, b = _system(gpu_ctx, M.box2d(40, 21, etype=M.QUAD4_STRAIN))
    x, i = gpu_ctx.solve(b, tol=1e-11)
    xs, js = gpu_ctx.solve(np.ldexp(b, e), tol=1e-11)
    assert i["iters"] == js["iters"]
    assert np.array_equal(np.ldexp(x, e), xs)


def test_several_launches_and_maxit(gpu_ctx):
    s, ad, al, b = _system(gpu_ctx, M.box2d(120, 60, etype=M.TRIA3_STRESS))
    x, i = gpu_ctx.solve(b, tol=1e-11, maxit=20000)
    assert i["iters"] > 1024  # more than two launches of 512 iterations
    x_o, i_o = O.pcg(s, ad, al, b, tol=1e-11, maxit=20000)
    assert rel_inf(x_o, x) <= 1e-10 and abs(i["iters"] - i_o["iters"]) <= 2
    for maxit in (1, 511, 512, 513, 1024):
        _, i = gpu_ctx.solve(b, tol=1e-11, maxit=maxit, raise_on_error=False)
        assert i["status"] == E.ERR_NO_CONVERGENCE and i["iters"] == maxit


def test_residual_far_from_the_matrix_scale(gpu_ctx):
    m = M.box_hexa8(5, 4, 4, E=1e-90)
    s, ad, al, b = _system(gpu_ctx, m)
    x_o, i_o = O.pcg(s, ad, al, b, tol=1e-11, maxit=5000)
    x, i = gpu_ctx.solve(b, tol=1e-11, maxit=5000)
    assert rel_inf(x_o, x) <= 1e-10 and abs(i["iters"] - i_o["iters"]) <= 2


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_load_that_is_not_finite_does_not_converge(gpu_ctx, bad):
    _, _, _, b = _system(gpu_ctx, M.box2d(30, 20, etype=M.QUAD4_STRESS))
    c = b.copy()
    c[17] = bad
    _, i = gpu_ctx.solve(c, tol=1e-10, maxit=200, raise_on_error=False)
    assert i["status"] == E.ERR_NO_CONVERGENCE
    x, i = gpu_ctx.solve(b, tol=1e-10)
    assert i["status"] == 0 and np.isfinite(x).all()


@pytest.mark.parametrize("name", ["hexa8 one slice", "quad4 152 slices", "tetra4"])
@pytest.mark.parametrize("nrhs", [1, 2, 3, 5, 6, 7])
def test_columns_match_single_solves(gpu_ctx, name, nrhs):
    """Each column's iterates are those of the single solve; a zero column and
    one that is solved early do not disturb the others."""
    _, _, _, b = _system(gpu_ctx, CASES[name]())
    rng = np.random.default_rng(nrhs)
    B = rng.standard_normal((b.size, nrhs))
    if nrhs > 2:
        B[:, 1] = 0.0
    X, infos = gpu_ctx.solve_block(B, precision=E.PREC_FP64, tol=1e-11, maxit=20000)
    for c in range(nrhs):
        x, i = gpu_ctx.solve(B[:, c], tol=1e-11, maxit=20000)
        assert infos[c]["status"] == 0 and abs(infos[c]["iters"] - i["iters"]) <= 2
        assert rel_inf(x, X[:, c]) <= 1e-10 if x.any() else not X[:, c].any()
        np.testing.assert_allclose(infos[c]["xkx"], i["xkx"], rtol=1e-10)
    # a column of another magnitude leaves the others' bits alone
    B[:, 0] *= 1e-30
    X2, infos2 = gpu_ctx.solve_block(B, precision=E.PREC_FP64, tol=1e-11, maxit=20000)
    assert rel_inf(1e-30 * X[:, 0], X2[:, 0]) <= 1e-10
    for c in range(1, nrhs):
        assert np.array_equal(X[:, c], X2[:, c]) and infos2[c]["iters"] == infos[c]["iters"]


@pytest.mark.parametrize("name", sorted(k for k in CASES if "rollers" not in k))
def test_mixed_meets_the_fp64_test(gpu_ctx, name):
    s, ad, al, b = _system(gpu_ctx, CASES[name]())
    x_o, _ = O.pcg(s, ad, al, b, tol=1e-13, maxit=20000)
    x, i = gpu_ctx.solve(b, precision=E.PREC_MIXED, tol=1e-10, maxit=20000)
    assert i["status"] == 0 and i["norm_m_r"] <= 3.16 * i["conv"]
    assert rel_inf(x_o, x) <= 1e-6
    x2, i2 = gpu_ctx.solve(b, precision=E.PREC_MIXED, tol=1e-10, maxit=20000)
    assert np.array_equal(x, x2) and i["inner_iters"] == i2["inner_iters"]


def test_mixed_maxit_and_bad_load(gpu_ctx):
    _, _, _, b = _system(gpu_ctx, M.box_hexa8(9, 8, 8, jitter=0.1))
    for maxit in (1, 6, 8):  # the test is made at every fourth iteration
        _, i = gpu_ctx.solve(b, precision=E.PREC_MIXED, tol=1e-12, maxit=maxit, raise_on_error=False)
        assert i["status"] == E.ERR_NO_CONVERGENCE and maxit <= i["iters"] < maxit + 4
    c = b.copy()
    c[5] = np.nan
    _, i = gpu_ctx.solve(c, precision=E.PREC_MIXED, tol=1e-10, maxit=100, raise_on_error=False)
    assert i["status"] == E.ERR_NO_CONVERGENCE
    _, i = gpu_ctx.solve(b, precision=E.PREC_MIXED, tol=1e-10)
    assert i["status"] == 0


# restart lengths around the 16 warps that share the basis vectors; k = 250
# does not fit the block's shared memory and takes the launches
@pytest.mark.parametrize("name,k", [("quad4 full slice", 1), ("quad4 two slices", 16),
                                    ("tetra4", 33), ("tria3 153 slices", 17),
                                    ("hexa8 rollers", 7), ("tetra4 rollers", 17),
                                    ("quad4 152 slices", 250)])
def test_gmres_cycle_matches_oracle(gpu_ctx, name, k):
    s, ad, al, b = _system(gpu_ctx, CASES[name]())
    k = min(k, s.neq)
    x_o, _ = O.gmres(s, ad, al, b, k=k, tol=1e-14, maxit=1)
    x, i = gpu_ctx.solve(b, solver=E.SOLVER_GMRES, tol=1e-14, maxit=1, ngram=k,
                         raise_on_error=False)
    assert i["refinements"] == 1 and i["iters"] <= k
    assert rel_inf(x_o, x) <= 1e-9
    x2, _ = gpu_ctx.solve(b, solver=E.SOLVER_GMRES, tol=1e-14, maxit=1, ngram=k,
                          raise_on_error=False)
    assert np.array_equal(x, x2)


def test_pack_with_teams_and_packed_launches(built_lib):
    """A load case too large for a team of the cooperative pack (above 160
    blocks of 768 rows) iterates in packed launches beside teams of one block
    and of several; each equals its own single solve."""
    meshes = [M.box2d(255, 250, etype=M.QUAD4_STRESS), M.box_hexa8(2, 2, 2),
              M.box_tetra4(9, 9, 9), M.box2d(40, 20, etype=M.TRIA3_STRAIN)]
    with E.Server(device=0, large_mode=-1) as srv, E.Context(device=0) as ctx:
        tickets = []
        for k, m in enumerate(meshes):
            F = np.random.default_rng(k).standard_normal((2,) + m.f.shape) * (m.id == 0)
            tickets.append((m, F, srv.submit(m, F, tol=1e-10, maxit=50000)))
        for m, F, t in tickets:
            U, infos, _, status = srv.wait(t, timeout=300)
            assert status == 0
            ctx.set_mesh(m)
            ctx.build_structure(True)
            st = ctx.structure()
            ctx.assemble(None, None)
            for k in range(2):
                m.f = F[k]
                b, u0 = E.pload(m, st.id)
                x, i = ctx.solve(b, tol=1e-10, maxit=50000)
                assert abs(infos[k]["iters"] - i["iters"]) <= max(2, 0.01 * i["iters"])
                assert rel_inf(ctx.update(x, u0), U[k]) <= 1e-8


# one column of a small matrix runs as one cluster of up to 16 blocks: one
# slice, 15 to 17, a last slice that is not full, partly fixed nodes, and the
# sizes on both sides of the rule (the larger of each pair runs as a grid)
SMALL = {
    "quad4 1 slice": lambda: M.box2d(4, 7, etype=M.QUAD4_STRESS),
    "quad4 15 slices": lambda: M.box2d(24, 19, etype=M.QUAD4_STRAIN),
    "tria3 16 slices": lambda: M.box2d(32, 15, etype=M.TRIA3_STRESS),
    "quad4 17 slices": lambda: M.box2d(32, 16, etype=M.QUAD4_STRESS),
    "quad4 rollers": lambda: rollers(M.box2d(23, 17, etype=M.QUAD4_STRAIN), 1),
    "hexa8 rollers": lambda: rollers(M.box_hexa8(7, 5, 6, jitter=0.1), 0),
    "tria3 cluster": lambda: M.box2d(60, 58, etype=M.TRIA3_STRESS),
    "tria3 grid": lambda: M.box2d(80, 56, etype=M.TRIA3_STRESS),
    "hexa8 cluster": lambda: M.box_hexa8(8, 8, 9),
    "hexa8 grid": lambda: M.box_hexa8(9, 10, 10),
}


@pytest.mark.parametrize("name", sorted(SMALL))
def test_small_matrices(gpu_ctx, name):
    s, ad, al, b = _system(gpu_ctx, SMALL[name]())
    x_o, i_o = O.pcg(s, ad, al, b, tol=1e-12, maxit=20000)
    x, i = gpu_ctx.solve(b, tol=1e-12, maxit=20000)
    assert rel_inf(x_o, x) <= 1e-10 and abs(i["iters"] - i_o["iters"]) <= 2
    for e in (-400, 0, 400):
        xs, js = gpu_ctx.solve(np.ldexp(b, e), tol=1e-12, maxit=20000)
        assert js["iters"] == i["iters"] and np.array_equal(np.ldexp(x, e), xs)
    for maxit in (1, 7, i["iters"] - 1):
        _, j = gpu_ctx.solve(b, tol=1e-12, maxit=maxit, raise_on_error=False)
        assert j["status"] == E.ERR_NO_CONVERGENCE and j["iters"] == maxit
    c = b.copy()
    c[-1] = np.nan
    _, j = gpu_ctx.solve(c, tol=1e-12, maxit=50, raise_on_error=False)
    assert j["status"] == E.ERR_NO_CONVERGENCE
    z, j = gpu_ctx.solve(0 * b, tol=1e-12)
    assert j["status"] == 0 and j["iters"] == 0 and not z.any()


# FP32 block products as one resident wave: 3 CTAs per SM on 152 SMs, 64, 32
# and 16 block rows a CTA at W = 16, 8 and 4; matrices whose passes are below
# the wave, equal to it at W = 16, above it, and several times it
@pytest.mark.parametrize("nz", [23, 24, 25])
@pytest.mark.parametrize("width", [4, 8, 16])
def test_block_products_of_one_wave(gpu_ctx, nz, width):
    s, ad, al, b = _system(gpu_ctx, M.box_hexa8(31, 37, nz))
    assert s.neq == 3 * 32 * 38 * nz
    B = np.random.default_rng(nz).standard_normal((b.size, width))
    X, infos = gpu_ctx.solve_block(B, precision=E.PREC_MIXED, tol=1e-9, maxit=20000, width=width)
    for i in infos:
        assert i["status"] == 0 and i["norm_m_r"] <= 3.16 * i["conv"]
    x_o, _ = O.pcg_omp(s, ad, al, B[:, -1], tol=1e-12, maxit=20000)
    assert rel_inf(x_o, X[:, -1]) <= 1e-6
    X2, _ = gpu_ctx.solve_block(B, precision=E.PREC_MIXED, tol=1e-9, maxit=20000, width=width)
    assert np.array_equal(X, X2)


@pytest.mark.parametrize("kind", ["fp64", "mixed", "gmres"])
def test_threads_with_matrices_of_different_sizes(built_lib, kind):
    """The same kernel launched by several threads for blocks of 3, 12 and 66 KB
    of vectors: the kernel's shared memory limit is no launch's own."""
    args = {"fp64": dict(maxit=4), "mixed": dict(precision=E.PREC_MIXED, maxit=4),
            "gmres": dict(solver=E.SOLVER_GMRES, ngram=4, maxit=1)}[kind]
    errors = []

    def work(n, count):
        try:
            with E.Context(device=0) as ctx:
                m = M.box_hexa8(n, n, n)
                ctx.set_mesh(m)
                ctx.build_structure(True)
                b, _ = E.pload(m, ctx.structure().id)
                ctx.assemble(None, b)
                x0 = None
                for _ in range(count):
                    x, i = ctx.solve(b, tol=1e-13, raise_on_error=False, **args)
                    assert i["status"] in (0, E.ERR_NO_CONVERGENCE) and x.any()
                    assert x0 is None or np.array_equal(x, x0)
                    x0 = x
        except Exception as e:  # noqa: BLE001 - reported by the main thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=a) for a in ((12, 300), (20, 200), (40, 60))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
