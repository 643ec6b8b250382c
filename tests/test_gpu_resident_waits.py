"""The bounded waits of the resident solvers: with one block that does not take
part (ELX_GRID_STALL_TEST=1; the others' waits run out after a second) each
solve returns ELX_ERR_TIMEOUT after the two launches in flight, whatever maxit
is, and the same context solves correctly once the stall is lifted."""
import time

import numpy as np
import pytest

import elastic_gb300 as E
import oracle as O
from elastic_gb300 import meshgen as M
from helpers import rel_inf, rollers

pytestmark = pytest.mark.gpu

KINDS = {
    "fp64": dict(),
    "mixed": dict(precision=E.PREC_MIXED),
    "gmres": dict(solver=E.SOLVER_GMRES, ngram=17),
}


@pytest.mark.parametrize("kind", sorted(KINDS) + ["rollers", "block"])
def test_a_wait_that_runs_out(built_lib, monkeypatch, kind):
    m = M.box2d(90, 80, etype=M.QUAD4_STRESS)  # too large for one cluster
    if kind == "rollers":
        m = rollers(m, 1)
    m.f = np.random.default_rng(3).standard_normal(m.f.shape) * (m.id == 0)
    with E.Context(device=0) as ctx:
        ctx.set_mesh(m)
        ctx.build_structure(True)
        s = O.structure(m, True)
        b0, u0 = O.loads(m, s)
        ad, al, b = O.assemble(m, s, u0, b0)
        ctx.assemble(u0, b0)
        x_o, _ = O.pcg(s, ad, al, b, tol=1e-11, maxit=20000)

        def solve(**kw):
            if kind == "block":
                X, infos = ctx.solve_block(np.outer(b, [1.0, 2.0, 4.0]), tol=1e-10,
                                           precision=E.PREC_FP64, maxit=20000)
                return X[:, 2] / 4, infos[2]
            return ctx.solve(b, maxit=kw.get("maxit", 20000), tol=1e-10, **KINDS.get(kind, {}))

        monkeypatch.setenv("ELX_GRID_STALL_TEST", "1")
        t0 = time.monotonic()
        with pytest.raises(E.ElasticError) as e:
            solve()
        assert e.value.code == E.ERR_TIMEOUT and "resident" in str(e.value)
        assert time.monotonic() - t0 < 4
        monkeypatch.delenv("ELX_GRID_STALL_TEST")
        if kind != "gmres":
            x, i = solve()
            assert i["status"] == 0 and rel_inf(x_o, x) <= (1e-5 if kind == "mixed" else 1e-8)
        else:
            g_o, _ = O.gmres(s, ad, al, b, k=17, tol=1e-14, maxit=1)
            x, _ = ctx.solve(b, solver=E.SOLVER_GMRES, ngram=17, tol=1e-14, maxit=1,
                             raise_on_error=False)
            assert rel_inf(g_o, x) <= 1e-9


def test_a_wait_of_the_pack_that_runs_out(built_lib, monkeypatch):
    m = M.box_hexa8(8, 9, 7)
    F = np.random.default_rng(3).standard_normal((2,) + m.f.shape) * (m.id == 0)
    monkeypatch.setenv("ELX_GRID_STALL_TEST", "1")
    with E.Server(device=0) as srv:
        t0 = time.monotonic()
        assert srv.wait(srv.submit(m, F, tol=1e-10), timeout=60)[3] == E.ERR_CUDA
        assert time.monotonic() - t0 < 5
    monkeypatch.delenv("ELX_GRID_STALL_TEST")
    with E.Server(device=0) as srv:
        U, _, _, status = srv.wait(srv.submit(m, F, tol=1e-10), timeout=60)
        assert status == 0 and U.any()
