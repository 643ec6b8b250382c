"""The resident solvers under a memory budget: whatever the budget leaves room
for without their plan still runs, on the launches of one iteration each, and
a solve that does not fit leaves a context that solves the next one."""
import numpy as np
import pytest

import elastic_gb300 as E
import oracle as O
from elastic_gb300 import meshgen as M
from helpers import rel_inf

pytestmark = pytest.mark.gpu


def _start(budget=0):
    m = M.box_hexa8(21, 22, 23)
    m.f = np.random.default_rng(1).standard_normal(m.f.shape) * (m.id == 0)
    ctx = E.Context(device=0, hbm_budget=budget)
    ctx.set_mesh(m)
    ctx.build_structure(True)
    b, _ = E.pload(m, ctx.structure().id)
    ctx.assemble(None, b)
    return ctx, m, b


@pytest.fixture(scope="module")
def system(built_lib):
    ctx, m, b = _start()
    with ctx:
        _, ad, al = ctx.assemble(None, b, want_matrix=True)
        s = O.structure(m, True)
        x, _ = O.pcg_omp(s, ad, al, b, tol=1e-12, maxit=20000)
        return ctx.device_bytes, b.size, b, x


def _block_bytes(width, precision):
    ctx, _, b = _start()
    with ctx:
        ctx.solve_block(np.ones((b.size, width)), precision=precision, width=width, maxit=1,
                        raise_on_error=False)
        return ctx.device_bytes


def test_block_solve_without_room_for_its_vectors(system):
    """A budget that holds the block buffers of an earlier mixed solve and the
    plan, but not the resident block solve's vectors: the block launches."""
    base, n, b, x = system
    budget = _block_bytes(8, E.PREC_MIXED) + 40 * n
    ctx, _, _ = _start(budget)
    with ctx:
        B = np.outer(b, 2.0 ** np.arange(5))
        ctx.solve_block(B, precision=E.PREC_MIXED, tol=1e-9, width=8)
        X, infos = ctx.solve_block(B, precision=E.PREC_FP64, tol=1e-11, width=8)
        assert all(i["status"] == 0 for i in infos)
        for k in range(5):
            assert rel_inf(x, X[:, k] / 2.0 ** k) <= 1e-9
        assert ctx.device_bytes <= budget


def test_block_solve_that_does_not_fit_leaves_the_context_usable(system):
    base, n, b, x = system
    ctx, _, _ = _start(base + 30 * n + (1 << 20))
    with ctx:
        assert rel_inf(x, ctx.solve(b, tol=1e-11)[0]) <= 1e-9
        with pytest.raises(E.ElasticError) as e:
            ctx.solve_block(np.outer(b, np.ones(6)), precision=E.PREC_FP64, tol=1e-11, width=16)
        assert e.value.code == E.ERR_OOM
        y, i = ctx.solve(b, solver=E.SOLVER_GMRES, ngram=2, tol=1e-11, maxit=1, raise_on_error=False)
        assert i["status"] in (E.OK, E.ERR_NO_CONVERGENCE) and np.isfinite(y).all() and y.any()
        assert rel_inf(x, ctx.solve(b, tol=1e-11)[0]) <= 1e-9


def test_other_solvers_take_the_place_of_the_plan(system):
    """Budgets that hold one solver's vectors but not the plan beside them."""
    base, n, b, x = system
    ctx, _, _ = _start(base + 24 * n + (64 << 10))
    with ctx:
        assert rel_inf(x, ctx.solve(b, tol=1e-11)[0]) <= 1e-9
        y, _ = ctx.solve(b, solver=E.SOLVER_BICGSTAB, tol=1e-11)  # 16 n bytes
        assert rel_inf(x, y) <= 1e-8
        assert rel_inf(x, ctx.solve(b, tol=1e-11)[0]) <= 1e-9
    k = 40
    ctx, _, _ = _start(base + 8 * n * (k + 1) + (128 << 10))
    with ctx:
        assert rel_inf(x, ctx.solve(b, tol=1e-11)[0]) <= 1e-9
        y, _ = ctx.solve(b, solver=E.SOLVER_GMRES, ngram=k, tol=1e-11)
        assert rel_inf(x, y) <= 1e-8
        y2, _ = ctx.solve(b, solver=E.SOLVER_GMRES, ngram=k, tol=1e-11)
        assert np.array_equal(y, y2)
