"""Where the blocks of a resident solve cannot all run at once (a process that
has a part of the GPU), the solvers take the launches of one iteration each.
ELX_RESIDENT_BLOCKS asks for 160 blocks, more than the GPU's SMs hold; the
cooperative launch is refused by the runtime."""
import numpy as np
import pytest

import elastic_gb300 as E
import oracle as O
from elastic_gb300 import meshgen as M
from helpers import rel_inf, rollers

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("blocks", [160, 40])
@pytest.mark.parametrize("name", ["clamped", "rollers"])
def test_more_blocks_than_fit(built_lib, monkeypatch, name, blocks):
    m = M.box2d(80, 75, etype=M.QUAD4_STRESS)
    if name == "rollers":
        m = rollers(m, 1)
    m.f = np.random.default_rng(3).standard_normal(m.f.shape) * (m.id == 0)
    monkeypatch.setenv("ELX_RESIDENT_BLOCKS", str(blocks))
    with E.Context(device=0) as ctx:
        ctx.set_mesh(m)
        ctx.build_structure(True)
        s = O.structure(m, True)
        b0, u0 = O.loads(m, s)
        ad, al, b = O.assemble(m, s, u0, b0)
        ctx.assemble(u0, b0)
        x_o, i_o = O.pcg(s, ad, al, b, tol=1e-11, maxit=20000)

        def launches(f):
            n0 = ctx.kernel_launches
            r = f()
            return r, ctx.kernel_launches - n0

        (x, i), n = launches(lambda: ctx.solve(b, tol=1e-11))
        assert rel_inf(x_o, x) <= 1e-9 and abs(i["iters"] - i_o["iters"]) <= 2
        assert (n > 3 * i["iters"]) == (blocks > 152)
        if name == "clamped":
            (x, i), n = launches(lambda: ctx.solve(b, precision=E.PREC_MIXED, tol=1e-9))
            assert i["status"] == 0 and rel_inf(x_o, x) <= 1e-6
            assert (n > 3 * i["inner_iters"]) == (blocks > 152)
            (X, infos), n = launches(lambda: ctx.solve_block(np.outer(b, [1.0, 2.0]), tol=1e-11,
                                                             precision=E.PREC_FP64))
            assert rel_inf(x_o, X[:, 1] / 2) <= 1e-9
            assert (n > 3 * infos[0]["iters"]) == (blocks > 152)
        g_o, _ = O.gmres(s, ad, al, b, k=17, tol=1e-14, maxit=1)
        (x, i), n = launches(lambda: ctx.solve(b, solver=E.SOLVER_GMRES, ngram=17, tol=1e-14,
                                               maxit=1, raise_on_error=False))
        assert rel_inf(g_o, x) <= 1e-9
        assert (n > 17) == (blocks > 152)


@pytest.mark.parametrize("blocks", [10000, 40])
def test_pack_of_more_blocks_than_fit(built_lib, monkeypatch, blocks):
    monkeypatch.setenv("ELX_RESIDENT_BLOCKS", str(blocks))
    m = M.box_hexa8(8, 9, 7)
    F = np.random.default_rng(3).standard_normal((2,) + m.f.shape) * (m.id == 0)
    with E.Server(device=0, poll_steps=1) as srv:
        U, infos, _, status = srv.wait(srv.submit(m, F, tol=1e-11), timeout=120)
        done = srv.stats()["iterations"]
    assert status == 0
    s = O.structure(m, True)
    for k in range(2):
        m.f = F[k]
        b0, u0 = O.loads(m, s)
        ad, al, b = O.assemble(m, s, u0, b0)
        x, i = O.pcg(s, ad, al, b, tol=1e-11, maxit=20000)
        assert abs(infos[k]["iters"] - i["iters"]) <= 2
        u = np.zeros(m.f.shape)
        u[s.id > 0] = x[s.id[s.id > 0] - 1]
        assert rel_inf(u, U[k]) <= 1e-9
    # a packed launch is one iteration; a resident one of HEXA8 four
    assert (done <= max(i["iters"] for i in infos) + 1) == (blocks > 608)
    assert done % 4 == 0 or blocks > 608
