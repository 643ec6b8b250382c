"""Which way a GMRES cycle goes, by its launches: one resident launch, or those
of every projection where the cycle is short for the size of the matrix; both
give the oracle's cycle."""
import numpy as np
import pytest

import elastic_gb300 as E
import oracle as O
from elastic_gb300 import meshgen as M
from helpers import rel_inf, rollers

pytestmark = pytest.mark.gpu

MESHES = {
    "quad4": lambda: M.box2d(64, 75, etype=M.QUAD4_STRESS),
    "quad4 rollers": lambda: rollers(M.box2d(64, 75, etype=M.QUAD4_STRESS), 1),
    "hexa8": lambda: M.box_hexa8(8, 8, 8),
    "tria3 large": lambda: M.box2d(500, 400, etype=M.TRIA3_STRESS),
    "tria3 large rollers": lambda: rollers(M.box2d(500, 400, etype=M.TRIA3_STRESS), 1),
}


@pytest.mark.parametrize("name,k,resident", [
    ("quad4", 1, False), ("quad4", 3, True), ("quad4 rollers", 1, False),
    ("quad4 rollers", 2, True), ("hexa8", 1, True), ("tria3 large", 3, False),
    ("tria3 large", 8, True), ("tria3 large rollers", 1, True)])
def test_route(gpu_ctx, name, k, resident):
    m = MESHES[name]()
    m.f = np.random.default_rng(3).standard_normal(m.f.shape) * (m.id == 0)
    gpu_ctx.set_mesh(m)
    gpu_ctx.build_structure(True)
    s = O.structure(m, True)
    b0, u0 = O.loads(m, s)
    ad, al, b = O.assemble(m, s, u0, b0)
    gpu_ctx.assemble(u0, b0)

    def solve(cycles):
        n0 = gpu_ctx.kernel_launches
        x, i = gpu_ctx.solve(b, solver=E.SOLVER_GMRES, tol=1e-14, maxit=cycles, ngram=k,
                             raise_on_error=False)
        return x, i, gpu_ctx.kernel_launches - n0

    solve(1)  # the plan
    x, i, one = solve(1)
    x_o, _ = O.gmres(s, ad, al, b, k=k, tol=1e-14, maxit=1)
    assert i["refinements"] == 1 and rel_inf(x_o, x) <= 1e-9
    assert (solve(3)[2] - one == 2) == resident
