"""Which way an FP64 block solve goes, by the launches it takes: one resident
launch for up to six load cases whatever the matrix; more of them in resident
chunks on large matrices, in blocks of 8 or 16 (three launches an iteration)
on small ones, where each chunk would wait again."""
import numpy as np
import pytest

import elastic_gb300 as E
from elastic_gb300 import meshgen as M

pytestmark = pytest.mark.gpu

MESHES = {
    "tria3 small": lambda: M.box2d(20, 10, etype=M.TRIA3_STRESS),
    "quad4 large": lambda: M.box2d(170, 130, etype=M.QUAD4_STRESS),
    "tetra4 small": lambda: M.box_tetra4(9, 9, 9),
    "hexa8 large": lambda: M.box_hexa8(27, 27, 27),
}
ROUTES = [("tria3 small", 6, True), ("tria3 small", 9, False), ("tria3 small", 12, False),
          ("tria3 small", 16, False), ("tria3 small", 24, False),
          ("quad4 large", 6, True), ("quad4 large", 9, True), ("quad4 large", 13, True),
          ("quad4 large", 24, True),
          ("tetra4 small", 7, True), ("tetra4 small", 13, False), ("tetra4 small", 16, False),
          ("hexa8 large", 8, True), ("hexa8 large", 13, True), ("hexa8 large", 16, False)]


@pytest.mark.parametrize("name,nrhs,resident", ROUTES)
def test_route(gpu_ctx, name, nrhs, resident):
    gpu_ctx.set_mesh(MESHES[name]())
    gpu_ctx.build_structure(True)
    gpu_ctx.assemble(None, None)
    n = gpu_ctx.sizes()[0]
    B = np.random.default_rng(nrhs).standard_normal((n, nrhs))
    gpu_ctx.solve_block(B, precision=E.PREC_FP64, tol=1e-9, width=16, maxit=1,
                        raise_on_error=False)  # the plan or the buffers
    n0 = gpu_ctx.kernel_launches
    X, infos = gpu_ctx.solve_block(B, precision=E.PREC_FP64, tol=1e-9, width=16)
    launches = gpu_ctx.kernel_launches - n0
    its = max(i["iters"] for i in infos)
    assert its > 60 and all(i["status"] == 0 for i in infos)
    # a chunk takes a launch per 512 iterations and two for each column's norms
    assert (launches < its + 2 * nrhs) == resident
    x, _ = gpu_ctx.solve(B[:, -1], tol=1e-9)
    assert np.abs(x - X[:, -1]).max() <= 1e-6 * np.abs(x).max()
