"""Mixed block solves whose grids are smaller than the slices of the last
block's sum (256 / W), equal and larger: each column meets the FP64 test and
the single FP64 solve (bars of the mixed solver's tests: ||r||_M within 3.16
of its target, x within 1e-6)."""
import numpy as np
import pytest

import elastic_gb300 as E
from elastic_gb300 import meshgen as M
from helpers import rel_inf

pytestmark = pytest.mark.gpu


# equations: 2 (nx + 1) ny of the clamped strip; at W = 16, VC = 4: 64 rows a block
@pytest.mark.parametrize("nx,ny", [(1, 1), (3, 4), (15, 30), (15, 32), (15, 33), (31, 64)])
@pytest.mark.parametrize("width", [1, 2, 4, 8, 16])
def test_small_grids(gpu_ctx, nx, ny, width):
    gpu_ctx.set_mesh(M.box2d(nx, ny, etype=M.QUAD4_STRAIN))
    gpu_ctx.build_structure(True)
    gpu_ctx.assemble(None, None)
    n = gpu_ctx.sizes()[0]
    B = np.random.default_rng(n + width).standard_normal((n, width))
    X, infos = gpu_ctx.solve_block(B, precision=E.PREC_MIXED, tol=1e-9, width=width)
    for c in range(width):
        assert infos[c]["status"] == 0 and infos[c]["norm_m_r"] <= 3.16 * infos[c]["conv"]
    for c in (0, width - 1):
        x, _ = gpu_ctx.solve(B[:, c], tol=1e-12)
        assert rel_inf(x, X[:, c]) <= 1e-6
    X2, _ = gpu_ctx.solve_block(B, precision=E.PREC_MIXED, tol=1e-9, width=width)
    assert np.array_equal(X, X2)
