"""Block solves on device or host arrays whose right-hand sides and solutions share
memory: the solutions and the reported norms are those of the same solve with
separate arrays, bit for bit."""
import numpy as np
import pytest

import elastic_gb300 as E
from elastic_gb300 import meshgen as M

pytestmark = pytest.mark.gpu

KEYS = ("iters", "status", "xkx", "norm_x", "norm_r", "norm_m_r", "conv")


@pytest.mark.parametrize("prec", [E.PREC_FP64, E.PREC_MIXED])
@pytest.mark.parametrize("nrhs", [1, 5, 7])
def test_in_place(gpu_ctx, prec, nrhs):
    torch = pytest.importorskip("torch")
    m = M.box2d(31, 17, etype=M.QUAD4_STRAIN)
    gpu_ctx.set_mesh(m)
    gpu_ctx.build_structure(True)
    gpu_ctx.assemble(None, None)
    n = gpu_ctx.sizes()[0]
    B = torch.from_numpy(np.random.default_rng(nrhs).standard_normal((nrhs, n))).cuda()
    X = torch.empty_like(B)
    torch.cuda.synchronize()
    args = dict(precision=prec, tol=1e-10, maxit=20000)
    want = gpu_ctx.solve_block_device(B.data_ptr(), X.data_ptr(), nrhs, **args)
    # the same array; the solutions a column ahead of the right-hand sides, and behind
    for at_b, at_x in ((0, 0), (1, 0), (0, 1)):
        buf = torch.empty((nrhs + 1, n), dtype=torch.float64, device="cuda")
        buf[at_b:at_b + nrhs] = B
        torch.cuda.synchronize()
        got = gpu_ctx.solve_block_device(buf[at_b:].data_ptr(), buf[at_x:].data_ptr(), nrhs, **args)
        assert torch.equal(buf[at_x:at_x + nrhs], X)
        for w, g in zip(want, got):
            assert all(w[k] == g[k] for k in KEYS), (at_b, at_x, w, g)
        hbuf = np.empty((nrhs + 1, n))
        hbuf[at_b:at_b + nrhs] = B.cpu().numpy()
        infos = (E.Info * nrhs)()
        st = E.load().elx_solve_block(gpu_ctx._h, nrhs, prec, 1e-10, 20000, 0,
                                      hbuf[at_b:].ctypes.data, hbuf[at_x:].ctypes.data, infos)
        assert st == E.OK and np.array_equal(hbuf[at_x:at_x + nrhs], X.cpu().numpy())
        for w, g in zip(want, infos):
            assert all(w[k] == g.as_dict()[k] for k in KEYS), (at_b, at_x)
