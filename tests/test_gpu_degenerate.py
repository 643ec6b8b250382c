"""Elements that name a node twice (a QUAD4 collapsed to a triangle, a HEXA8 to
a wedge): refused where the node has free dofs, solved where it is fixed."""
import numpy as np
import pytest

import elastic_gb300 as E
import oracle as O
from elastic_gb300 import meshgen as M
from helpers import rel_inf

pytestmark = pytest.mark.gpu

MESHES = {
    "quad4": (lambda: M.box2d(5, 4, etype=M.QUAD4_STRESS), [(3, 2)]),
    "hexa8": (lambda: M.box_hexa8(3, 3, 3), [(4, 0), (7, 3)]),
}


def _collapsed(name, fixed):
    make, pairs = MESHES[name]
    m = make()
    ix = m.ix.copy()
    for el in (0, m.numel // 2):  # node a takes node b's place
        for a, b in pairs:
            ix[el, a] = ix[el, b]
    m.ix, m.id = ix, m.id.copy()
    if fixed:
        for el in (0, m.numel // 2):
            for _, b in pairs:
                m.id[ix[el, b] - 1] = 1
    m.f = np.random.default_rng(1).standard_normal(m.f.shape) * (m.id == 0)
    return m


@pytest.mark.parametrize("name", sorted(MESHES))
def test_free_node_twice_is_refused(gpu_ctx, built_lib, name):
    m = _collapsed(name, False)
    gpu_ctx.set_mesh(m)
    with pytest.raises(E.ElasticError) as e:
        gpu_ctx.build_structure(True)
    assert e.value.code == E.ERR_ARG and "twice" in str(e.value)
    with E.Server(device=0) as srv:
        assert srv.wait(srv.submit(m, m.f, tol=1e-8), timeout=60)[3] == E.ERR_ARG


@pytest.mark.parametrize("name", sorted(MESHES))
def test_fixed_node_twice_is_solved(gpu_ctx, name):
    m = _collapsed(name, True)
    gpu_ctx.set_mesh(m)
    gpu_ctx.build_structure(True)
    s = O.structure(m, True)
    b0, u0 = O.loads(m, s)
    ad, al, b = O.assemble(m, s, u0, b0)
    b_g = gpu_ctx.assemble(u0, b0)
    assert rel_inf(b, b_g) <= 1e-13
    x_o, _ = O.pcg(s, ad, al, b, tol=1e-12, maxit=5000)
    x, i = gpu_ctx.solve(b_g, tol=1e-12, maxit=5000)
    assert i["status"] == 0 and rel_inf(x_o, x) <= 1e-10
