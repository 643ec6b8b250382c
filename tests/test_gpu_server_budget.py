"""The memory that a request's teams share with one another counts against the
server's budget: 16 KB for each load case in the pack."""
import numpy as np
import pytest

import elastic_gb300 as E
from elastic_gb300 import meshgen as M

pytestmark = pytest.mark.gpu

SYNC = 15 * 1024  # of one load case, at least


def test_words_of_the_pack_are_counted(built_lib):
    m = M.box_hexa8(2, 2, 2)
    peak = {}
    for nrhs in (1, 129):
        F = np.random.default_rng(1).standard_normal((nrhs,) + m.f.shape) * (m.id == 0)
        with E.Server(device=0) as srv:
            U, infos, _, status = srv.wait(srv.submit(m, F, tol=1e-10), timeout=120)
            assert status == 0 and np.isfinite(U).all()
            peak[nrhs] = srv.stats()["peak_bytes"]
    n = 3 * 3 * 3 * 2  # free dofs
    assert peak[129] - peak[1] >= 128 * (5 * 8 * n + SYNC)


def test_a_budget_without_room_for_them_refuses(built_lib):
    m = M.box_hexa8(2, 2, 2)
    F = np.random.default_rng(1).standard_normal((200,) + m.f.shape) * (m.id == 0)
    with E.Server(device=0, hbm_budget=2 << 20) as srv:
        _, _, _, status = srv.wait(srv.submit(m, F, tol=1e-10), timeout=120)
        assert status == E.ERR_OOM
        U, _, _, status = srv.wait(srv.submit(m, F[:8], tol=1e-10), timeout=120)
        assert status == 0 and srv.stats()["peak_bytes"] <= 2 << 20
