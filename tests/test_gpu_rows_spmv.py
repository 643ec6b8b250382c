"""elx_spmv_dot_noalloc at the edges of its loops: blocks of 128 rows, rows of
no entries, of one step of two lanes (16 entries), one more and many, and
infinities, against the product formed from the same arrays.  Bars: the product's (1e-14 of the largest |y|) and the dot's
(1e-13 of sum |x y|)."""
import ctypes as C

import numpy as np
import pytest

import elastic_gb300 as E
from test_zz_no_alloc import upper_csr

pytestmark = pytest.mark.gpu


def _random_lower(neq, per_row, seed):
    """A strict lower CSR with up to per_row entries a row, some rows empty."""
    rng = np.random.default_rng(seed)
    ia, ja = [1], []
    for i in range(neq):
        n = 0 if rng.random() < 0.05 else min(i, per_row)
        ja.append(np.sort(rng.choice(i, n, replace=False)) + 1 if n else np.zeros(0, int))
        ia.append(ia[-1] + n)
    ja = np.concatenate(ja).astype(np.int32)
    return np.array(ia, np.int32), ja, rng.standard_normal(neq) + 4.0, rng.standard_normal(ja.size)


def _call(ia, ja, ad, al, x):
    torch = pytest.importorskip("torch")
    neq = ad.size
    iat, jat, pt = upper_csr(ia, ja, neq)
    # one element more: an empty array has no address, and null is refused
    d = [torch.from_numpy(np.append(a, a[:1] if a.size else a.dtype.type(0))).cuda()
         for a in (ia, ja, ad, al, iat, jat, al[pt], x)]
    y = torch.full((neq,), np.nan, dtype=torch.float64, device="cuda")
    xy = torch.full((1,), np.nan, dtype=torch.float64, device="cuda")
    st = E.load().elx_spmv_dot_noalloc(neq, *[C.c_void_p(t.data_ptr()) for t in d],
                                       C.c_void_p(y.data_ptr()), C.c_void_p(xy.data_ptr()),
                                       C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert st == E.OK
    torch.cuda.synchronize()
    return y.cpu().numpy(), xy.item()


def _expected(ia, ja, ad, al, x):
    rows = np.repeat(np.arange(ad.size), np.diff(ia))
    y = ad * x
    np.add.at(y, rows, al * x[ja - 1])
    np.add.at(y, ja - 1, al * x[rows])
    return y


@pytest.mark.parametrize("neq,per_row", [(1, 0), (127, 5), (128, 16), (129, 17), (700, 15),
                                         (700, 32), (900, 300), (60000, 3)])
def test_matches_reference(built_lib, neq, per_row):
    ia, ja, ad, al = _random_lower(neq, per_row, neq + per_row)
    x = np.random.default_rng(2).standard_normal(neq)
    want = _expected(ia, ja, ad, al, x)
    for _ in range(2):  # the ticket is left at zero
        y, xy = _call(ia, ja, ad, al, x)
        assert np.abs(y - want).max() <= 1e-14 * max(np.abs(want).max(), 1.0) * max(1, per_row) ** 0.5
        assert abs(xy - x @ want) <= 1e-13 * np.abs(x * want).sum()


def test_infinities_and_nan_reach_the_dot(built_lib):
    ia, ja, ad, al = _random_lower(300, 10, 5)
    x = np.ones(300)
    x[200] = np.inf
    y, xy = _call(ia, ja, np.abs(ad), np.abs(al), x)
    assert y[200] == np.inf and xy == np.inf
    x[100] = np.nan
    assert np.isnan(_call(ia, ja, ad, al, x)[1])
