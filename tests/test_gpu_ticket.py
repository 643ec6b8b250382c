"""elx_spmv_dot_noalloc after calls that overlapped: those race for the scratch
and their dots are undefined, but the next call by itself is right again."""
import ctypes as C

import numpy as np
import pytest

import elastic_gb300 as E
from test_gpu_rows_spmv import _call, _expected, _random_lower
from test_zz_no_alloc import upper_csr

pytestmark = pytest.mark.gpu


def test_a_call_after_overlapping_calls(built_lib):
    torch = pytest.importorskip("torch")
    streams = [torch.cuda.Stream() for _ in range(2)]
    calls = []
    for neq, st in zip((200000, 77777), streams):
        ia, ja, ad, al = _random_lower(neq, 3, neq)
        iat, jat, pt = upper_csr(ia, ja, neq)
        d = [torch.from_numpy(a).cuda() for a in (ia, ja, ad, al, iat, jat, al[pt], np.ones(neq))]
        d += [torch.empty(neq, dtype=torch.float64, device="cuda"),
              torch.empty(1, dtype=torch.float64, device="cuda")]
        calls.append((neq, d, [C.c_void_p(t.data_ptr()) for t in d], C.c_void_p(st.cuda_stream)))
    ia, ja, ad, al = _random_lower(5000, 7, 1)
    x = np.random.default_rng(2).standard_normal(5000)
    want = _expected(ia, ja, ad, al, x)
    fn = E.load().elx_spmv_dot_noalloc
    for rounds in (1, 7, 50):
        torch.cuda.synchronize()
        for _ in range(rounds):
            for neq, _, p, st in calls:
                assert fn(neq, *p, st) == E.OK
        torch.cuda.synchronize()
        y, xy = _call(ia, ja, ad, al, x)
        assert np.abs(y - want).max() <= 1e-14 * np.abs(want).max() * 7 ** 0.5
        assert abs(xy - x @ want) <= 1e-13 * np.abs(x * want).sum()
