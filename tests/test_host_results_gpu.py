"""C in host memory: results that are alive together, released in another
order than they were made and made again in sizes around the smallest kept
array (256 KiB), hold their own values throughout, bit for bit."""

import ctypes as C

import numpy as np
import pytest

import rvsp_b200 as rv
from rvsp_b200 import gen
from test_parity_gpu import assert_same, oracle_full

pytestmark = pytest.mark.gpu


def _arrays(c, rows):
    def view(p, t, n):
        return np.ctypeslib.as_array(C.cast(p, C.POINTER(t)), (n,)).copy()
    return (view(c.row_ptr, C.c_int32, rows + 1), view(c.col_idx, C.c_int32, c.nnz),
            view(c.values, C.c_float, c.nnz))


def test_results_alive_together(gpu_lib):
    L = rv.lib()
    rng = np.random.default_rng(2)
    pairs = []
    for rows in (1000, 1024, 1025, 3000, 4096, 9000):  # C: 0.25 to 2.3 MB an array
        A = gen.uniform_fixed(rows, rows, 8, seed=rows)
        pairs.append((A, oracle_full(A, A)))
    opts = rv.SpgemmOptions(rv.RVSP_BACKEND_CUDA, rv.RVSP_DTYPE_FP32, rv.RVSP_DTYPE_FP32)
    for _ in range(3):
        live = []
        for i in rng.permutation(np.repeat(np.arange(len(pairs)), 2)):
            A = pairs[i][0]
            a, c = rv.from_csr(A), rv.CsrMatrix()
            rv.check(L.rvsp_spgemm_csr(C.byref(a), C.byref(a), C.byref(c), C.byref(opts)))
            live.append((i, c))
            if len(live) > 4:  # one goes while the others stay
                j, d = live.pop(int(rng.integers(len(live))))
                assert_same(_arrays(d, pairs[j][0].rows), pairs[j][1], "released")
                L.rvsp_csr_destroy(C.byref(d))
        for j, d in live:
            assert_same(_arrays(d, pairs[j][0].rows), pairs[j][1], "live")
            L.rvsp_csr_destroy(C.byref(d))
