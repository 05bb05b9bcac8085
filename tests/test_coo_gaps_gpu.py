"""COO lists whose entries leave runs of empty rows: none, a few, a warp's
width and far more, before the first entry, between entries and after the
last one."""

import ctypes as C

import numpy as np
import pytest

import rvsp_b200 as rv
from gpu_util import d2h, dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cols", [1, 1 << 20])
@pytest.mark.parametrize("gaps,after", [
    ([0], 0), ([31, 32, 33, 34, 1, 0, 1], 31), ([100, 0, 1000, 5, 70000], 32),
    ([64] * 300, 500000), (list(range(130)), 1),
])
def test_empty_rows(gpu_lib, cols, gaps, after):
    rng = np.random.default_rng(len(gaps))
    row = np.cumsum(np.array(gaps) + 1) - 1
    row = np.repeat(row, rng.integers(1, 4, row.size))
    rows = int(row[-1]) + 1 + after
    col = rng.integers(0, cols, row.size)
    _, keep = np.unique(row * cols + col, return_index=True)  # no repeats
    row, col = row[keep], col[keep]
    order = rng.permutation(row.size)
    val = rng.uniform(-1, 1, row.size).astype(np.float32)
    r, c, v = dev(row[order].astype(np.int32)), dev(col[order].astype(np.int32)), dev(val[order])
    p, n = [C.c_void_p() for _ in range(3)], C.c_int32()
    rv.check(rv.lib().rvsp_cuda_coo_to_csr(rows, cols, row.size, rv.ptr(r), rv.ptr(c), rv.ptr(v),
                                           0, 1, *[C.byref(x) for x in p], C.byref(n)))
    got = [d2h(p[0].value, rows + 1, np.int32), d2h(p[1].value, n.value, np.int32),
           d2h(p[2].value, n.value, np.float32)]
    for x in p:
        rv.free_device(x.value)
    want = np.concatenate([[0], np.cumsum(np.bincount(row, minlength=rows))])
    assert np.array_equal(got[0], want)
    assert np.array_equal(got[1], col) and np.array_equal(got[2], val)
