"""Heavy rows times a B that the segment lists cannot describe: rows that
repeat columns keep the reference's sums, rows whose columns run backwards
are refused, and what lies in B's arrays outside every row is never read as a
column."""

import numpy as np
import pytest

import rvsp_b200 as rv
from gpu_util import oneshot
from rvsp_b200 import gen
from test_parity_gpu import assert_same, oracle_full

pytestmark = pytest.mark.gpu

ALGOS = [rv.RVSP_CUDA_ALGO_EXACT, rv.RVSP_CUDA_ALGO_LEARNED]
COLS, K = 40000, 2000


@pytest.fixture(autouse=True)
def heavy_params(gpu_lib):
    rv.check(rv.set_default_params((32, 2, 64, 11)))  # rows of some 50 columns and more
    yield
    rv.check(rv.set_default_params(None))


def _b(rows, rng):
    rp = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    ci = np.concatenate(rows).astype(np.int32)
    return gen.CSR(K, COLS, rp, ci, rng.uniform(-1, 1, ci.size).astype(np.float32))


def _a(rng):
    counts = np.array([300, 500, 64, 65, 1200, 0, 7])
    return gen.from_keys(counts.size, K, gen._distinct_rows(counts, K, rng), None, rng)


@pytest.mark.parametrize("algo", ALGOS)
def test_repeated_columns(algo):
    rng = np.random.default_rng(1)
    rows = [np.sort(rng.integers(0, COLS, 5)) for _ in range(K)]
    for r in rows[::3]:
        r[1:3] = r[1]  # next to each other, in every third row
    rows[4][:] = rows[4][0]
    A, B = _a(rng), _b(rows, rng)
    assert_same(oneshot(A, B, algo=algo), oracle_full(A, B))


@pytest.mark.parametrize("algo", ALGOS)
def test_columns_backwards(algo):
    rng = np.random.default_rng(2)
    rows = [np.sort(rng.choice(COLS, 5, replace=False)) for _ in range(K)]
    rows[K // 2] = np.array([2, 1, 3]) * 2048 + 7  # first column below the last one
    A, B = _a(rng), _b(rows, rng)
    assert (A.col_idx == K // 2).any()
    with pytest.raises(rv.RvspError) as e:
        oneshot(A, B, algo=algo)
    assert e.value.status == rv.RVSP_ERROR_INVALID_CSR


@pytest.mark.parametrize("algo", ALGOS)
def test_entries_outside_every_row(algo):
    rng = np.random.default_rng(3)
    rows = [np.sort(rng.choice(COLS, 5, replace=False)) for _ in range(K)]
    A, B = _a(rng), _b(rows, rng)
    want = oracle_full(A, B)
    junk = np.array([-1, COLS, 2**31 - 1, -2**31, 9, 3, 1 << 20], np.int32)
    P = gen.CSR(K, COLS, B.row_ptr + junk.size, np.concatenate([junk, B.col_idx]),
                np.concatenate([np.full(junk.size, np.nan, np.float32), B.values]))
    assert_same(oneshot(A, P, algo=algo), want)
