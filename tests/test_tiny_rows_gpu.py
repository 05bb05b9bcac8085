"""Rows of at most 32 products (k_tiny_sort): every product count from 0 to
32, empty and repeated B rows' columns, rows that are neighbours in C and rows
scattered among longer ones, column counts at the limit of the packed words
and past it, bit for bit against the oracle: one-shot exact and learned, and a
descriptor's fill and its replay on new values."""

import numpy as np
import pytest

import oracle
import rvsp_b200 as rv
from gpu_util import DevCSR, dev, oneshot
from rvsp_b200 import gen
from test_parity_gpu import assert_same, oracle_full

pytestmark = pytest.mark.gpu


def _product(cols, most, long_rows, rows=413, seed=3):
    """Rows of A with 0 .. `most` products (33 .. 40 for the share
    `long_rows`), from B rows of 0 .. 7 entries that repeat columns."""
    rng = np.random.default_rng(seed)
    lens = np.tile(np.arange(8), 60)
    pool = np.unique(np.concatenate([[0, cols - 1], rng.integers(0, cols, 23)]))
    brp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    bci = np.concatenate([np.sort(rng.choice(pool, n, replace=False)) for n in lens])
    B = gen.CSR(lens.size, cols, brp, bci.astype(np.int32),
                rng.uniform(-1, 1, bci.size).astype(np.float32))
    picks = []
    for r in range(rows):
        left = int(rng.integers(33, 41)) if rng.random() < long_rows else r % (most + 1)
        pick = set(rng.choice(np.flatnonzero(lens == 0), r % 4, replace=False).tolist())
        while left:
            n = int(rng.integers(1, min(left, 7) + 1))
            pick.add(int(rng.choice(np.setdiff1d(np.flatnonzero(lens == n), list(pick)))))
            left -= n
        picks.append(np.array(sorted(pick), np.int32))
    arp = np.concatenate([[0], np.cumsum([p.size for p in picks])]).astype(np.int32)
    A = gen.CSR(rows, B.rows, arp, np.concatenate(picks).astype(np.int32),
                rng.uniform(-1, 1, int(arp[-1])).astype(np.float32))
    return A, B


@pytest.mark.parametrize("cols,most,long_rows", [
    (200, 8, 0.0), (200, 16, 0.0), (200, 24, 0.0), (200, 28, 0.0), (200, 32, 0.0),
    (30, 32, 0.2), (1 << 27, 32, 0.02), ((1 << 27) + 1, 32, 0.02)])
def test_every_product_count(gpu_lib, cols, most, long_rows):
    A, B = _product(cols, most, long_rows)
    want = oracle_full(A, B)
    assert_same(oneshot(A, B), want, "exact")
    assert_same(oneshot(A, B, algo=rv.RVSP_CUDA_ALGO_LEARNED), want, "learned")
    d = rv.Descriptor(rv.RVSP_SPGEMM_ALGO_CUDA)
    dA, dB = DevCSR(A), DevCSR(B)
    st, ws, nnz = d.work_estimation(dA.struct(), dB.struct())
    rv.check(st)
    crp, cci, cv = (dev(np.zeros(A.rows + 1, np.int32)), dev(np.zeros(nnz, np.int32)),
                    dev(np.zeros(nnz, np.float32)))
    c = rv.csr_struct(A.rows, B.cols, nnz, crp, cci, cv)
    rng = np.random.default_rng(5)
    for _ in range(2):  # the fill, then the replay of its position maps
        rv.check(d.compute(dA.struct(), dB.struct(), c, np.zeros(256, np.uint8)))
        assert_same((crp.cpu().numpy(), cci.cpu().numpy(), cv.cpu().numpy()), want, "descriptor")
        A = gen.CSR(A.rows, A.cols, A.row_ptr, A.col_idx,
                    rng.uniform(-1, 1, A.nnz).astype(np.float32))
        dA.values.copy_(dev(A.values))
        want = (want[0], want[1], oracle.spgemm_f32(A, B)[2])
    d.close()
