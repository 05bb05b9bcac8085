"""Heavy rows by segment lists: rows of one and of several list units, every
chunk width, B rows inside one chunk, across all of them and empty, and a B
too wide for the lists (the lookup kernel), bit for bit against the oracle:
one-shot exact and learned, a descriptor's fill and its replay."""

import numpy as np
import pytest

import oracle
import rvsp_b200 as rv
from gpu_util import DevCSR, bits, dev, oneshot
from rvsp_b200 import gen
from test_parity_gpu import assert_same, oracle_full

pytestmark = pytest.mark.gpu


def _product(cols, seed):
    rng = np.random.default_rng(seed)
    K = 3000
    lens = np.concatenate([np.zeros(200, np.int64), rng.integers(1, 4, 1000),
                           rng.integers(4, 60, 1600), rng.integers(500, 4000, 200)])
    rng.shuffle(lens)
    parts = []
    for i, n in enumerate(lens):
        span = cols if i % 3 else min(cols, 900)  # a third of the rows within 900 columns
        lo = int(rng.integers(0, cols - span + 1))
        parts.append(np.unique(lo + rng.integers(0, span, n)))
    blen = np.array([p.size for p in parts])
    B = gen.CSR(K, cols, np.concatenate([[0], np.cumsum(blen)]).astype(np.int32),
                np.concatenate(parts).astype(np.int32),
                rng.uniform(-1, 1, int(blen.sum())).astype(np.float32))
    # 511, 512, 513 entries and several units beside short rows of long B rows
    counts = np.array([511, 512, 513, 1024, 1025, 2900, 3000, 40, 60, 0, 5, 700])
    A = gen.from_keys(counts.size, K, gen._distinct_rows(counts, K, rng), None, rng)
    return A, B


CASES = [(40000, 11), (40000, 9), (40000, 13), (2048, 11), (2049, 11), (1 << 20, 9),
         ((1 << 22) + 1, 11), (1 << 22, 11)]


@pytest.mark.parametrize("cols,cw", CASES)
def test_heavy_rows_match_oracle(gpu_lib, cols, cw):
    A, B = _product(cols, cols % 89 + cw)
    want = oracle_full(A, B)
    try:
        rv.check(rv.set_default_params((32, 2, 64, cw)))
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
        for _ in range(2):
            rv.check(d.compute(dA.struct(), dB.struct(), c, np.zeros(256, np.uint8)))
            assert_same((crp.cpu().numpy(), cci.cpu().numpy(), cv.cpu().numpy()), want, "descriptor")
            A = gen.CSR(A.rows, A.cols, A.row_ptr, A.col_idx,
                        rng.uniform(-1, 1, A.nnz).astype(np.float32))
            dA.values.copy_(dev(A.values))
            want = (want[0], want[1], oracle.spgemm_f32(A, B)[2])
        d.close()
    finally:
        rv.set_default_params(None)


def test_zero_sums_and_non_finite_values(gpu_lib):
    """Sums that cancel, that are zero of either sign and that are not finite
    in dense chunks and sparse stretches: every occurring column is there, bit
    for bit (a NaN as a NaN: its payload is not specified)."""
    A, B = _product(40000, 7)
    rng = np.random.default_rng(11)
    A.values[:] = rng.choice(np.float32([1, -1, 0.0, -0.0]), A.nnz)
    B.values[:] = rng.choice(np.float32([1, -1, 0.0, -0.0, 2]), B.nnz)
    B.values[5::997] = np.inf
    want = oracle_full(A, B)
    assert (want[2] == 0).sum() > 1000 and np.isnan(want[2]).any()
    nan = np.isnan(want[2])
    try:
        rv.check(rv.set_default_params((32, 2, 64, 11)))
        for algo in (rv.RVSP_CUDA_ALGO_EXACT, rv.RVSP_CUDA_ALGO_LEARNED):
            got = oneshot(A, B, algo=algo)
            assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
            assert np.array_equal(np.isnan(got[2]), nan)
            assert np.array_equal(bits(got[2])[~nan], bits(want[2])[~nan])
    finally:
        rv.check(rv.set_default_params(None))
