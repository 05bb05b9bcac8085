"""Heavy rows on both sides of the rule that weighs segment lists against
lookups, at the widest B that lists take (2048 chunks), in one chunk and with
B rows of one entry, bit for bit against the oracle: one-shot exact and
learned, a descriptor's fill and its replay."""

import numpy as np
import pytest

import oracle
import rvsp_b200 as rv
from gpu_util import DevCSR, dev, oneshot
from rvsp_b200 import gen
from test_parity_gpu import assert_same, oracle_full

pytestmark = pytest.mark.gpu

# heavy rows, their entries, rows of B, their entries, columns, chunk width
CASES = [
    (300, 500, 3000, 40, 1 << 20, 9),    # lists: many pairs
    (300, 500, 3000, 40, 1 << 22, 11),
    (2, 500, 3000, 40, 1 << 22, 11),     # lookups: few rows, many chunks
    (1, 2100, 3000, 1, 5000, 11),        # lists: a short launch
    (3000, 64, 3000, 40, 2048, 11),      # lists: one chunk, many products an entry
    (17000, 300, 3000, 2, 4096, 11),     # lookups: two products an entry
]


@pytest.mark.parametrize("rows,alen,K,blen,cols,cw", CASES)
def test_both_sides(gpu_lib, rows, alen, K, blen, cols, cw):
    rng = np.random.default_rng(rows + cols)
    counts = np.full(rows + 5, alen)
    counts[rng.choice(counts.size, 5, replace=False)] = [0, 1, 2, 3, K]
    A = gen.from_keys(counts.size, K, gen._distinct_rows(counts, K, rng), None, rng)
    B = gen.from_keys(K, cols, gen._distinct_rows(np.full(K, blen), cols, rng), None, rng)
    want = oracle_full(A, B)
    try:
        rv.check(rv.set_default_params((32, 2, 64, cw)))
        for algo in (rv.RVSP_CUDA_ALGO_EXACT, rv.RVSP_CUDA_ALGO_LEARNED):
            assert_same(oneshot(A, B, algo=algo), want, str(algo))
        d = rv.Descriptor(rv.RVSP_SPGEMM_ALGO_CUDA)
        dA, dB = DevCSR(A), DevCSR(B)
        st, ws, nnz = d.work_estimation(dA.struct(), dB.struct())
        rv.check(st)
        crp, cci, cv = (dev(np.zeros(A.rows + 1, np.int32)), dev(np.zeros(nnz, np.int32)),
                        dev(np.zeros(nnz, np.float32)))
        c = rv.csr_struct(A.rows, B.cols, nnz, crp, cci, cv)
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
