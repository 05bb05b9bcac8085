"""Rows sorted by column (k_sort): row sizes at the bins' edges, short and
long B rows with empty ones between, repeated columns, and column counts at
the limit of the packed words and past it (where the hash kernel takes the
rows), bit for bit against the oracle: one-shot exact and learned, and a
descriptor's fill and its replay on new values."""

import numpy as np
import pytest

import oracle
import rvsp_b200 as rv
from gpu_util import DevCSR, bits, dev, oneshot
from rvsp_b200 import gen
from test_legacy_dtypes_gpu import assert_typed_same, cuda_typed, typed_pair
from test_parity_gpu import assert_same, oracle_full

pytestmark = pytest.mark.gpu

EDGES = [33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 511, 512, 513, 1023, 1024, 1025,
         2047, 2048, 2049]
LENGTHS = [0, 1, 2, 3, 7, 16, 33, 100, 300]


def _edge_product(cols, repeats, seed, clustered=False):
    """A's rows have EDGES products each, made of B rows of LENGTHS entries
    (empty ones among them), every B row used up to `repeats` times."""
    rng = np.random.default_rng(seed)
    per = 120  # B rows of each length
    counts = np.minimum(np.repeat(LENGTHS, per), cols)
    parts = [np.sort(rng.choice(cols, n, replace=False)) if cols < 1 << 20
             else np.unique(rng.integers(0, cols, 2 * n))[:n] for n in counts]
    if clustered:  # runs of columns, few of them: crowded buckets
        parts = [int(rng.integers(0, 6)) * (cols // 7) + np.arange(n) for n in counts]
    for p in parts:  # the outermost columns occur
        if p.size > 1:
            p[0], p[-1] = 0, cols - 1
    lens = np.array([p.size for p in parts])
    brp = np.concatenate([[0], np.cumsum(lens)])
    B = gen.CSR(len(parts), cols, brp.astype(np.int32), np.concatenate(parts).astype(np.int32),
                rng.uniform(-1, 1, int(brp[-1])).astype(np.float32))
    # A has `repeats` columns for each B row of its pool: the rows of B are
    # stacked that many times, so an A row can use one B row's columns again
    S = gen.CSR(B.rows * repeats, cols,
                np.concatenate([[0], np.cumsum(np.tile(lens, repeats))]).astype(np.int32),
                np.tile(B.col_idx, repeats), rng.uniform(-1, 1, B.nnz * repeats).astype(np.float32))
    slen = S.row_lengths()
    rows = []
    for target in EDGES * 4:
        left, pick = target, set()
        for length in rng.permutation(LENGTHS).tolist() + [16, 7, 3, 2, 1, 1, 1]:
            pool = np.flatnonzero(slen == length)
            if length == 0:
                pick.update(rng.choice(pool, 40, replace=False).tolist())
                continue
            if pool.size == 0:
                continue
            most = left // length if length == 1 else min(left // length, rng.integers(1, 20))
            free = np.setdiff1d(pool, list(pick))
            take = free[:min(most, free.size)]
            pick.update(take.tolist())
            left -= length * take.size
        rows.append(np.array(sorted(pick)))
    rp = np.concatenate([[0], np.cumsum([r.size for r in rows])]).astype(np.int32)
    A = gen.CSR(len(rows), S.rows, rp, np.concatenate(rows).astype(np.int32),
                rng.uniform(-1, 1, int(rp[-1])).astype(np.float32))
    return A, S


CASES = [(5000, 1, False), (400, 4, False), (1044480, 1, False), (1044481, 2, False),
         ((1 << 26) + 1, 1, False), (100000, 1, True), (3000, 4, True)]


@pytest.mark.parametrize("cols,repeats,clustered", CASES)
def test_row_sizes_at_the_bins_edges(gpu_lib, cols, repeats, clustered):
    A, B = _edge_product(cols, repeats, cols % 97, clustered)
    ops = gen.row_products(A, B)
    assert {64, 65, 128, 256, 512, 1024, 2048} & set(ops.tolist())
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


def test_signed_zeros_and_non_finite_values(gpu_lib):
    """Runs start from +0.0f; infinities and NaN pass through like the
    reference's (compared as values: a NaN's payload is not specified)."""
    A, B = _edge_product(5000, 1, 3)
    A.values[::5] = -0.0
    B.values[::7] = 0.0
    B.values[3::11] = np.inf
    want = oracle_full(A, B)
    got = oneshot(A, B)
    assert np.array_equal(got[1], want[1])
    nan = np.isnan(want[2])
    assert np.array_equal(np.isnan(got[2]), nan)
    assert np.array_equal(bits(got[2])[~nan], bits(want[2])[~nan])


@pytest.mark.parametrize("dtype", ["f64", "i8"])
@pytest.mark.parametrize("cols,repeats,clustered", [(5000, 1, False), (400, 4, False),
                                                    (1044480, 1, False), (3000, 4, True)])
def test_typed_rows_at_the_bins_edges(gpu_lib, dtype, cols, repeats, clustered):
    """FP64 and INT8 through the sorting pass (rows of up to 2048 products; the
    2049-product rows dropped), zero sums left out."""
    A, B = _edge_product(cols, repeats, cols % 97, clustered)
    keep = np.flatnonzero(gen.row_products(A, B) <= 2048)
    rp = A.row_ptr
    A = gen.CSR(keep.size, A.cols,
                np.concatenate([[0], np.cumsum(np.diff(rp)[keep])]).astype(np.int32),
                np.concatenate([A.col_idx[rp[r]:rp[r + 1]] for r in keep]),
                np.concatenate([A.values[rp[r]:rp[r + 1]] for r in keep]))
    A, B = typed_pair(A, B, dtype, seed=3)
    want = oracle.spgemm_typed(A, B, dtype)
    for device in (True, False):
        assert_typed_same(cuda_typed(A, B, dtype, device), want, dtype, f"{cols} {device}")
