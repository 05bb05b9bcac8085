"""Batches whose products hold none, one, a warp's and many warps' worth of A
entries side by side, each product bit for bit against the oracle."""

import numpy as np
import pytest

import oracle
import rvsp_b200 as rv
from gpu_util import DevCSR, bits, d2h
from rvsp_b200 import gen

pytestmark = pytest.mark.gpu


def _matrix(entries, n, rng):
    counts = np.bincount(rng.integers(0, n, entries), minlength=n)
    return gen.from_keys(n, n, gen._distinct_rows(np.minimum(counts, n), n, rng), None, rng)


@pytest.mark.parametrize("algo", [rv.RVSP_CUDA_ALGO_EXACT, rv.RVSP_CUDA_ALGO_LEARNED])
@pytest.mark.parametrize("seed,sizes", [
    (0, [0, 1, 0, 0, 31, 32, 33, 0, 511, 512, 513, 1, 1, 1, 8192, 0]),
    (1, [1] * 700),
    (2, [0] * 40 + [20000] + [3] * 200 + [0] * 40),
    (3, [0, 0]),
])
def test_batched_products(gpu_lib, algo, seed, sizes):
    rng = np.random.default_rng(seed)
    pairs = []
    for e in sizes:
        n = max(4, int(e ** 0.5) * 2)
        pairs.append((_matrix(e, n, rng), _matrix(2 * e, n, rng)))
    dev = [(DevCSR(a), DevCSR(b)) for a, b in pairs]
    (prp, pci, pv), nnz, rows, entries = rv.spgemm_batched(dev, algo)
    rp = d2h(prp, int(rows[-1]) + len(pairs), np.int32)
    ci, v = d2h(pci, nnz, np.int32), d2h(pv, nnz, np.float32)
    for p in (prp, pci, pv):
        rv.free_device(p)
    for i, (a, b) in enumerate(pairs):
        wrp, wci, wv = oracle.spgemm_f32(a, b)
        r0, e0, e1 = int(rows[i]) + i, int(entries[i]), int(entries[i + 1])
        assert np.array_equal(rp[r0:r0 + a.rows + 1], wrp)
        assert np.array_equal(ci[e0:e1], wci)
        assert np.array_equal(bits(v[e0:e1]), bits(wv))
