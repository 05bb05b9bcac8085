"""One-shot exact products whose rows go to C through slots: which rows do
(where most are tiny, those are counted and written in place), bit for bit
against the oracle."""

import numpy as np
import pytest

import rvsp_b200 as rv
from gpu_util import oneshot
from rvsp_b200 import gen
from test_parity_gpu import assert_same, oracle_full

pytestmark = pytest.mark.gpu


def _mixed(tiny, rng):
    """Rows of 20 x 20 products, more than 2^22 in all, between `tiny` short ones."""
    K = 3000
    B = gen.from_keys(K, K, gen._distinct_rows(np.full(K, 20), K, rng), None, rng)
    counts = np.concatenate([np.full(11000, 20), np.full(tiny, 1)])
    rng.shuffle(counts)
    return gen.from_keys(counts.size, K, gen._distinct_rows(counts, K, rng), None, rng), B


def _timed(A, B):
    rv.kernel_timing(True)
    try:
        got = oneshot(A, B)
    finally:
        times = rv.kernel_times()
        rv.kernel_timing(False)
    return got, {k: n for k, (_, n) in times.items()}


def test_stencil_rows_are_counted(gpu_lib):
    A = gen.poisson2d(500)
    got, n = _timed(A, A)
    assert n["k_tiny<COUNT>"] == 1 and n["k_compact"] == 0
    assert_same(got, oracle_full(A, A))


@pytest.mark.parametrize("tiny,counted", [(15000, True), (4000, False)])
def test_mixed_rows(gpu_lib, tiny, counted):
    A, B = _mixed(tiny, np.random.default_rng(tiny))
    got, n = _timed(A, B)
    assert n["k_tiny<COUNT>"] == (1 if counted else 0) and n["k_compact"] == 1
    assert_same(got, oracle_full(A, B))
