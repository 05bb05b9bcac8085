"""Tiles of rows that hold most of A's entries (k_analyze_big): a hub tile at
the start, in the middle, across two tiles and as the ragged last one, rows
long and short in it, and too few tiles or entries to be split. Bit for bit
against the oracle, exact and learned."""

import numpy as np
import pytest

import rvsp_b200 as rv
from gpu_util import oneshot
from rvsp_b200 import gen
from test_parity_gpu import assert_same, oracle_full

pytestmark = pytest.mark.gpu


def _product(rows, hubs, entries, seed):
    rng = np.random.default_rng(seed)
    K = 2000
    counts = rng.integers(0, 4, rows)
    counts[hubs] = entries
    B = gen.from_keys(K, 3000, gen._distinct_rows(rng.integers(0, 5, K), 3000, rng), None, rng)
    A = gen.from_keys(rows, K, gen._distinct_rows(counts, K, rng), None, rng)
    return A, B


# rows of A, first row of the hubs, their entries
CASES = [(256 * 32, 0, [1000] * 9), (256 * 40 + 6, 256 * 40, [2000] * 6),
         (256 * 64 + 200, 256 * 64 + 10, [1800] * 20),
         (256 * 50, 256 * 20 + 5, [33, 32, 31] + [2000] * 30),
         (256 * 33, 250, [1900] * 40), (256 * 31, 0, [2000] * 30), (256 * 32, 0, [1024] * 8),
         (256 * 32, 256, [1021] * 4)]


@pytest.mark.parametrize("rows,first,entries", CASES)
def test_hub_tiles(gpu_lib, rows, first, entries):
    hubs = np.arange(first, min(first + len(entries), rows))
    A, B = _product(rows, hubs, entries[:hubs.size], rows % 83)
    want = oracle_full(A, B)
    assert_same(oneshot(A, B), want, "exact")
    assert_same(oneshot(A, B, algo=rv.RVSP_CUDA_ALGO_LEARNED), want, "learned")
