"""COO canonicalisation: list lengths at the sort's tile edges, key widths from
no bits to seven passes, all entries in one row or one cell, and lists long
enough that tiles wait on each other's counts; bit for bit against the oracle."""

import numpy as np
import pytest

import oracle
from test_coo_gpu import coo_to_csr, same

pytestmark = pytest.mark.gpu

TILE = 4096
SHAPES = [(1, 1), (3, 2), (1, 2 ** 31 - 1), (200, 300), (1 << 16, 1 << 16), ((1 << 16) + 1, 1 << 16),
          (1 << 20, 2 ** 31 - 1)]


@pytest.mark.parametrize("rows,cols", SHAPES)
@pytest.mark.parametrize("n", [1, TILE - 1, TILE, TILE + 1, 3 * TILE + 17])
def test_lengths_and_key_widths(gpu_lib, rows, cols, n):
    rng = np.random.default_rng(n + cols % 1000)
    r = rng.integers(0, rows, n).astype(np.int32)
    c = rng.integers(0, cols, n).astype(np.int32)
    half = rng.integers(0, n, n // 2)  # repeats
    r[: n // 2], c[: n // 2] = r[half], c[half]
    v = rng.uniform(-1, 1, n).astype(np.float32)
    v[::9] = -0.0
    for vals in (v, None):
        st, got = coo_to_csr(rows, cols, r, c, vals, False, True, True)
        assert st == 0
        same(got, oracle.coo_to_csr(rows, cols, r, c, vals, False), f"{rows} x {cols}, {n}")


@pytest.mark.parametrize("symmetric", [False, True])
def test_skewed_long_list(gpu_lib, symmetric):
    """2 M entries, half of them in 16 rows and columns (full digits beside
    empty ones), several hundred tiles in flight at once."""
    rng = np.random.default_rng(8)
    m, n = 1 << 18, 2_000_000
    r = rng.integers(0, m, n)
    c = rng.integers(0, m, n)
    hot = rng.random(n) < 0.5
    r[hot] &= 15
    c[hot] &= 15
    v = rng.uniform(-1, 1, n).astype(np.float32)
    st, got = coo_to_csr(m, m, r.astype(np.int32), c.astype(np.int32), v, symmetric, True, True)
    assert st == 0
    same(got, oracle.coo_to_csr(m, m, r.astype(np.int32), c.astype(np.int32), v, symmetric), "skewed")


def test_index_out_of_range_in_a_long_list(gpu_lib):
    n = 5 * TILE
    r = np.zeros(n, np.int32)
    c = np.arange(n, dtype=np.int32)
    for sym in (False, True):
        bad = c.copy()
        bad[n - 2] = n
        st, _ = coo_to_csr(n, n, r, bad, None, sym, True, True)
        assert st == -2
