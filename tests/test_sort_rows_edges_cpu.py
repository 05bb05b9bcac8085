"""The operands of the sorted rows' GPU tests hold rows at both sides of every
bin's edge."""

import pytest

import test_sort_rows_gpu as gpu_tests
from rvsp_b200 import gen

EDGES = {64, 65, 128, 129, 256, 257, 512, 513, 1024, 1025, 2048, 2049}


@pytest.mark.parametrize("cols,repeats,clustered", gpu_tests.CASES)
def test_edges_occur(cols, repeats, clustered):
    A, B = gpu_tests._edge_product(cols, repeats, cols % 97, clustered)
    ops = set(gen.row_products(A, B).tolist())
    assert EDGES <= ops, sorted(EDGES - ops)
