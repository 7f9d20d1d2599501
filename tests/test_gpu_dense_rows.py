"""Dense gates on 3 to 6 wires at many rows, whose tiles the CTAs share out across row borders: more rows
than CTAs, rows of one and of several tiles, one matrix and one a row.  Oracle and tolerance of
test_gpu_dense_tile.py."""
import pytest

from tests import test_gpu_dense_tile as dense

pytestmark = pytest.mark.gpu

CASES = [(14, 3, 153, [13, 0, 6], True), (13, 4, 305, [1, 12, 5, 8], False), (13, 5, 457, [12, 11, 0, 1, 2], True),
         (14, 6, 229, [3, 0, 13, 7, 9, 10], True), (6, 6, 700, [5, 4, 3, 2, 1, 0], True), (8, 5, 913, [7, 1, 4, 0, 2], False),
         (9, 3, 1999, [0, 8, 4], True), (12, 6, 311, [0, 2, 4, 6, 8, 10], False)]


@pytest.mark.parametrize("n,k,bsz,wires,per_row", CASES)
def test_many_rows(n, k, bsz, wires, per_row):
    dense.test_dense_tile_kernels(n, k, bsz, wires, per_row)
