"""Block products where blocks and rows are more than the SMs, so that a CTA keeps more columns: every width, with and
without a batch, and both sides of the line.  Oracle and tolerances of test_gpu_block_build.py."""
import pytest

from tests import test_gpu_block_build as build

pytestmark = pytest.mark.gpu

# k, blocks, batch rows, ops, bits the ops may touch
CASES = [(1, 160, 1, 3, 1), (2, 200, 2, 20, 2), (3, 151, 1, 33, 3), (3, 152, 1, 33, 3), (3, 31, 5, 40, 2), (4, 153, 1, 12, 4),
         (4, 20, 8, 35, 4), (5, 152, 1, 9, 5), (5, 26, 6, 33, 3), (6, 160, 1, 10, 6), (6, 20, 8, 12, 5)]


@pytest.mark.parametrize("k,nblocks,batch,nops,nbits", CASES)
def test_many_blocks(k, nblocks, batch, nops, nbits):
    build.test_block_build_and_reverse(k, nblocks, batch, nops, nbits)
