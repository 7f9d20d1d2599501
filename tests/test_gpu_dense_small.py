"""In-place gates on 3 to 6 wires on both sides of the line between the kernel of one output at a time and the
tiles: rows of few groups and small states.  Oracle and tolerance of test_gpu_dense_tile.py; and the two kernels
give the same states bit for bit: a row of a large batch and the same row in a small one."""
import pytest
import torch

from tests import test_gpu_dense_tile as dense

pytestmark = pytest.mark.gpu

# (k, n, rows): amplitudes just below and above 2^15, 2^16 and 2^18 at 0 to 4 column bits and more
CASES = [(3, 3, 7), (3, 5, 1024), (3, 6, 513), (3, 12, 16), (3, 15, 1), (3, 16, 2), (4, 6, 512), (4, 7, 300), (4, 8, 257), (4, 9, 64),
         (5, 5, 1030), (5, 7, 256), (5, 8, 2000), (5, 9, 65), (6, 6, 700), (6, 8, 128), (6, 9, 129), (6, 10, 32), (6, 7, 4097)]


@pytest.mark.parametrize("per_row", [False, True])
@pytest.mark.parametrize("k,n,bsz", CASES)
def test_small_states(k, n, bsz, per_row):
    wires = [(3 * j + 1) % n for j in range(n)] if n % 3 else list(range(n))[::-1]
    dense.test_dense_tile_kernels(n, k, bsz, wires[:k], per_row)


@pytest.mark.parametrize("k,n", [(3, 6), (4, 7), (5, 8), (6, 9), (3, 13), (5, 14), (6, 13)])
def test_the_same_states_in_small_and_large_batches(k, n):
    from torchquantum_gb300 import _lib

    gen = torch.Generator(device="cuda").manual_seed(n)
    rows = max(4, (1 << 19) >> n)
    x, lam = (torch.randn(rows, 1 << n, dtype=torch.complex64, device="cuda", generator=gen) for _ in range(2))
    u = torch.linalg.qr(torch.randn(1 << k, 1 << k, dtype=torch.complex64, device="cuda", generator=gen))[0].contiguous()
    wires = list(range(n - k, n))
    for m in (1, 2, rows // 3, rows):
        a, p, q = x[:m].clone(), x[:m].clone(), lam[:m].clone()
        _lib.apply_matrix(a, n, wires, u, 1)
        _lib.adjoint_matrix(p, q, n, wires, u, 1, None)
        if m == 1:
            first = a[0].clone(), p[0].clone(), q[0].clone()
        assert all(torch.equal(t[0], f) for t, f in zip((a, p, q), first))
