"""Matrix cotangents of gates on 3 to 6 wires are float32 over at most 32 columns and as good as
float64 beyond: with the identity as the gate and amplitudes that are whole numbers below 512, a
sum of 32 products stays below 2^24 and is exact, and so must the whole sum be.  Sizes with many
tiles a CTA, with one, and with fewer columns than threads share; one matrix and one a row."""
import pytest
import torch

from tests.test_gpu_dense_tile import _split

pytestmark = pytest.mark.gpu

# n, k, batch rows, wires, a matrix for each row
CASES = [(22, 3, 4, [21, 3, 10], False), (22, 4, 4, [0, 20, 7, 21], False), (22, 5, 4, [2, 9, 21, 0, 13], False),
         (22, 6, 4, [1, 21, 20, 8, 3, 15], False), (21, 3, 8, [0, 1, 2], True), (21, 4, 8, [20, 19, 18, 17], True),
         (21, 5, 8, [4, 0, 20, 11, 7], True), (21, 6, 8, [20, 1, 14, 5, 9, 0], True), (14, 3, 33, [13, 0, 6], False),
         (13, 6, 40, [0, 2, 4, 6, 8, 12], False), (9, 6, 700, [0, 1, 2, 3, 4, 5], True), (12, 5, 130, [11, 0, 5, 6, 7], True),
         (6, 6, 5, [5, 4, 3, 2, 1, 0], False), (7, 5, 3, [6, 2, 4, 0, 1], True), (16, 4, 20, [15, 8, 4, 0], True)]


@pytest.mark.parametrize("n,k,bsz,wires,per_row", CASES)
def test_cotangents_of_whole_numbers_are_exact(n, k, bsz, wires, per_row):
    from torchquantum_gb300 import _lib, binding

    gen = torch.Generator(device="cuda").manual_seed(31 * n + k)

    def whole():
        v = torch.randint(0, 512, (bsz, 1 << n, 2), device="cuda", generator=gen)
        return torch.view_as_complex(v.to(torch.float32))

    rows, d = (bsz if per_row else 1), 1 << k
    u = torch.eye(d, dtype=torch.complex64, device="cuda").repeat(rows, 1, 1)
    x, lam = whole(), whole()
    ref = torch.zeros(rows, d, d, dtype=torch.complex128, device="cuda")
    for b in range(bsz):
        l1, x1 = (_split(t[b:b + 1], n, wires)[0].to(torch.complex128) for t in (lam, x))
        ref[b if per_row else 0] += l1 @ x1.conj().T
    for unc in (None, u):
        psi, la = x.clone(), lam.clone()
        g = torch.zeros(rows * d * d * 2, dtype=torch.float64, device="cuda")
        _lib.adjoint_matrix(psi, la, n, wires, u, rows, g, unc)
        assert torch.equal(torch.view_as_complex(g.view(rows, d, d, 2)), ref)
        assert torch.equal(psi, x) and torch.equal(la, lam)
    m = (u if per_row else u[0]).clone().requires_grad_(True)
    out = binding.apply_unitary_bmm(x.view([bsz] + [2] * n), m, wires)
    gm, = torch.autograd.grad(out, (m,), lam.view(out.shape))
    assert torch.equal(gm, (ref if per_row else ref[0]).to(torch.complex64))
