"""Expectation values of strings with several X-masks are float32 over at most 64 visits of amplitude
pairs and as good as float64 beyond: on amplitudes that are whole numbers below 180 the sum of 64 visits
(4 products, counted twice) stays below 2^24 and is exact, and so must the whole value be.  Strings of X
alone, whose terms all have one sign, so that longer float32 sums would leave the range of exact ones."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,bsz,count", [(9, 7, 11), (12, 3, 11), (13, 5, 11), (17, 3, 2), (17, 1, 1), (20, 2, 11)])
def test_values_of_whole_numbers_are_exact(n, bsz, count):
    from torchquantum_gb300 import _lib

    gen = torch.Generator(device="cuda").manual_seed(n)
    psi = torch.view_as_complex(torch.randint(0, 180, (bsz, 1 << n, 2), device="cuda", generator=gen).to(torch.float32))
    bit = lambda b: 1 << min(n - 1, b)  # noqa: E731
    masks = [(1 << n) - 1, bit(10), 0, 1, 2, 3, bit(5), bit(6) | 1, bit(9), bit(11) | 2, 1 << (n - 1)][:count]
    if count == 1:
        masks = masks + [0]  # one string beside the norm: both have few visits
    got = _lib.pauli_expval(psi, n, masks, [0] * len(masks))
    p = psi.to(torch.complex128)
    index = torch.arange(1 << n, device="cuda")
    want = torch.stack([(p.conj() * p[:, index ^ x]).sum(1).real for x in masks], 1)
    assert torch.equal(got, want)
