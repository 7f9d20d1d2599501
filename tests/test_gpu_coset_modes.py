"""Coset passes over every way a string's partner can lie: diagonal, in the same pair, told apart
by the lane, by the warp and by each bit of a thread's pair index, even and odd numbers of Y,
signs that do and do not differ inside a pair -- on stages smaller than, equal to and cut from a
row, with one and several groups of strings; expectation values and their gradient, against
torch in complex128.

Tolerance: products and sums of amplitudes of a normalised row, float32 over at most 16 terms in
sequence: 32 x 2^-24; the gradient sums 2 x strings products: 4 x strings x 2^-24 of its norm."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _strings(n):
    # X-mask bits (amplitude index bit b is wire n - 1 - b), each with Z and Y decorations
    masks = [0, 1, 2, 3, 1 << min(n - 1, 5), (1 << min(n - 1, 6)) | 1, 1 << min(n - 1, 9), 1 << min(n - 1, 10),
             (1 << min(n - 1, 11)) | 2, (1 << (n - 1)) | 5, (1 << n) - 1]
    out = []
    for i, x in enumerate(masks):
        for z in (1, x, (1 << (n - 1)) | (x & -x) | (i & 1)):
            z &= (1 << n) - 1
            s = "".join("IXZY"[(x >> b & 1) | (z >> b & 1) << 1] for b in range(n - 1, -1, -1))
            if set(s) != {"I"} and s not in out:
                out.append(s)
    return out


def _apply(s, psi):
    n = len(s)
    i = torch.arange(1 << n, device=psi.device)
    x = sum(1 << (n - 1 - w) for w, c in enumerate(s) if c in "XY")
    z = sum(1 << (n - 1 - w) for w, c in enumerate(s) if c in "ZY")
    par = torch.zeros_like(i)
    for b in range(n):
        if z >> b & 1:
            par ^= (i ^ x) >> b & 1
    return (1j ** s.count("Y")) * (1 - 2 * par) * psi[:, i ^ x]


@pytest.mark.parametrize("n,bsz", [(4, 3), (8, 5), (11, 2), (12, 1), (13, 3), (14, 200), (17, 2)])
def test_coset_modes(n, bsz):
    import torchquantum_gb300 as tq

    dev = torch.device("cuda", 0)
    gen = torch.Generator(device=dev).manual_seed(n)
    psi = torch.randn(bsz, 1 << n, dtype=torch.complex128, device=dev, generator=gen)
    psi = (psi / psi.norm(dim=1, keepdim=True)).to(torch.complex64)
    strings = _strings(n)
    w = torch.randn(len(strings), device=dev, generator=gen)
    st = psi.clone().requires_grad_(True)
    q = tq.QuantumDevice(n_wires=n, bsz=bsz, device=dev)
    q.set_states(st)
    ev = tq.expval_joint_analytical_batch(q, strings)
    (ev * w).sum().backward()
    p = psi.to(torch.complex128)
    images = [_apply(s, p) for s in strings]
    want = torch.stack([(p.conj() * v).sum(1).real for v in images], 1)
    assert float((ev.detach().double() - want).abs().max()) <= 32 * 2.0 ** -24
    grad = 2 * sum(float(c) * v for c, v in zip(w, images))
    assert float((st.grad - grad).norm(dim=1).max()) <= 4 * len(strings) * 2.0 ** -24 * float(w.abs().sum())
