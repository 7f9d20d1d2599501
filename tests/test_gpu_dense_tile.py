"""Dense gates on 3 to 6 wires: forward, in-place reverse step (with U^H and with an explicit
inverse) and the reverse step against a kept input, at the edges of a tile (no other wire, one
column, fewer than four columns, several tiles) and with targets on the lowest, highest and
mixed index bits, against torch in complex128.

Tolerance 1e-5 of the largest entry: sums of D <= 64 products in float32, cotangents in
float32 over at most 32 columns and compensated beyond."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

CASES = [(3, 3, 2, [0, 1, 2], False), (4, 3, 1, [3, 0, 2], True), (6, 6, 3, [5, 4, 3, 2, 1, 0], True),
         (7, 6, 1, [0, 1, 2, 4, 5, 6], False), (7, 5, 2, [6, 2, 4, 0, 1], False), (8, 4, 5, [7, 6, 5, 4], True),
         (11, 3, 2, [10, 0, 5], False), (12, 5, 1, [11, 10, 9, 8, 7], True), (12, 6, 2, [0, 2, 4, 6, 8, 10], False),
         (14, 4, 3, [13, 1, 7, 12], False), (16, 5, 2, [3, 15, 9, 0, 14], True), (17, 6, 1, [16, 15, 1, 0, 8, 5], False),
         (18, 3, 2, [17, 16, 15], False), (19, 4, 1, [0, 18, 9, 1], True), (18, 5, 3, [2, 3, 4, 5, 17], False)]


def _split(v, n, wires):
    order = [0] + [w + 1 for w in wires] + [i + 1 for i in range(n) if i not in wires]
    return v.view([-1] + [2] * n).permute(order).reshape(v.shape[0], 1 << len(wires), -1)


def _join(x, n, wires):
    order = [0] + [w + 1 for w in wires] + [i + 1 for i in range(n) if i not in wires]
    return x.reshape([-1] + [2] * n).permute([order.index(i) for i in range(n + 1)]).reshape(x.shape[0], -1)


def _close(got, want):
    assert float((got - want).abs().max()) <= 1e-5 * max(1.0, float(want.abs().max()))


@pytest.mark.parametrize("n,k,bsz,wires,per_row", CASES)
def test_dense_tile_kernels(n, k, bsz, wires, per_row):
    from torchquantum_gb300 import _lib, binding

    gen = torch.Generator(device="cuda").manual_seed(97 * n + k)
    rand = lambda *s: torch.randn(*s, dtype=torch.complex64, device="cuda", generator=gen)  # noqa: E731
    rows, d = (bsz if per_row else 1), 1 << k
    u = torch.linalg.qr(rand(rows, d, d))[0].contiguous()
    inv = (torch.linalg.inv(u) * 0.5).contiguous()  # not U^H: an explicit uncompute matrix is used as given
    x, lam = rand(bsz, 1 << n) / np.sqrt(1 << n), rand(bsz, 1 << n)
    u2, i2, x2, l2 = (t.to(torch.complex128) for t in (u, inv, x, lam))
    out = x.clone()
    _lib.apply_matrix(out, n, wires, u, rows)
    _close(out, _join(u2 @ _split(x2, n, wires), n, wires))
    for unc, m2 in ((None, u2.conj().transpose(1, 2)), (inv, i2)):
        for want_grad in (True, False):
            psi, la = x.clone(), lam.clone()
            g = torch.zeros(rows * d * d * 2, dtype=torch.float64, device="cuda") if want_grad else None
            _lib.adjoint_matrix(psi, la, n, wires, u, rows, g, unc)
            y = m2 @ _split(x2, n, wires)
            _close(psi, _join(y, n, wires))
            _close(la, _join(u2.conj().transpose(1, 2) @ _split(l2, n, wires), n, wires))
            if want_grad:
                ref = _split(l2, n, wires) @ y.conj().transpose(1, 2)
                _close(torch.view_as_complex(g.view(rows, d, d, 2)), ref if per_row else ref.sum(0, keepdim=True))
    s = x.view([bsz] + [2] * n).clone().requires_grad_(True)
    m = (u if per_row else u[0]).clone().requires_grad_(True)
    res = binding.apply_unitary_bmm(s, m, wires)
    gs, gm = torch.autograd.grad(res, (s, m), lam.view(s.shape))
    _close(res.detach().view(bsz, -1), _join(u2 @ _split(x2, n, wires), n, wires))
    _close(gs.view(bsz, -1), _join(u2.conj().transpose(1, 2) @ _split(l2, n, wires), n, wires))
    ref = _split(l2, n, wires) @ _split(x2, n, wires).conj().transpose(1, 2)
    _close(gm, ref if per_row else ref.sum(0))
    assert torch.equal(s.detach().view(bsz, -1), x)
