"""Drop-in gate application out of place (tqk_apply_matrix_to / tqk_adjoint_matrix_stored):
result, state gradient and matrix gradient against torch in complex128, for both wire counts,
shared and per-row matrices, every alignment of the lowest bit, sizes at the edges of a
thread's work, and states that are conjugated, strided or misaligned views.

Tolerance: a result sums D <= 4 products and a matrix gradient 2^n / D * bsz of them, float32
within a block of at most 2 * 16 * 256 groups: 1e-5 of the largest entry covers both."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _reference(x, m, wires, g):
    bsz, n, k = x.shape[0], x.dim() - 1, len(wires)
    order = [0] + [w + 1 for w in wires] + [i + 1 for i in range(n) if i not in wires]
    back = [order.index(i) for i in range(n + 1)]
    x, m, g = (t.detach().to(torch.complex128) for t in (x, m, g))
    m3 = m if m.dim() == 3 else m[None]
    flat = lambda t: t.permute(order).reshape(bsz, 1 << k, -1)  # noqa: E731
    unflat = lambda t: t.reshape([bsz] + [2] * n).permute(back)  # noqa: E731
    gm = flat(g) @ flat(x).conj().transpose(1, 2)
    return unflat(m3 @ flat(x)), unflat(m3.conj().transpose(1, 2) @ flat(g)), gm if m.dim() == 3 else gm.sum(0)


@pytest.mark.parametrize("view", ["plain", "conj", "strided", "misaligned"])
@pytest.mark.parametrize("n,bsz,wires,per_row", [
    (1, 1, [0], False), (2, 5, [1], True), (2, 1, [1, 0], False), (3, 2, [0, 2], True), (9, 3, [8], True),
    (10, 1, [4, 9], False), (13, 2, [0], False), (14, 3, [13, 2], True), (17, 1, [3, 7], False), (17, 2, [16], False),
    (19, 2, [18, 0], False)])
def test_apply_unitary_out_of_place(n, bsz, wires, per_row, view):
    from torchquantum_gb300 import binding

    gen = torch.Generator(device="cuda").manual_seed(n * 10 + bsz)
    rand = lambda *s: torch.randn(*s, dtype=torch.complex64, device="cuda", generator=gen)  # noqa: E731
    d = 1 << len(wires)
    base = rand(bsz * (1 << n) * 2 + 1) / np.sqrt(1 << n)
    if view == "strided":
        x = base[:bsz * (1 << n) * 2].view([bsz] + [2] * n + [2])[..., 1]
    elif view == "misaligned":
        x = base[1:1 + bsz * (1 << n)].view([bsz] + [2] * n)
    else:
        x = base[:bsz * (1 << n)].view([bsz] + [2] * n)
    if view == "conj":
        x = x.conj()
    x = x.detach().requires_grad_(True)
    m = (rand(bsz, d, d) if per_row else rand(d, d)).requires_grad_(True)
    g = rand(*([bsz] + [2] * n))
    keep = x.detach().clone(), g.clone()
    out = binding.apply_unitary_bmm(x, m, wires)
    gx, gm = torch.autograd.grad(out, (x, m), g.conj() if view == "conj" else g)
    ref = _reference(x, m, wires, g.conj() if view == "conj" else g)
    for got, want in zip((out, gx, gm), ref):
        assert got.shape == want.shape
        assert float((got.detach() - want).abs().max()) <= 1e-5 * max(1.0, float(want.abs().max()))
    assert torch.equal(x.detach(), keep[0]) and torch.equal(g, keep[1])  # neither input is written
    only_state = torch.autograd.grad(binding.apply_unitary_bmm(x, m.detach(), wires), x, g)[0]
    assert torch.equal(only_state, torch.autograd.grad(binding.apply_unitary_bmm(x, m, wires), x, g)[0])


def test_entry_points_refuse_aliases_and_wide_gates():
    import ctypes

    from torchquantum_gb300 import _lib, binding

    lib = binding._load()
    s = torch.zeros(1, 256, dtype=torch.complex64, device="cuda")
    m = torch.eye(128, dtype=torch.complex64, device="cuda")
    w = (ctypes.c_int32 * 7)(*range(7))
    st = torch.cuda.current_stream().cuda_stream
    p, o = s.data_ptr(), torch.zeros_like(s)
    assert lib.tqk_apply_matrix_to(p, p, 1, 8, w, 1, m.data_ptr(), 1, st) != 0
    assert lib.tqk_apply_matrix_to(p, o.data_ptr(), 1, 8, w, 7, m.data_ptr(), 1, st) != 0
    assert lib.tqk_adjoint_matrix_stored(p, p, p, 1, 8, w, 1, m.data_ptr(), 1, None, st) != 0
    assert lib.tqk_adjoint_matrix_stored(p, p, o.data_ptr(), 1, 8, w, 7, m.data_ptr(), 1, None, st) != 0
    assert _lib.load() is not None
