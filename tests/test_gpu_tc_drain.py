"""Tensor-core blocks whose targets hold index bit 0, bit 1, both or neither (every way the
outputs are stored), forward in place and out of place and both reverse steps, against torch in
complex128.

Tolerance 5e-5 of the largest entry: three bf16 products of split operands (about 2^-16 of a
64-term sum of a unit vector's entries by a unitary's)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

BITS = [[0, 5, 7, 9, 10, 12], [0, 2, 3, 4, 5, 6], [1, 3, 4, 8, 9, 11], [1, 5, 6, 10, 11, 12], [0, 1, 4, 6, 8, 12],
        [1, 2, 3, 5, 7, 9], [2, 3, 6, 8, 10, 11], [7, 8, 9, 10, 11, 12], [0, 8, 9, 10, 11, 12]]


@pytest.mark.parametrize("bits", BITS)
@pytest.mark.parametrize("n,bsz", [(13, 3), (15, 2)])
def test_block_outputs_land_in_place(bits, n, bsz):
    from torchquantum_gb300 import _lib

    dev = torch.device("cuda", 0)
    gen = torch.Generator(device=dev).manual_seed(sum(bits) * n)
    rand = lambda *s: torch.randn(*s, dtype=torch.complex128, device=dev, generator=gen)  # noqa: E731
    wires = [n - 1 - b for b in bits]
    u = torch.linalg.qr(rand(1, 64, 64))[0].contiguous()
    psi, lam = rand(bsz, 1 << n), rand(bsz, 1 << n)
    psi, lam = psi / psi.norm(dim=1, keepdim=True), lam / lam.norm(dim=1, keepdim=True)
    psi, lam = psi.to(torch.complex64), lam.to(torch.complex64)

    def apply(m, x):
        order = [0] + [w + 1 for w in wires] + [i + 1 for i in range(n) if i not in wires]
        y = x.to(torch.complex128).view([-1] + [2] * n).permute(order).reshape(bsz, 64, -1)
        y = (m @ y).reshape([bsz] + [2] * n)
        return y.permute([order.index(i) for i in range(n + 1)]).reshape(bsz, -1)

    def close(got, want):
        assert float((got - want).abs().max()) <= 5e-5 * float(want.abs().max())

    lib, w6 = _lib.load(), _lib._i32(wires)
    status = _lib.status_word(dev)
    st = torch.cuda.current_stream().cuda_stream
    image = _lib.fused_prepare(u, wires)
    image_h = torch.empty_like(image)
    _lib._check(lib.tqk_fused_prepare_adjoint(u.data_ptr(), 1, w6, image_h.data_ptr(), st))
    out = torch.empty_like(psi)
    _lib._check(lib.tqk_fused_apply_to(psi.data_ptr(), out.data_ptr(), bsz, n, w6, image.data_ptr(), 1,
                                       status.data_ptr(), st))
    close(out, apply(u, psi))
    back, cot = out.clone(), lam.clone()
    _lib._check(lib.tqk_fused_adjoint(back.data_ptr(), cot.data_ptr(), bsz, n, w6, image_h.data_ptr(), 1, None,
                                      status.data_ptr(), st))
    want = apply(u.conj().transpose(1, 2), lam)
    close(back, psi.to(torch.complex128))
    close(cot, want)
    kept, got = lam.clone(), torch.empty_like(lam)
    _lib._check(lib.tqk_fused_adjoint_stored_to(psi.data_ptr(), kept.data_ptr(), got.data_ptr(), bsz, n, w6,
                                                image_h.data_ptr(), 1, None, status.data_ptr(), st))
    assert torch.equal(got, cot) and torch.equal(kept, lam)
    _lib._check(lib.tqk_fused_apply(kept.data_ptr(), bsz, n, w6, image.data_ptr(), 1, status.data_ptr(), st))
    close(kept, apply(u, lam))
