"""The reverse sweep reads the incoming cotangent where it is: the tensor handed to backward is
unchanged, and the gradients are those of a sweep that works in place on a copy of it, whichever
step comes first (tile pass, staged run, lone gate, tensor-core block with and without a stored
input, none at all), also for a cotangent the kernels cannot read in place (odd offset, lazy
conjugate).

The initial state's gradient has the same operations in both: equal.  Parameter gradients add
float64 sums in any order and round to float32: 4 x 2^-24 of the largest."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _gradients(n, method, checkpoint, last, form, depth, monkeypatch, in_place):
    import torchquantum_gb300 as tq
    import torchquantum_gb300.functional as tqf
    from torchquantum_gb300 import program

    monkeypatch.setattr(program, "TILE_SHORT_ROW_AMPS", 0)  # small states take the tile passes too
    monkeypatch.setattr(program, "TILE_MIN_AMPS", 0)
    dev, bsz = torch.device("cuda", 0), 2
    gen = torch.Generator(device=dev).manual_seed(10 * n + depth)
    init = torch.randn(bsz, 1 << n, dtype=torch.complex64, device=dev, generator=gen)
    init = (init / init.norm(dim=1, keepdim=True)).requires_grad_(True)
    theta = (torch.rand(depth + 1, device=dev, generator=gen) * 6 - 3).requires_grad_(True)
    q = tq.QuantumDevice(n_wires=n, bsz=bsz, device=dev)
    q.method, q.checkpoint = "plain" if method == "none" else method, checkpoint
    if method == "fused":
        q.fuse_wires, q.fused_backend = 6, "tc"
    q.set_states(init)
    for i in range(depth):
        tqf.ry(q, wires=i % n, params=theta[i])
        tqf.cnot(q, wires=[i % n, (i + 2) % n])
    wide = torch.linalg.qr(torch.randn(128, 128, dtype=torch.complex128, device=dev, generator=gen))[0]
    if last == "ry":
        tqf.ry(q, wires=1, params=theta[depth])
    elif last == "unitary":  # a gate that no block takes
        tqf.qubitunitaryfast(q, wires=list(range(7)), params=wide.to(torch.complex64))
    out = q.get_states_1d()
    g = torch.randn(bsz * (1 << n) + 1, dtype=torch.complex64, device=dev, generator=gen)
    g = (g[1:] if form == "offset" else g[:-1]).view(bsz, -1)
    given = g.conj() if form == "conj" else g
    before = given.clone()
    if in_place:
        inner = program.Segment.backward

        def on_a_copy(self, psi, lam, need_grads, inputs=None, lam_end=None):
            if lam_end is not None:
                lam.copy_(lam_end)
            return inner(self, psi, lam, need_grads, inputs)

        monkeypatch.setattr(program.Segment, "backward", on_a_copy)
    out.backward(gradient=given)
    assert torch.equal(given, before)
    return init.grad, theta.grad


@pytest.mark.parametrize("n,method,checkpoint,last", [
    (5, "plain", True, "ry"), (10, "plain", True, "ry"), (12, "plain", True, "cnot"), (14, "plain", True, "ry"),
    (14, "fused", True, "ry"), (14, "fused", False, "ry"), (13, "fused", True, "unitary"), (9, "none", True, "")])
@pytest.mark.parametrize("form", ["plain", "offset", "conj"])
def test_cotangent_is_only_read(n, method, checkpoint, last, form, monkeypatch):
    depth = 0 if method == "none" else 30
    got = _gradients(n, method, checkpoint, last, form, depth, monkeypatch, False)
    want = _gradients(n, method, checkpoint, last, form, depth, monkeypatch, True)
    assert torch.equal(got[0], want[0])
    if depth:
        assert float((got[1] - want[1]).abs().max()) <= 4 * 2.0 ** -24 * float(want[1].abs().max())
