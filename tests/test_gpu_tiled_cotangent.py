"""Operand cotangents of tile passes are float32 over at most 64 terms and as good as float64 beyond:
with identities as gates and amplitudes that are whole numbers below 360, a sum of 64 products stays
below 2^24 and is exact, and so must the whole sum be.  Every kind of op, targets and controls inside and
outside of tiles and registers, one operand and one a row, runs of up to 64 ops with cotangents."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# n, batch rows, ops
CASES = [(9, 1, 12), (9, 37, 64), (10, 5, 30), (12, 3, 64), (13, 20, 40), (14, 330, 9), (16, 4, 64), (20, 2, 50)]


@pytest.mark.parametrize("n,bsz,nops", CASES)
def test_cotangents_of_whole_numbers_are_exact(n, bsz, nops):
    from torchquantum_gb300 import _lib

    rng = np.random.default_rng(100 * n + nops)
    gen = torch.Generator(device="cuda").manual_seed(n)
    whole = lambda: torch.view_as_complex(  # noqa: E731
        torch.randint(0, 360, (bsz, 1 << n, 2), device="cuda", generator=gen).to(torch.float32))
    psi, lam = whole(), whole()
    prod = lam.to(torch.complex128), psi.to(torch.complex128)
    tile = [0, 1, 2, 3] + sorted(int(b) for b in rng.choice(np.arange(4, n), min(n, 12) - 4, replace=False))
    mask = sum(1 << b for b in tile)
    index = torch.arange(1 << n, device="cuda")
    bit = lambda w: (index >> (n - 1 - w)) & 1  # noqa: E731
    ops, want, keep = [], [], []
    for _ in range(nops):
        kind = [_lib.S_DENSE1, _lib.S_PHASE, _lib.S_DIAG][int(rng.choice(3, p=[0.6, 0.2, 0.2]))]
        rows = int(rng.choice([1, bsz]))
        others = [int(w) for w in rng.choice(n, int(rng.integers(0, 3)), replace=False)]
        op = _lib.StagedOp()
        l2, p2 = prod
        if kind == _lib.S_DENSE1:
            t = n - 1 - int(rng.choice(tile))
            wires = [w for w in others if w != t] + [t]
            on = index[torch.stack([bit(w) == 1 for w in wires[:-1]] + [bit(t) == 0]).all(0)]
            pair = torch.stack([on, on ^ (1 << (n - 1 - t))])
            g = torch.einsum("bra,bca->brc", l2[:, pair], p2[:, pair].conj()).reshape(bsz, 4)
            val = torch.eye(2, dtype=torch.complex64, device="cuda").reshape(1, 4).repeat(rows, 1)
        elif kind == _lib.S_PHASE:
            wires = others or [int(rng.integers(n))]
            on = torch.stack([bit(w) == 1 for w in wires]).all(0)
            g = (l2[:, on] * p2[:, on].conj()).sum(1, keepdim=True)
            val = torch.ones(rows, 1, dtype=torch.complex64, device="cuda")
        else:
            wires = others or [int(rng.integers(n))]
            entry = sum(bit(w) << (len(wires) - 1 - j) for j, w in enumerate(wires))
            g = torch.stack([(l2[:, entry == e] * p2[:, entry == e].conj()).sum(1) for e in range(1 << len(wires))], 1)
            val = torch.ones(rows, 1 << len(wires), dtype=torch.complex64, device="cuda")
        grad = torch.zeros(rows, val.shape[1], dtype=torch.complex128, device="cuda")
        op.kind, op.nwires, op.ctrl_val, op.batch = kind, len(wires), 1, rows
        op.operand, op.grad = val.data_ptr(), grad.data_ptr()
        for j, w in enumerate(wires):
            op.wires[j] = w
        ops.append(op)
        want.append(g if rows == bsz else g.sum(0, keepdim=True))
        keep.append((val, grad))
    p1, l1 = psi.clone(), lam.clone()
    _lib.staged_adjoint(p1, l1, n, ops, mask)
    assert torch.equal(p1, psi) and torch.equal(l1, lam)
    for g, (_, grad) in zip(want, keep):
        assert torch.equal(grad, g)
