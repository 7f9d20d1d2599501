"""Tile passes of the plain method (tqk_tiled_apply / tqk_tiled_adjoint).

* CPU: a pass plan holds every op once, applies an order equivalent to the recorded one and
  keeps every target inside its tile; the tile layout in shared memory is a bijection whose
  16-byte accesses are conflict free for the lane bits the host picks; the register / thread
  / copy mappings visit every amplitude of every row exactly once.
* GPU: states, expvals and gradients with tile passes equal the gate-by-gate plain method
  and the oracle (1e-5: complex64 against complex128, as for every plain kernel), at widths
  around the edges of the tile and warp sizes and with odd batches.
"""
import numpy as np
import pytest
import torch

from oracle import statevec as O
from torchquantum_gb300 import _lib
from torchquantum_gb300 import engine
from torchquantum_gb300 import program as P

D, C, X, PH, DG, SW = (engine.KIND_DENSE, engine.KIND_CTRL, engine.KIND_X, engine.KIND_PHASE, engine.KIND_DIAG,
                       engine.KIND_SWAP)


def _random_ops(rng, n, count):
    ops = []
    for _ in range(count):
        kind = [D, C, X, PH, DG, SW][int(rng.choice(6, p=[0.35, 0.15, 0.2, 0.15, 0.1, 0.05]))]
        w = [int(v) for v in rng.choice(n, size=2, replace=False)]
        m = torch.eye(2, dtype=torch.complex64)[None]
        if kind == D:
            op = engine.TapeOp(D, w[:1], operand=m)
        elif kind == C:
            op = engine.TapeOp(C, w, controls=w[:1], targets=w[1:], operand=m)
        elif kind == X:
            op = engine.TapeOp(X, w, controls=w[:1], targets=w[1:])
        elif kind == PH:
            op = engine.TapeOp(PH, w, operand=torch.ones(1, dtype=torch.complex64))
        elif kind == DG:
            op = engine.TapeOp(DG, w, operand=torch.ones(1, 4, dtype=torch.complex64))
        else:
            op = engine.TapeOp(SW, w, targets=w)
        ops.append(op)
    return ops


@pytest.mark.parametrize("n,count,small", [(13, 40, True), (16, 150, False), (24, 90, False), (34, 60, True), (9, 70, True),
                                           (12, 40, False)])
def test_plan_holds_every_op_in_an_equivalent_order(n, count, small):
    ops = _random_ops(np.random.default_rng(n), n, count)
    plan = P.plan_tiles(ops, n, small)
    order = [i for idx, _ in plan for i in idx]
    assert sorted(order) == list(range(count))
    place = {i: k for k, i in enumerate(order)}
    for i in range(count):
        for j in range(i + 1, count):  # ops that share a wire keep their order
            if set(ops[i].wires) & set(ops[j].wires):
                assert place[i] < place[j]
    for idx, mask in plan:
        if not mask:
            assert len(idx) == 1
            continue
        assert bin(mask).count("1") == min(n, _lib.STAGED_MAX_TILE_BITS) and mask & 15 == 15 and mask < 1 << n
        assert 2 <= len(idx) <= _lib.STAGED_MAX_OPS
        for i in idx:
            op = ops[i]
            assert op.kind != SW
            if op.kind in (D, C, X):
                t = op.targets[0] if op.kind != D else op.wires[0]
                assert (mask >> (n - 1 - t)) & 1
        if not small:
            assert sum(P._pass_share(ops[i]) for i in idx) >= 1.0


def _swz(l):
    return l ^ ((((l >> 4) ^ (l >> 7) ^ (l >> 10)) & 7) << 1)


def _thread_bits(m, regs):
    """Local bit of each thread bit: three lowest lanes from different classes, then the
    other tile bits ascending."""
    free = [b for b in range(1, m) if b not in regs]
    first = []
    for cls in range(3):
        first += [b for b in free if (b - 1) % 3 == cls][:1]
    return first + [b for b in free if b not in first]


@pytest.mark.parametrize("m", range(9, 13))
def test_tile_mappings_visit_every_amplitude_once(m):
    size, threads = 1 << m, 1 << (m - 4)
    rng = np.random.default_rng(m)
    assert sorted(_swz(l) for l in range(size)) == list(range(size))
    assert all(_swz(l ^ k) == _swz(l) ^ _swz(k) for l, k in rng.integers(0, size, (50, 2)))
    assert all(_swz(l | 1) == _swz(l) | 1 for l in range(0, size, 2))  # 16-byte pairs stay whole
    # copies: thread t, piece group i -> local 2 (t + i threads)
    assert sorted(2 * t + 2 * threads * i for t in range(threads) for i in range(8)) == list(range(0, size, 2))
    for _ in range(8):
        regs = sorted(int(b) for b in rng.choice(np.arange(1, m), size=3, replace=False))
        pos = _thread_bits(m, regs)
        assert len(pos) == m - 4
        seen = []
        for t in range(threads):
            tl = sum(((t >> j) & 1) << b for j, b in enumerate(pos))
            for q in range(8):
                l = tl | sum(((q >> j) & 1) << b for j, b in enumerate(regs))
                assert _swz(l) == _swz(tl) ^ _swz(l ^ tl)
                seen.append(l)
        assert sorted(seen) == list(range(0, size, 2))
        if len({(b - 1) % 3 for b in pos[:3]}) == 3:  # 8 lanes hit 8 different 16-byte banks
            banks = {(_swz(sum(((t >> j) & 1) << b for j, b in enumerate(pos))) >> 1) & 7 for t in range(8)}
            assert len(banks) == 8


def _circuit(rng, n, depth, bsz):
    from torchquantum_gb300 import gates as G

    one = ["u3", "rx", "ry", "rz", "hadamard", "sx", "t"]
    two = ["cnot", "cz", "crx", "crz", "cu1", "rzz", "cu3", "swap", "rxx"]
    gates = []
    for _ in range(depth):
        r = rng.random()
        name = one[int(rng.integers(len(one)))] if r < 0.5 or n == 1 else "toffoli" if r > 0.93 and n > 2 else \
            two[int(rng.integers(len(two)))]
        gd = G.GATES[G.canonical_name(name)]
        wires = [int(w) for w in rng.choice(n, size=gd.num_wires, replace=False)]
        p = None
        if gd.num_params:
            p = rng.uniform(-np.pi, np.pi, size=(bsz if rng.random() < 0.5 else 1, gd.num_params))
        gates.append({"name": name, "wires": wires, "params": p})
    return gates


@pytest.mark.gpu
@pytest.mark.parametrize("n,bsz,depth", [(9, 2, 80), (10, 5, 150), (11, 5, 80), (12, 1, 140), (13, 3, 90), (15, 2, 150),
                                         (18, 1, 60)])
def test_tile_passes_match_gate_by_gate_and_oracle(n, bsz, depth, monkeypatch):
    monkeypatch.setattr(P, "TILE_SHORT_ROW_AMPS", 0)  # small states take the tiled kernels too
    monkeypatch.setattr(P, "TILE_MIN_AMPS", 0)
    import torchquantum_gb300 as tq
    import torchquantum_gb300.functional as tqf

    rng = np.random.default_rng(100 * n + bsz)
    gates = _circuit(rng, n, depth, bsz)
    paulis = ["".join(rng.choice(list("IXYZ"), size=n)) for _ in range(3)]
    dev = torch.device("cuda")
    res = {}
    for stage in (True, False):
        q = tq.QuantumDevice(n_wires=n, bsz=bsz, device=dev)
        q.stage_low = stage
        leaves = []
        for g in gates:
            p = None
            if g["params"] is not None:
                p = torch.tensor(g["params"], dtype=torch.float32, device=dev, requires_grad=True)
                leaves.append(p)
            tqf.func_name_dict[g["name"]](q, wires=g["wires"], params=p)
        ev = tq.expval_joint_analytical_batch(q, paulis)
        ev.sum().backward()
        runs = [o for sg in q._tape for o in sg.exec_ops if isinstance(o, P.StagedRun)]
        assert bool(runs) == stage
        assert all(o.tile_bits > 64 for o in runs)
        if stage and n > 12:
            assert any(o.tile_bits >> 12 for o in runs)
        res[stage] = (q.get_states_1d().detach().cpu().numpy(), ev.detach().cpu().numpy(),
                      [l.grad.cpu().numpy() for l in leaves])
    ref = O.run(n, bsz, [dict(g, params=None if g["params"] is None else np.asarray(g["params"])) for g in gates])
    assert np.abs(res[True][0] - ref).max() < 1e-5
    assert np.abs(res[True][1] - res[False][1]).max() < 1e-5
    for a, b in zip(res[True][2], res[False][2]):
            assert np.abs(a - b).max() < 1e-5 * max(1, bsz / 4)


@pytest.mark.gpu
def test_tiled_abi_checks_mask_and_targets():
    n = 15
    psi = torch.zeros(1, 1 << n, dtype=torch.complex64, device="cuda")
    psi[:, 0] = 1
    m = torch.tensor([[[0, 1], [1, 0]]], dtype=torch.complex64, device="cuda")
    d = _lib.StagedOp()
    d.kind, d.nwires, d.batch, d.operand = _lib.S_DENSE1, 1, 1, m.data_ptr()
    d.wires[0] = 0  # bit 14
    low = (1 << 12) - 1
    with pytest.raises(_lib.TQKError, match="outside the tile"):
        _lib.staged_apply(psi, n, [d], low)
    for bad in (low >> 1 << 1 | 1 << 13, low | 1 << 12, low ^ 1 | 1 << 15):
        with pytest.raises(_lib.TQKError, match="tile holds"):
            _lib.staged_apply(psi, n, [d], bad)
    _lib.staged_apply(psi, n, [d], low ^ (1 << 11) | 1 << 14)
    assert int(psi[0].abs().argmax()) == 1 << 14
