"""Tile passes at more rows than CTAs fit the GPU, whose tiles the CTAs share out across row borders: rows of one and
of several tiles, angles of a row's own and shared ones.  Against the kernels of one gate, 1e-5 an entry of the
states and the per-row gradients (complex64 against complex64, as in test_tiled.py); shared gradients are sums over
the rows, 1e-5 of their largest with sqrt(rows) such errors."""
import numpy as np
import pytest
import torch

from torchquantum_gb300 import program as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shared", [False, True])
@pytest.mark.parametrize("n,bsz", [(9, 1300), (12, 457), (13, 153), (13, 305), (14, 229), (14, 611)])
def test_rows_are_those_of_one_gate_at_a_time(n, bsz, shared, monkeypatch):
    monkeypatch.setattr(P, "TILE_SHORT_ROW_AMPS", 0)
    monkeypatch.setattr(P, "TILE_MIN_AMPS", 0)
    import torchquantum_gb300 as tq
    import torchquantum_gb300.functional as tqf

    rng = np.random.default_rng(n + bsz)
    gen = torch.Generator(device="cuda").manual_seed(n)
    init = torch.randn(bsz, 1 << n, dtype=torch.complex64, device="cuda", generator=gen)
    init = init / init.norm(dim=1, keepdim=True)
    gates = [(str(rng.choice(["u3", "rx", "rz", "crx", "cnot", "cz", "rzz"])), [int(w) for w in rng.permutation(n)[:2]])
             for _ in range(24)]
    theta = torch.randn(1 if shared else bsz, 72, device="cuda", generator=gen)
    got = []
    for stage in (True, False):
        q = tq.QuantumDevice(n_wires=n, bsz=bsz, device="cuda")
        q.stage_low = stage
        q.set_states(init)
        th = theta.clone().requires_grad_(True)
        for i, (name, ws) in enumerate(gates):
            k = {"u3": 3, "cnot": 0, "cz": 0}.get(name, 1)
            tqf.func_name_dict[name](q, wires=ws if name in ("crx", "cnot", "cz", "rzz") else ws[:1],
                                     params=th[:, 3 * i:3 * i + k] if k else None)
        ev = tq.expval_joint_analytical_batch(q, ["Z" + "I" * (n - 1), "I" * (n - 1) + "X", "Y" * n])
        ev.sum().backward()
        runs = [o for sg in q._tape for o in sg.exec_ops if isinstance(o, P.StagedRun)]
        assert bool(runs) == stage and all(o.tile_bits > 64 for o in runs)
        got.append((q.get_states_1d().detach(), ev.detach(), th.grad))
    for a, b in zip(got[0][:2], got[1][:2]):
        assert float((a - b).abs().max()) < 1e-5
    assert float((got[0][2] - got[1][2]).abs().max()) < 1e-5 * (max(bsz ** 0.5, float(got[1][2].abs().max())) if shared else 1)
