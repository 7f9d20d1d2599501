"""Circuit batches run in register sweeps: every kernel variant on widths around the smallest
swept tile, one tile and several tiles, with random one-qubit, controlled, CZ (any pair) and
partial-ladder ops (controls and pairs inside and outside registers and tiles), against numpy.

Tolerance: an op rounds a state by at most 4 x 2^-24 of its norm: ops x 4 x 2^-24."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

CONFIGS = [(14, 512, 1), (14, 256, 1), (13, 256, 3), (13, 128, 3), (12, 128, 6), (11, 256, 2), (10, 128, 8)]
WIDTHS = [1, 2, 5, 8, 9, 10, 11, 12, 14, 15]


def _random_ir(rng, n, count):
    from torchquantum_gb300 import batch as B

    ops, mats = [], []
    for _ in range(count):
        kind = [B.DENSE1, B.CTRL1, B.CZ, B.CZ_LADDER][rng.choice(4, p=[0.55, 0.2, 0.15, 0.1])] if n > 1 else B.DENSE1
        if kind in (B.DENSE1, B.CTRL1):
            q, _ = np.linalg.qr(rng.normal(size=(2, 2)) + 1j * rng.normal(size=(2, 2)))
            mats.append(q)
        w = [int(v) for v in rng.choice(n, min(n, 2), replace=False)]
        if kind == B.CZ_LADDER:
            w = sorted(w)
        ops.append((kind, w[0], w[1] if kind != B.DENSE1 else 0, len(mats) - 1 if kind in (B.DENSE1, B.CTRL1) else -1))
    return np.array(ops, dtype=B.OP_T), np.array(mats).reshape(-1, 2, 2)


def _simulate(n, ops, mats):
    from torchquantum_gb300 import batch as B

    s = np.zeros(1 << n, dtype=complex)
    s[0] = 1.0
    index = np.arange(1 << n)
    bit = lambda w: (index >> (n - 1 - w)) & 1  # noqa: E731
    for kind, w0, w1, m in ops.tolist():
        if kind in (B.DENSE1, B.CTRL1):
            t = w0 if kind == B.DENSE1 else w1
            g = mats[m].astype(np.complex64).astype(complex)
            flip = index ^ (1 << (n - 1 - t))
            new = np.where(bit(t) == 0, g[0, 0] * s + g[0, 1] * s[flip], g[1, 1] * s + g[1, 0] * s[flip])
            s = new if kind == B.DENSE1 else np.where(bit(w0) == 1, new, s)
        else:
            for a, b in [(w0, w1)] if kind == B.CZ else [(w, w + 1) for w in range(w0, w1)]:
                s = np.where((bit(a) & bit(b)) == 1, -s, s)
    return s


@pytest.mark.parametrize("config", CONFIGS)
def test_sweeps_match_numpy(config):
    from torchquantum_gb300 import batch as B

    rng = np.random.default_rng(sum(config))
    cb, want = B.CircuitBatch(), []
    counts = [0, 1, 33, 90]
    for i, n in enumerate(WIDTHS):
        ops, mats = _random_ir(rng, n, counts[(i + sum(config)) % 4])
        cb.add_ops(n, ops, mats, z_wire=int(rng.integers(n)))
        want.append(_simulate(n, ops, mats))
    res = cb.run(torch.device("cuda", 0), return_states=True, config=B.BatchConfig(*config))
    for i, n in enumerate(WIDTHS):
        tol = 4 * 2.0 ** -24 * max(1, len(cb._ops[i]))
        assert np.linalg.norm(res.states[i].cpu().numpy() - want[i]) <= tol
        sign = 1.0 - 2.0 * ((np.arange(1 << n) >> (n - 1 - cb._z[i])) & 1)
        assert abs(res.z[i] - float((sign * abs(want[i]) ** 2).sum())) <= 2 * tol
