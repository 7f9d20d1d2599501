"""Register sweeps (tile passes, circuit batches) round gates near the identity as the products of
small size first and the large one last would: 1 + e + e' with e = e' = 0.6 x 2^-24 is 1 + 2^-23, not
1 (each e by itself is less than half of 2^-23).  So every output is the float32 nearest to its value in
64 bits."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

E = float(np.float32(0.6 * 2.0 ** -24))
UPPER = np.array([[1 - 1j * E, E], [0, 1]], dtype=np.complex64)   # on (1 + i, 1): 1 + 2 e + i (1 - e)
LOWER = np.array([[1, 0], [E, 1 - 1j * E]], dtype=np.complex64)   # on (1, 1 + i): the same below


def _want(m, pair):
    return (m.astype(np.complex128) @ np.array(pair, dtype=np.complex128)).astype(np.complex64)


@pytest.mark.parametrize("m,pair", [(UPPER, (1 + 1j, 1)), (LOWER, (1, 1 + 1j))])
@pytest.mark.parametrize("n,controlled", [(9, False), (12, False), (14, False), (12, True)])
def test_tile_pass(n, controlled, m, pair):
    from torchquantum_gb300 import _lib

    mt = torch.tensor(m, device="cuda")[None].contiguous()
    want = _want(m, pair)
    index = np.arange(1 << n)
    for w in range(n):
        bit = (index >> (n - 1 - w)) & 1
        state = np.array(pair, dtype=np.complex64)[bit]
        expect = want[bit]
        wires = [w]
        if controlled:
            c = (w + 5) % n
            wires = [c, w]
            expect = np.where((index >> (n - 1 - c)) & 1, expect, state)
        op = _lib.StagedOp()
        op.kind, op.nwires, op.ctrl_val, op.batch, op.operand = _lib.S_DENSE1, len(wires), 1, 1, mt.data_ptr()
        for j, v in enumerate(wires):
            op.wires[j] = v
        st = torch.tensor(state, device="cuda")[None].contiguous()
        mask = ((1 << min(n, 12)) - 1) if n - 1 - w < 12 else (((1 << 11) - 1) | 1 << (n - 1 - w))
        _lib.staged_apply(st, n, [op], mask)
        assert np.array_equal(st.cpu().numpy()[0], expect)


@pytest.mark.parametrize("config", [(14, 512, 1), (14, 256, 1), (13, 256, 3), (13, 128, 3), (11, 128, 6)])
@pytest.mark.parametrize("m,pair", [(UPPER, (1 + 1j, 1)), (LOWER, (1, 1 + 1j))])
def test_circuit_batch(config, m, pair):
    from torchquantum_gb300 import batch as B

    first = np.array([[pair[0], 0], [pair[1], 1]], dtype=np.complex64)
    cb, want = B.CircuitBatch(), []
    for n in (1, 4, 5, 9, 11, 13):
        for w in range(n):
            cb.add_ops(n, np.array([(B.DENSE1, w, 0, 0), (B.DENSE1, w, 0, 1)], dtype=B.OP_T), np.stack([first, m]))
            s = np.zeros(1 << n, dtype=np.complex64)
            s[0], s[1 << (n - 1 - w)] = _want(m, pair)
            want.append(s)
    res = cb.run(torch.device("cuda", 0), return_states=True, config=B.BatchConfig(*config))
    for got, s in zip(res.states, want):
        assert np.array_equal(got.cpu().numpy(), s)
