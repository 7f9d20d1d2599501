"""Ops outside the limits of a block's table are skipped, also at the end of a chunk of 32, where
the next chunk is read over the skipped ops' records: the product and the cotangents are those of
the other ops.  Several blocks and rows, so that CTAs meet the chunk's end at different times.

Tolerances as in test_gpu_block_build.py: float64 products of unitary ops, 8e-15 an op; the
reverse in float32, (8 ops + 16) 2^-24 |X| |W|."""
import numpy as np
import pytest
import torch

from tests.test_gpu_block_build import _cotangent, _matrix, _random_op

pytestmark = pytest.mark.gpu

# block width, ops, skipped ops
CASES = [(6, 70, (30, 31)), (6, 100, (31, 63)), (4, 65, tuple(range(20, 32))), (3, 96, tuple(range(32, 64))),
         (5, 64, (31, 32, 63)), (2, 33, (0, 31))]
BLOCKS, BATCH = 40, 3


def _break(bo, how, k):
    """One of the ways an op can lie outside the limits."""
    if how == 0:
        bo.kind = 99
    elif how == 1:
        bo.pos[0] = k
    elif how == 2:
        bo.nw = 0
    else:
        bo.nctrl = bo.nw + 1


@pytest.mark.parametrize("k,nops,skipped", CASES)
def test_skipped_ops(k, nops, skipped):
    from torchquantum_gb300 import _lib, engine, program

    rng = np.random.default_rng(7 * k + nops)
    dev, d = torch.device("cuda", 0), 1 << k
    flips = (engine.KIND_X, engine.KIND_SWAP)
    row = [_random_op(rng, range(k), engine) for _ in range(nops)]
    gu = rng.normal(size=(BLOCKS, BATCH, d, d)) + 1j * rng.normal(size=(BLOCKS, BATCH, d, d))
    gu_t = torch.tensor(gu, device=dev)
    u_t = torch.full((BLOCKS, BATCH, d, d), float("nan"), dtype=torch.complex128, device=dev)
    keep, descs, ops = [], [], []
    for i in range(BLOCKS):
        bd = program.BlockDesc()
        bd.first_op, bd.num_ops, bd.k, bd.batch = len(ops), nops, k, BATCH
        bd.u, bd.gu = u_t[i].data_ptr(), gu_t[i].data_ptr()
        descs.append(bd)
        for j, (kind, pos, nc, cv, o) in enumerate(row):
            bo = program.BlockOp()
            bo.kind, bo.nw, bo.nctrl, bo.ctrl_val = program.KIND_ID[kind], len(pos), nc, cv
            for q, p in enumerate(pos):
                bo.pos[q] = p
            bo.batch, bo.op_size = 1, len(o)
            val = torch.tensor(o[None], device=dev)
            grad = torch.zeros_like(val)
            bo.operand = val.data_ptr()
            bo.grad = None if kind in flips else grad.data_ptr()
            if j in skipped:
                _break(bo, j % 4, k)
            keep.append((val, grad))
            ops.append(bo)
    bt, bh = program._to_device_table(descs, dev)
    ot, oh = program._to_device_table(ops, dev)
    for _ in range(5):
        for _, grad in keep:
            grad.zero_()
        u_t.fill_(float("nan"))
        _lib.block_build(bt, BLOCKS, BATCH, ot, dev)
        _lib.block_unbuild(bt, BLOCKS, BATCH, ot, dev)
        torch.cuda.synchronize()
        mats = [None if j in skipped else _matrix(op, k, engine) for j, op in enumerate(row)]
        w = np.eye(d, dtype=complex)
        for g in mats:
            w = w if g is None else g @ w
        assert np.abs(u_t.cpu().numpy() - w).max() <= 8e-15 * nops
        for i in (0, BLOCKS - 1):
            ws, xs = w, [gu[i, b] for b in range(BATCH)]
            tol = sum((8 * nops + 16) * 2.0 ** -24 * np.linalg.norm(x) * np.linalg.norm(w) for x in xs)
            for j in range(nops - 1, -1, -1):
                got = keep[i * nops + j][1][0].cpu().numpy()
                if mats[j] is None:
                    assert not got.any()
                    continue
                ws = mats[j].conj().T @ ws
                want = sum(_cotangent(row[j], x, ws, k, engine) for x in xs) if row[j][0] not in flips else 0
                assert np.abs(got - want).max() <= tol
                xs = [mats[j].conj().T @ x for x in xs]
