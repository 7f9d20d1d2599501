"""Block products and their reverse (k_block_build, k_block_unbuild): widths 1 to 6, every op
kind, ops that reach the block's bits late or never, more ops than one chunk, and block counts
on both sides of the column split, against numpy in complex128.

Tolerances: the build is float64, 1e-15 x 8 roundings per op on unitary products; the reverse
keeps W and X in float32, each op rounding both by at most 8 x 2^-24 of their norm, and sums
chains of at most 16 terms: (8 ops + 16) 2^-24 |X| |W|."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# k, blocks, batch rows, ops, bits the ops may touch
CASES = [(1, 1, 1, 3, 1), (2, 3, 2, 0, 2), (2, 5, 1, 31, 2), (3, 2, 3, 33, 2), (4, 1, 1, 64, 4), (4, 200, 1, 12, 3),
         (5, 7, 2, 65, 5), (5, 90, 1, 40, 5), (6, 1, 1, 70, 6), (6, 30, 1, 25, 4), (6, 60, 1, 32, 6), (6, 40, 4, 20, 6)]


def _unitary(rng, d):
    q, r = np.linalg.qr(rng.normal(size=(d, d)) + 1j * rng.normal(size=(d, d)))
    return q * (np.diag(r) / abs(np.diag(r)))


def _random_op(rng, bits, engine):
    """(kind, wire bits, nctrl, ctrl_val, operand)"""
    kinds = [engine.KIND_DENSE, engine.KIND_CTRL, engine.KIND_X, engine.KIND_SWAP, engine.KIND_PHASE, engine.KIND_DIAG]
    while True:
        kind = kinds[rng.integers(len(kinds))]
        nc = 0 if kind == engine.KIND_DENSE else int(rng.integers(0, 3))
        kt = {engine.KIND_X: 1, engine.KIND_SWAP: 2}.get(kind, int(rng.integers(1, 3)))
        if kind == engine.KIND_DIAG:
            nc, kt = 0, int(rng.integers(1, 7))
        if kind == engine.KIND_CTRL and nc == 0:
            continue
        if nc + kt <= len(bits):
            break
    pos = [int(v) for v in rng.permutation(bits)[:nc + kt]]
    unit = lambda m: np.exp(2j * np.pi * rng.random(m))  # noqa: E731
    opnd = {engine.KIND_PHASE: lambda: unit(1), engine.KIND_DIAG: lambda: unit(1 << kt)}.get(
        kind, lambda: _unitary(rng, 1 << kt).reshape(-1))()
    return kind, pos, nc, int(rng.integers(0, 2)) if kind == engine.KIND_X else 1, opnd


def _rows(pos, val):
    return sum(1 << p for j, p in enumerate(pos) if (val >> (len(pos) - 1 - j)) & 1)


def _matrix(op, k, engine):
    kind, pos, nc, cv, opnd = op
    g = np.eye(1 << k, dtype=complex)
    nw, kt = len(pos), len(pos) - nc
    for base in (r for r in range(1 << k) if not any((r >> p) & 1 for p in pos)):
        if kind == engine.KIND_PHASE:
            r = base | _rows(pos, (1 << nw) - 1)
            g[r, r] = opnd[0]
            continue
        if kind == engine.KIND_DIAG:
            for a in range(1 << nw):
                r = base | _rows(pos, a)
                g[r, r] = opnd[a]
            continue
        ctl = base | (_rows(pos[:nc], (1 << nc) - 1) if kind != engine.KIND_X or cv else 0)
        rows = [ctl | _rows(pos[nc:], a) for a in range(1 << kt)]
        m = {engine.KIND_X: lambda: np.eye(2)[::-1], engine.KIND_SWAP: lambda: np.eye(4)[[0, 2, 1, 3]]}.get(
            kind, lambda: opnd.reshape(1 << kt, 1 << kt))()
        g[np.ix_(rows, rows)] = m
    return g


def _cotangent(op, x, w, k, engine):
    kind, pos, nc, _, opnd = op
    nw, kt = len(pos), len(pos) - nc
    out = np.zeros(len(opnd), dtype=complex)
    for base in (r for r in range(1 << k) if not any((r >> p) & 1 for p in pos)):
        if kind in (engine.KIND_PHASE, engine.KIND_DIAG):
            for a in [(1 << nw) - 1] if kind == engine.KIND_PHASE else range(1 << nw):
                r = base | _rows(pos, a)
                out[0 if kind == engine.KIND_PHASE else a] += x[r] @ w[r].conj()
            continue
        rows = [base | _rows(pos[:nc], (1 << nc) - 1) | _rows(pos[nc:], a) for a in range(1 << kt)]
        out += (x[rows] @ w[rows].conj().T).reshape(-1)
    return out


@pytest.mark.parametrize("k,nblocks,batch,nops,nbits", CASES)
def test_block_build_and_reverse(k, nblocks, batch, nops, nbits):
    from torchquantum_gb300 import _lib, engine, program

    rng = np.random.default_rng(1000 * k + nops)
    dev, d = torch.device("cuda", 0), 1 << k
    flips = (engine.KIND_X, engine.KIND_SWAP)
    # a few distinct blocks with an operand row per batch row; the others repeat them
    distinct = min(nblocks, 2)
    blocks = []
    for _ in range(distinct):
        bits = rng.permutation(k)[:nbits]
        late = [_random_op(rng, bits[:max(1, nbits // 2)] if i < nops // 2 else bits, engine) for i in range(nops)]
        rows = [[(kind, pos, nc, cv, o if b == 0 or kind in flips else _random_same(rng, kind, o, engine))
                 for kind, pos, nc, cv, o in late] for b in range(batch)]
        blocks.append(rows)
    gu = rng.normal(size=(nblocks, batch, d, d)) + 1j * rng.normal(size=(nblocks, batch, d, d))
    gu_t = torch.tensor(gu, device=dev)
    u_t = torch.full((nblocks, batch, d, d), float("nan"), dtype=torch.complex128, device=dev)
    keep, descs, ops = [], [], []
    for i in range(nblocks):
        bd = program.BlockDesc()
        bd.first_op, bd.num_ops, bd.k, bd.batch = len(ops), nops, k, batch
        bd.u, bd.gu = u_t[i].data_ptr(), gu_t[i].data_ptr()
        descs.append(bd)
        for j in range(nops):
            kind, pos, nc, cv, o = blocks[i % distinct][0][j]
            bo = program.BlockOp()
            bo.kind, bo.nw, bo.nctrl, bo.ctrl_val = program.KIND_ID[kind], len(pos), nc, cv
            for q, p in enumerate(pos):
                bo.pos[q] = p
            bo.batch, bo.op_size = batch, len(o)
            val = torch.tensor(np.stack([blocks[i % distinct][b][j][4] for b in range(batch)]), device=dev)
            grad = torch.zeros_like(val)
            bo.operand = val.data_ptr()
            bo.grad = None if kind in flips or j % 7 == 6 else grad.data_ptr()
            keep.append((val, grad))
            ops.append(bo)
    bt, bh = program._to_device_table(descs, dev)
    ot, oh = program._to_device_table(ops if ops else [program.BlockOp()], dev)
    _lib.block_build(bt, nblocks, batch, ot, dev)
    _lib.block_unbuild(bt, nblocks, batch, ot, dev)
    torch.cuda.synchronize()
    for i in {0, nblocks // 2, nblocks - 1}:
        for b in range(batch):
            row = blocks[i % distinct][b]
            mats = [_matrix(op, k, engine) for op in row]
            w = np.eye(d, dtype=complex)
            for g in mats:
                w = g @ w
            assert np.abs(u_t[i, b].cpu().numpy() - w).max() <= 8e-15 * max(1, nops)
            x = gu[i, b]
            tol = (8 * nops + 16) * 2.0 ** -24 * np.linalg.norm(x) * np.linalg.norm(w)
            for j in range(nops - 1, -1, -1):
                w = mats[j].conj().T @ w
                got = keep[i * nops + j][1][b].cpu().numpy()
                want = _cotangent(row[j], x, w, k, engine) if ops[i * nops + j].grad else np.zeros_like(got)
                assert np.abs(got - want).max() <= tol
                x = mats[j].conj().T @ x


def _random_same(rng, kind, o, engine):
    if kind in (engine.KIND_PHASE, engine.KIND_DIAG):
        return np.exp(2j * np.pi * rng.random(len(o)))
    return _unitary(rng, int(round(len(o) ** 0.5))).reshape(-1)
