"""The tile planner: the same passes as a walk over all pending ops, on circuits of every kind of op, and
a time that grows with the number of ops, not with its square, on circuits that no pass can hold."""
import time

import numpy as np
import pytest
import torch

from torchquantum_gb300 import _lib, engine
from torchquantum_gb300 import program as P


def _walk(ops, n, small):
    """Passes by the planner's definition: each walks all pending ops in order."""
    tb = min(n, _lib.STAGED_MAX_TILE_BITS)
    pending, out = list(range(len(ops))), []
    while pending:
        mask, free, blocked, take, rest = 15, tb - 4, 0, [], []
        for i in pending:
            op = ops[i]
            wires = sum(1 << (n - 1 - w) for w in op.wires)
            if not (wires & blocked) and len(take) < _lib.STAGED_MAX_OPS and P.stageable(op, n, n):
                tgt = 0
                if op.kind not in (engine.KIND_PHASE, engine.KIND_DIAG):
                    tgt = 1 << (n - 1 - (op.targets[0] if op.kind != engine.KIND_DENSE else op.wires[0]))
                if not tgt & ~mask or free:
                    free -= bool(tgt & ~mask)
                    mask |= tgt
                    take.append(i)
                    continue
            blocked |= wires or (1 << n) - 1
            rest.append(i)
        if len(take) < 2 or not (small or sum(P._pass_share(ops[i]) for i in take) >= P.TILE_MIN_SHARE):
            out.append(([pending[0]], 0))
            pending = pending[1:]
            continue
        for b in range(n):
            if free and not (mask >> b) & 1:
                mask |= 1 << b
                free -= 1
        out.append((take, mask))
        pending = rest
    return out


def _ops(rng, n, count, kinds, wires=None):
    one, two = torch.eye(2, dtype=torch.complex64)[None], torch.eye(4, dtype=torch.complex64)[None]
    out = []
    for _ in range(count):
        k = kinds[int(rng.integers(len(kinds)))]
        w = [int(v) for v in rng.choice(n if wires is None else wires, 3, replace=False)]
        out.append({"dense": lambda: engine.TapeOp("dense", w[:1], operand=one),
                    "dense2": lambda: engine.TapeOp("dense", w[:2], operand=two),
                    "inverse": lambda: engine.TapeOp("dense", w[:1], operand=one, uncompute=one),
                    "ctrl": lambda: engine.TapeOp("ctrl", w[:2], controls=w[:1], targets=w[1:2], operand=one),
                    "ctrl2": lambda: engine.TapeOp("ctrl", w, controls=w[:2], targets=w[2:], operand=one),
                    "x": lambda: engine.TapeOp("x", w[:2], controls=w[:1], targets=w[1:2]),
                    "xfirst": lambda: engine.TapeOp("x", w[:2], controls=w[1:2], targets=w[:1]),
                    "phase": lambda: engine.TapeOp("phase", w, operand=one[:, 0, 0]),
                    "all": lambda: engine.TapeOp("phase", [], operand=one[:, 0, 0]),
                    "diag": lambda: engine.TapeOp("diag", w[:2], operand=two[:, 0]),
                    "diag3": lambda: engine.TapeOp("diag", w, operand=torch.ones(1, 8, dtype=torch.complex64)),
                    "swap": lambda: engine.TapeOp("swap", w[:2], targets=w[:2])}[k]())
    return out


KINDS = [["dense"], ["dense2", "swap"], ["dense", "x", "ctrl"], ["dense", "dense2", "phase", "diag"], ["all", "dense", "x"],
         ["dense", "inverse", "ctrl2", "xfirst", "diag3", "swap", "phase"], ["diag", "phase", "x", "diag3"]]


@pytest.mark.parametrize("small", [False, True])
@pytest.mark.parametrize("kinds", KINDS)
def test_same_passes_as_a_walk_over_all_ops(kinds, small):
    for n, count, wires in ((9, 0, None), (9, 1, None), (9, 80, None), (13, 300, None), (20, 500, None), (34, 260, None),
                            (24, 120, [0, 1, 2]), (24, 200, [23, 5, 11, 12])):
        ops = _ops(np.random.default_rng(n + count), n, count, kinds, wires)
        assert P.plan_tiles(ops, n, small) == _walk(ops, n, small)


@pytest.mark.parametrize("kinds,tail", [(["dense2"], []), (["swap", "dense", "x"], []), (["dense2"], ["dense"])])
def test_time_grows_with_the_ops(kinds, tail):
    def best(count):
        rng = np.random.default_rng(count)
        # (with a tail on wires of its own, which stays pending until the end or leaves in the first pass)
        ops = _ops(rng, 20, count, kinds, list(range(12))) + _ops(rng, 20, 3, tail or kinds, [17, 18, 19])
        runs = []
        for _ in range(3):
            t = time.perf_counter()
            P.plan_tiles(ops, 20, False)
            runs.append(time.perf_counter() - t)
        return min(runs)

    assert best(8000) <= 8 * best(2000)  # four times the ops; the walk takes sixteen times as long


def test_light_ops_wait_for_company():
    one = torch.eye(2, dtype=torch.complex64)[None]
    u3 = lambda w: engine.TapeOp("dense", [w], operand=one)  # noqa: E731
    swap = lambda a, b: engine.TapeOp("swap", [a, b], targets=[a, b])  # noqa: E731
    crx = lambda c, t: engine.TapeOp("ctrl", [c, t], controls=[c], targets=[t], operand=one)  # noqa: E731
    # two half passes gain nothing ..
    assert [m for _, m in P.plan_tiles([crx(0, 1), crx(2, 3)], 20, False)] == [0, 0]
    assert [len(i) for i, _ in P.plan_tiles([crx(0, 1), crx(2, 3), crx(4, 5)], 20, False)] == [3]
    # .. and an op that comes free alone waits for the next
    plan = P.plan_tiles([swap(0, 1), swap(2, 3), u3(0), u3(2)], 20, False)
    assert [i for i, _ in plan] == [[0], [1], [2, 3]] and [bool(m) for _, m in plan] == [False, False, True]
