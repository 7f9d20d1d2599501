"""Gate programs: how a recorded sequence of gates becomes GPU work.

Gates are recorded cheaply by ``gate_wrapper`` and compiled into a ``Segment`` when
the state is read:

* every parameterised gate of a supported type (``NATIVE``) gets its operand built
  on the GPU by one ``tqk_gate_operands`` launch for the whole segment, reading its
  parameters in place through their strides (no per-gate torch ops);
* the plain method then applies the ops in tile passes that gates on any wires share
  (``tile_runs``), or each with its own kernel; the fused method plans
  blocks of up to 6 wires (``fusion.plan_blocks``; width, planner variant and kernel
  per block chosen by ``autotune.choose_fusion`` from measured pass costs when
  ``fuse_wires == "auto"``), builds every block unitary in float64 with one
  ``tqk_block_build`` launch, and applies each block with the tensor-core kernel or
  the CUDA-core dense kernel -- out of place, keeping the block's input state, when a
  backward can follow and memory allows (``QuantumDevice.checkpoint``);
* the backward walks the segment in reverse with the adjoint kernels (a tensor-core
  block with a stored input reads it instead of uncomputing the state; the images and
  cotangents of all tensor-core blocks take one launch each), turns block cotangents
  into gate-operand cotangents with ``tqk_block_unbuild``, and gate-operand cotangents
  into parameter gradients with ``tqk_param_grads`` (analytic derivatives), accumulated
  in float64 into one buffer per parameter base tensor.

Gates with no native type (qubitunitary, multirz, qft, user matrices, ...) keep the
torch-built operand and its autograd graph (``generic`` ops).
"""
from __future__ import annotations

import ctypes
import heapq
import math
import struct
import weakref
from typing import Dict, List, Optional

import numpy as np
import torch

from . import _lib
from . import engine

# canonical gate name -> (TQK_G_* type id, number of parameters)
NATIVE = {
    "u3": (0, 3), "rx": (1, 1), "ry": (2, 1), "rz": (3, 1), "phaseshift": (4, 1), "u1": (4, 1), "rot": (5, 3),
    "u2": (6, 2), "r": (7, 2), "crx": (8, 1), "cry": (9, 1), "crz": (10, 1), "cu3": (11, 3), "cu1": (12, 1),
    "crot": (13, 3), "cu": (14, 4), "rzz": (15, 1), "rxx": (16, 1), "ryy": (17, 1), "rzx": (18, 1),
    "singleexcitation": (19, 1),
}
_DIAG_TYPES = {3: 2, 4: 1, 12: 1, 10: 4, 15: 4}  # type -> operand size for diagonal / phase operands
_WIDE_TYPES = {16, 17, 18, 19}                    # 4x4 dense operands

KIND_ID = {engine.KIND_DENSE: 0, engine.KIND_CTRL: 1, engine.KIND_X: 2, engine.KIND_PHASE: 3,
           engine.KIND_DIAG: 4, engine.KIND_SWAP: 5}


_CONTROLLED = (engine.KIND_CTRL, engine.KIND_X, engine.KIND_SWAP)


def operand_size(type_id: int) -> int:
    if type_id in _DIAG_TYPES:
        return _DIAG_TYPES[type_id]
    return 16 if type_id in _WIDE_TYPES else 4


# ---------------------------------------------------------------- ctypes descriptor layouts
class GateDesc(ctypes.Structure):
    _fields_ = [("type", ctypes.c_int32), ("inverse", ctypes.c_int32), ("batch", ctypes.c_int32),
                ("nparam", ctypes.c_int32), ("p", ctypes.c_void_p), ("p_row_stride", ctypes.c_int64),
                ("p_col_stride", ctypes.c_int64), ("p_is_double", ctypes.c_int32), ("pad0", ctypes.c_int32),
                ("op128", ctypes.c_void_p), ("op64", ctypes.c_void_p), ("op_grad", ctypes.c_void_p),
                ("grad", ctypes.c_void_p)]


class BlockOp(ctypes.Structure):
    _fields_ = [("kind", ctypes.c_int32), ("nw", ctypes.c_int32), ("pos", ctypes.c_int32 * 6),
                ("nctrl", ctypes.c_int32), ("ctrl_val", ctypes.c_int32), ("batch", ctypes.c_int32),
                ("op_size", ctypes.c_int32), ("operand", ctypes.c_void_p), ("grad", ctypes.c_void_p)]


class BlockDesc(ctypes.Structure):
    _fields_ = [("first_op", ctypes.c_int32), ("num_ops", ctypes.c_int32), ("k", ctypes.c_int32),
                ("batch", ctypes.c_int32), ("u", ctypes.c_void_p), ("gu", ctypes.c_void_p)]


assert ctypes.sizeof(GateDesc) == 80 and ctypes.sizeof(BlockOp) == 64 and ctypes.sizeof(BlockDesc) == 32


# The same records packed by one call each (fields in order), for tables built every step:
# setting the fields of a ctypes record one by one took 4 to 8 us a gate.
_GATE = struct.Struct("=4iQ2q2i4Q")
_BLOCK_OP = struct.Struct("=12i2Q")
_BLOCK_DESC = struct.Struct("=4i2Q")
_GATE_T = np.dtype({"names": ["op128", "op64", "op_grad", "grad"], "formats": ["u8"] * 4,
                    "offsets": [48, 56, 64, 72], "itemsize": 80})
_BLOCK_OP_T = np.dtype({"names": ["grad"], "formats": ["u8"], "offsets": [56], "itemsize": 64})
_BLOCK_DESC_T = np.dtype({"names": ["gu"], "formats": ["u8"], "offsets": [24], "itemsize": 32})
assert (_GATE.size, _BLOCK_OP.size, _BLOCK_DESC.size) == tuple(map(ctypes.sizeof, (GateDesc, BlockOp, BlockDesc)))


def _upload(data, device):
    """Packed records (bytes-like) -> (device uint8 tensor, its pinned staging copy)."""
    src = np.frombuffer(data, dtype=np.uint8)
    host = torch.empty(max(src.size, 1), dtype=torch.uint8, pin_memory=True)
    host.numpy()[:src.size] = src
    return host.to(device, non_blocking=True), host


def _to_device_table(structs, device) -> torch.Tensor:
    """Array of ctypes structures -> device uint8 tensor (via a pinned staging copy)."""
    n = len(structs)
    size = ctypes.sizeof(structs[0]) * n if n else 0
    host = torch.empty(max(size, 1), dtype=torch.uint8, pin_memory=True)
    arr = (type(structs[0]) * n)(*structs)
    ctypes.memmove(host.data_ptr(), ctypes.addressof(arr), size)
    dev = host.to(device, non_blocking=True)
    return dev, host  # keep the staging buffer alive until the copy has run


# ---------------------------------------------------------------- recorded native gate
class NativeGate:
    """A parameterised gate whose operand the GPU builds from ``params`` in place."""

    __slots__ = ("name", "type_id", "nparam", "wires", "params", "inverse", "kind", "nctrl", "batch")

    def __init__(self, name, wires, params, inverse, kind, nctrl):
        self.name = name
        self.type_id, self.nparam = NATIVE[name]
        self.wires = list(wires)
        self.params = params          # [B, P] float32/float64 on the device (may require grad)
        self.inverse = bool(inverse)
        self.kind = kind              # engine.KIND_*
        self.nctrl = nctrl
        self.batch = int(params.shape[0])


def _param_base(p: torch.Tensor):
    """(base tensor to differentiate, element offset of p[0, 0] inside base's storage)."""
    base = p._base if p._base is not None else p
    if base.dtype not in (torch.float32, torch.float64) or not _dense(base):
        return p, 0
    return base, p.storage_offset() - base.storage_offset()


def _dense(t: torch.Tensor) -> bool:
    try:
        return t.is_contiguous() or t.is_non_overlapping_and_dense()
    except AttributeError:
        return t.is_contiguous()


# ---------------------------------------------------------------- segment
class Segment:
    """A compiled run of gates: forward applied at construction, ``backward`` on demand."""

    def __init__(self, qdev, records: List, method: str):
        from . import fusion

        self.n = qdev.n_wires
        self.bsz = qdev.bsz
        self.device = qdev.device
        dev = self.device
        n = self.n
        # ---- native gate operands (one launch)
        natives = [r for r in records if isinstance(r, NativeGate)]
        self.natives = natives
        # operands laid out by shape: the natives of one operand shape are consecutive, so
        # their views come from one view + unbind per shape instead of per-gate slicing
        by_shape: Dict[tuple, List[int]] = {}
        shape_of: Dict[tuple, tuple] = {}
        for i, g in enumerate(natives):
            shp = shape_of.get((g.type_id, g.batch))
            if shp is None:
                shp = shape_of[g.type_id, g.batch] = _operand_shape(g, operand_size(g.type_id))
            by_shape.setdefault(shp, []).append(i)
        offsets = [0] * len(natives)
        total = 0
        for shp, idx in by_shape.items():
            numel = math.prod(shp)
            for i in idx:
                offsets[i] = total
                total += numel
        self.op128 = torch.empty(max(total, 1), dtype=torch.complex128, device=dev)
        self.op64 = torch.empty(max(total, 1), dtype=torch.complex64, device=dev)
        views64, views128 = [None] * len(natives), [None] * len(natives)
        for shp, idx in by_shape.items():
            a, cnt = offsets[idx[0]], len(idx)
            size = cnt * math.prod(shp)
            for i, v64, v128 in zip(idx, self.op64[a:a + size].view(cnt, *shp).unbind(0),
                                    self.op128[a:a + size].view(cnt, *shp).unbind(0)):
                views64[i], views128[i] = v64, v128
        self.gate_offsets = offsets
        self._keep = []
        p64, p128 = self.op64.data_ptr(), self.op128.data_ptr()
        table = bytearray()
        pack = _GATE.pack
        for g, off in zip(natives, offsets):
            p = g.params
            table += pack(g.type_id, g.inverse, g.batch, g.nparam, p.data_ptr(), p.stride(0) if g.batch > 1 else 0,
                          p.stride(1), p.dtype == torch.float64, 0, p128 + 16 * off, p64 + 8 * off, 0, 0)
        self.gate_table = np.frombuffer(table, dtype=np.uint8).reshape(-1, _GATE.size)
        if natives:
            dev_table, host = _upload(table, dev)
            self._keep += [dev_table, host]
            _lib.gate_operands(dev_table, len(natives), dev)
        # ---- exec ops: one TapeOp per record (operands point into op64 / op128)
        ops = []
        gi = 0
        for r in records:
            if isinstance(r, NativeGate):
                op = engine.TapeOp(r.kind, r.wires, controls=r.wires[:r.nctrl], targets=r.wires[r.nctrl:],
                                   operand=views64[gi])
                op.native = r
                op.op128 = views128[gi]
                op.ptr128 = p128 + 16 * offsets[gi]
                gi += 1
            else:
                op = r
            ops.append(op)
        self.records = ops
        # ---- plan
        self.blocks = []
        if method == "fused":
            wl = planner_wires(ops, n)
            fw = qdev.fuse_wires
            backend = getattr(qdev, "fused_backend", "auto")
            tc_ok = backend != "cuda" and n >= fusion.TC_MIN_WIRES
            if fw == "auto" and self.device.type == "cuda":
                from . import autotune

                with_adj = any(isinstance(r, NativeGate) and r.params.requires_grad for r in records) or \
                    any(not isinstance(r, NativeGate) and r.needs_grad for r in records)
                stored = with_adj and getattr(qdev, "checkpoint", "auto") is not False
                # how a gate left alone by a plan runs: a dense or controlled gate may still
                # run as a tensor-core block (its own kernel is a dense pass with a
                # cotangent, and on large states a 6-wire block's forward + reverse step
                # costs less); structured gates keep their light kernels
                lone_kind = [autotune.LONE_OTHER if not fusable(op) else
                             autotune.LONE_DENSE if op.kind in (engine.KIND_DENSE, engine.KIND_CTRL) else
                             autotune.LONE_LIGHT for op in ops]
                plan, tc_flags, k, _ = autotune.choose_fusion(wl, n, self.bsz, dev, tc_ok, with_adj, stored=stored,
                                                              lone_kind=lone_kind)
                lone_tc = [len(idxs) == 1 and tc for (_, idxs), tc in zip(plan, tc_flags)]
                if backend == "tc":
                    tc_flags = [tc_ok for _ in plan]
            else:
                k = max(1, min(6 if fw == "auto" else int(fw), n, 6))
                plan = fusion.plan_cached(wl, k, 8, 4)
                tc_flags = [fusion.use_tensor_cores(qdev, len(bw)) for bw, _ in plan]
                lone_tc = [False] * len(plan)
            self.fuse_width = k
            exec_ops = []
            for (bwires, idxs), tc, lone in zip(plan, tc_flags, lone_tc):
                members = [ops[i] for i in idxs]
                if len(members) == 1 and not (lone and fusable(members[0])):  # a lone gate on its own kernel
                    exec_ops.append(members[0])
                    continue
                exec_ops.append(self._make_block(qdev, members, bwires, tc))
            self.exec_ops = exec_ops
            self._build_blocks()
        else:
            self.exec_ops = tile_runs(ops, n, self.bsz) if getattr(qdev, "stage_low", True) else ops
        # ---- differentiable inputs
        self.bases: Dict[int, tuple] = {}
        self.grad_gates = []  # (gate, its base's id, element offset of its parameters in the base)
        for i, g in enumerate(natives):
            if g.params.requires_grad:
                base, eoff = _param_base(g.params)
                self.bases.setdefault(id(base), (base, None))
                self.grad_gates.append((i, id(base), eoff))
        self.generic_sources = [op for op in ops if op.native is None and op.needs_grad]
        self.diff_inputs = [b for b, _ in self.bases.values()] + [op.source for op in self.generic_sources]

    # -------------------------------------------------------------- blocks
    def _make_block(self, qdev, members, bwires, tc):
        from . import fusion

        if len(bwires) > 6 or not all(fusable(m) for m in members):
            raise _lib.TQKError(1, f"a fused block holds at most 6 wires of fusable ops (got {len(bwires)} wires)")
        if tc:
            bwires = fusion._pad_wires(bwires, self.n)
        k = len(bwires)
        batch = max(m.batch if m.batch else 1 for m in members)
        blk = engine.TapeOp(engine.KIND_DENSE, bwires)
        blk.members = members
        blk.block_batch = batch
        blk.tc = tc
        blk.batch = batch
        blk.k = k
        self.blocks.append(blk)
        return blk

    def _build_blocks(self):
        if not self.blocks:
            return
        dev = self.device
        sizes = [b.block_batch * (1 << (2 * b.k)) for b in self.blocks]
        self.u128 = torch.empty(max(sum(sizes), 1), dtype=torch.complex128, device=dev)
        off = 0
        # one upload: the ops' records, then the blocks'
        table, descs = bytearray(), []
        nops, p_u = 0, self.u128.data_ptr()
        for blk, sz in zip(self.blocks, sizes):
            d = 1 << blk.k
            blk.u128 = self.u128[off:off + sz].view(blk.block_batch, d, d)
            blk.ptr_u = p_u + 16 * off
            off += sz
            where = {w: blk.k - 1 - i for i, w in enumerate(blk.wires)}
            descs.append((nops, len(blk.members), blk.k, blk.block_batch, blk.ptr_u, 0))
            nops += len(blk.members)
            for m in blk.members:
                table += self._block_op(m, where)
        self.num_block_ops = nops
        for d in descs:
            table += _BLOCK_DESC.pack(*d)
        self.block_table = table
        self.max_block_batch = max(b.block_batch for b in self.blocks)
        dev_table, host = _upload(table, dev)
        self._keep += [dev_table, host]
        _lib.block_build(dev_table[64 * nops:], len(descs), self.max_block_batch, dev_table, dev)
        for blk in self.blocks:
            if not blk.tc:
                blk.operand = blk.u128.to(torch.complex64)
        self._prepare_images(adjoint=False)
        # keep operands of non-native members alive in complex128
        self._member128 = [m._op128_keep for b in self.blocks for m in b.members]

    def _prepare_images(self, adjoint: bool) -> None:
        """Tensor-core operand images of every block of the segment (of U, or of U^H for
        the reverse sweep) in one buffer and one launch: ``blk.image`` / ``blk.image_h``."""
        tcb = [b for b in self.blocks if b.tc]
        if not tcb:
            return
        lib = _lib.load()
        sizes = [lib.tqk_fused_image_bytes(b.block_batch) for b in tcb]
        buf = torch.empty(sum(sizes), dtype=torch.uint8, device=self.device)
        jobs, off = [], 0
        for b, sz in zip(tcb, sizes):
            img = buf[off:off + sz]  # every image is a multiple of 64 KB: offsets stay aligned
            off += sz
            setattr(b, "image_h" if adjoint else "image", img)
            j = _lib.ImageJob()
            j.u, j.image, j.u_batch, j.adjoint = b.u128.data_ptr(), img.data_ptr(), b.block_batch, int(adjoint)
            for i, w in enumerate(b.wires):
                j.wires[i] = w
            jobs.append(j)
        table, host = _to_device_table(jobs, self.device)
        # the pinned staging copy must outlive its asynchronous upload (one slot per
        # direction, so repeated reverse sweeps do not accumulate them)
        setattr(self, "_keep_images_h" if adjoint else "_keep_images", (table, host))
        _lib.fused_prepare_many(table, len(jobs), max(b.block_batch for b in tcb))

    def _block_op(self, m, where) -> bytes:
        """The ``tqk_block_op`` record of a block's member (no cotangent slot)."""
        pos = [where[w] for w in m.wires]
        nw = len(pos)
        pos += [0] * (6 - nw)
        k = m.kind
        nctrl = len(m.controls) if k in _CONTROLLED else 0
        if k in (engine.KIND_X, engine.KIND_SWAP):
            return _BLOCK_OP.pack(KIND_ID[k], nw, *pos, nctrl, m.ctrl_val, 1, 1, self._dummy_ptr(), 0)
        if m.native is not None:
            return _BLOCK_OP.pack(KIND_ID[k], nw, *pos, nctrl, m.ctrl_val, m.native.batch,
                                  operand_size(m.native.type_id), m.ptr128, 0)
        o128 = _generic128(m)
        return _BLOCK_OP.pack(KIND_ID[k], nw, *pos, nctrl, m.ctrl_val, o128.shape[0], o128[0].numel(),
                              o128.data_ptr(), 0)

    def _dummy_ptr(self):
        if not hasattr(self, "_dummy"):
            self._dummy = torch.zeros(1, dtype=torch.complex128, device=self.device)
        return self._dummy.data_ptr()

    # -------------------------------------------------------------- forward
    def apply(self, buf: torch.Tensor, store_inputs: bool = False, zero_input: bool = False) -> torch.Tensor:
        """Run the segment on ``buf``; returns the buffer holding the result.  With
        ``store_inputs`` every tensor-core block writes its output to a new buffer and
        keeps its input for the backward (``buf`` itself may become one of those stored
        inputs, so the result is then a different tensor).  ``zero_input``: ``buf`` is
        |0...0> in every row and no initial state or earlier segment precedes it (the
        device's first segment from its default state)."""
        _lib.nvtx_push(f"tqk.segment.forward[{len(self.exec_ops)} passes]")
        try:
            return self._apply(buf, store_inputs, zero_input)
        finally:
            _lib.nvtx_pop()

    def _apply(self, buf: torch.Tensor, store_inputs: bool, zero_input: bool) -> torch.Tensor:
        recs, keep = [], []
        cur = buf
        for i, op in enumerate(self.exec_ops):
            if isinstance(op, StagedRun):
                recs.append(_staged_record(op, op.descs(), keep))
            elif getattr(op, "members", None) is not None:
                if not op.tc:
                    recs.append(_exec(_lib.X_BLOCK_DENSE, op.wires, batch=op.block_batch, operand=op.operand))
                    continue
                if zero_input and i == 0:
                    # a first block on |0...0>: its output is column 0 of U at the block's 64
                    # patterns (every other amplitude stays 0), written directly instead of a
                    # pass over the state; its reverse step needs neither its input nor the
                    # cotangent before it (nothing precedes it), so nothing is kept
                    op.zero_input = True
                    recs.append(_exec(_lib.X_BLOCK_ZERO, op.wires, batch=op.block_batch, u=op.u128))
                    continue
                r = _exec(_lib.X_BLOCK_TC, op.wires, batch=op.block_batch, image=op.image)
                out = None
                if store_inputs:
                    out = _new_state(cur)
                    if out is None:  # out of memory: the remaining blocks run in place
                        store_inputs = False
                if out is not None:
                    r.out = out.data_ptr()
                    op.stored_input = cur
                    op.kept_input = True
                    cur = out
                recs.append(r)
            else:
                recs.append(_plain_record(op))
        if recs:
            table = (_lib.ExecOp * len(recs))(*recs)
            final = _lib.segment_forward(buf, self.n, table, len(recs))
            assert final == cur.data_ptr(), "segment runner ended on an unexpected buffer"
        return cur

    def take_stored_inputs(self) -> list:
        """(block, stored input) pairs for an autograd node to save; the segment keeps weak
        references, so later nodes over the same segment still find the inputs while one
        node holds them, and the memory goes when the last node releases them."""
        out = []
        for op in self.blocks:
            t = getattr(op, "stored_input", None)
            if t is None and getattr(op, "stored_ref", None) is not None:
                t = op.stored_ref()
            if t is None:
                continue
            op.stored_ref = weakref.ref(t)
            op.stored_input = None
            out.append((op, t))
        return out

    def stored_bytes(self, state: torch.Tensor) -> int:
        """Device memory ``apply(..., store_inputs=True)`` keeps for the backward."""
        return sum(1 for b in self.blocks if b.tc) * state.numel() * state.element_size()

    # -------------------------------------------------------------- backward
    def backward(self, psi: "engine.StateCursor", lam: torch.Tensor, need_grads: bool,
                 inputs: Optional[dict] = None, lam_end: Optional[torch.Tensor] = None) -> List[Optional[torch.Tensor]]:
        """Reverse sweep over this segment (``psi`` at its end on entry, at its start on
        return; ``lam`` updated in place, or written from ``lam_end``, which is only read);
        ``inputs`` maps id(block) to the block's stored
        input state, where the forward kept one and it is still held.  Returns grads for
        ``self.diff_inputs``."""
        _lib.nvtx_push(f"tqk.segment.backward[{len(self.exec_ops)} passes]")
        try:
            return self._backward(psi, lam, need_grads, inputs or {}, lam_end)
        finally:
            _lib.nvtx_pop()

    def _backward(self, psi: "engine.StateCursor", lam: torch.Tensor, need_grads: bool,
                  inputs: dict, lam_end: Optional[torch.Tensor] = None) -> List[Optional[torch.Tensor]]:
        dev = self.device
        n = self.n
        opg = torch.zeros_like(self.op128) if (need_grads and self.natives) else None
        gslots = {}
        for op in self.generic_sources:
            gslots[id(op)] = torch.zeros(op.operand.shape, dtype=torch.complex128, device=dev)
        gu = torch.zeros_like(self.u128) if (need_grads and self.blocks) else None
        # tensor-core blocks: U^H images in one launch, one zeroed buffer for the cross
        # terms of the blocks that need a cotangent, stored-input cotangents added in one
        # launch after the sweep
        self._prepare_images(adjoint=True)
        mr_of = {}
        tc_grad = [b for b in self.blocks if b.tc and gu is not None and _block_needs_grad(b)]
        if tc_grad:
            mr_all = torch.zeros(sum(b.block_batch for b in tc_grad), 128, 128, dtype=torch.float64, device=dev)
            row = 0
            for b in tc_grad:
                mr_of[id(b)] = mr_all[row:row + b.block_batch]
                row += b.block_batch
        cross_jobs, recs, keep, stored_at = [], [], [], {}
        zero_block = None
        # a native gate's cotangent slot: the place of its operand in op128, inside opg
        dopg = opg.data_ptr() - self.op128.data_ptr() if opg is not None else 0
        for op in self.exec_ops:  # forward order; the runner walks it backwards
            if isinstance(op, StagedRun):
                slots = []
                for m in op.ops:
                    slot = None
                    if need_grads:
                        if m.native is not None and m.native.params.requires_grad:
                            slot = m.ptr128 + dopg
                        elif id(m) in gslots:
                            slot = torch.view_as_real(gslots[id(m)]).view(-1)
                    slots.append(slot)
                recs.append(_staged_record(op, op.descs(slots), keep))
                continue
            if getattr(op, "members", None) is not None:
                slot = None
                if gu is not None and _block_needs_grad(op):
                    slot = _as_real(gu, op.u128, self.u128)
                if not op.tc:
                    recs.append(_exec(_lib.X_BLOCK_DENSE, op.wires, batch=op.block_batch, operand=op.operand,
                                      grad=slot))
                    continue
                stored = inputs.get(id(op))
                mr = mr_of.get(id(op)) if slot is not None else None
                r = _exec(_lib.X_BLOCK_TC, op.wires, batch=op.block_batch, image_h=op.image_h, u=op.u128, grad=slot,
                          mr=mr)
                if getattr(op, "zero_input", False):
                    # the last reverse step of the circuit, from |0...0>: the runner stops
                    # before it; the cotangent of U is lam conj(e_0)^T (taken below)
                    r.skip_reverse = 1
                    zero_block = (op, slot)
                elif stored is not None:
                    r.stored = stored.data_ptr()
                    stored_at[stored.data_ptr()] = stored
                    if mr is not None:  # the cross term against the stored input is the cotangent
                        j = _lib.CrossJob()
                        j.mr, j.gu, j.batch = mr.data_ptr(), slot.data_ptr(), op.block_batch
                        cross_jobs.append(j)
                recs.append(r)
                continue
            slot = None
            if need_grads:
                if op.native is not None and op.native.params.requires_grad:
                    slot = op.ptr128 + dopg
                elif id(op) in gslots:
                    slot = torch.view_as_real(gslots[id(op)]).view(-1)
            recs.append(_plain_record(op, slot))
        if recs:
            # the sweep writes its state only on a work buffer: the cursor's own when it
            # already owns one, else one state more, when any reverse step uncomputes
            uncomputes = any(not (r.kind == _lib.X_BLOCK_TC and (r.stored or r.skip_reverse)) for r in recs)
            work = psi.state if psi.owned else (psi.work_buffer() if uncomputes else None)
            table = (_lib.ExecOp * len(recs))(*recs)
            start = _lib.segment_backward(psi.state, lam, work, n, table, len(recs), lam_end)
            if work is not None and start == work.data_ptr():
                psi.state, psi.owned = work, True
            elif start in stored_at:
                psi.state, psi.owned = stored_at[start], False
        elif lam_end is not None:
            lam.copy_(lam_end)
        if zero_block is not None and zero_block[1] is not None:
            _add_zero_input_cotangent(lam, zero_block[0], zero_block[1], n)
        if cross_jobs:
            table, host = _to_device_table(cross_jobs, dev)
            self._keep_cross = (table, host)  # the cross terms themselves are stream-ordered
            _lib.fused_cross_add_many(table, len(cross_jobs), max(j.batch for j in cross_jobs))
        if not need_grads:
            return [None] * len(self.diff_inputs)
        # block cotangents -> member operand cotangents
        if self.blocks and gu is not None:
            nops = self.num_block_ops
            table = bytearray(self.block_table)
            grad_col = np.frombuffer(table, dtype=_BLOCK_OP_T, count=nops)["grad"]
            gu_col = np.frombuffer(table, dtype=_BLOCK_DESC_T, offset=64 * nops)["gu"]
            dgu = gu.data_ptr() - self.u128.data_ptr()
            slots = []
            for m in (m for blk in self.blocks for m in blk.members):
                if m.native is not None and m.native.params.requires_grad:
                    slots.append(m.ptr128 + dopg)
                else:
                    g = gslots.get(id(m))
                    slots.append(0 if g is None else g.data_ptr())
            grad_col[:] = slots
            gu_col[:] = [blk.ptr_u + dgu if _block_needs_grad(blk) else 0 for blk in self.blocks]
            dev_table, host = _upload(table, dev)
            _lib.block_unbuild(dev_table[64 * nops:], len(self.blocks), self.max_block_batch, dev_table, dev)
            self._keep_bw = [dev_table, host]
        # operand cotangents -> parameter gradients
        grads = []
        if self.natives and self.bases:
            # one float64 buffer for every base tensor's gradient (each base's part laid out
            # like the base's own storage), one conversion back to the bases' dtype
            bases = [b for b, _ in self.bases.values()]
            spans = [max(0, sum((sz - 1) * st for sz, st in zip(b.shape, b.stride()))) + 1 for b in bases]
            starts = np.cumsum([0] + spans[:-1]).tolist()
            flat = torch.zeros(max(sum(spans), 1), dtype=torch.float64, device=dev)
            start_of = {k: st for k, st in zip(self.bases.keys(), starts)}
            if self.grad_gates:
                rows = [i for i, _, _ in self.grad_gates]
                table = self.gate_table[rows]  # a copy
                col = table.reshape(-1).view(_GATE_T)
                col["op128"] = 0
                col["op64"] = 0
                col["op_grad"] = [opg.data_ptr() + 16 * self.gate_offsets[i] for i in rows]
                col["grad"] = [flat.data_ptr() + 8 * (start_of[base] + eoff) for _, base, eoff in self.grad_gates]
                dev_table, host = _upload(table, dev)
                _lib.param_grads(dev_table, len(rows), dev)
                self._keep_pg = [dev_table, host]
            dtypes = {b.dtype for b in bases}
            conv = flat.to(bases[0].dtype) if len(dtypes) == 1 else None
            for b, st in zip(bases, starts):
                src = conv if conv is not None else flat
                gb = src.as_strided(b.shape, b.stride(), st)
                grads.append(gb if conv is not None else gb.to(b.dtype))
        else:
            grads += [None] * len(self.bases)
        for op in self.generic_sources:
            grads.append(gslots[id(op)].to(op.source.dtype).view(op.source.shape))
        return grads


_PLAIN_KIND = {engine.KIND_DENSE: _lib.X_DENSE, engine.KIND_CTRL: _lib.X_CTRL, engine.KIND_X: _lib.X_MCX,
               engine.KIND_PHASE: _lib.X_PHASE, engine.KIND_DIAG: _lib.X_DIAG, engine.KIND_SWAP: _lib.X_SWAP}


EXEC_MAX_WIRES = len(_lib.ExecOp().wires)


def _address(t):
    return t if t is None or isinstance(t, int) else t.data_ptr()


def _exec(kind: int, wires, nctrl: int = 0, ctrl_val: int = 1, batch: int = 1, operand=None, uncompute=None,
          image=None, image_h=None, u=None, grad=None, mr=None) -> "_lib.ExecOp":
    """One ``tqk_exec_op`` record (tensors, or device addresses as ints)."""
    if len(wires) > EXEC_MAX_WIRES:
        raise _lib.TQKError(1, f"an op on {len(wires)} wires exceeds the {EXEC_MAX_WIRES} one op may touch")
    return _lib.ExecOp(kind, len(wires), nctrl, ctrl_val, tuple(wires), batch, _address(operand), _address(uncompute),
                       _address(image), _address(image_h), _address(u), None, None, _address(grad), _address(mr))


def _plain_record(op, grad=None) -> "_lib.ExecOp":
    """A plain tape op (engine.TapeOp) as a ``tqk_exec_op``: wires are controls first,
    then targets, for the controlled kinds."""
    k = op.kind
    if k in (engine.KIND_CTRL, engine.KIND_X, engine.KIND_SWAP):
        wires, nctrl = op.controls + op.targets, len(op.controls)
    else:
        wires, nctrl = op.wires, 0
    return _exec(_PLAIN_KIND[k], wires, nctrl=nctrl, ctrl_val=op.ctrl_val, batch=op.batch, operand=op.operand,
                 uncompute=op.uncompute, grad=grad)


def _staged_record(run, descs, keep: list) -> "_lib.ExecOp":
    arr = (_lib.StagedOp * len(descs))(*descs)
    keep.append(arr)  # alive until the runner returns (it reads the table on the host)
    r = _lib.ExecOp()
    r.staged, r.nstaged = ctypes.addressof(arr), len(descs)
    if run.tile_bits > 64:
        r.kind, r.batch = _lib.X_TILED, run.tile_bits
    else:
        r.kind, r.tile_bits = _lib.X_STAGED, run.tile_bits
    return r


def _zero_input_index(blk, n: int, device) -> torch.Tensor:
    """Amplitude offsets of a 6-wire block's 64 patterns with every other bit clear
    (wires[0] is the pattern's most significant bit), on the device; built once per block."""
    idx = getattr(blk, "_zero_idx", None)
    if idx is None:
        offs = [sum(1 << (n - 1 - w) for i, w in enumerate(blk.wires) if (j >> (5 - i)) & 1) for j in range(64)]
        # a pinned staging copy: a copy from pageable memory would block the stream (and
        # with it the host's run-ahead into the next step)
        host = torch.tensor(offs, dtype=torch.long).pin_memory()
        idx = host.to(device, non_blocking=True)
        blk._zero_idx_host = host  # alive until the copy has run
        blk._zero_idx = idx
    return idx


def _add_zero_input_cotangent(lam: torch.Tensor, blk, slot: torch.Tensor, n: int) -> None:
    """gu[b][j][0] += lam[b, offset of pattern j] for a block applied to |0...0> (wires[0] is
    the pattern's most significant bit; the sum over rows when one U serves every row)."""
    vals = lam.index_select(1, _zero_input_index(blk, n, lam.device)).to(torch.complex128)  # [bsz, 64]
    g = torch.view_as_complex(slot.view(-1, 2)).view(blk.block_batch, 64, 64)
    if blk.block_batch == 1:
        g[0, :, 0] += vals.sum(0)
    else:
        g[:, :, 0] += vals


def _new_state(like: torch.Tensor) -> Optional[torch.Tensor]:
    """A buffer for a block's output when its input is kept, or None when the device is out
    of memory (the caller then continues in place; the reverse sweep uncomputes through
    the blocks without a stored input)."""
    try:
        return torch.empty_like(like)
    except torch.cuda.OutOfMemoryError:
        return None


# ---------------------------------------------------------------- staged runs
class StagedRun:
    """Ops applied in one pass through tiles held on chip and reversed in one adjoint pass.
    ``tile_bits``: the number of lowest index bits a tile spans (``tqk_staged_apply``), or,
    above 64, the mask of its index bits (``tqk_tiled_apply``)."""

    def __init__(self, ops, tile_bits):
        self.ops = ops
        self.tile_bits = tile_bits
        self.wires = sorted({w for o in ops for w in o.wires})

    def descs(self, grads=None):
        """The run's ``tqk_staged_op`` records; ``grads``: per-op cotangent slots (tensor,
        device address or None) for the reverse pass.  The records without slots are built
        once per run (operands do not move) and copied when slots are set."""
        base = getattr(self, "_descs", None)
        if base is None:
            base = self._build_descs()
            self._descs = base
        if grads is None:
            return base
        out = []
        for d, g in zip(base, grads):
            if g is None:
                out.append(d)
                continue
            e = _lib.StagedOp.from_buffer_copy(d)
            e.grad = g if isinstance(g, int) else g.data_ptr()
            out.append(e)
        return out

    def _build_descs(self):
        out = []
        for o in self.ops:
            kind, ctrl_val = _lib.S_DIAG, 0
            ws = o.wires
            if o.kind == engine.KIND_X:
                ws, kind, ctrl_val = o.controls + o.targets, _lib.S_X, o.ctrl_val
            elif o.kind == engine.KIND_CTRL:
                ws, kind = o.controls + o.targets, _lib.S_DENSE1
            elif o.kind == engine.KIND_DENSE:
                kind = _lib.S_DENSE1
            elif o.kind == engine.KIND_PHASE:
                kind = _lib.S_PHASE
            flip = o.kind == engine.KIND_X
            out.append(_lib.StagedOp(kind, len(ws), tuple(ws), ctrl_val, 0, None if flip else o.operand.data_ptr(),
                                     1 if flip else o.operand.shape[0], None))
        return out


def stageable(op, n: int, tile_bits: int) -> bool:
    """Ops ``tqk_staged_apply`` can run: one target inside the low tile (dense, controlled,
    controlled-X), or diagonal ops anywhere (phase on any wires, diagonal on <= 2)."""
    if getattr(op, "uncompute", None) is not None or getattr(op, "image", None) is not None:
        return False
    if not op.wires or len(op.wires) > _lib.STAGED_MAX_WIRES:
        return False
    low = n - tile_bits  # wires >= low have their bit inside the tile
    k = op.kind
    if k == engine.KIND_DENSE:
        return len(op.wires) == 1 and op.wires[0] >= low and _mat2(op)
    if k == engine.KIND_CTRL:
        return len(op.targets) == 1 and op.targets[0] >= low and _mat2(op)
    if k == engine.KIND_X:
        return len(op.targets) == 1 and op.targets[0] >= low
    if k == engine.KIND_PHASE:
        return op.operand is not None and op.operand.numel() == int(op.operand.shape[0])
    if k == engine.KIND_DIAG:
        return len(op.wires) <= 2 and op.operand is not None and op.operand.shape[-1] == (1 << len(op.wires))
    return False


def _mat2(op) -> bool:
    t = op.operand
    return t is not None and t.dtype == torch.complex64 and tuple(t.shape[1:]) == (2, 2) and t.is_contiguous()


def stage_runs(ops, n: int, min_run: int = 2):
    """Group maximal runs of consecutive stageable ops into ``StagedRun`` passes (tile of
    2^min(n, 12) amplitudes; at most ``STAGED_MAX_OPS`` ops per pass)."""
    tb = min(n, _lib.STAGED_MAX_TILE_BITS)
    out, run = [], []

    def close():
        if len(run) >= min_run:
            out.append(StagedRun(list(run), tb))
        else:
            out.extend(run)
        run.clear()

    for op in ops:
        if stageable(op, n, tb):
            run.append(op)
            if len(run) == _lib.STAGED_MAX_OPS:
                close()
        else:
            close()
            out.append(op)
    close()
    return out


# A tile pass moves the state once (2 S bytes forward, 4 S in reverse) whatever its ops are; an op on its
# own kernel moves its share of that.  Ops share a pass when their shares add up to more than the pass
# costs: TILE_MIN_SHARE, or TILE_L2_SHARE on states that stay in L2, where a pass is bound by its
# instructions (us forward + reverse, tile pass / own kernels: 268 MB two CRX 377 / 314, three 416 / 440, U3
# and CNOT 350 / 365; 32 MB three CRX 66 / 58, four 73 / 85, U3 and CNOT 53 / 49).  States up to
# TILE_SMALL_BYTES always share: launches cost more than bytes there (8 MB: two CRX 18 / 26; 16 MB: two
# gates with the rest of a step 86 / 106).
TILE_MIN_SHARE = 1.2
TILE_L2_SHARE = 1.75
TILE_L2_BYTES = 64 << 20
TILE_SMALL_BYTES = 16 << 20
# Where a step is bound by the host (35 us a gate, forward and backward), the kernels of one gate
# and the staged runs stay, whose order of operations results are known by.  Rows of at most 2^12
# amplitudes are one tile either way: up to 2^21 amplitudes in all (n = 10, bsz = 256, 100 gates:
# 162 us of 3.3 ms in the staged kernels, 128 us in the tiled ones).  Longer rows: below 2^20 in all
# (60 gates with backward, ms: n = 13, bsz = 64 2.20 so and 2.11 in tile passes; n = 16, bsz = 16,
# 2^20 amplitudes, 2.21 and 2.00; n = 18, bsz = 8, 2^21, 2.42 and 2.02).
TILE_SHORT_ROW_AMPS = 1 << 22
TILE_MIN_AMPS = 1 << 20
_TILE_PLANS: dict = {}


def _pass_share(op) -> float:
    """Share of a pass over the state (2 S forward, 4 S reverse) of an op's own kernel."""
    if op.kind in (engine.KIND_CTRL, engine.KIND_X):
        return 0.5 ** len(op.controls)
    if op.kind == engine.KIND_PHASE:
        return 0.5 ** len(op.wires)
    return 1.0


def plan_tiles(ops, n: int, small: bool, share: float = TILE_MIN_SHARE) -> List[tuple]:
    """Cut the ops into passes: (op indices, tile mask), mask 0 for an op on its own kernel.

    A pass starts from the lowest four index bits (whole 128-byte lines) and walks the
    pending ops in order: an op joins when no wire of it was touched by an op left out and
    its target (if any) is or fits among the tile's bits; ops on disjoint wires commute, so
    the passes apply an equivalent order.  Free bits are filled from the lowest.  Unless
    ``small``, the ops of a pass move the state ``share`` times at least on their own kernels; where
    they would not, the first pending op runs on its own and the others wait.

    The ops of a wire leave in order, so each wire has a queue, and a pass looks at the queues'
    fronts only: every op left out closes a wire for the pass, which takes at most
    ``STAGED_MAX_OPS`` and leaves out at most n (a walk over all pending ops a pass took 1.9 s
    for 4000 gates that no pass can hold)."""
    tb = min(n, _lib.STAGED_MAX_TILE_BITS)
    queues, places = [[] for _ in range(n)], []
    for i, op in enumerate(ops):
        bits = [n - 1 - w for w in op.wires] or range(n)  # an op without wires: after and before all others
        places.append(bits)
        for b in bits:
            queues[b].append(i)
    front, out, left = [0] * n, [], len(ops)

    def leave(i):  # -> the ops that come to the front of a queue
        fresh = []
        for b in places[i]:
            front[b] += 1
            if front[b] < len(queues[b]):
                fresh.append(queues[b][front[b]])
        return fresh

    while left:
        mask, free, blocked, take = 15, tb - 4, 0, []
        heap = [q[f] for q, f in zip(queues, front) if f < len(q)]
        heapq.heapify(heap)
        first, last, fronts = heap[0], -1, list(front)
        while heap and len(take) < _lib.STAGED_MAX_OPS:
            i = heapq.heappop(heap)
            if i == last:  # at the front of another wire's queue too
                continue
            last, op = i, ops[i]
            wires = 0
            for b in places[i]:
                wires |= 1 << b
            if not (wires & blocked) and stageable(op, n, n):
                tgt = 0
                if op.kind not in (engine.KIND_PHASE, engine.KIND_DIAG):
                    tgt = 1 << (n - 1 - (op.targets[0] if op.kind != engine.KIND_DENSE else op.wires[0]))
                if not tgt & ~mask or free:
                    free -= bool(tgt & ~mask)
                    mask |= tgt
                    take.append(i)
                    for j in leave(i):
                        heapq.heappush(heap, j)
                    continue
            blocked |= wires
        if len(take) < 2 or not (small or sum(_pass_share(ops[i]) for i in take) >= share):
            front = fronts  # the others may join ops that are not free yet
            leave(first)
            out.append(([first], 0))
            left -= 1
            continue
        left -= len(take)
        for b in range(n):
            if free and not (mask >> b) & 1:
                mask |= 1 << b
                free -= 1
        out.append((take, mask))
    return out


def tile_runs(ops, n: int, bsz: int):
    """The plain method's execution list: ``StagedRun`` passes and ops on their own kernels.
    Small states take ``stage_runs``; the others are cut by ``plan_tiles``, memoised on the
    circuit's structure."""
    if n < _lib.TILED_MIN_WIRES or \
            (bsz << n) < (TILE_SHORT_ROW_AMPS if n <= _lib.STAGED_MAX_TILE_BITS else TILE_MIN_AMPS):
        return stage_runs(ops, n)
    small = (bsz << (n + 3)) <= TILE_SMALL_BYTES
    share = TILE_L2_SHARE if (bsz << (n + 3)) <= TILE_L2_BYTES else TILE_MIN_SHARE
    key = (n, small, share, tuple((op.kind, tuple(op.wires), len(op.controls), stageable(op, n, n)) for op in ops))
    plan = _TILE_PLANS.get(key)
    if plan is None:
        if len(_TILE_PLANS) > 256:
            _TILE_PLANS.clear()
        plan = plan_tiles(ops, n, small, share)
        _TILE_PLANS[key] = plan
    return [StagedRun([ops[i] for i in idx], mask) if mask else ops[idx[0]] for idx, mask in plan]


def _operand_shape(r: NativeGate, sz: int):
    if r.type_id in _DIAG_TYPES:
        return (r.batch,) if sz == 1 else (r.batch, sz)
    d = 4 if r.type_id in _WIDE_TYPES else 2
    return (r.batch, d, d)


def _as_real(buf: torch.Tensor, view: torch.Tensor, base: torch.Tensor) -> torch.Tensor:
    """float64 interleaved view of ``buf`` at the position ``view`` occupies inside ``base``."""
    off = (view.data_ptr() - base.data_ptr()) // 16
    return torch.view_as_real(buf[off:off + view.numel()]).view(-1)


def _block_needs_grad(blk) -> bool:
    return any((m.native is not None and m.native.params.requires_grad) or m.needs_grad for m in blk.members)


def _generic128(m) -> torch.Tensor:
    const = m.const
    if const is not None and const._op128_keep is not None:
        m._op128_keep = const._op128_keep
        return m._op128_keep
    src = m.source if m.source is not None else m.operand
    t = engine.kernel_operand(src.to(torch.complex128))
    m._op128_keep = t
    if const is not None and t.data_ptr() == src.data_ptr():  # a view of the constant: no work was queued for it
        const._op128_keep = t
    return t


def planner_wires(ops, n: int) -> List[List[int]]:
    """Wire lists the fusion planners see: an op's wires, or for an op the block kernels
    cannot hold (``fusable`` false) a barrier -- every wire (nothing moves across it) plus
    7 placeholder wires, wider than any block, so every planner leaves it alone (also when
    n <= 6, where all n wires would fit in one block)."""
    barrier = list(range(n)) + [-1 - i for i in range(7)]
    return [op.wires if fusable(op) else barrier for op in ops]


def fusable(op) -> bool:
    """Ops the block kernels can fold into a fused block."""
    if not op.wires or getattr(op, "uncompute", None) is not None:
        return False
    nw = len(op.wires)
    if op.kind in (engine.KIND_X, engine.KIND_SWAP, engine.KIND_PHASE):
        return nw <= 6
    if op.kind == engine.KIND_DIAG:
        return nw <= 4
    if op.kind == engine.KIND_CTRL:
        return len(op.targets) <= 2 and nw <= 6
    return nw <= 2
