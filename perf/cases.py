"""The work a user of this package gives it, as cases that can be timed and checked.

A case is a dict of plain values; ``kind`` says which part of the public API it runs:

* ``model``       a trainable circuit model built from modules (encoder, U3 layers, CNOT
                  rings, ``MeasureAll``), forward and backward;
* ``train``       a circuit recorded through the functional API with the plain (default) or
                  the fused method, Pauli-string expectation values, backward to the angles;
* ``forward``     the same without gradients, returning the final states;
* ``observables`` many Pauli strings on a state in hand, and the gradient to that state;
* ``sampling``    expectation values estimated from shots;
* ``apply``       the drop-in ``apply_unitary_bmm``, forward and backward;
* ``unitary``     wide unitary gates given as matrices, forward and backward to them;
* ``batch``       many uneven circuits in one prepared batch, new angles on every pass.

Angles are drawn near zero, as variational circuits are initialised, and the strings are
those of spin and molecular Hamiltonians, so expectation values and gradients are of
order one.
"""
import math
import random

import numpy as np
import torch

import torchquantum_gb300 as tq
import torchquantum_gb300.functional as tqf
from torchquantum_gb300 import batch as tqb
from torchquantum_gb300 import binding

DEV = "cuda"


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the four-qubit classifier of the package's small configuration: latency and launches
        dict(name="model-4", kind="model", n=4, bsz=32, layers=2),
        # the same architecture on ten qubits with an image-sized batch of samples
        dict(name="model-10", kind="model", n=10, bsz=256, layers=3),
        # gate-by-gate training at an odd size: the default method just above the size that
        # one shared-memory tile holds
        dict(name="plain-13", kind="train", circuit="random", method="plain", n=13, bsz=7, depth=60, strings=5, seed=1),
        # gate-by-gate training on a state larger than L2, the default method at scale
        dict(name="plain-22", kind="train", circuit="random", method="plain", n=22, bsz=8, depth=40, strings=4, seed=2),
        # a hardware-efficient ansatz with shared angles and per-sample inputs, many strings
        dict(name="ansatz-20", kind="train", circuit="ansatz", method="fused", n=20, bsz=16, depth=5, strings=20,
             seed=3),
        # the headline: depth-400 random circuit on 24 qubits, 16 samples, 8 strings
        dict(name="headline-24", kind="train", circuit="random", method="fused", n=24, bsz=16, depth=400, strings=8,
             seed=0),
        # inference: a fused forward pass at an odd width and an odd batch, states returned
        dict(name="forward-25", kind="forward", circuit="random", method="fused", n=25, bsz=3, depth=150, strings=8,
             seed=4),
        # a Hamiltonian of many terms on a given state, value and gradient
        dict(name="observables-22", kind="observables", n=22, bsz=4, strings=24, seed=5),
        # expectation values from shots, as on hardware
        dict(name="sampling-20", kind="sampling", n=20, bsz=4, strings=3, shots=8192, seed=6),
        # upstream code routed through the drop-in gate application: one per-sample gate and
        # one shared two-qubit gate
        dict(name="apply-21", kind="apply", n=21, bsz=8, seed=7),
        # Trotter blocks given as five-qubit unitaries, trained through
        dict(name="unitary-18", kind="unitary", n=18, bsz=8, k=5, gates=4, strings=3, seed=8),
        # 256 uneven circuits per step with new angles every step
        dict(name="batch-256", kind="batch", circuits=256, low=8, high=20, layers=40, seed=9),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["model", "train", "train", "train", "forward", "observables", "sampling", "apply", "unitary",
                       "batch"])
    seed = rng.randrange(1 << 20)
    if kind == "model":
        n = rng.randint(2, 12)
        return dict(kind=kind, n=n, bsz=_log_int(rng, 1, 512), layers=rng.randint(1, max(1, min(4, 48 // n))))
    if kind == "train":
        method = rng.choice(["plain", "fused"])
        n = rng.randint(8, 23)
        bsz = _log_int(rng, 1, min(64, 1 << (26 - n if n > 20 else 6)))
        if rng.random() < 0.4:
            return dict(kind=kind, circuit="ansatz", method=method, n=n, bsz=bsz, depth=rng.randint(1, 4),
                        strings=rng.randint(1, 24), seed=seed)
        return dict(kind=kind, circuit="random", method=method, n=n, bsz=bsz, depth=_log_int(rng, 10, 120),
                    strings=rng.randint(1, 12), seed=seed)
    if kind == "forward":
        n = rng.randint(14, 25)
        return dict(kind=kind, circuit="random", method=rng.choice(["plain", "fused"]), n=n,
                    bsz=_log_int(rng, 1, 1 << min(4, 26 - n)), depth=_log_int(rng, 10, 120),
                    strings=rng.randint(1, 8), seed=seed)
    if kind == "observables":
        n = rng.randint(9, 23)
        return dict(kind=kind, n=n, bsz=_log_int(rng, 1, 1 << min(6, 25 - n)), strings=_log_int(rng, 1, 50), seed=seed)
    if kind == "sampling":
        n = rng.randint(6, 22)
        return dict(kind=kind, n=n, bsz=_log_int(rng, 1, 1 << min(5, 24 - n)), strings=rng.randint(1, 5),
                    shots=_log_int(rng, 256, 65536), seed=seed)
    if kind == "apply":
        n = rng.randint(6, 23)
        return dict(kind=kind, n=n, bsz=_log_int(rng, 1, 1 << min(6, 25 - n)), seed=seed)
    if kind == "unitary":
        n = rng.randint(8, 19)
        return dict(kind=kind, n=n, bsz=_log_int(rng, 1, 16), k=rng.randint(3, 6), gates=rng.randint(1, 5),
                    strings=rng.randint(1, 4), seed=seed)
    low = rng.randint(4, 12)
    return dict(kind=kind, circuits=_log_int(rng, 16, 256), low=low, high=rng.randint(low, 19),
                layers=rng.randint(2, 30), seed=seed)


# ------------------------------------------------------------------ circuits and strings
def _gates(case):
    """The circuit as (name, wires, first angle column, number of angles), and the columns."""
    n, out, col = case["n"], [], 0
    if case["kind"] == "model":
        for g in range(4):
            for w in range(n):
                out.append((("rx", "ry", "rz", "rx")[g], [w], col, 1))
                col += 1
        for _ in range(case["layers"]):
            for w in range(n):
                out.append(("u3", [w], col, 3))
                col += 3
            for w in range(n):
                out.append(("cnot", [w, (w + 1) % n], 0, 0))
        return out, col
    if case["circuit"] == "ansatz":  # column block 0 is the per-sample input layer
        for w in range(n):
            out.append(("ry", [w], col, 1))
            col += 1
        for _ in range(case["depth"]):
            for name in ("ry", "rz"):
                for w in range(n):
                    out.append((name, [w], col, 1))
                    col += 1
            for w in range(n - 1):
                out.append(("cz", [w, w + 1], 0, 0))
        return out, col
    r = random.Random("circuit %d %d %d" % (case["seed"], n, case["depth"]))
    for _ in range(case["depth"]):
        if r.random() < 0.6:
            name, wires, k = "u3", [r.randrange(n)], 3
        else:
            name = r.choice(["cnot", "cz", "crx"])
            wires, k = r.sample(range(n), 2), 1 if name == "crx" else 0
        out.append((name, wires, col if k else 0, k))
        col += k
    return out, max(col, 1)


def _strings(case):
    """Terms of a Hamiltonian: Z, X, ZZ, and hopping terms (X or Y at both ends, Z between)."""
    n, r, out = case["n"], random.Random("strings %d %d" % (case["seed"], case["n"])), []
    for _ in range(case["strings"]):
        s, t = ["I"] * n, r.randrange(4)
        i, j = sorted(r.sample(range(n), 2))
        if t == 0:
            s[i] = "Z"
        elif t == 1:
            s[i] = "X"
        elif t == 2:
            s[i] = s[j] = "Z"
        else:
            s[i:j + 1] = ["Z"] * (j + 1 - i)
            s[i] = s[j] = r.choice("XY")
        out.append("".join(s))
    return out


def _normal(shape, g, scale=1.0, dtype=torch.float32):
    return torch.randn(shape, generator=g, device=DEV, dtype=torch.float64).mul_(scale).to(dtype)


def _product_state(n, bsz, g):
    """[bsz, 2^n] states of independent qubits, each rotated a little away from |0>."""
    s = torch.ones(bsz, 1, dtype=torch.complex128, device=DEV)
    th, ph = _normal((n, bsz), g, 0.5, torch.float64), _normal((n, bsz), g, 0.5, torch.float64)
    for w in range(n):
        q = torch.stack([torch.cos(th[w]).to(torch.complex128), torch.polar(torch.sin(th[w]), ph[w])], dim=1)
        s = (s[:, :, None] * q[:, None, :]).reshape(bsz, -1)
    return s.to(torch.complex64)


def _unitaries(count, k, g):
    z = torch.randn(count, 1 << k, 1 << k, generator=g, device=DEV, dtype=torch.complex128)
    h = (z + z.conj().transpose(1, 2)) * (0.3 / math.sqrt(1 << k))  # exp(-i h) of a small Hermitian h
    return torch.matrix_exp(-1j * h).to(torch.complex64)


def _model(n, layers):
    class Model(tq.QuantumModule):
        def __init__(self):
            super().__init__()
            self.enc = tq.GeneralEncoder([{"input_idx": [n * g + w], "func": ["rx", "ry", "rz", "rx"][g], "wires": [w]}
                                          for g in range(4) for w in range(n)])
            self.u3 = tq.QuantumModuleList([tq.Op1QAllLayer(op=tq.U3, n_wires=n, has_params=True, trainable=True)
                                            for _ in range(layers)])
            self.cx = tq.QuantumModuleList([tq.Op2QAllLayer(op=tq.CNOT, n_wires=n, circular=True)
                                            for _ in range(layers)])
            self.meas = tq.MeasureAll(tq.PauliZ)

        def forward(self, x):
            q = tq.QuantumDevice(n_wires=n, bsz=x.shape[0], device=DEV)
            self.enc(q, x)
            for a, b in zip(self.u3, self.cx):
                a(q)
                b(q)
            return self.meas(q)

    return Model().to(DEV)


def _apply_wires(case):
    r = random.Random("wires %d %d" % (case["seed"], case["n"]))
    return r.randrange(case["n"]), r.sample(range(case["n"]), 2)


def _unitary_wires(case):
    r = random.Random("wires %d %d" % (case["seed"], case["n"]))
    return [r.sample(range(case["n"]), case["k"]) for _ in range(case["gates"])]


def _batch_specs(case):
    r = random.Random("batch %d" % case["seed"])
    return [(r.randint(case["low"], case["high"]), r.randint(2, case["layers"])) for _ in range(case["circuits"])]


def _batch_angles(case, seed):
    r = np.random.default_rng([seed, 11])
    return [(r.normal(0, 0.4, (L, n)), r.normal(0, 0.4, (L, n))) for n, L in _batch_specs(case)]


# ------------------------------------------------------------------ what a program has in hand
def prepare(case, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    kind = case["kind"]
    st = {"case": case}
    if kind == "model":
        n = case["n"]
        model = _model(n, case["layers"])
        with torch.no_grad():
            for p in model.parameters():
                p.copy_(_normal(p.shape, g, 0.6))
        return st | {"model": model, "x": _normal((case["bsz"], 4 * n), g, 0.6),
                     "w": _normal((case["bsz"], n), g)}
    if kind in ("train", "forward"):
        gates, cols = _gates(case)
        st |= {"gates": gates, "strings": _strings(case), "w": _normal((case["strings"],), g)}
        if case["circuit"] == "ansatz":
            st |= {"x": _normal((case["bsz"], case["n"]), g, 0.5), "theta": _normal((1, cols - case["n"]), g, 0.3)}
        else:
            st["theta"] = _normal((case["bsz"], cols), g, 0.2)
        if kind == "train":
            st["theta"].requires_grad_(True)
        return st
    if kind == "observables":
        s = _product_state(case["n"], case["bsz"], g).requires_grad_(True)
        return st | {"state": s, "strings": _strings(case), "w": _normal((case["strings"],), g)}
    if kind == "sampling":
        q = tq.QuantumDevice(n_wires=case["n"], bsz=case["bsz"], device=DEV)
        q.set_states(_product_state(case["n"], case["bsz"], g))
        r = random.Random("z strings %d %d" % (case["seed"], case["n"]))
        obs = ["".join(r.choice("IZ") for _ in range(case["n"])) for _ in range(case["strings"])]
        return st | {"q": q, "strings": [o if "Z" in o else "Z" + o[1:] for o in obs], "seed": seed,
                     "generator": torch.Generator(device=DEV)}
    if kind == "apply":
        n, bsz = case["n"], case["bsz"]
        return st | {"state": _product_state(n, bsz, g).view([bsz] + [2] * n).requires_grad_(True),
                     "m1": _unitaries(bsz, 1, g).requires_grad_(True),
                     "m2": _unitaries(1, 2, g)[0].requires_grad_(True),
                     "grad": torch.randn([bsz] + [2] * n, generator=g, device=DEV, dtype=torch.complex64)}
    if kind == "unitary":
        return st | {"state": _product_state(case["n"], case["bsz"], g), "strings": _strings(case),
                     "w": _normal((case["strings"],), g),
                     "u": [u.clone().requires_grad_(True) for u in _unitaries(case["gates"], case["k"], g)]}
    cb = tqb.CircuitBatch()
    angles = _batch_angles(case, seed)
    for (n, _), (ry, rz) in zip(_batch_specs(case), angles):
        cb.add_layered(n, ry, rz)
    pb = cb.prepare(DEV, config="auto")
    pb.capture()
    mats = np.concatenate([tqb.layered_matrices(n, ry, rz) for (n, _), (ry, rz) in zip(_batch_specs(case), angles)])
    return st | {"pb": pb, "mats": mats}


# ------------------------------------------------------------------ one pass
def _record(q, st):
    case = st["case"]
    fns, theta, n = tqf.func_name_dict, st["theta"], case["n"]
    shift = 0
    gates = st["gates"]
    if case["circuit"] == "ansatz":
        for w in range(n):
            tqf.ry(q, wires=w, params=st["x"][:, w:w + 1])
        gates, shift = gates[n:], n
    for name, wires, col, k in gates:
        fns[name](q, wires=wires, params=theta[:, col - shift:col - shift + k] if k else None)


def run(st):
    case, kind = st["case"], st["case"]["kind"]
    if kind == "model":
        model = st["model"]
        model.zero_grad(set_to_none=True)
        out = model(st["x"])
        (out * st["w"]).sum().backward()
        return [out.detach()] + [p.grad for p in model.parameters()]
    if kind in ("train", "forward"):
        q = tq.QuantumDevice(n_wires=case["n"], bsz=case["bsz"], device=DEV)
        q.method = case["method"]
        if kind == "forward":
            with torch.no_grad():
                _record(q, st)
                return [tq.expval_joint_analytical_batch(q, st["strings"]), q.get_states_1d()]
        st["theta"].grad = None
        _record(q, st)
        ev = tq.expval_joint_analytical_batch(q, st["strings"])
        (ev * st["w"]).sum().backward()
        return [ev.detach(), st["theta"].grad]
    if kind == "observables":
        q = tq.QuantumDevice(n_wires=case["n"], bsz=1, device=DEV)
        st["state"].grad = None
        q.set_states(st["state"])
        ev = tq.expval_joint_analytical_batch(q, st["strings"])
        (ev * st["w"]).sum().backward()
        return [ev.detach(), st["state"].grad]
    if kind == "sampling":
        gen = st["generator"].manual_seed(st["seed"])
        got = tq.expval_joint_sampling_grouping(st["q"], sorted(set(st["strings"])), case["shots"], generator=gen)
        got["first"] = tq.expval_joint_sampling(st["q"], st["strings"][0], case["shots"], generator=gen)
        return [got[k] for k in sorted(got)]
    if kind == "apply":
        w, pair = _apply_wires(case)
        out = binding.apply_unitary_bmm(binding.apply_unitary_bmm(st["state"], st["m1"], [w]), st["m2"], pair)
        return [out.detach()] + list(torch.autograd.grad(out, (st["state"], st["m1"], st["m2"]), st["grad"]))
    if kind == "unitary":
        q = tq.QuantumDevice(n_wires=case["n"], bsz=1, device=DEV)
        q.set_states(st["state"])
        for u, wires in zip(st["u"], _unitary_wires(case)):
            u.grad = None
            tqf.qubitunitary(q, wires=wires, params=u)
        ev = tq.expval_joint_analytical_batch(q, st["strings"])
        (ev * st["w"]).sum().backward()
        return [ev.detach()] + [u.grad for u in st["u"]]
    pb = st["pb"]
    pb.set_matrices(st["mats"])
    pb.launch()
    # states are complex64: the values carry single precision
    return torch.from_numpy(pb.result().z).to(torch.float32)


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    kind = case["kind"]
    if kind == "batch":
        amps = [(1 << n, n, L) for n, L in _batch_specs(case)]
        return {"bytes": sum(n * L * 32 + 8 for _, n, L in amps), "flops": sum(a * n * L * 14 + a * 3 for a, n, L in amps)}
    n, bsz = case["n"], case["bsz"]
    amps = float(bsz << n)
    if kind in ("model", "train", "forward"):
        gates, cols = _gates(case)
        per = {"u3": 14, "rx": 14, "ry": 14, "rz": 6, "crx": 7, "cnot": 0, "cz": 0.5}
        fwd = amps * sum(per[g[0]] for g in gates)
        m = n if kind == "model" else case["strings"]
        rows = 1 if kind == "model" or case["circuit"] == "ansatz" else bsz
        if kind == "forward":
            return {"bytes": rows * cols * 4 + bsz * m * 4 + amps * 8, "flops": fwd + amps * m * 4}
        # the reverse sweep takes both states back and forms each trained gate's cotangent
        return {"bytes": rows * cols * 8 + bsz * m * 4, "flops": 4 * fwd + amps * m * 8}
    if kind == "observables":
        return {"bytes": amps * 16 + bsz * case["strings"] * 8, "flops": amps * case["strings"] * 8}
    if kind == "sampling":
        shots = bsz * case["shots"]
        return {"bytes": amps * 8 + shots * 8, "flops": amps * 4}
    if kind == "apply":  # state, gradient in; result, state gradient out
        return {"bytes": amps * 8 * 4, "flops": amps * (14 + 30) * 3}
    d = 1 << case["k"]
    return {"bytes": amps * 8 + case["gates"] * d * d * 16, "flops": amps * d * 8 * case["gates"] * 4 + amps * 8 * case["strings"]}


# ------------------------------------------------------------------ the same in 64 bits, by plain torch
C = torch.complex128


def _matrix(name, p):
    """[B, 2, 2] of a one-qubit gate (a controlled gate's lower block) at angles p [B, k]."""
    if name == "cnot":
        return torch.tensor([[[0, 1], [1, 0]]], dtype=C, device=DEV)
    if name == "cz":
        return torch.tensor([[[1, 0], [0, -1]]], dtype=C, device=DEV)
    c, s = torch.cos(p[:, 0] / 2).to(C), torch.sin(p[:, 0] / 2).to(C)
    if name in ("rx", "crx"):
        m = [c, -1j * s, -1j * s, c]
    elif name == "ry":
        m = [c, -s, s, c]
    elif name == "rz":
        e = torch.exp(0.5j * p[:, 0].to(C))
        m = [e.conj(), 0 * e, 0 * e, e]
    else:
        f, l = torch.exp(1j * p[:, 1].to(C)), torch.exp(1j * p[:, 2].to(C))
        m = [c, -l * s, f * s, f * l * c]
    return torch.stack(m, dim=1).view(-1, 2, 2)


def _parts(v, n, control, target):
    """The two halves (views) of v [B, 2^n] on which a (controlled) one-qubit gate acts."""
    if control is None:
        t = v.view(v.shape[0], 1 << target, 2, -1)
        return t[:, :, 0], t[:, :, 1]
    a, b = sorted((control, target))
    t = v.view(v.shape[0], 1 << a, 2, 1 << (b - a - 1), 2, -1)
    t = t.select(2 if control == a else 4, 1)
    d = 3 if control == a else 2
    return t.select(d, 0), t.select(d, 1)


def _apply2(v, n, control, target, m):
    x, y = _parts(v, n, control, target)
    e = lambda r, c: m[:, r, c].view([-1] + [1] * (x.dim() - 1))  # noqa: E731
    new = e(0, 0) * x + e(0, 1) * y
    y.mul_(e(1, 1)).add_(e(1, 0) * x)
    x.copy_(new)


def _pauli(v, n, s):
    """P v for a Pauli string s."""
    idx = torch.arange(1 << n, device=DEV)
    x = sum(1 << (n - 1 - w) for w, ch in enumerate(s) if ch in "XY")
    z = sum(1 << (n - 1 - w) for w, ch in enumerate(s) if ch in "YZ")
    par = (idx ^ x) & z
    for sh in (16, 8, 4, 2, 1):
        par = par ^ (par >> sh)
    sign = 1.0 - 2.0 * (par & 1).to(torch.float64)
    out = v[:, idx ^ x] if x else v.clone()
    return out.mul_(sign).mul_(1j ** s.count("Y"))


def _observe(v, n, strings, w):
    """Expectation values [B, m] and lam = sum_j w_j P_j v (w: [m] or [B, m])."""
    ev, lam = [], torch.zeros_like(v)
    for j, s in enumerate(strings):
        pv = _pauli(v, n, s)
        ev.append((v.real * pv.real).sum(1) + (v.imag * pv.imag).sum(1))
        lam += pv.mul_(w[..., j].reshape(-1, 1))
    return torch.stack(ev, dim=1), lam


def _circuit64(case, angles, strings, w, grad):
    """(expectation values, final state, d/d angles [rows of each gate] as a list per gate)."""
    n, bsz = case["n"], case["bsz"]
    v = torch.zeros(bsz, 1 << n, dtype=C, device=DEV)
    v[:, 0] = 1
    todo = [(name, wires[0] if len(wires) == 2 else None, wires[-1], p) for (name, wires, _, _), p in angles]
    for name, c, t, p in todo:
        _apply2(v, n, c, t, _matrix(name, p))
    ev, lam = _observe(v, n, strings, w)
    if not grad:
        return ev, v, None
    grads = []
    for name, c, t, p in reversed(todo):
        m = _matrix(name, p)
        mh = m.conj().transpose(1, 2)
        _apply2(v, n, c, t, mh)
        if p is None:
            grads.append(None)
        else:
            x, l = _parts(v, n, c, t), _parts(lam, n, c, t)
            cot = torch.stack([torch.stack([(l[r].conj() * x[k]).reshape(bsz, -1).sum(1) for k in range(2)], 1)
                               for r in range(2)], 1)
            q = p.detach().clone().requires_grad_(True)
            with torch.enable_grad():
                (2 * (cot * _matrix(name, q)).real.sum()).backward()
            grads.append(q.grad)
        _apply2(lam, n, c, t, mh)
    return ev, v, grads[::-1]


def _exact_unitary(case, st):
    n, k = case["n"], case["k"]
    d = 1 << k

    def split(v, wires):
        t = v.view([v.shape[0]] + [2] * n)
        return t.permute([0] + [w + 1 for w in wires] + [i + 1 for i in range(n) if i not in wires])

    def mul(v, wires, m):
        t = split(v, wires)
        shape = t.shape
        t.copy_((m @ t.reshape(v.shape[0], d, -1)).view(shape))

    v, wires = st["state"].to(C), _unitary_wires(case)
    us = [u.detach().to(C) for u in st["u"]]
    for u, ws in zip(us, wires):
        mul(v, ws, u)
    ev, lam = _observe(v, n, st["strings"], st["w"].double())
    lam *= 2  # torch's gradient of a real loss to a complex leaf
    grads = []
    for u, ws in zip(reversed(us), reversed(wires)):
        # u is unitary to single precision only: the state before the gate is its exact inverse's
        mul(v, ws, torch.linalg.inv(u))
        a, b = split(lam, ws).reshape(v.shape[0], d, -1), split(v, ws).reshape(v.shape[0], d, -1)
        grads.append((a @ b.conj().transpose(1, 2)).sum(0))
        mul(lam, ws, u.conj().T)
    return [ev] + grads[::-1]


def _exact_apply(case, st):
    n, bsz = case["n"], case["bsz"]
    w, (a, b) = _apply_wires(case)

    def mul(v, wires, m):
        t = v.view([bsz] + [2] * n).permute([0] + [q + 1 for q in wires] +
                                            [i + 1 for i in range(n) if i not in wires])
        x = t.reshape(bsz, 1 << len(wires), -1)
        out = torch.empty_like(v)
        o = out.view([bsz] + [2] * n).permute([0] + [q + 1 for q in wires] +
                                              [i + 1 for i in range(n) if i not in wires])
        o.copy_((m @ x).view(o.shape))
        return out, x

    x, g = st["state"].detach().to(C), st["grad"].to(C)
    m1, m2 = st["m1"].detach().to(C), st["m2"].detach().to(C)
    y, x1 = mul(x, [w], m1)
    out, y2 = mul(y, [a, b], m2)
    g1, _ = mul(g, [a, b], m2.conj().T)
    g0, _ = mul(g1, [w], m1.conj().transpose(1, 2))
    cot = lambda gv, wires, xv: mul(gv, wires, torch.eye(1 << len(wires), dtype=C, device=DEV))[1] @ xv.conj().transpose(1, 2)  # noqa: E731
    return [out, g0, cot(g1, [w], x1), cot(g, [a, b], y2).sum(0)]


def _exact_batch(case, seed):
    out = []
    for (n, L), (ry, rz) in zip(_batch_specs(case), _batch_angles(case, seed)):
        m = torch.from_numpy(tqb_matrices(ry, rz)).to(DEV)
        idx = torch.arange(1 << n, device=DEV)
        par = idx & (idx >> 1)
        for sh in (16, 8, 4, 2, 1):
            par = par ^ (par >> sh)
        sign = 1.0 - 2.0 * (par & 1).to(torch.float64)
        v = torch.zeros(1, 1 << n, dtype=C, device=DEV)
        v[:, 0] = 1
        for l in range(L):
            for w in range(n):
                v = (m[l, w] @ v.view(1 << w, 2, -1)).view(1, -1)
            if n > 1:
                v = v * sign
        p = v.abs().square().view(2, -1).sum(1)
        out.append(p[0] - p[1])
    return torch.stack(out)


def tqb_matrices(ry, rz):
    """[L, n, 2, 2] of RZ(rz) RY(ry)."""
    c, s, e = np.cos(ry / 2), np.sin(ry / 2), np.exp(0.5j * rz)
    return np.stack([np.conj(e) * c, -np.conj(e) * s, e * s, e * c], axis=-1).reshape(ry.shape + (2, 2))


@torch.no_grad()
def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return _exact_batch(case, seed)
    if kind == "sampling":  # estimates from shots: no value of their own in 64 bits
        return None
    st = prepare(case, seed)
    if kind == "observables":
        ev, lam = _observe(st["state"].to(C), case["n"], st["strings"], st["w"].double())
        return [ev, 2 * lam]
    if kind == "apply":
        return _exact_apply(case, st)
    if kind == "unitary":
        return _exact_unitary(case, st)
    gates, cols = _gates(case)
    n = case["n"]
    if kind == "model":
        p = [q.detach().double() for q in st["model"].parameters()]
        x, at, angles = st["x"].double(), 0, []
        for g in gates:
            if g[0] == "u3":
                angles.append((g, p[at]))
                at += 1
            else:
                angles.append((g, x[:, g[2]:g[2] + 1] if g[3] else None))
        strings = ["I" * w + "Z" + "I" * (n - 1 - w) for w in range(n)]
        ev, _, grads = _circuit64(case, angles, strings, st["w"].double(), True)
        return [ev] + [q for g, q in zip(gates, grads) if g[0] == "u3"]
    theta = st["theta"].detach().double()
    shift = n if case["circuit"] == "ansatz" else 0
    angles = [(g, None if not g[3] else st["x"].double()[:, g[2]:g[2] + 1] if g[2] < shift else
               theta[:, g[2] - shift:g[2] - shift + g[3]]) for g in gates]
    ev, v, grads = _circuit64(case, angles, st["strings"], st["w"].double(), kind == "train")
    if kind == "forward":
        return [ev, v]
    out = torch.zeros_like(theta)
    for g, q in zip(gates, grads):
        if q is not None and g[2] >= shift:
            out[:, g[2] - shift:g[2] - shift + g[3]] += q
    return [ev, out]
