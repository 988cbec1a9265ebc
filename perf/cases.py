"""Performance cases: what programs on this library have it do, over the sizes they do it at.

Every case goes through the public Python API (``CudaCvdv``, ``BatchedCircuits``,
``VariationalCircuit``).  ``listed()`` names the fixed cases, ``draw(rng)`` gives another one of
the same kinds and ranges, ``prepare``/``run`` are what a user's program does before and in the
timed part, ``work`` is the least traffic and arithmetic of one pass, and ``exact`` is the same
result in 64-bit torch, without the library.

Kinds
  transfer     CV-to-DV state transfer: initialise from register arrays, squeeze and displace the
               mode, then H / cd / Rz per qubit, and read every qubit's marginal and the state.
  network      two-mode Gaussian network: layers of beam splitter, rotations and displacements.
  mixed        random circuits over every gate the API has, on layouts of qubit, qudit and mode
               registers in any order.
  readouts     scalar readouts of a resident state: norm, marginals, photon numbers, fidelities.
  phase_space  Wigner and Husimi functions of one mode of a resident state.
  batched      many independent small circuits, one stage launch per gate.
  variational  fidelity loss and its gradient for a batch of parameter sets.

Single-precision contexts return their double-typed readouts rounded to float32: that is all the
precision a complex64 state carries.
"""

from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cuda-cvdv_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

SQRT2 = math.sqrt(2.0)


# ------------------------------------------------------------------ cases
def listed():
    return [
        # the reference's own first example: a qubit and a small mode, five gates, full readout;
        # a program that sweeps parameters makes thousands of these, so launches and latency count
        dict(name="qubit_mode", kind="transfer", layout="1,10", precision="complex128", rounds=1),
        # a mid-size transfer (2^20 amplitudes, 32 MB with its second buffer: L2-resident)
        dict(name="transfer_9_11", kind="transfer", layout="1,1,1,1,1,1,1,1,1,11", precision="complex128", rounds=9),
        # the headline workload: 14 qubits and a 2^14-point mode, both precisions
        dict(name="transfer_14_14_c128", kind="transfer", layout="1,1,1,1,1,1,1,1,1,1,1,1,1,1,14",
             precision="complex128", rounds=14),
        dict(name="transfer_14_14_c64", kind="transfer", layout="1,1,1,1,1,1,1,1,1,1,1,1,1,1,14",
             precision="complex64", rounds=14),
        # the two-mode network at its benchmark size, both precisions, and a smaller uneven one
        dict(name="network_13_13_c128", kind="network", layout="13,13", precision="complex128", layers=3),
        dict(name="network_13_13_c64", kind="network", layout="13,13", precision="complex64", layers=3),
        dict(name="network_9_10", kind="network", layout="9,10", precision="complex128", layers=6),
        # every gate, on a layout with a qudit, a mode that is not last and a trailing qubit
        dict(name="mixed_2_8_9_1", kind="mixed", layout="2,8,9,1", precision="complex128", gates=60),
        # scalar readouts of a 2^22 state with a strided and a contiguous mode
        dict(name="readouts_1_9_12", kind="readouts", layout="1,9,12", precision="complex128"),
        # phase-space pictures of a mode entangled with two qubits
        dict(name="phase_space_1_1_11", kind="phase_space", layout="1,1,11", precision="complex128", register=2),
        # uneven circuits run as one batch (the ranges of the batched benchmark, fewer instances)
        dict(name="batched_96", kind="batched", precision="complex64", count=96, gates=50, m_low=8, m_high=13),
        # a training step of the variational benchmark: 64 parameter sets, 40 layers
        dict(name="variational_64_12", kind="variational", layout="1,12", precision="complex64", batch=64, layers=40,
             graphs=True),
    ]


def _log_int(rng, lo, hi):
    """An integer of [lo, hi], uniform in its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["transfer", "transfer", "network", "network", "mixed", "readouts", "phase_space", "batched",
                       "variational"])
    prec = rng.choice(["complex128", "complex64"])
    if kind == "transfer":
        nq, m = rng.randint(1, 14), rng.randint(8, 14)
        return dict(kind=kind, layout=",".join(["1"] * nq + [str(m)]), precision=prec, rounds=rng.randint(1, nq))
    if kind == "network":
        q0, q1 = rng.randint(6, 13), rng.randint(6, 13)
        return dict(kind=kind, layout="%d,%d" % (q0, q1), precision=prec, layers=rng.randint(1, 6 if q0 + q1 < 25 else 3))
    if kind == "mixed":
        regs = [rng.randint(7, 11), rng.randint(6, 9)] + [rng.choice([1, 1, 1, 2, 3]) for _ in range(rng.randint(1, 4))]
        rng.shuffle(regs)
        return dict(kind=kind, layout=",".join(map(str, regs)), precision=prec, gates=_log_int(rng, 10, 120))
    if kind == "readouts":
        regs = [rng.randint(6, 12), rng.randint(6, 10)] + [rng.choice([1, 1, 2]) for _ in range(rng.randint(0, 3))]
        rng.shuffle(regs)
        return dict(kind=kind, layout=",".join(map(str, regs)), precision=prec)
    if kind == "phase_space":
        regs = [1] * rng.randint(0, 6) + [rng.randint(6, 11)]
        rng.shuffle(regs)
        return dict(kind=kind, layout=",".join(map(str, regs)), precision=prec, register=regs.index(max(regs)))
    if kind == "batched":
        lo = rng.randint(8, 12)
        return dict(kind=kind, precision=prec, count=_log_int(rng, 3, 128), gates=rng.randint(10, 50), m_low=lo,
                    m_high=rng.randint(lo, 13))
    nq = rng.randint(1, 2)
    return dict(kind=kind, layout=",".join(["1"] * nq + [str(rng.randint(8, 12))]), precision=prec,
                batch=_log_int(rng, 1, 64), layers=rng.randint(3, 40), graphs=rng.random() < 0.5)


# ------------------------------------------------------------------ inputs
def _layout(case):
    return [int(v) for v in case["layout"].split(",")]


def _rng(case, seed):
    return np.random.default_rng([int(seed), 20241])


def _cnormal(rng, sigma=1.0):
    return complex(sigma * (rng.standard_normal() + 1j * rng.standard_normal()) / SQRT2)


def _grid(N, device="cuda"):
    return (torch.arange(N, dtype=torch.float64, device=device) - 0.5 * (N - 1)) * math.sqrt(2.0 * math.pi / N)


def _packet(N, rng, device="cuda", sigma=0.7):
    """A normalised superposition of two coherent states near the origin, as a mode's array."""
    x = _grid(N, device)
    out = torch.zeros(N, dtype=torch.complex128, device=device)
    for _ in range(2):
        a, c = _cnormal(rng, sigma), _cnormal(rng) + 0.5
        out += c * torch.exp(-0.5 * (x - SQRT2 * a.real) ** 2 + 1j * SQRT2 * a.imag * x)
    return out / torch.linalg.vector_norm(out)


def _registers(case, seed, device="cuda"):
    """The initial register arrays of a circuit (complex128)."""
    rng = np.random.default_rng([int(seed), 11])
    out = []
    for q in _layout(case):
        if q >= 4:
            out.append(_packet(1 << q, rng, device))
        elif case["kind"] in ("transfer", "variational"):
            a = torch.zeros(1 << q, dtype=torch.complex128, device=device)
            a[0] = 1.0
            out.append(a)
        else:
            v = rng.standard_normal(1 << q) + 1j * rng.standard_normal(1 << q)
            out.append(torch.from_numpy(v / np.linalg.norm(v)).to(device))
    return out


def _circuit(case, seed):
    """The circuit's gates as (method, arguments) of the CudaCvdv API."""
    rng, qs, g = _rng(case, seed), _layout(case), []
    if case["kind"] == "transfer":
        mode = len(qs) - 1
        g += [("s", (mode, float(rng.uniform(0.05, 0.5)))), ("d", (mode, _cnormal(rng, 1.5)))]
        for k in range(1, int(case["rounds"]) + 1):
            beta = math.sqrt(math.pi / 2.0) * 2.0 ** (-k)
            g += [("h", (k - 1, 0)), ("cd", (mode, k - 1, 0, beta)), ("rz", (k - 1, 0, float(rng.uniform(0, 2 * math.pi))))]
        return g
    if case["kind"] == "network":
        same = qs[0] == qs[1]
        g += [("s", (r, float(rng.uniform(0.2, 0.8)))) for r in (0, 1)]
        for _ in range(int(case["layers"])):
            g += [("bs", (0, 1, float(rng.uniform(0, math.pi / 2 if same else 1.5))))]
            g += [("r", (r, float(rng.uniform(0, 2 * math.pi)))) for r in (0, 1)]
            g += [("d", (r, _cnormal(rng))) for r in (0, 1)]
        return g
    return _mixed_gates(case, rng, qs)


def _mixed_gates(case, rng, qs):
    modes = [r for r, q in enumerate(qs) if q >= 4]
    small = [r for r, q in enumerate(qs) if q < 4]
    g = []

    def qubit():
        r = int(rng.choice(small))
        return r, int(rng.integers(qs[r]))

    kinds = ["d", "cd", "cr", "rx", "ry", "rz", "h", "p", "cp", "sheer", "phaseCubic", "r", "s", "cs", "bs", "cbs",
             "q1q2", "x", "ftQ2P", "swap"]
    for i in range(int(case["gates"])):
        k = kinds[i] if i < len(kinds) else str(rng.choice(kinds))
        t, u = int(rng.choice(modes)), float(rng.uniform(-1.2, 1.2))
        c = qubit()
        if k in ("h", "x"):
            g.append((k, c))
        elif k in ("rx", "ry", "rz"):
            g.append((k, c + (float(rng.uniform(0, 2 * math.pi)),)))
        elif k == "d":
            g.append((k, (t, _cnormal(rng, 0.4))))
        elif k == "cd":
            g.append((k, (t,) + c + (_cnormal(rng, 0.4),)))
        elif k == "cr":
            g.append((k, (t,) + c + (float(rng.uniform(0, 2 * math.pi)),)))
        elif k == "cs":
            g.append((k, (t,) + c + (0.2 * u if abs(u) > 0.1 else 0.1,)))
        elif k == "cp":
            g.append((k, (t,) + c))
        elif k in ("p", "ftQ2P"):
            g.append((k, (t,)))
        elif k == "r":
            g.append((k, (t, float(rng.uniform(0, 2 * math.pi)))))
        elif k in ("s", "sheer"):
            g.append((k, (t, 0.25 * u)))
        elif k == "phaseCubic":
            g.append((k, (t, 0.02 * u)))
        elif k == "bs":
            g.append((k, (modes[0], modes[1], u)))
        elif k == "cbs":
            g.append((k, (modes[1], modes[0]) + c + (u,)))
        elif k == "q1q2":
            g.append((k, (modes[0], modes[1], 0.2 * u)))
        else:  # swap of two registers of one size, where the layout has them
            pairs = [(a, b) for a in range(len(qs)) for b in range(a) if qs[a] == qs[b]]
            if pairs:
                g.append((k, pairs[int(rng.integers(len(pairs)))]))
    return g


def _resident_circuit(case, seed):
    """Gates that entangle the registers of a state that is then read out."""
    rng, qs = _rng(case, seed), _layout(case)
    modes = [r for r, q in enumerate(qs) if q >= 4]
    small = [r for r, q in enumerate(qs) if q < 4]
    g = [("s", (m, float(rng.uniform(0.05, 0.3)))) for m in modes]
    for r in small:
        g.append(("h", (r, 0)))
        for m in modes:
            g.append(("cd", (m, r, 0, _cnormal(rng, 0.8))))
    if len(modes) > 1:
        g.append(("bs", (modes[0], modes[1], float(rng.uniform(0.2, 1.2)))))
    return g


def _instances(case, seed):
    """The uneven circuits of a batch and their start states (each a flat complex128 tensor)."""
    shapes, rng, out = np.random.default_rng(int(case["count"])), _rng(case, seed), []
    for _ in range(int(case["count"])):
        Q, m = int(shapes.integers(1, 4)), int(shapes.integers(int(case["m_low"]), int(case["m_high"]) + 1))
        g = []
        for _ in range(int(case["gates"])):
            k, c = int(rng.integers(7)), int(rng.integers(Q))
            if k == 0:
                g.append(("h", (c, 0)))
            elif k in (1, 2):
                g.append((("rx", "rz")[k - 1], (c, 0, float(rng.uniform(0, 2 * math.pi)))))
            elif k == 3:
                g.append(("cd", (Q, c, 0, _cnormal(rng))))
            elif k == 4:
                g.append(("d", (Q, _cnormal(rng))))
            elif k == 5:
                g.append(("s", (Q, float(rng.uniform(0.02, 0.5)))))
            else:
                g.append(("r", (Q, float(rng.uniform(0, 2 * math.pi)))))
        out.append(dict(qubits=[1] * Q + [m], gates=g))
    return out


def _start_states(insts, seed, device="cuda"):
    rng, out = np.random.default_rng([int(seed), 12]), []
    for inst in insts:
        mode = _packet(1 << inst["qubits"][-1], rng, device)
        psi = torch.zeros(1 << (len(inst["qubits"]) - 1), mode.numel(), dtype=torch.complex128, device=device)
        psi[0] = mode
        out.append(psi.reshape(-1))
    return out


def _variational(case, seed, device="cuda"):
    """Parameters, start state and target of a variational problem; gates in the circuit's form."""
    rng, qs = _rng(case, seed), _layout(case)
    layers, B, nq = int(case["layers"]), int(case["batch"]), len(qs) - 1
    gates, p = [], np.empty((B, 2 * layers))
    for l in range(layers):
        gates += [("rx", l % nq, 0), ("cd", nq, l % nq, 0)]
        p[:, 2 * l] = rng.uniform(0, 2 * math.pi, B)
        p[:, 2 * l + 1] = rng.normal(0, 0.5, B)
    x = _grid(1 << qs[-1], device)
    start = torch.zeros(1 << nq, x.numel(), dtype=torch.complex128, device=device)
    start[0] = torch.exp(-0.5 * x * x)
    target = torch.zeros_like(start)
    a = SQRT2 * float(rng.uniform(1.5, 2.5))
    target[0] = torch.exp(-0.5 * (x - a) ** 2) + torch.exp(-0.5 * (x + a) ** 2)
    start, target = (v.reshape(-1) / torch.linalg.vector_norm(v) for v in (start, target))
    dt = torch.float32 if case["precision"] == "complex64" else torch.float64
    return gates, torch.from_numpy(p).to(device=device, dtype=dt), start, target


# ------------------------------------------------------------------ the library
def _separable(qs, arrays):
    from cvdv_b200 import SeparableState
    sep = SeparableState(qs)
    for r, a in enumerate(arrays):
        sep.setCoeffs(r, a)
    return sep


def _apply(sim, gates):
    for name, args in gates:
        getattr(sim, name)(*args)


def prepare(case, seed):
    from cvdv_b200 import CudaCvdv
    kind = case["kind"]
    if kind == "batched":
        from cvdv_b200.batch import BatchedCircuits
        insts = _instances(case, seed)
        return dict(case=case, batch=BatchedCircuits(insts, precision=case["precision"]),
                    start=_start_states(insts, seed), sizes=[1 << sum(i["qubits"]) for i in insts])
    if kind == "variational":
        from cvdv_b200.variational import VariationalCircuit
        gates, params, start, target = _variational(case, seed)
        circ = VariationalCircuit(_layout(case), gates, precision=case["precision"], graphs=bool(case["graphs"]))
        return dict(case=case, circ=circ, params=params, start=start.to(circ.cdtype), target=target.to(circ.cdtype))
    qs = _layout(case)
    sim = CudaCvdv(qs, precision=case["precision"])
    sep = _separable(qs, _registers(case, seed))
    state = dict(case=case, sim=sim, sep=sep)
    if kind in ("readouts", "phase_space"):
        sim.initStateVector(sep)
        _apply(sim, _resident_circuit(case, seed))
        sim.synchronize()
        if kind == "readouts":  # a second state to compare with: the product state
            state["other"] = CudaCvdv(qs, precision=case["precision"])
            state["other"].initStateVector(sep)
            state["other"].synchronize()
    else:
        state["gates"] = _circuit(case, seed)
    return state


def _as_state_precision(case, v):
    """Readouts come as float64; those of a complex64 state are kept as float32."""
    if case["precision"] == "complex128":
        return v
    if isinstance(v, dict):
        return {k: _as_state_precision(case, x) for k, x in v.items()}
    if isinstance(v, list):
        return [_as_state_precision(case, x) for x in v]
    return np.asarray(v, dtype=np.float32) if isinstance(v, (float, np.ndarray)) else v


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "batched":
        b = state["batch"]
        b.set_initial(state["start"])
        b.run(graph=True)
        return b.states
    if kind == "variational":
        p = state["params"].detach().requires_grad_(True)
        loss = state["circ"].fidelity_loss(p, state["start"], state["target"]).to(p.dtype)
        loss.sum().backward()
        return dict(loss=loss.detach(), grad=p.grad)
    sim = state["sim"]
    regs = range(sim.num_registers)
    if kind == "readouts":
        modes = [r for r in regs if sim.register_dims[r] >= 16]
        small = [r for r in regs if sim.register_dims[r] < 16]
        out = dict(norm=sim.m(), marginals=[sim.m(r) for r in regs], photons=[sim.getPhotonNumber(r) for r in modes],
                   product=sim.getFidelity(state["sep"]), pair=sim.fidelityWith(state["other"]))
        if small:
            out["joint"] = sim.m(small[0], modes[1])
        return _as_state_precision(case, out)
    if kind == "phase_space":
        r = int(case["register"])
        return _as_state_precision(case, dict(wigner=sim.getWigner(r), husimi=sim.getHusimiQ(r)))
    sim.initStateVector(state["sep"])
    _apply(sim, state["gates"])
    out = dict(marginals=_as_state_precision(case, sim.mEach(_read_registers(case))))
    out["state"] = sim.stateTensor()
    out["state"].simulator = sim  # the tensor is a view of the simulator's buffer: it keeps it alive
    return out


def _read_registers(case):
    """The registers whose marginals a circuit ends with: a transfer's qubits, the others' all."""
    n = len(_layout(case))
    return list(range(n - 1)) if case["kind"] == "transfer" and n > 2 else list(range(n))


# ------------------------------------------------------------------ the least work
#: transforms, diagonal passes and 2x2 updates that each gate's definition is made of
_GATE_OPS = {"d": (2, 2, 0), "cd": (2, 2, 0), "r": (2, 3, 0), "cr": (2, 3, 0), "s": (4, 4, 0), "cs": (4, 4, 0),
             "bs": (4, 3, 0), "cbs": (4, 3, 0), "ftQ2P": (1, 0, 0), "h": (0, 0, 1), "rx": (0, 0, 1), "ry": (0, 0, 1),
             "x": (0, 0, 1)}


def _gate_flops(gates, qs):
    n, fl = float(1 << sum(qs)), 0.0
    for name, args in gates:
        t, d, p = _GATE_OPS.get(name, (0, 1, 0))
        fl += t * 5.0 * n * qs[args[0]] + d * 6.0 * n + p * 14.0 * n
    return fl


def work(case):
    kind, b = case["kind"], 16.0 if case["precision"] == "complex128" else 8.0
    if kind == "batched":
        insts = _instances(case, 0)
        size = float(sum(1 << sum(i["qubits"]) for i in insts))
        return dict(bytes=size * (16.0 + b), flops=sum(_gate_flops(i["gates"], i["qubits"]) for i in insts))
    qs = _layout(case)
    n = float(1 << sum(qs))
    regs = 16.0 * sum(1 << q for q in qs)
    if kind == "variational":
        B, L = float(case["batch"]), float(case["layers"])
        # forward: one state per set; the adjoint walks the state and the target back
        return dict(bytes=(2 * n + 4 * B * L) * b, flops=3 * B * L * (10.0 * n * qs[-1] + 26.0 * n))
    if kind == "readouts":
        modes = sum(1 for q in qs if q >= 4)
        return dict(bytes=2 * n * b + regs * 1.5, flops=n * (4.0 * (len(qs) + 3) + 16.0)
                    + modes * 8 * n + sum(5.0 * n * q for q in qs if q >= 4))
    if kind == "phase_space":
        N = float(1 << qs[int(case["register"])])
        return dict(bytes=n * b + 16.0 * N * N,
                    flops=2.0 * N * n + 2.5 * N * N * math.log2(N) + n * N * (5.0 * math.log2(N) + 8.0))
    return dict(bytes=regs + n * b, flops=_gate_flops(_circuit(case, 0), qs))


# ------------------------------------------------------------------ the same in 64-bit torch
class _Plain:
    """A dense state as a torch tensor with one axis a register, each gate by its definition."""

    def __init__(self, qs, arrays):
        self.q = qs
        t = arrays[0]
        for a in arrays[1:]:
            t = torch.outer(t.reshape(-1), a).reshape(-1)
        self.t = t.reshape([1 << q for q in qs]).clone()

    def _axis(self, v, r):
        shape = [1] * len(self.q)
        shape[r] = -1
        return v.reshape(shape)

    def x(self, r):
        return self._axis(_grid(1 << self.q[r], self.t.device), r)

    def z(self, r, k):
        j = torch.arange(1 << self.q[r], device=self.t.device)
        return self._axis(1.0 - 2.0 * ((j >> (self.q[r] - 1 - k)) & 1).double(), r)

    def phase(self, v):
        self.t *= torch.polar(torch.ones_like(v), v)

    def ft(self, r, sign):
        """Centred unitary transform with kernel exp(-i sign x p) / sqrt(N)."""
        N = 1 << self.q[r]
        j = torch.arange(N, device=self.t.device)
        tw = torch.polar(torch.ones(N, dtype=torch.float64, device=j.device),
                         sign * math.pi * (((N - 1) * j) % (2 * N)).double() / N)
        self.t *= self._axis(tw, r)
        self.t = (torch.fft.fft if sign > 0 else torch.fft.ifft)(self.t, dim=r, norm="ortho")
        a = -sign * math.pi * (((N - 1) ** 2) % (4 * N)) / (2 * N)
        self.t *= self._axis(tw, r) * complex(math.cos(a), math.sin(a))

    def two(self, r, k, m):
        shape = list(self.t.shape)
        b = self.q[r] - 1 - k
        v = self.t.reshape(shape[:r] + [shape[r] >> (b + 1), 2, 1 << b] + shape[r + 1:])
        a0, a1 = v.select(r + 1, 0), v.select(r + 1, 1)
        self.t = torch.stack((m[0] * a0 + m[1] * a1, m[2] * a0 + m[3] * a1), dim=r + 1).reshape(shape)

    def rx(self, r, k, th):
        c, s = math.cos(th / 2), math.sin(th / 2)
        self.two(r, k, (c, -1j * s, -1j * s, c))

    def ry(self, r, k, th):
        c, s = math.cos(th / 2), math.sin(th / 2)
        self.two(r, k, (c, -s, s, c))

    def rz(self, r, k, th):
        self.phase(-0.5 * th * self.z(r, k))

    def h(self, r, k):
        s = 1 / SQRT2
        self.two(r, k, (s, s, s, -s))

    def gate_x(self, r, k):
        self.rx(r, k, math.pi)

    def p(self, r):
        self.t = self.t.flip(r)

    def cp(self, r, cr, ck):
        self.t = torch.where(self.z(cr, ck) < 0, self.t.flip(r), self.t)

    def swap(self, a, b):
        self.t = self.t.transpose(a, b).contiguous()

    def sheer(self, r, t):
        self.phase(t * self.x(r) ** 2)

    def phaseCubic(self, r, t):
        self.phase(t * self.x(r) ** 3)

    def ftQ2P(self, r):
        self.ft(r, 1)

    def _shift(self, r, a, z):
        if abs(a.imag) > 1e-12:
            self.phase(SQRT2 * a.imag * self.x(r) * z)
        if abs(a.real) > 1e-12:
            self.ft(r, 1)
            self.phase(-SQRT2 * a.real * self.x(r) * z)
            self.ft(r, -1)

    def d(self, r, a):
        self._shift(r, complex(a), 1.0)

    def cd(self, r, cr, ck, a):
        self._shift(r, complex(a), self.z(cr, ck))

    def _turn(self, r, th, z):
        if abs(th) < 1e-15:
            return
        t, s, x2 = math.tan(th / 2), math.sin(th), self.x(r) ** 2 * z
        self.phase(-0.5 * t * x2)
        self.ft(r, 1)
        self.phase(-0.5 * s * x2)
        self.ft(r, -1)
        self.phase(-0.5 * t * x2)

    @staticmethod
    def _quarter(th):
        k = int(np.rint(th / (math.pi / 2)))
        return k % 4, th - k * (math.pi / 2)

    def r(self, r, th):
        k, rest = self._quarter(th)
        if k == 2:
            self.p(r)
        elif k:
            self.ft(r, 1 if k == 1 else -1)
        self._turn(r, rest, 1.0)

    def cr(self, r, cr, ck, th):
        k, rest = self._quarter(th)
        if k == 2:
            self.p(r)
            self.rz(cr, ck, math.pi)
        elif k:
            sg = 1 if k == 1 else -1
            self.ft(r, sg)
            self.cp(r, cr, ck)
            self.rz(cr, ck, sg * math.pi / 2)
        self._turn(r, rest, self.z(cr, ck))

    def s(self, r, v):
        a, b, c = math.exp(0.5 * v), math.exp(-0.5 * v), math.sqrt(abs(math.exp(v) - 1.0))
        sg, x2 = (1.0 if v >= 0 else -1.0), self.x(r) ** 2
        for coeff, sign in ((-0.5 * a * c, 1), (0.5 * b * c * sg, -1), (0.5 * b * c, 1), (-0.5 * a * c * sg, -1)):
            self.ft(r, sign)
            self.phase(coeff * x2)

    def cs(self, r, cr, ck, v):
        ch, sh, c = math.cosh(v), math.sinh(v), math.sqrt(2.0 * abs(math.sinh(0.5 * v)))
        z, x2 = self.z(cr, ck), self.x(r) ** 2
        self.phase((0.5 * c * ch - 0.5 * c * sh * z) * x2)
        self.ft(r, 1)
        self.phase((0.5 * (ch - 1) / c + 0.5 * sh / c * z) * x2)
        self.ft(r, -1)
        self.phase(-0.5 * c * x2)
        self.ft(r, 1)
        self.phase((0.5 * (ch - 1) / c - 0.5 * sh / c * z) * x2)
        self.ft(r, -1)

    def _mix(self, a, b, th, z):
        if abs(th) < 1e-15:
            return
        xx = self.x(a) * self.x(b) * z
        self.phase(-math.tan(0.25 * th) * xx)
        self.ft(a, 1)
        self.ft(b, 1)
        self.phase(-math.sin(0.5 * th) * xx)
        self.ft(a, -1)
        self.ft(b, -1)
        self.phase(-math.tan(0.25 * th) * xx)

    def bs(self, a, b, th):  # the cases' angles stay below pi / 2: no half turns
        self._mix(a, b, th, 1.0)

    def cbs(self, a, b, cr, ck, th):
        self._mix(a, b, th, self.z(cr, ck))

    def q1q2(self, a, b, c):
        self.phase(c * self.x(a) * self.x(b))

    def apply(self, gates):
        for name, args in gates:
            getattr(self, "gate_x" if name == "x" else name)(*args)

    def prob(self, keep):
        p = self.t.real ** 2 + self.t.imag ** 2
        drop = [r for r in range(len(self.q)) if r not in keep]
        p = p.sum(dim=drop) if drop else p
        order = sorted(keep)
        return p.permute([order.index(r) for r in keep])

    def slices(self, r):
        return self.t.movedim(r, -1).reshape(-1, 1 << self.q[r])


def _exact_wigner(sim, r):
    """W[jc][i] from G[i][d] = sum conj(psi[i + d]) psi[i - d], d = k - (N - 1) // 2."""
    N, v = 1 << sim.q[r], sim.slices(r)
    i = torch.arange(N, device=v.device)[:, None]
    d = torch.arange(N, device=v.device)[None, :] - (N - 1) // 2
    ok = (i + d >= 0) & (i + d < N) & (i - d >= 0) & (i - d < N)
    up, dn = (i + d).clamp(0, N - 1), (i - d).clamp(0, N - 1)
    G = torch.zeros(N, N, dtype=torch.complex128, device=v.device)
    for row in v:
        G += torch.where(ok, row[up].conj() * row[dn], 0.0)
    H = torch.fft.ifft(G, dim=1, norm="forward")
    s = torch.arange(N, device=v.device) - N // 2
    ph = torch.polar(torch.ones(N, dtype=torch.float64, device=v.device),
                     math.pi * ((-s * (N - 1)) % (2 * N)).double() / N)
    return ((H[:, s % N] * ph).real * (math.sqrt(2 * math.pi / N) / math.pi)).T.contiguous()


def _exact_husimi(sim, r):
    N, v = 1 << sim.q[r], sim.slices(r)
    dx = math.sqrt(2 * math.pi / N)
    k = torch.arange(N, device=v.device)
    p = 2 * math.pi * torch.where(k <= N // 2, k, k - N).double() / (N * dx)
    g = math.pi ** 0.25 * math.sqrt(2 / dx) * torch.exp(-0.5 * p * p)
    at = (k[:, None] + k[None, :]) % N
    acc = torch.zeros(N, N, dtype=torch.float64, device=v.device)
    for row in torch.fft.fft(v, dim=1):
        H = torch.fft.ifft(row[at] * g, dim=1, norm="forward")
        acc += H.real ** 2 + H.imag ** 2
    return acc.roll(N // 2, 0) / (math.pi * N * N)


def _exact_variational(case, seed):
    gates, params, start, target = _variational(case, seed)
    qs = _layout(case)
    p = params.double().requires_grad_(True)
    B, nq, N = p.shape[0], len(qs) - 1, 1 << qs[-1]
    x = _grid(N)
    j = torch.arange(N, device="cuda")
    one = torch.ones(N, dtype=torch.float64, device="cuda")
    tw = torch.polar(one, math.pi * (((N - 1) * j) % (2 * N)).double() / N)
    psi = start.expand(B, -1).reshape(B, 1 << nq, N)
    for g, gate in enumerate(gates):
        k = gate[1] if gate[0] == "rx" else gate[2]
        v = psi.reshape(B, 1 << k, 2, 1 << (nq - 1 - k), N)
        if gate[0] == "rx":
            c, s = (f(p[:, g] / 2).reshape(B, 1, 1, 1, 1) for f in (torch.cos, torch.sin))
            v = c * v - 1j * s * v.flip(2)
        else:
            ph = -SQRT2 * p[:, g].reshape(B, 1, 1, 1, 1) * x
            ph = torch.cat((ph, -ph), dim=2)
            v = torch.fft.fft(v * tw, norm="ortho") * tw * torch.polar(torch.ones_like(ph), ph)
            v = torch.fft.ifft(v * tw.conj(), norm="ortho") * tw.conj()
        psi = v.reshape(B, 1 << nq, N)
    ov = (target.conj() * psi.reshape(B, -1)).sum(dim=1)
    loss = 1.0 - (ov.real ** 2 + ov.imag ** 2)
    loss.sum().backward()
    return dict(loss=loss.detach(), grad=p.grad)


def exact(case, seed):
    kind = case["kind"]
    if kind == "variational":
        return _exact_variational(case, seed)
    if kind == "batched":
        insts, out = _instances(case, seed), []
        for inst, psi in zip(insts, _start_states(insts, seed)):
            sim = _Plain(inst["qubits"], [psi])
            sim.apply(inst["gates"])
            out.append(sim.t.reshape(-1))
        return torch.cat(out)
    arrays, qs = _registers(case, seed), _layout(case)
    sim = _Plain(qs, arrays)
    if kind not in ("readouts", "phase_space"):
        sim.apply(_circuit(case, seed))
        marg = [sim.prob([r]).cpu().numpy() for r in _read_registers(case)]
        return dict(marginals=marg, state=sim.t.reshape(-1))
    sim.apply(_resident_circuit(case, seed))
    if kind == "phase_space":
        r = int(case["register"])
        return dict(wigner=_exact_wigner(sim, r), husimi=_exact_husimi(sim, r))
    first = _Plain(qs, arrays)
    modes = [r for r, q in enumerate(qs) if q >= 4]
    small = [r for r, q in enumerate(qs) if q < 4]
    photons = []
    for r in modes:
        x2 = (sim.prob([r]) * _grid(1 << qs[r]) ** 2).sum()
        sim.ft(r, 1)
        p2 = (sim.prob([r]) * _grid(1 << qs[r]) ** 2).sum()
        sim.ft(r, -1)
        photons.append(float(0.5 * (x2 + p2 - 1.0)))
    fid = float((first.t.conj() * sim.t).sum().abs() ** 2)
    out = dict(norm=float(sim.prob([0]).sum()), marginals=[sim.prob([r]) for r in range(len(qs))], photons=photons,
               product=fid, pair=fid)
    if small:
        out["joint"] = sim.prob([small[0], modes[1]])
    return out
