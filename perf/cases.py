"""Timed cases of the engine's public entry points.

Each case is one call (or one short sequence of calls) that a user's program makes, at the sizes
that the benchmark configurations and the tests use: the drop-in port on host buffers, one-shot and
planned evolution of resident states, dense fused gates, energies, sampling, monitored circuits,
variational gradients and noise trajectories, in both precisions.

  listed()          the fixed cases
  draw(rng)         one more case from the same ranges
  prepare(case, s)  inputs made from seed s, with the plans and states a program keeps
  run(state)        one pass
  work(case)        bytes and flops that one pass cannot do without
  exact(case, s)    run's outputs in 64 bits from plain torch, where that is quick enough
"""
from __future__ import annotations

import math

import numpy as np
import torch

from quantummatter_b200 import QuantumCircuit, SingleQubitUnitary
from quantummatter_b200.algorithms import QuantumFourierTransform
from quantummatter_b200.backend import (FP32, FP64, B200BackendOptions, B200Context, B200StateVectorBackend,
                                        DeviceState, Plan)
from quantummatter_b200.noise import NoiseChannel, NoisyCircuit
from quantummatter_b200.observables import PauliHamiltonian, PauliString, PauliTerm
from quantummatter_b200.trajectories import B200NoisySimulator
from quantummatter_b200.variational import B200VariationalEnergyEvaluator, ParameterizedCircuit

GIB = 1 << 30
_context = None


def context() -> B200Context:
    """The program's one context: an engine instance lives as long as the program does."""
    global _context
    if _context is None:
        _context = B200Context(B200BackendOptions(DeviceMemoryBudgetBytes=96 * GIB, StagingMemoryBudgetBytes=32 * GIB))
    return _context


# ------------------------------------------------------------------------------------ the cases

def listed():
    return [
        # The drop-in port on a small register, where launches and host work count: a caller's loop over
        # small circuits (teaching material, unit tests, small algorithm instances).
        {"name": "port_small", "kind": "port", "qubits": 10, "depth": 10, "pinned": False},
        # The drop-in port at the reference's own benchmark size (20 qubits, depth 20, 590 gates).
        {"name": "port_20q", "kind": "port", "qubits": 20, "depth": 20, "pinned": True},
        # One-shot evolution of a resident state: a program that builds a circuit and runs it once, the
        # path of the server and of the dynamic simulator's single trajectories.
        {"name": "evolve_brick_21q", "kind": "evolve", "circuit": "brick", "qubits": 21, "depth": 24, "precision": FP32},
        {"name": "evolve_qft_25q", "kind": "evolve", "circuit": "qft", "qubits": 25, "depth": 0, "precision": FP64},
        # A plan made once and run many times: the 30-qubit random circuit of the headline benchmark, and
        # a complex64 one of odd size.
        {"name": "plan_30q_fp64", "kind": "plan", "qubits": 30, "depth": 40, "width": 0, "precision": FP64},
        {"name": "plan_27q_fp32", "kind": "plan", "qubits": 27, "depth": 17, "width": 0, "precision": FP32},
        # Dense fused gates of at most k qubits (the benchmark's width sweep, k = 2..6).
        {"name": "dense_k4_fp64", "kind": "plan", "qubits": 26, "depth": 12, "width": 4, "precision": FP64},
        # Energy of a resident state: the XXZ chain of the variational benchmark, as an optimiser or a
        # time-evolution loop reads it after each step.
        {"name": "energy_28q_fp64", "kind": "energy", "model": "xxz", "qubits": 28, "precision": FP64},
        # Terminal sampling of a resident state: the 1000 shots of a served request.
        {"name": "sample_27q_fp64", "kind": "sample", "qubits": 27, "shots": 1000, "precision": FP64},
        # A monitored circuit: unitary layer, amplitude damping, a marginal and a mid-circuit measurement
        # on a resident state (the steps of the noisy dynamic simulator).
        {"name": "monitored_26q_fp64", "kind": "monitored", "qubits": 26, "rounds": 3, "precision": FP64},
        # One optimiser step over a batch of parameter vectors: energies and parameter-shift gradients of
        # the 4-layer hardware-efficient ansatz.
        {"name": "vqe_18q_fp32", "kind": "vqe", "qubits": 18, "vectors": 8, "precision": FP32},
        # Noise trajectories: RY layers and CZ ladders with depolarizing and damping channels.
        {"name": "trajectories_22q_fp32", "kind": "trajectories", "qubits": 22, "depth": 10, "trajectories": 48,
         "precision": FP32},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["port", "evolve", "plan", "dense", "energy", "sample", "monitored", "vqe", "trajectories"])
    precision = rng.choice([FP64, FP32])
    if kind == "port":
        n = rng.randint(4, 23)
        return {"kind": kind, "qubits": n, "depth": _log_int(rng, 4, 40), "pinned": rng.random() < 0.5}
    if kind == "evolve":
        circuit = rng.choice(["brick", "qft"])
        return {"kind": kind, "circuit": circuit, "qubits": rng.randint(10, 27),
                "depth": _log_int(rng, 6, 40) if circuit == "brick" else 0, "precision": precision}
    if kind == "plan":
        return {"kind": "plan", "qubits": rng.randint(16, 29), "depth": _log_int(rng, 6, 40), "width": 0,
                "precision": precision}
    if kind == "dense":
        return {"kind": "plan", "qubits": rng.randint(20, 27), "depth": _log_int(rng, 4, 16),
                "width": rng.randint(2, 6), "precision": precision}
    if kind == "energy":
        return {"kind": kind, "model": rng.choice(["xxz", "tfim"]), "qubits": rng.randint(10, 29),
                "precision": precision}
    if kind == "sample":
        return {"kind": kind, "qubits": rng.randint(10, 29), "shots": _log_int(rng, 1, 20000), "precision": precision}
    if kind == "monitored":
        return {"kind": kind, "qubits": rng.randint(10, 28), "rounds": rng.randint(1, 6), "precision": precision}
    if kind == "vqe":
        n = rng.randint(12, 20)
        return {"kind": kind, "qubits": n, "vectors": rng.randint(1, 16 if n < 18 else 6), "precision": precision}
    n = rng.randint(14, 23)
    return {"kind": kind, "qubits": n, "depth": rng.randint(3, 16),
            "trajectories": rng.randint(8, 256 if n < 20 else 48), "precision": precision}


# ------------------------------------------------------------------------------------ inputs

def _rng(seed, salt):
    return np.random.default_rng([seed & 0xFFFFFFFF, salt])


def _brick(n, depth, seed):
    """U3 with uniform angles on every qubit, then CNOTs on alternating neighbour pairs, as
    ("u", qubit, 2x2 matrix) and ("cx", control, target)."""
    rng, ops = _rng(seed, 1), []
    for layer in range(depth):
        for q, (t, p, l) in enumerate(rng.uniform(0, 2 * math.pi, (n, 3))):
            c, s = math.cos(t / 2), math.sin(t / 2)
            e = [complex(math.cos(x), math.sin(x)) for x in (l, p, p + l)]
            ops.append(("u", q, ((complex(c), -e[0] * s), (e[1] * s, e[2] * c))))
        ops += [("cx", q, q + 1) for q in range(layer % 2, n - 1, 2)]
    return ops


def _circuit(n, ops):
    c = QuantumCircuit(n)
    for op in ops:
        if op[0] == "u":
            c.U(op[1], SingleQubitUnitary.Create(op[2]))
        else:
            c.CNot(op[1], op[2])
    return c


def _chain(case, seed):
    """(coefficient, {qubit: label}) terms of an open XXZ or transverse-field Ising chain."""
    rng, n, terms = _rng(seed, 2), case["qubits"], []
    if case.get("model") == "tfim":
        terms += [(-j, {i: "Z", i + 1: "Z"}) for i, j in enumerate(rng.uniform(0.5, 1.5, n - 1))]
        terms += [(-h, {i: "X"}) for i, h in enumerate(rng.uniform(0.5, 1.5, n))]
        return terms
    for i, (j, d) in enumerate(zip(rng.uniform(0.5, 1.5, n - 1), rng.uniform(0, 2, n - 1))):
        terms += [(j, {i: p, i + 1: p}) for p in "XY"] + [(j * d, {i: "Z", i + 1: "Z"})]
    return terms + [(h, {i: "Z"}) for i, h in enumerate(rng.normal(0, 0.3, n))]


def _hamiltonian(n, terms):
    def label(at):
        return "".join(at.get(q, "I") for q in reversed(range(n)))
    return PauliHamiltonian(n, [PauliTerm(float(c), PauliString(label(at))) for c, at in terms])


def _amplitudes(n, precision, seed):
    """A normalised random state on the GPU: what a deep random circuit leaves."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    kind = torch.complex128 if precision == FP64 else torch.complex64
    v = torch.randn(1 << n, dtype=kind, device="cuda", generator=g)
    # the norm in pieces: linalg.norm of the whole would hold a second copy
    total = sum(torch.linalg.vector_norm(x).item() ** 2 for x in v.split(1 << 24))
    return v.div_(math.sqrt(total))


class _Buffer:
    """A state's device memory for torch.as_tensor; a tensor made from it keeps the state alive."""

    def __init__(self, state):
        self.state = state
        kind = "<c16" if state.precision == FP64 else "<c8"
        self.__cuda_array_interface__ = {"shape": (state.Length,), "typestr": kind, "version": 3, "strides": None,
                                         "data": (state.device_pointer(), False)}


def _view(state):
    """The state's amplitudes as a torch tensor, without a copy."""
    return torch.as_tensor(_Buffer(state), device="cuda")


def _resident(case, seed):
    state = DeviceState(context(), case["qubits"], case["precision"])
    _view(state).copy_(_amplitudes(case["qubits"], case["precision"], seed))
    torch.cuda.synchronize()
    return state


def _monitored_steps(case, seed):
    """Per round: the layer's operations, a damped qubit, a marginal's qubits, a measured pair, draws."""
    rng, n, steps = _rng(seed, 3), case["qubits"], []
    for k in range(case["rounds"]):
        pick = [int(q) for q in rng.permutation(n)]
        steps.append({"ops": _brick(n, 1, seed * 7 + k), "damped": pick[0], "gamma": 0.05, "marginal": pick[1:3],
                      "measured": pick[3:5], "draws": [float(x) for x in rng.uniform(0, 1, 2)]})
    return steps


def _ansatz(n, layers=4):
    c, p = ParameterizedCircuit(n, 2 * n * layers), 0
    for _ in range(layers):
        for rotation in (c.Ry, c.Rz):
            for q in range(n):
                rotation(q, p)
                p += 1
        ladder = QuantumCircuit(n)
        for q in range(n - 1):
            ladder.CZ(q, q + 1)
        c.Append(ladder)
    return c


def _noisy(case, seed):
    """("ry", q, angle), ("cz", a, b), ("dep", q, p) and ("damp", q, gamma) in program order."""
    rng, n, steps = _rng(seed, 4), case["qubits"], []
    for _ in range(case["depth"]):
        for q, a in enumerate(rng.uniform(0, 2 * math.pi, n)):
            steps += [("ry", q, float(a)), ("dep", q, 1e-3)]
        for q in range(n - 1):
            steps += [("cz", q, q + 1), ("dep", q, 1e-2), ("dep", q + 1, 1e-2)]
        steps += [("damp", q, 1e-3) for q in range(n)]
    draws = rng.uniform(0, 1, (case["trajectories"], sum(s[0] in ("dep", "damp") for s in steps)))
    return steps, draws


def _z_observables(n):
    return [{i: "Z"} for i in range(n)] + [{i: "Z", i + 1: "Z"} for i in range(n - 1)]


class _Draws:
    """The program's random source (NextDouble) for one pass."""

    def __init__(self, values):
        self.values, self.at = values, 0

    def NextDouble(self):
        self.at += 1
        return self.values[self.at - 1]


def prepare(case, seed):
    kind, n = case["kind"], case["qubits"]
    s = {"case": case, "kind": kind}
    if kind == "port":
        s["backend"] = B200StateVectorBackend(context=context())
        s["circuit"] = _circuit(n, _brick(n, case["depth"], seed))
        if case["pinned"]:
            s["host"] = context().host_array(1 << n)
            s["amplitudes"] = s["host"].array
        else:
            s["amplitudes"] = np.empty(1 << n, dtype=np.complex128)
        s["amplitudes"][:] = 0
        s["amplitudes"][0] = 1
    elif kind == "evolve":
        s["circuit"] = (QuantumFourierTransform.CreateCircuit(n) if case["circuit"] == "qft"
                        else _circuit(n, _brick(n, case["depth"], seed)))
        s["state"] = _resident(case, seed)
    elif kind == "plan":
        s["plan"] = Plan(context(), _circuit(n, _brick(n, case["depth"], seed)), case["precision"], case["width"])
        s["state"] = DeviceState(context(), n, case["precision"])
    elif kind == "energy":
        s["state"] = _resident(case, seed)
        s["hamiltonian"] = _hamiltonian(n, _chain(case, seed))
    elif kind == "sample":
        s["state"] = _resident(case, seed)
        s["draws"] = _rng(seed, 5).uniform(0, 1, case["shots"])
    elif kind == "monitored":
        s["state"] = _resident(case, seed)
        s["steps"] = _monitored_steps(case, seed)
        for step in s["steps"]:
            step["plan"] = Plan(context(), _circuit(n, step["ops"]), case["precision"])
    elif kind == "vqe":
        s["evaluator"] = B200VariationalEnergyEvaluator(context(), case["precision"])
        s["ansatz"] = _ansatz(n)
        s["hamiltonian"] = _hamiltonian(n, _chain(case, seed))
        s["parameters"] = _rng(seed, 6).uniform(-math.pi, math.pi, (case["vectors"], s["ansatz"].ParameterCount))
    else:
        s["simulator"] = B200NoisySimulator(context(), precision=case["precision"])
        steps, s["draws"] = _noisy(case, seed)
        s["circuit"] = noisy = NoisyCircuit(n)
        for name, a, b in steps:
            if name == "ry":
                noisy.Append(QuantumCircuit(n).Ry(a, b))
            elif name == "cz":
                noisy.Append(QuantumCircuit(n).CZ(a, b))
            else:
                noisy.ApplyNoise(NoiseChannel.Depolarizing(b) if name == "dep" else NoiseChannel.AmplitudeDamping(b), a)
        s["observables"] = [t.Observable for t in _hamiltonian(n, [(1.0, at) for at in _z_observables(n)]).Terms]
    return s


# ------------------------------------------------------------------------------------ one pass

def _numbers(values, precision):
    """A complex64 state's observables carry single precision, and its optimiser keeps them so."""
    return np.asarray(values, dtype=np.float64 if precision == FP64 else np.float32)


def run(s):
    kind, case = s["kind"], s["case"]
    if kind == "port":
        s["backend"].Execute(s["circuit"], s["amplitudes"])
        return s["amplitudes"]
    if kind == "evolve":
        s["state"].Evolve(s["circuit"])
        return _view(s["state"])
    if kind == "plan":
        s["plan"].execute(s["state"])
        return _view(s["state"])
    if kind == "energy":
        return s["state"].ExpectationEnergy(s["hamiltonian"])
    if kind == "sample":
        return s["state"].Sample(s["draws"])[0]
    if kind == "monitored":
        state, read = s["state"], []
        for step in s["steps"]:
            step["plan"].execute(state)
            draws = _Draws(step["draws"])
            state.ApplyNoise(NoiseChannel.AmplitudeDamping(step["gamma"]), step["damped"], draws)
            marginal = state.MarginalProbability(step["marginal"], 1)
            read.append((state.Measure(step["measured"], draws.NextDouble())[0], _numbers(marginal, case["precision"])))
        return {"read": read, "state": _view(state)}
    if kind == "vqe":
        r = s["evaluator"].EvaluateBatch(s["ansatz"], s["hamiltonian"], s["parameters"])
        return {"energies": _numbers(r.Energies, case["precision"]), "gradients": _numbers(r.Gradients, case["precision"])}
    r = s["simulator"].RunBatch(s["circuit"], s["draws"], s["observables"], branches=True)
    return {"values": _numbers(r.values, case["precision"]), "branches": r.branches, "consumed": r.consumed}


# ------------------------------------------------------------------------------------ the least work

def work(case):
    """Each input read once and each output written once; 8 flops an amplitude for a general 2x2 gate, 4 for
    a real one, 2 for a phase or a mass."""
    kind, n = case["kind"], case["qubits"]
    amps = 1 << n
    size = amps * (8 if case.get("precision", FP64) == FP32 else 16)
    if kind in ("port", "evolve", "plan"):
        gates = 2 * n if case.get("circuit") == "qft" else n * case["depth"]
        return {"bytes": 2 * size, "flops": 8 * gates * amps}
    if kind in ("energy", "sample"):
        return {"bytes": size, "flops": (8 * (4 * n - 3) if kind == "energy" else 2) * amps}
    if kind == "monitored":
        # a layer (read, write), masses (read) and damping (read, write), a marginal (read), a draw (read)
        # and the projection of a quarter of the state (read a quarter, write all)
        return {"bytes": int(case["rounds"] * 8.25 * size), "flops": case["rounds"] * (8 * n + 12) * amps}
    if kind == "vqe":
        circuits = case["vectors"] * (1 + 2 * 8 * n)
        return {"bytes": circuits * 2 * size, "flops": circuits * (4 * n * 6 + 8 * (4 * n - 3)) * amps}
    return {"bytes": case["trajectories"] * 2 * size, "flops": case["trajectories"] * case["depth"] * 8 * n * amps}


# ------------------------------------------------------------------------------------ in 64 bits

def _u(psi, q, m):
    """Applies the 2x2 matrix m to qubit q in place."""
    v = psi.view(-1, 2, 1 << q)
    x = v[:, 0].clone()
    v[:, 0].mul_(m[0][0]).add_(v[:, 1], alpha=m[0][1])
    v[:, 1].mul_(m[1][1]).add_(x, alpha=m[1][0])


def _pair(psi, a, b):
    """psi by the bits of qubits a < b: [.., bit of b, .., bit of a, ..]."""
    return psi.view(-1, 2, 1 << (b - a - 1), 2, 1 << a)


def _apply(psi, ops):
    for op in ops:
        if op[0] == "u":
            _u(psi, op[1], op[2])
        else:  # CNOT of neighbours, control below target
            v = _pair(psi, op[1], op[2])
            x = v[:, 0, :, 1].clone()
            v[:, 0, :, 1] = v[:, 1, :, 1]
            v[:, 1, :, 1] = x
    return psi


def _zero(n):
    psi = torch.zeros(1 << n, dtype=torch.complex128, device="cuda")
    psi[0] = 1
    return psi


def _on(probabilities, n, at):
    """sum of probabilities times the Z signs of the qubits in `at`."""
    v = probabilities
    for q in sorted(at, reverse=True):
        v = v.view(-1, 2, 1 << q)
        v = (v[:, 0] - v[:, 1]).reshape(-1)
    return v.sum()


def _expect(psi, n, at):
    """<psi|P|psi> of a Pauli string {qubit: label} on at most two qubits."""
    if set(at.values()) == {"Z"}:
        return _on(psi.real.square() + psi.imag.square(), n, at)
    if len(at) == 1:
        v = psi.view(-1, 2, 1 << next(iter(at)))
        return 2 * (v[:, 0].conj() * v[:, 1]).real.sum()
    a, b = sorted(at)
    v = _pair(psi, a, b)
    sign = -1 if at[a] == "Y" else 1
    return 2 * ((v[:, 1, :, 1].conj() * v[:, 0, :, 0]).real.sum() * sign
                + (v[:, 1, :, 0].conj() * v[:, 0, :, 1]).real.sum())


def _exact_vqe(case, seed):
    n, rng = case["qubits"], _rng(seed, 6)
    terms = _chain(case, seed)
    energies, gradients = [], []
    bits = torch.arange(1 << n, device="cuda")
    ladder = torch.zeros(1 << n, dtype=torch.int64, device="cuda")
    for q in range(n - 1):
        ladder += (bits >> q) & (bits >> (q + 1)) & 1
    sign = (1 - 2 * (ladder & 1)).to(torch.float64)
    for vector in rng.uniform(-math.pi, math.pi, (case["vectors"], 8 * n)):
        t = torch.tensor(vector, dtype=torch.float64, device="cuda", requires_grad=True)
        psi = _zero(n)
        for layer in range(4):
            for q in range(n):
                a, z = t[2 * n * layer + q] / 2, t[2 * n * layer + n + q] / 2
                v = psi.view(-1, 2, 1 << q)
                c, s, phase = torch.cos(a), torch.sin(a), torch.polar(torch.ones_like(z), z)
                psi = torch.stack(((c * v[:, 0] - s * v[:, 1]) * phase.conj(), (s * v[:, 0] + c * v[:, 1]) * phase),
                                  dim=1).reshape(-1)
            psi = psi * sign
        energy = sum(c * _expect(psi, n, at) for c, at in terms)
        energy.backward()
        energies.append(energy.item())
        gradients.append(t.grad.cpu().numpy())
    return {"energies": np.array(energies), "gradients": np.array(gradients)}


def _damp(psi, q, gamma, u):
    """Amplitude damping with the draw u; whether it was needed to choose the branch."""
    v = psi.view(-1, 2, 1 << q)
    zero, one = ((v[:, k].real.square() + v[:, k].imag.square()).sum().item() for k in (0, 1))
    jump, stay = gamma * one, zero + (1 - gamma) * one
    if jump > 0 and (stay == 0 or u < jump / (jump + stay)):
        v[:, 0] = v[:, 1] * math.sqrt(gamma / jump)
        v[:, 1] = 0
    else:
        v[:, 0].mul_(1 / math.sqrt(stay))
        v[:, 1].mul_(math.sqrt((1 - gamma) / stay))
    return jump > 0 and stay > 0


def _exact_monitored(case, seed):
    psi, read = _amplitudes(case["qubits"], case["precision"], seed).to(torch.complex128), []
    for step in _monitored_steps(case, seed):
        draws = _Draws(step["draws"])
        _apply(psi, step["ops"])
        if _damp(psi, step["damped"], step["gamma"], step["draws"][0]):
            draws.NextDouble()
        p = psi.real.square() + psi.imag.square()
        bits = torch.arange(p.numel(), device="cuda")
        (a, b), total = step["marginal"], p.sum()
        marginal = (p[((bits >> a) & 1 == 1) & ((bits >> b) & 1 == 0)].sum() / total).item()
        cdf = torch.cumsum(p, 0)
        basis = int(torch.searchsorted(cdf, draws.NextDouble() * cdf[-1:], right=True).item())
        mask = sum(1 << q for q in step["measured"])
        psi[(bits & mask) != (basis & mask)] = 0
        psi /= torch.linalg.vector_norm(psi)
        read.append((None, np.asarray(marginal)))
    return {"read": read, "state": psi}


def _exact_trajectories(case, seed):
    n = case["qubits"]
    steps, draws = _noisy(case, seed)
    values = []
    for row in draws:
        psi, at = _zero(n), 0
        for name, a, b in steps:
            if name == "ry":
                c, s = math.cos(b / 2), math.sin(b / 2)
                _u(psi, a, ((c, -s), (s, c)))
            elif name == "cz":
                _pair(psi, a, b)[:, 1, :, 1].neg_()
            elif name == "dep":
                u, at = row[at], at + 1
                if u < b / 4:
                    _u(psi, a, ((0, 1), (1, 0)))
                elif u < b / 2:
                    _u(psi, a, ((0, -1j), (1j, 0)))
                elif u < 3 * b / 4:
                    psi.view(-1, 2, 1 << a)[:, 1].neg_()
            elif _damp(psi, a, b, row[at]):
                at += 1
        p = psi.real.square() + psi.imag.square()
        p /= p.sum()
        values.append([_on(p, n, o).item() for o in _z_observables(n)])
    return {"values": np.array(values), "branches": None, "consumed": None}


def exact(case, seed):
    kind, n = case["kind"], case["qubits"]
    if kind == "port":
        return _apply(_zero(n), _brick(n, case["depth"], seed)).cpu().numpy()
    if kind in ("evolve", "plan"):
        if n > 27 or case["depth"] * n * (1 << n) > 1.2e11:
            return None
        if kind == "plan":
            return _apply(_zero(n), _brick(n, case["depth"], seed))
        psi = _amplitudes(n, case["precision"], seed).to(torch.complex128)
        if case["circuit"] == "qft":
            return torch.fft.ifft(psi, norm="ortho")
        return _apply(psi, _brick(n, case["depth"], seed))
    if kind == "energy":
        psi = _amplitudes(n, case["precision"], seed).to(torch.complex128)
        total = (psi.real.square() + psi.imag.square()).sum()
        return float(sum(c * _expect(psi, n, at) for c, at in _chain(case, seed)) / total)
    if kind == "monitored" and n <= 27:
        return _exact_monitored(case, seed)
    if kind == "vqe" and n <= 20:
        return _exact_vqe(case, seed)
    if kind == "trajectories" and case["trajectories"] * case["depth"] * n * (2e-4 + (1 << n) * 2e-10) < 18:
        return _exact_trajectories(case, seed)
    return None
