"""One-shot executions on the interpreting pass kernel: matrices with a 1 in their first column, phases
and scales moved forward past every other gate kind, and circuits long enough for the scale to be taken
up on the way (complex64 does so about every forty matrices), against the oracle."""
from __future__ import annotations

import math

import numpy as np
import pytest

import oracle as orc
from circuits import random_circuit, random_state
from quantummatter_b200.backend import FP32, FP64, DeviceState, Plan
from quantummatter_b200.circuit import QuantumCircuit, SingleQubitUnitary, u3
from quantummatter_b200.workloads import brick_circuit

pytestmark = pytest.mark.gpu


def edges(n: int) -> QuantumCircuit:
    """Matrices whose split is degenerate: diagonal, antidiagonal, real, equal columns, and one
    left pending before each kind of gate that its phase cannot pass."""
    c = QuantumCircuit(n)
    i = 1j
    for q in range(n):
        c.U(q, SingleQubitUnitary.Create(1, 0, 0, i)).U(q, SingleQubitUnitary.Create(0, -i, i, 0))
        c.U(q, u3(math.pi / 2, 0.3, -0.2)).H(q).Ry(q, math.pi).Rx(q, math.pi).Y(q).Rz(q, 0.7).Rx(q, 0.2).Z(q)
    for q in range(n - 2):
        c.U(q, u3(0.4 + q, 0.1, 0.9)).X(q).U(q, u3(1.4 + q, 0.5, -0.9)).Swap(q, q + 1)
        c.U(q, u3(2.4, 0.1 * q, 0.9)).CNot(q + 1, q).U(q + 2, u3(0.3, 1.0, 2.0)).Toffoli(q, q + 1, q + 2)
        c.Rz(q, 0.3).CRz(q, q + 1, 0.4).U(q + 1, u3(0.2, 0.1, 0.9)).CH(q + 1, q).T(q)
    return c


@pytest.mark.parametrize("precision,tol", [(FP64, 5e-12), (FP32, 2e-5)], ids=["fp64", "fp32"])
@pytest.mark.parametrize("n", [12, 15])
def test_one_shot_circuits_match_the_oracle(gpu_context, n, precision, tol):
    psi = random_state(n, n)
    for c in (edges(n), random_circuit(n, 400, seed=n), random_circuit(n, 2500, seed=n + 1), brick_circuit(n, 90)):
        want = orc.execute(c, psi)
        for width in (0, 9):
            with DeviceState(gpu_context, n, precision) as st:
                st.Upload(psi)
                st.Evolve(c, fusion_width=width)
                got = st.Download()
            assert np.max(np.abs(got - want)) <= tol, width
            assert abs(np.sum(np.abs(got) ** 2) - np.sum(np.abs(psi) ** 2)) <= 50 * tol


@pytest.mark.parametrize("precision,tol", [(FP64, 5e-13), (FP32, 2e-6)], ids=["fp64", "fp32"])
def test_large_states_without_compiled_passes(gpu_context, precision, tol):
    """26 qubits, no kernel of the circuit's structure compiled yet: the interpreter's form of the circuit
    against the compiled plan (amplitudes of about 1e-4, tolerances of 1e-2 of them and less)."""
    n, c = 26, brick_circuit(26, 5, seed=61)
    with DeviceState(gpu_context, n, precision) as st:
        st.Evolve(c)
        got = st.Download()
    p = Plan(gpu_context, c, FP64, 0)
    with DeviceState(gpu_context, n, FP64) as st:
        p.execute(st)
        want = st.Download()
    p.Dispose()
    assert np.max(np.abs(got - want)) <= tol
