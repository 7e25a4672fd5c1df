"""Runs of constant phases in the interpreting pass kernel: their rounding error against one launch per
gate, and angles at the ends of a turn, moduli other than 1 and qubits on register, thread and outer bits
against a product in extended precision."""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import pytest

import oracle as orc
from circuits import random_state
from quantummatter_b200 import _lib
from quantummatter_b200.algorithms import QuantumFourierTransform
from quantummatter_b200.backend import FP32, FP64, DeviceState
from quantummatter_b200.circuit import GateKind, GateOperation, QuantumCircuit, prepare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [13, 16, 18])
def test_transform_error_is_no_larger_than_with_a_launch_per_gate(gpu_context, n):
    """complex64: a ladder's phases applied together round no more than one multiplication of the
    amplitudes per phase does."""
    psi = random_state(n, n).astype(np.complex64).astype(np.complex128)
    circuit = QuantumFourierTransform.CreateCircuit(n)
    want = orc.execute(circuit, psi)
    error = {}
    for width in (0, 1):
        with DeviceState(gpu_context, n, FP32) as st:
            st.Upload(psi)
            st.Evolve(circuit, fusion_width=width)
            error[width] = float(np.linalg.norm(st.Download() - want))
    assert error[0] <= error[1]


@pytest.mark.parametrize("precision,tol", [(FP64, 1e-15), (FP32, 7.5e-7)], ids=["fp64", "fp32"])
@pytest.mark.parametrize("n", [12, 15])
def test_phases_of_every_angle_and_place(gpu_context, n, precision, tol):
    """One multiplication per amplitude by phases of up to three qubits: half an ulp from the phase, its
    product with the amplitude and the final rounding, and up to eight further ones where a phase has
    two register bits: ten of 1e-16 (complex64: 7.5e-8) of the amplitude's modulus."""
    rng = np.random.default_rng(n)
    angles = [math.pi / 2, -math.pi / 2, math.nextafter(math.pi, 0), -math.nextafter(math.pi, 0), math.pi / 4,
              3 * math.pi / 4, 1e-9, -1e-9, 2.5, -0.7]
    c = QuantumCircuit(n)
    for a in angles + [float(x) for x in rng.uniform(-math.pi, math.pi, 14)]:
        q = [int(x) for x in rng.choice(n, size=3, replace=False)]
        if rng.random() < 0.3:
            c.AppendValidated(GateOperation(GateKind.Phase, q[0], q[1], a, q[2]))
        else:
            c.CPhase(q[0], q[1], a)
    gates, count = prepare(c)
    gates[3].d[0], gates[3].d[1] = 0.3, -0.4  # not of modulus 1: applied by itself
    psi = random_state(n, 5).astype(np.complex64).astype(np.complex128)
    factor = np.ones(1 << n, dtype=np.clongdouble)
    index = np.arange(1 << n)
    for g in gates[:count]:
        mask = g.control_mask | 1 << g.target
        factor[(index & mask) == mask] *= np.longdouble(g.d[0]) + 1j * np.longdouble(g.d[1])
    with DeviceState(gpu_context, n, precision) as st:
        st.Upload(psi)
        _lib.check(_lib.load().qm_execute(st.handle, gates, count, 0, None))
        got = st.Download()
    want = (psi * factor).astype(np.complex128)
    assert np.all(np.abs(got - want) <= tol * np.abs(psi))
