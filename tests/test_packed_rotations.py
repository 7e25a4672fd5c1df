"""complex64 passes with both parts of an amplitude in one packed multiply-add: rotations of both
forms (small and large angles), with no phase, a sign, a fixed phase and one chosen at run time, and
real matrices under controls, against the oracle."""
from __future__ import annotations

import math

import numpy as np
import pytest

import oracle as orc
from circuits import random_state
from quantummatter_b200.backend import FP32, FP64, DeviceState, Plan
from quantummatter_b200.circuit import QuantumCircuit, u3

pytestmark = pytest.mark.gpu


def circuit(n: int, angle: float) -> QuantumCircuit:
    c = QuantumCircuit(n)
    for layer in range(4):
        for q in range(n):
            c.Ry(q, angle + 0.01 * q)
            if layer == 1:
                c.Z(q)
            if layer == 2:
                c.U(q, u3(angle, 0.4 + q, -0.3))
            if layer == 3:
                c.H(q).Rx(q, angle)
        for q in range(layer % 2, n - 1, 2):
            c.CNot(q, q + 1)
        c.CRy(0, n - 1, angle).CRy(n - 1, 1, angle).CH(2, 3)
    return c


@pytest.mark.parametrize("n", [9, 12, 16, 25])
@pytest.mark.parametrize("angle", [0.2, math.pi / 2, 2.9, math.pi])
def test_packed_rotations_match_the_oracle(gpu_context, n, angle):
    c, psi = circuit(n, angle), random_state(n, n)
    if n < 25:
        want = orc.execute(c, psi)
    else:  # from 25 qubits on the packed form runs; the complex128 plan in the oracle's place
        wide = Plan(gpu_context, c, FP64, 0)
        with DeviceState(gpu_context, n, FP64) as st:
            st.Upload(psi)
            wide.execute(st)
            want = st.Download()
        wide.Dispose()
    p = Plan(gpu_context, c, FP32, 0)
    with DeviceState(gpu_context, n, FP32) as st:
        st.Upload(psi)
        p.execute(st)
        got = st.Download()
    p.Dispose()
    # about 300 gates, a few roundings of 6e-8 each on amplitudes of at most 1
    assert np.max(np.abs(got - want)) <= 2e-5
