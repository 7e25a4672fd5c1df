"""Kernels whose blocks take several pieces of work on large states: masses, measurements and projections
from 21 qubits on, and complex64 plans in packed form from 25."""
from __future__ import annotations

import math

import numpy as np
import pytest

import oracle as orc
from circuits import random_state
from quantummatter_b200.backend import FP32, FP64, DeviceState, Plan
from quantummatter_b200.circuit import QuantumCircuit, u3

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [(FP64, 1e-14), (FP32, 1e-7)], ids=["fp64", "fp32"])
@pytest.mark.parametrize("n", [21, 22])
def test_masses_and_projections(gpu_context, n, precision, tol):
    """tol: of a mass (sums of 2^n products in compensated FP64; complex64 states hold their amplitudes to
    6e-8), and of an amplitude relative to the largest."""
    psi = random_state(n, n) * 1.3
    if precision == FP32:
        psi = psi.astype(np.complex64).astype(np.complex128)
    p, index = np.abs(psi) ** 2, np.arange(1 << n)
    for qubits, u in (([0], 0.3), ([n - 1], 0.8), ([1, 12, n - 2], 0.55), ([n - 1, 0, 5, 13, 18], 0.1)):
        with DeviceState(gpu_context, n, precision) as st:
            st.Upload(psi)
            m0, m1 = st.QubitMasses(qubits[-1])
            bit = (index >> qubits[-1]) & 1
            assert abs(m0 - p[bit == 0].sum()) <= 1e-13 and abs(m1 - p[bit == 1].sum()) <= 1e-13
            pattern = sum((k & 1) << q for k, q in enumerate(qubits))
            mask = sum(1 << q for q in qubits)
            marginal = st.MarginalProbability(qubits, sum((k & 1) << k for k in range(len(qubits))))
            assert abs(marginal - p[(index & mask) == pattern].sum() / p.sum()) <= 1e-13
            outcome, _ = st.Measure(qubits, u)
            got = st.Download()
        # the oracle draws; its norm is a running sum of 2^n terms, so the state is projected with numpy's
        _, want = orc.measure(psi, qubits, u)
        assert outcome == want
        branch = (index & mask) == sum(((want >> k) & 1) << q for k, q in enumerate(qubits))
        want_state = np.where(branch, psi, 0) / math.sqrt(p[branch].sum())
        assert np.max(np.abs(got - want_state)) <= tol * np.max(np.abs(want_state))


@pytest.mark.parametrize("angle", [0.2, math.pi / 2, 2.9, math.pi])
def test_packed_plans_keep_the_precision_of_complex64(gpu_context, angle):
    """25 qubits, amplitudes of 1.7e-4: 2e-9 is 200 roundings of one. The complex128 plan stands in for
    the oracle."""
    n, c = 25, QuantumCircuit(25)
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
    psi, got = random_state(n, n).astype(np.complex64).astype(np.complex128), {}
    for precision in (FP64, FP32):
        plan = Plan(gpu_context, c, precision, 0)
        with DeviceState(gpu_context, n, precision) as st:
            st.Upload(psi)
            plan.execute(st)
            got[precision] = st.Download()
        plan.Dispose()
    assert np.max(np.abs(got[FP32] - got[FP64])) <= 2e-9
