"""Whole gate lists in one block (one-shot executions of up to 11 qubits, plans below 9) against the
oracle: every gate kind, controls and swaps inside and across the 64 amplitudes of a warp, and lists
longer than one launch takes."""
from __future__ import annotations

import numpy as np
import pytest

import oracle as orc
from circuits import random_circuit, random_state
from quantummatter_b200.backend import FP32, FP64, B200StateVectorBackend, DeviceState, Plan
from quantummatter_b200.circuit import QuantumCircuit

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [(FP64, 1e-12), (FP32, 1e-5)], ids=["fp64", "fp32"])
@pytest.mark.parametrize("n", [3, 5, 6, 7, 8, 9, 11])
@pytest.mark.parametrize("gates", [1, 48, 49, 384, 385, 900])
def test_gate_lists_match_the_oracle(gpu_context, n, gates, precision, tol):
    c = random_circuit(n, gates, seed=10 * n + gates)
    psi = random_state(n, n + gates)
    want = orc.execute(c, psi)
    with DeviceState(gpu_context, n, precision) as st:
        st.Upload(psi)
        prof = st.Evolve(c, profile=True)
        assert prof.KernelLaunches <= 3 and prof.Passes == 0
        assert np.max(np.abs(st.Download() - want)) <= tol
        if n < 9:
            p = Plan(gpu_context, c, precision)
            st.Upload(psi)
            p.execute(st)
            assert np.max(np.abs(st.Download() - want)) <= tol
            st.Upload(psi)
            p.capture(st).launch()
            assert np.max(np.abs(st.Download() - want)) <= tol
            p.Dispose()


def test_one_and_two_qubits_and_no_gates(gpu_context):
    for n in (1, 2):
        c = QuantumCircuit(n).H(0).T(0).Rx(n - 1, 0.3)
        if n == 2:
            c.CNot(0, 1).Swap(0, 1).CPhase(1, 0, 0.4).I(0)
        psi = random_state(n, n)
        buf = psi.copy()
        B200StateVectorBackend(context=gpu_context).Execute(c, buf)
        assert np.max(np.abs(buf - orc.execute(c, psi))) <= 1e-14
        B200StateVectorBackend(context=gpu_context).Execute(QuantumCircuit(n), buf)
        assert np.max(np.abs(buf - orc.execute(c, psi))) <= 1e-14
