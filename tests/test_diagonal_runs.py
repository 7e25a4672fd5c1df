"""Runs of diagonals in the interpreting pass kernel (one-shot executions) against the oracle: phases
and controlled phases with the target and up to three controls on register, thread and outer bits."""
from __future__ import annotations

import math

import numpy as np
import pytest

import oracle as orc
from circuits import random_state
from quantummatter_b200.algorithms import QuantumFourierTransform
from quantummatter_b200.backend import FP32, FP64, DeviceState
from quantummatter_b200.circuit import GateKind, GateOperation, QuantumCircuit

pytestmark = pytest.mark.gpu


def ladder(n: int, seed: int) -> QuantumCircuit:
    rng = np.random.default_rng(seed)
    c = QuantumCircuit(n)
    for _ in range(12):
        for q in rng.choice(n, size=4, replace=False):  # moves the register layout around
            c.Ry(int(q), float(rng.uniform(0, 2 * math.pi)))
        for _ in range(int(rng.integers(2, 14))):
            q = [int(x) for x in rng.choice(n, size=3, replace=False)]
            a = float(rng.uniform(-math.pi, math.pi))
            kind = int(rng.integers(0, 6))
            if kind == 0:
                c.Rz(q[0], a)
            elif kind == 1:
                c.CPhase(q[0], q[1], a)
            elif kind == 2:
                c.CRz(q[0], q[1], a)
            elif kind == 3:
                c.T(q[0])
            elif kind == 4:
                c.CZ(q[0], q[1])
            else:  # two controls: beyond the builders, as a prepared circuit may hold it
                c.AppendValidated(GateOperation(GateKind.Rz, q[0], q[1], a, q[2]))
    return c


@pytest.mark.parametrize("precision,tol", [(FP64, 1e-12), (FP32, 5e-6)], ids=["fp64", "fp32"])
@pytest.mark.parametrize("n", [12, 13, 17])
def test_one_shot_diagonal_runs_match_the_oracle(gpu_context, n, precision, tol):
    psi = random_state(n, n)
    for c in [QuantumFourierTransform.CreateCircuit(n), QuantumFourierTransform.CreateCircuit(n, inverse=True)] + \
            [ladder(n, 7 * n + k) for k in range(4)]:
        want = orc.execute(c, psi)
        for width in (0, 9, 12):
            with DeviceState(gpu_context, n, precision) as st:
                st.Upload(psi)
                st.Evolve(c, fusion_width=width)
                assert np.max(np.abs(st.Download() - want)) <= tol, width
