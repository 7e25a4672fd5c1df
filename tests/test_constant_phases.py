"""Rounding of constant diagonals in compiled passes (complex64), against extended precision."""
from __future__ import annotations

import math

import numpy as np
import pytest

from circuits import random_state
from quantummatter_b200.backend import FP32, DeviceState, Plan
from quantummatter_b200.circuit import QuantumCircuit, prepare

pytestmark = pytest.mark.gpu


def clifford_t(n: int, rng) -> QuantumCircuit:
    c = QuantumCircuit(n)
    for _ in range(12):
        for q in range(n):
            [c.H, c.S, c.T, c.X, c.Y][int(rng.integers(5))](q)
        for _ in range(n // 2):
            a, b = [int(v) for v in rng.choice(n, 2, replace=False)]
            (c.CZ if rng.random() < 0.5 else c.CNot)(a, b)
    return c


def exact(circuit: QuantumCircuit, psi: np.ndarray) -> np.ndarray:
    gates, count = prepare(circuit)
    x, index = psi.astype(np.clongdouble), np.arange(psi.size)
    for g in gates[:count]:
        low = index[((index >> g.target) & 1 == 0) & ((index & g.control_mask) == g.control_mask)]
        high = low | 1 << g.target
        if g.kernel == 3:  # exchange
            x[low], x[high] = x[high], x[low]
            continue
        m = [np.longdouble(v[0]) + 1j * np.longdouble(v[1]) for v in (g.a, g.b, g.c, g.d)]
        x[low], x[high] = m[0] * x[low] + m[1] * x[high], m[2] * x[low] + m[3] * x[high]
    return x


@pytest.mark.parametrize("n,bound", [(12, 3.5e-7), (14, 4.4e-7)])
def test_constant_phases_round_no_more_than_one_by_one(gpu_context, n, bound):
    """Layers of S, T and H: multiplying the amplitudes by one member of a group after the other leaves
    3.05e-7 at 12 qubits and 3.80e-7 at 14 (bounds: 15 % above), products of the members' rounded factors
    4.0e-7 and 5.3e-7."""
    total = 0.0
    for seed in range(1, 5):
        circuit = clifford_t(n, np.random.default_rng(seed))
        psi = random_state(n, seed).astype(np.complex64).astype(np.complex128)
        plan = Plan(gpu_context, circuit, FP32)
        with DeviceState(gpu_context, n, FP32) as st:
            st.Upload(psi)
            plan.execute(st)
            got = st.Download()
        plan.Dispose()
        total += float(np.sum(np.abs(got.astype(np.clongdouble) - exact(circuit, psi)) ** 2))
    assert math.sqrt(total / 4) <= bound
