"""Rounding error of one-shot complex128 executions against one launch per gate, both measured against
the gates' own coefficients in extended precision."""
from __future__ import annotations

import math

import numpy as np
import pytest

from circuits import random_state
from quantummatter_b200.backend import FP64, DeviceState
from quantummatter_b200.circuit import QuantumCircuit, prepare, u3

pytestmark = pytest.mark.gpu


def layers(kind: str, n: int, rng) -> QuantumCircuit:
    c = QuantumCircuit(n)
    for _ in range(12):
        for q in range(n):
            a = [float(x) for x in rng.uniform(0, 2 * math.pi, 3)]
            if kind == "hea":
                c.Ry(q, a[0]).Rz(q, a[1])
            else:
                c.U(q, u3(*a))
        for q in range(n - 1):
            (c.CNot if kind == "cnot" else c.CZ)(q, q + 1)
    return c


def exact(circuit: QuantumCircuit, psi: np.ndarray) -> np.ndarray:
    """2x2 matrices, exchanges and controls in extended precision."""
    gates, count = prepare(circuit)
    x, index = psi.astype(np.clongdouble), np.arange(psi.size)
    for g in gates[:count]:
        on = (index >> g.target) & 1 == 0
        low = index[on & ((index & g.control_mask) == g.control_mask)]
        high = low | 1 << g.target
        if g.kernel == 3:  # exchange
            x[low], x[high] = x[high], x[low]
            continue
        m = [np.longdouble(v[0]) + 1j * np.longdouble(v[1]) for v in (g.a, g.b, g.c, g.d)]
        x[low], x[high] = m[0] * x[low] + m[1] * x[high], m[2] * x[low] + m[3] * x[high]
    return x


@pytest.mark.parametrize("kind,most", [("u3", 1.25), ("hea", 1.25), ("cnot", 1.5)])
@pytest.mark.parametrize("n", [12, 13])
def test_fused_gates_round_like_single_ones(gpu_context, n, kind, most):
    """A pass multiplies the amplitudes by the same matrices as a launch per gate, with the same number
    of roundings: a quarter above the latter's error covers the two orders of addition.  CNOTs planned as
    CZs round the matrices beside them once more (twice that), and nothing else."""
    total = {0: 0.0, 1: 0.0}
    for seed in range(3):
        circuit, psi = layers(kind, n, np.random.default_rng(seed)), random_state(n, seed)
        want = exact(circuit, psi)
        for width in total:
            with DeviceState(gpu_context, n, FP64) as st:
                st.Upload(psi)
                st.Evolve(circuit, fusion_width=width)
                total[width] += float(np.sum(np.abs(st.Download().astype(np.clongdouble) - want) ** 2))
    assert math.sqrt(total[0]) <= most * math.sqrt(total[1])
