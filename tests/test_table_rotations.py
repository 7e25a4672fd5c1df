"""Rotations whose angles come from a batch's table, as one scaled shear pair, and register phases
formed once per state: angles at which the form changes or an entry is zero, passes with one such
matrix and with more than take the form, and phases that meet thread factors, against the oracle."""
from __future__ import annotations

import math

import numpy as np
import pytest

import ref_variational as ref
from quantummatter_b200.backend import FP32, FP64, jit_info
from quantummatter_b200.circuit import QuantumCircuit
from quantummatter_b200.variational import B200VariationalEnergyEvaluator, ParameterizedCircuit
from quantummatter_b200.workloads import hardware_efficient_ansatz, uniform_parameters, xxz_chain

pytestmark = pytest.mark.gpu

SPECIAL = [0.0, math.pi, -math.pi, math.pi / 2, -math.pi / 2, 2 * math.pi, 3 * math.pi / 2, 1e-9, math.pi - 1e-9, 0.3]


def single(n: int) -> ParameterizedCircuit:
    """One parameterised RY, and parameterised phases on a few qubits only."""
    c = ParameterizedCircuit(n, 4)
    fixed = QuantumCircuit(n)
    for q in range(n):
        fixed.H(q).T(q)
    c.Append(fixed).Ry(n // 2, 0).Rz(0, 1).Rz(n - 1, 2).Rz(n // 2, 3)
    return c.Append(QuantumCircuit(n).CNot(0, n - 1).H(0))


@pytest.mark.parametrize("precision,tol", [(FP64, 5e-12), (FP32, 1e-6)], ids=["fp64", "fp32"])
@pytest.mark.parametrize("n,layers", [(9, 1), (9, 30), (11, 3), (13, 2), (14, 3), (10, 0)])
def test_table_rotations_match_the_oracle(gpu_context, n, layers, precision, tol):
    c = hardware_efficient_ansatz(n, layers) if layers else single(n)
    h = xxz_chain(n)
    params = uniform_parameters(c.ParameterCount, 3, -math.pi, math.pi, seed=n)
    params[1] = np.resize(SPECIAL, c.ParameterCount)
    params[2] = np.resize(SPECIAL[::-1] + [math.pi], c.ParameterCount)
    before = jit_info()
    got = B200VariationalEnergyEvaluator(gpu_context, precision).EvaluateBatch(c, h, params, withGradient=layers < 3)
    assert jit_info()["failed"] == before["failed"]
    scale = max(1.0, sum(abs(t.Coefficient) for t in h.Terms))
    for v in range(3):
        if layers < 3:
            energy, gradient = ref.energy_and_gradient(c, h, params[v])
            assert np.max(np.abs(got.Gradients[v] - gradient)) <= tol * scale
        else:
            energy = ref.energy(c, h, params[v])
        assert abs(got.Energies[v] - energy) <= tol * scale
