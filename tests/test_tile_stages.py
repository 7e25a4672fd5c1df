"""Batched Pauli sums on compiled tiles against the oracle: flips on every run of tile bits, flips that
share a stage, flips too wide for one, none, and zero to many diagonal terms, from the smallest tile to
sizes with qubits outside it."""
from __future__ import annotations

import math

import numpy as np
import pytest

import ref_variational as ref
from quantummatter_b200.backend import FP32, FP64, jit_info
from quantummatter_b200.observables import PauliHamiltonian, PauliString, PauliTerm
from quantummatter_b200.variational import B200VariationalEnergyEvaluator
from quantummatter_b200.workloads import hardware_efficient_ansatz, uniform_parameters

pytestmark = pytest.mark.gpu


def hamiltonian(n: int, diagonal: int, flips, seed: int) -> PauliHamiltonian:
    """Terms with the given numbers of flipped qubits, neighbouring ones and random ones, and Z signs
    anywhere; the coefficients differ, so that no two terms can be exchanged."""
    rng, terms = np.random.default_rng(seed), []

    def add(at):
        label = "".join(at.get(q, "I") for q in reversed(range(n)))
        terms.append(PauliTerm(float(rng.uniform(0.5, 1.5)), PauliString(label)))

    for count in flips:
        sets = [[int(q) for q in rng.choice(n, size=count, replace=False)] for _ in range(4)]
        sets += [list(range(q, q + count)) for q in range(n - count + 1)]
        for qubits in sets:
            for _ in range(2):
                at = {q: str(rng.choice(list("XY"))) for q in qubits}
                at.update({q: "Z" for q in range(n) if q not in at and rng.random() < 0.3})
                add(at)
    for _ in range(diagonal):
        add({q: "Z" for q in range(n) if rng.random() < 0.4})
    return PauliHamiltonian(n, terms)


@pytest.mark.parametrize("precision,tol", [(FP64, 5e-12), (FP32, 1e-6)], ids=["fp64", "fp32"])
@pytest.mark.parametrize("diagonal,flips", [(0, (1,)), (1, (2, 3)), (2, ()), (3, (4,)), (40, (1, 2, 5, 8)), (5, ())])
@pytest.mark.parametrize("n", [9, 10, 11, 12, 14])
def test_staged_tiles_match_the_oracle(gpu_context, n, diagonal, flips, precision, tol):
    c = hardware_efficient_ansatz(n, 2)
    h = hamiltonian(n, diagonal, flips, 100 * n + diagonal)
    params = uniform_parameters(c.ParameterCount, 2, -math.pi, math.pi, seed=n)
    before = jit_info()
    got = B200VariationalEnergyEvaluator(gpu_context, precision).EvaluateBatch(c, h, params, withGradient=False)
    assert jit_info()["failed"] == before["failed"]
    scale = max(1.0, sum(abs(t.Coefficient) for t in h.Terms))
    for v in range(2):
        assert abs(got.Energies[v] - ref.energy(c, h, params[v])) <= tol * scale
