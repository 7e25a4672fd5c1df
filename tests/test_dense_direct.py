"""Dense fused gates through the register kernel (up to 4 qubits) and the FP64 tensor kernel (5 and 6
qubits) against the oracle: the smallest states of each, one tile, half-size tiles and full ones, with
the gate at the bottom (adjacent amplitudes move together), at the top, straddling and scattered."""
from __future__ import annotations

import numpy as np
import pytest

import oracle as orc
from circuits import random_state
from quantummatter_b200.backend import FP32, FP64, DeviceState
from quantummatter_b200.circuit import QuantumCircuit

pytestmark = pytest.mark.gpu


def placements(n: int, m: int):
    rng = np.random.default_rng(100 * n + m)
    yield list(range(m))
    yield list(range(n - m, n))
    if n > m:
        yield list(range(1, m + 1))
        yield [0] + list(range(n - m + 1, n))
        yield sorted(rng.choice(n, size=m, replace=False).tolist())
    if n > m + 1 and m >= 2:
        yield [0, 1] + list(range(n - m + 2, n))


@pytest.mark.parametrize("precision,tol", [(FP64, 1e-12), (FP32, 2e-6)], ids=["fp64", "fp32"])
@pytest.mark.parametrize("n", [4, 7, 9, 10, 11, 12, 13, 16])
@pytest.mark.parametrize("m", [2, 3, 4, 5, 6])
def test_dense_gates_match_the_oracle(gpu_context, m, n, precision, tol):
    if m > n:
        pytest.skip("the gate is wider than the register")
    rng = np.random.default_rng(n)
    for qubits in placements(n, m):
        c = QuantumCircuit(n)
        for _ in range(2):
            for q in qubits:
                c.Ry(q, float(rng.uniform(0, 6.28))).Rz(q, float(rng.uniform(0, 6.28)))
            for a, b in zip(qubits, qubits[1:]):
                c.CNot(a, b)
        psi = random_state(n, n + m)
        want = orc.execute(c, psi)
        with DeviceState(gpu_context, n, precision) as st:
            st.Upload(psi)
            st.Evolve(c, fusion_width=m)
            assert np.max(np.abs(st.Download() - want)) <= tol, qubits


@pytest.mark.parametrize("qubits", [list(range(6)), list(range(17, 23)), [0, 4, 9, 13, 18, 22], [0, 1, 2, 20, 21, 22],
                                    [7, 8, 9, 10, 11, 12]], ids=lambda q: "-".join(map(str, q)))
def test_full_tiles_match_a_launch_per_gate(gpu_context, qubits):
    """Six qubits of 23, complex128: tiles of 4096 amplitudes, fourteen per block in a ring of three.
    Amplitudes of 3.5e-4; 1e-17 is some hundred roundings of one."""
    n, rng = 23, np.random.default_rng(qubits[-1])
    c = QuantumCircuit(n)
    for _ in range(2):
        for q in qubits:
            c.Ry(q, float(rng.uniform(0, 6.28))).Rz(q, float(rng.uniform(0, 6.28)))
        for a, b in zip(qubits, qubits[1:]):
            c.CNot(a, b)
    psi, got = random_state(n, qubits[0]), {}
    for width in (6, 1):
        with DeviceState(gpu_context, n, FP64) as st:
            st.Upload(psi)
            st.Evolve(c, fusion_width=width)
            got[width] = st.Download()
    assert np.max(np.abs(got[6] - got[1])) <= 1e-17
