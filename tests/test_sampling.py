"""Born-rule draws through the two-level mass table (512-amplitude fine chunks, coarse chunks of 4096
and more) against the oracle, at the sizes where a level appears and on states with runs of zeros."""
from __future__ import annotations

import numpy as np
import pytest

import oracle as orc
from circuits import random_state
from quantummatter_b200.backend import FP32, FP64, DeviceState
from quantummatter_b200.errors import MassError

pytestmark = pytest.mark.gpu


def sparse(psi: np.ndarray, seed: int) -> np.ndarray:
    """Runs of zeros over whole chunks, at both ends and between single amplitudes."""
    rng = np.random.default_rng(seed)
    out = psi.copy()
    for _ in range(6):
        a, b = sorted(int(x) for x in rng.integers(0, psi.size, 2))
        out[a:b:int(rng.integers(1, 4))] = 0
    out[:psi.size // 5] = 0
    out[-(psi.size // 7):] = 0
    out[psi.size // 2] = 0.25  # never empty
    return out


@pytest.mark.parametrize("precision", [FP64, FP32], ids=["fp64", "fp32"])
@pytest.mark.parametrize("n", [1, 4, 8, 9, 10, 12, 13, 16, 21])
def test_draws_match_the_oracle(gpu_context, n, precision):
    rng = np.random.default_rng(n)
    draws = np.concatenate([[0.0, 0.5, 1 - 2.0 ** -53], rng.random(301)])
    dense = random_state(n, 5 + n)
    for psi in (dense, sparse(dense, n)):
        if precision == FP32:
            psi = psi.astype(np.complex64).astype(np.complex128)
        with DeviceState(gpu_context, n, precision) as st:
            st.Upload(psi)
            got, ambiguous = st.Sample(draws)
            one, _ = st.Sample(draws[7:8])
        want = orc.sample(psi, draws)
        # the largest draw below 1 lies within rounding of the total, so only its flag is fixed
        assert np.array_equal(np.delete(got, 2), np.delete(want, 2))
        assert psi[got[2]] != 0
        assert ambiguous <= 2 and one[0] == got[7]


def test_draws_of_a_basis_state(gpu_context):
    for n, k in ((13, 0), (13, 511), (13, 512), (13, 4095), (13, 4096), (13, 8191)):
        psi = np.zeros(1 << n, dtype=np.complex128)
        psi[k] = 1.0
        with DeviceState(gpu_context, n, FP64) as st:
            st.Upload(psi)
            got, _ = st.Sample([0.0, 0.25, 1 - 2.0 ** -53])
        assert list(got) == [k, k, k]


@pytest.mark.parametrize("precision,tol", [(FP64, 1e-12), (FP32, 2e-6)], ids=["fp64", "fp32"])
@pytest.mark.parametrize("n", [1, 2, 5, 11, 13])
def test_projection_onto_any_selection(gpu_context, n, precision, tol):
    """The branch's amplitudes are enumerated by their free bits: single qubits from lowest to highest,
    neighbours, scattered selections and the whole register."""
    psi = random_state(n, 40 + n) * 1.7
    rng = np.random.default_rng(n)
    selections = [[0], [n - 1], list(range(n)), sorted(rng.choice(n, size=(n + 1) // 2, replace=False).tolist())]
    for qubits in selections:
        u = float(rng.random())
        with DeviceState(gpu_context, n, precision) as st:
            st.Upload(psi)
            m0, m1 = st.QubitMasses(qubits[-1])
            outcome, _ = st.Measure(qubits, u)
            got = st.Download()
        bit = (np.arange(1 << n) >> qubits[-1]) & 1
        p = np.abs(psi) ** 2
        assert abs(m0 - p[bit == 0].sum()) <= tol * p.sum() and abs(m1 - p[bit == 1].sum()) <= tol * p.sum()
        want_state, want = orc.measure(psi, qubits, u)
        assert outcome == want
        assert np.max(np.abs(got - want_state)) <= tol


def test_a_state_without_mass_is_left_alone(gpu_context):
    for bad in (0.0, np.inf, np.nan):
        psi = np.full(1 << 10, bad, dtype=np.complex128)
        with DeviceState(gpu_context, 10, FP64) as st:
            st.Upload(psi)
            for call in (lambda: st.Sample([0.5]), lambda: st.Measure([3], 0.5), lambda: st.MeasureAll(0.5),
                         lambda: st.MarginalProbability([2], 1)):
                with pytest.raises(MassError):
                    call()
            assert np.array_equal(st.Download(), psi, equal_nan=True)
