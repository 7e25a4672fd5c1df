"""Born-rule draws through the two-level mass table (512-amplitude fine chunks, coarse chunks of 4096
and more) against the oracle, at the sizes where a level appears and on states with runs of zeros."""
from __future__ import annotations

import numpy as np
import pytest

import oracle as orc
from circuits import random_state
from quantummatter_b200.backend import FP32, FP64, DeviceState

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
