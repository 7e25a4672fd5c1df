"""Pauli sums of one resident state against the oracle: chains, all-to-all and random term lists at the
sizes where tiles, outer qubits, further passes and the wide terms' fallback appear."""
from __future__ import annotations

import numpy as np
import pytest

import oracle as orc
from circuits import random_state
from quantummatter_b200.backend import FP32, FP64, DeviceState
from quantummatter_b200.observables import PauliHamiltonian, PauliString, PauliTerm

pytestmark = pytest.mark.gpu


def label(n: int, at: dict[int, str]) -> str:
    return "".join(at.get(q, "I") for q in reversed(range(n)))


def chain(n: int) -> list[str]:
    out = [label(n, {i: p, i + 1: p}) for i in range(n - 1) for p in "XYZ"]
    return out + [label(n, {i: p}) for i in range(n) for p in "ZXY"]


def all_pairs(n: int) -> list[str]:
    return [label(n, {a: "Z", b: "Z"}) for a in range(n) for b in range(a)] + [label(n, {0: "X", n - 1: "X"})]


def scattered(n: int, seed: int) -> list[str]:
    """Terms that flip zero to n qubits, with Z signs anywhere: single-register flips, wide ones, the
    identity, repeated terms and more distinct diagonal parts than one pass holds."""
    rng = np.random.default_rng(seed)
    out = ["I" * n, "X" * n, "Y" * n, "Z" * n]
    for flips in (0, 0, 1, 2, 3, 4, 4, 5, 7):
        for _ in range(8):
            at = {int(q): str(rng.choice(list("XY"))) for q in rng.choice(n, size=min(flips, n), replace=False)}
            for q in range(n):
                if q not in at and rng.random() < 0.4:
                    at[q] = "Z"
            out.append(label(n, at))
    return out + out[5:9]


@pytest.mark.parametrize("precision", [FP64, FP32], ids=["fp64", "fp32"])
@pytest.mark.parametrize("n", [9, 10, 12, 13, 14, 17])
def test_term_lists_match_the_oracle(gpu_context, n, precision):
    psi = random_state(n, 70 + n) * 1.4
    if precision == FP32:
        psi = psi.astype(np.complex64).astype(np.complex128)
    with DeviceState(gpu_context, n, precision) as st:
        st.Upload(psi)
        for labels in (chain(n), all_pairs(n), scattered(n, n), [], ["Z" * n]):
            strings = [PauliString(s) for s in labels]
            got, mass = st.ExpectationValues(strings)
            assert abs(mass - float(np.sum(np.abs(psi) ** 2))) <= 1e-12
            for s, value in zip(strings, got):
                # sums of 2^n products in FP64: 1e-12 is far above their rounding
                assert abs(value - orc.expectation(psi, s)) <= 1e-12, s
            terms = [PauliTerm(0.1 * (i % 7) - 0.3, s) for i, s in enumerate(strings)]
            energy = st.ExpectationEnergy(PauliHamiltonian(n, terms))
            assert abs(energy - sum(t.Coefficient * v for t, v in zip(terms, got))) <= 1e-11


def test_terms_that_are_zero_for_every_state(gpu_context):
    """A phase that does not match the signs (possible through the C ABI only) cancels between the
    members of each pair; so does the imaginary part of a probability."""
    import ctypes as C
    from quantummatter_b200 import _lib
    n = 13
    psi = random_state(n, 4)
    recs = (_lib.PauliTermC * 4)()
    for r, (flip, sign, y) in zip(recs, ((1, 1, 0), (6, 2, 2), (0, 5, 1), (3, 0, 0))):
        r.flip_mask, r.sign_mask, r.y_count, r.coefficient = flip, sign, y, 1.0
    out, mass = (C.c_double * 4)(), C.c_double()
    with DeviceState(gpu_context, n, FP64) as st:
        st.Upload(psi)
        _lib.check(_lib.load().qm_expectation_pauli(st.handle, recs, 4, out, C.byref(mass)))
    assert max(abs(v) for v in list(out)[:3]) <= 1e-15
    assert abs(out[3] - orc.expectation(psi, PauliString(label(n, {0: "X", 1: "X"})))) <= 1e-12
