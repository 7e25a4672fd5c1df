"""Pauli sums of one resident state whose blocks work through several tiles: more tiles of 12 qubits than
blocks, so that running sums, outer signs and tile starts carry from one tile to the next."""
from __future__ import annotations

import ctypes as C
from fractions import Fraction

import numpy as np
import pytest

import oracle as orc
from circuits import random_state
from quantummatter_b200 import _lib
from quantummatter_b200.backend import FP32, FP64, DeviceState
from quantummatter_b200.observables import PauliString

pytestmark = pytest.mark.gpu


def label(n: int, at: dict[int, str]) -> str:
    return "".join(at.get(q, "I") for q in reversed(range(n)))


@pytest.mark.parametrize("precision", [FP64, FP32], ids=["fp64", "fp32"])
def test_small_contributions_of_many_tiles_are_kept(gpu_context, precision):
    """Sums that start at 1 in the first tile and get e = 2^-54 from each other one, which a plain addition
    drops: the pair 0, 3 (flips) and the amplitude 16 (17 balances its 1).  A sum may be plain over twelve
    tiles of a block, which drops 11 e: 33 e of the mass of 4 (whose last rounding takes 8 e) and 22 e of a
    flip's raw sum, with the mass 10 e of its value (whose rounding takes 1).  Plain over the 55 tiles of a
    block, the mass loses 165 e and a value 14 to 41 e."""
    n, tiles, e = 26, 1 << 14, Fraction(1, 1 << 54)
    psi = np.zeros(1 << n, dtype=np.complex64 if precision == FP32 else np.complex128)
    psi[0::4096] = psi[3::4096] = psi[16::4096] = 2.0 ** -27
    psi[0], psi[3], psi[16], psi[17] = 1.0, -1.0, 1.0, 1.0
    tail = (tiles - 1) * e
    mass = 4 + 3 * tail
    want = {"X0 X1": -2 + 2 * tail, "Y0 Y1": 2 - 2 * tail, "X0 X1 Z5": -2 + 2 * tail, "Z0": tail, "Z0 Z7": tail}
    with DeviceState(gpu_context, n, precision) as st:
        st.Upload(psi)
        got, total = st.ExpectationValues([PauliString(label(n, {int(f[1:]): f[0] for f in t.split()})) for t in want])
    assert abs(Fraction(total) - mass) <= 42 * e
    for name, value in zip(want, got):
        assert abs(Fraction(value) - want[name] / mass) <= 12 * e, name


def rounded(psi: np.ndarray, precision: int) -> np.ndarray:
    return psi.astype(np.complex64).astype(np.complex128) if precision == FP32 else psi


@pytest.mark.parametrize("precision", [FP64, FP32], ids=["fp64", "fp32"])
@pytest.mark.parametrize("n", [21, 23])
def test_terms_on_states_of_many_tiles_match_the_oracle(gpu_context, n, precision):
    """Flips inside the first tile, across its edge and outside it, with signs on tile and outer qubits, and
    diagonal terms of both kinds: two to seven tiles per block."""
    psi = rounded(random_state(n, n), precision)
    terms = [{0: "X", 1: "X"}, {5: "Y", 11: "Y"}, {11: "X", 12: "Y"}, {12: "Y", 13: "Y"}, {n - 2: "X", n - 1: "X"},
             {3: "X", n - 1: "Z"}, {n - 1: "Y", 0: "Z", 14: "Z"}, {0: "X", n - 1: "X", 7: "Z"}, {2: "Z"}, {n - 1: "Z"},
             {4: "Z", 13: "Z"}, {q: "Z" for q in range(n)}]
    strings = [PauliString(label(n, t)) for t in terms]
    with DeviceState(gpu_context, n, precision) as st:
        st.Upload(psi)
        got, mass = st.ExpectationValues(strings)
    assert abs(mass - float(np.sum(np.abs(psi) ** 2))) <= 1e-12
    for s, value in zip(strings, got):
        assert abs(value - orc.expectation(psi, s)) <= 1e-12, s


@pytest.mark.parametrize("precision", [FP64, FP32], ids=["fp64", "fp32"])
@pytest.mark.parametrize("n,count,flips", [(13, 300, 0), (14, 40, 0), (18, 300, 0), (18, 80, 40), (20, 600, 0), (20, 90, 30),
                                           (22, 10, 0), (23, 10, 0), (23, 40, 0), (23, 40, 3)])
def test_long_lists_of_diagonal_terms(gpu_context, n, count, flips, precision):
    """Z strings with any phase (2: the negative; 1 and 3, possible through the C ABI only: zero), alone and
    beside flips, on both sides of the lines where the tiled kernel takes them."""
    rng = np.random.default_rng(n + count)
    psi = rounded(random_state(n, n + count), precision)
    p, index = np.abs(psi) ** 2, np.arange(1 << n, dtype=np.uint32)
    recs = (_lib.PauliTermC * (count + flips))()
    want = []
    for i, r in enumerate(recs):
        r.coefficient = 1.0
        if i % 3 == 0 and i // 3 < flips:  # X on neighbours, everywhere
            r.flip_mask = 3 << (i % (n - 1))
            want.append(float(np.vdot(psi[index ^ r.flip_mask], psi).real))
            continue
        r.sign_mask, r.y_count = int(rng.integers(0, 1 << n)), int(rng.choice([0, 0, 0, 1, 2, 3]))
        odd = np.bitwise_count(index & np.uint32(r.sign_mask)) & 1
        value = float(np.sum(np.where(odd, -p, p)))
        want.append([value, 0.0, -value, 0.0][r.y_count])
    out, mass = (C.c_double * len(recs))(), C.c_double()
    with DeviceState(gpu_context, n, precision) as st:
        st.Upload(psi)
        _lib.check(_lib.load().qm_expectation_pauli(st.handle, recs, len(recs), out, C.byref(mass)))
    assert abs(mass.value - float(np.sum(p))) <= 1e-12
    assert np.max(np.abs(np.array(list(out)) * mass.value - np.array(want))) <= 1e-12
