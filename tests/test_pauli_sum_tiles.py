"""Pauli sums of one resident state whose blocks work through several tiles: more tiles of 12 qubits than
blocks, so that running sums, outer signs and tile starts carry from one tile to the next."""
from __future__ import annotations

from fractions import Fraction

import numpy as np
import pytest

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
