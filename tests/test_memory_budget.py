"""Device memory that a context keeps after a batch call."""
from __future__ import annotations

import numpy as np
import pytest

from quantummatter_b200.backend import FP32, FP64, B200BackendOptions, B200Context, DeviceState
from quantummatter_b200.circuit import QuantumCircuit
from quantummatter_b200.observables import PauliHamiltonian, PauliString, PauliTerm
from quantummatter_b200.variational import B200VariationalEnergyEvaluator, ParameterizedCircuit

pytestmark = pytest.mark.gpu
MIB = 1 << 20


def free_bytes() -> int:
    import torch
    return torch.cuda.mem_get_info()[0]


def gradient_step(context, n: int = 18) -> None:
    ansatz = ParameterizedCircuit(n, 2 * n)
    for q in range(n):
        ansatz.Ry(q, q)
    ladder = QuantumCircuit(n)
    for q in range(n - 1):
        ladder.CZ(q, q + 1)
    ansatz.Append(ladder)
    for q in range(n):
        ansatz.Rz(q, n + q)
    h = PauliHamiltonian(n, [PauliTerm(1.0, PauliString("Z" * n)), PauliTerm(0.5, PauliString("X" + "I" * (n - 1)))])
    B200VariationalEnergyEvaluator(context, FP32).EvaluateBatch(ansatz, h, np.full((1, 2 * n), 0.3))


def test_kept_memory_leaves_the_budget_to_states(gpu_context):
    """A gradient step of 73 circuits runs 32 states of 2 MiB at a time. With 64 MiB of states after it,
    a context of 96 MiB holds no more than that: 24 MiB on top for scratch, tables and what the driver
    allots in pieces."""
    gradient_step(gpu_context)  # kernels compiled and loaded
    options = B200BackendOptions(DeviceMemoryBudgetBytes=96 * MIB, StagingMemoryBudgetBytes=64 * MIB)
    context = B200Context(options)
    try:
        before = free_bytes()
        gradient_step(context)
        with DeviceState(context, 22, FP64):
            assert before - free_bytes() <= (96 + 24) * MIB
            gradient_step(context)
            assert before - free_bytes() <= (96 + 24) * MIB
    finally:
        context.Dispose()
