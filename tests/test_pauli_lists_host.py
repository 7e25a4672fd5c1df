"""Plans of long Pauli lists on one state (no GPU): how often the state is read."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

from quantummatter_b200 import _lib, build

ROOT = Path(__file__).resolve().parents[1]
GXX = shutil.which("g++")


@pytest.fixture(scope="module")
def plans(tmp_path_factory):
    exe = tmp_path_factory.mktemp("plans") / "pauli_plan_test"
    cuda = Path(build.nvcc()).resolve().parents[1] / "include"
    lib = Path(_lib.LIB_PATH)
    res = subprocess.run([GXX, "-std=c++17", "-O1", "-I", str(ROOT / "include"), "-I", str(cuda),
                          "-I", str(ROOT / "quantummatter_b200" / "csrc"), str(ROOT / "tests" / "pauli_plan_test.cpp"),
                          str(lib), f"-Wl,-rpath,{lib.parent}", "-Wl,--unresolved-symbols=ignore-in-shared-libs",
                          "-o", str(exe)], capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stderr[-2000:]
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert run.returncode == 0, run.stderr
    return [line.split() for line in run.stdout.splitlines()]


@pytest.mark.skipif(GXX is None, reason="g++ not found")
def test_diagonal_lists_take_few_reads(plans):
    """Lists of nothing else go to the tiled kernel (no passes here), 256 terms a read; beside flips, more
    than 32 distinct tile parts do. What stays is a pass per 22 sums and tile of the flips, 16 parts each."""
    for qubits, _, kind, count, passes, left_out, parts in plans:
        qubits, count, passes, left_out, parts = int(qubits), int(count), int(passes), int(left_out), int(parts)
        if kind == "diagonal":
            assert passes == 0, (qubits, count)
        elif qubits >= 18:
            assert parts <= 32, (qubits, count)
            assert left_out == 0 if count == 64 else left_out >= count // 2 - qubits, (qubits, count)
            assert passes <= 2 + qubits // 4 + count // 2 // 16, (qubits, count, passes)
