"""Device memory of a sum over quadratic forms: the reduced terms and their
forms, no term tables."""
from __future__ import annotations

import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

_CHILD = r"""
import sys
sys.path.insert(0, {root!r})
import torch
import stab_decomp_simulator_rust_gb300 as pkg
from stab_decomp_simulator_rust_gb300 import workloads as W
ident = pkg.PauliString.identity()
free = lambda: torch.cuda.mem_get_info()[0]
small = pkg.QuantumState.from_gates(44, W.random_clifford_t_circuit(44, 880, 24, 1))  # every kernel is loaded
small.exp_value(ident)
st = pkg.QuantumState.from_gates(64, W.random_clifford_t_circuit(64, 1280, 38, 2))
before = free()
if {plan}:
    plan = pkg.BatchPlan([st], [[ident]])
    value = plan.run()[0][0]
else:
    value = st.exp_value(ident)
print(st.stabilizer_rank, value, before - free())
"""


@pytest.mark.parametrize("plan", [False, True])
def test_no_tables_beside_forms(gpu_pkg, plan):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    run = subprocess.run([sys.executable, "-c", _CHILD.format(root=root, plan=plan)], check=True, capture_output=True,
                         text=True)
    chi, value, used = run.stdout.split()[-3:]
    chi = int(chi)
    assert chi >= 15000 and abs(float(value) - 1.0) <= 1e-9
    # a reduced term takes at most 3 * 64 * 8 + 48 bytes, its form 1,072; tables
    # and frames would take 3,000 besides up to 32 qubits, 9,000 above
    assert int(used) <= chi * 2800, int(used) / chi
