"""Qubits projected again and again, gates in between: the carried generators stay those of the state."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import random_full_circuit
from stab_decomp_simulator_rust_gb300 import workloads as W
from test_gpu_reduction import noalloc

pytestmark = pytest.mark.gpu


def test_values_after_repeated_projections(gpu_pkg):
    n = 48
    st = gpu_pkg.QuantumState.from_gates(n, W.random_clifford_t_circuit(n, 20 * n, 24, 4800))
    ps = [gpu_pkg.PauliString.sparse([3], [q]) for q in range(0, n, 5)]
    ps += [gpu_pkg.PauliString.dense(p) for p in W.random_dense_paulis(n, 4, 4801)] + [gpu_pkg.PauliString.identity()]
    for step in range(3):
        for _ in range(3):
            st.measure(range(0, 36), 4810 + step)
        st.apply_gates(random_full_circuit(n, 60, 0, 4820 + step))
        want = [noalloc(st, p) for p in ps]
        for _ in range(2):
            np.testing.assert_allclose(st.exp_values(ps), want, rtol=0, atol=1e-12)
