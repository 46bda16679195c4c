"""One and a few shots of nine to twelve qubits of a wide state, which are drawn
from the tree of projections: possible outcomes, the same for the same seed, and
at their frequencies over many seeds."""
from __future__ import annotations

import numpy as np
import pytest

from stab_decomp_simulator_rust_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k,shots", [(24, 9, 1), (25, 9, 2), (26, 12, 1), (26, 9, 3)])
def test_few_shots(gpu_pkg, n, k, shots):
    st = gpu_pkg.QuantumState.from_gates(n, W.random_clifford_t_circuit(n, 12 * n, 8, 6300 + n))
    for seed in range(3):
        vals, counts = st.sample_raw(range(k), shots, seed)
        assert (vals, counts) == st.sample_raw(range(k), shots, seed) and sum(counts) == shots
        for v in vals:
            c = st.clone()
            for q in range(k):
                c.project_normalized(q, bool((v >> q) & 1))  # raises where it is impossible
            assert abs(c.norm() - 1.0) <= 1e-9


def test_frequencies_of_single_shots(gpu_pkg):
    n, k, runs = 24, 9, 600
    st = gpu_pkg.QuantumState.from_gates(n, W.random_clifford_t_circuit(n, 12 * n, 6, 6400))
    p = [0.5 * (1.0 - st.exp_value(gpu_pkg.PauliString.sparse([3], [q]))) for q in range(k)]
    drawn = np.asarray([st.sample_raw(range(k), 1, s)[0][0] for s in range(runs)])
    for q in range(k):
        freq = ((drawn >> q) & 1).mean()
        assert abs(freq - p[q]) <= 5 * np.sqrt(max(p[q] * (1 - p[q]), 1e-12) / runs)
