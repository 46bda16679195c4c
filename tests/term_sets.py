"""States of unrelated terms, for tests that need pairs over more than 32 qubits:
nothing is shared, so a sum over quadratic forms keeps the full width."""
from __future__ import annotations

import numpy as np

from stab_decomp_simulator_rust_gb300 import workloads as W


def unrelated_terms(pkg, n, chi, seed):
    """The term dump of `chi` deep random stabilizer states of n qubits, global factor 1/chi."""
    rng = np.random.default_rng(seed)
    circuits = [(n, W.random_clifford_t_circuit(n, 12 * n, 0, int(rng.integers(1 << 30)))) for _ in range(chi)]
    parts = [s.export_terms() for s in pkg.QuantumState.from_gates_many(circuits)]
    d = {k: np.concatenate([p[k] for p in parts]) for k in
         ("G", "F", "M", "gamma", "v", "s", "phase", "coef_phase", "coef_r", "coef_zero")}
    d["coef_phase"] = rng.integers(0, 8, chi).astype(np.uint8)
    d.update(n=n, global_factor=np.asarray([1.0 / chi, 0.0]))
    return d
