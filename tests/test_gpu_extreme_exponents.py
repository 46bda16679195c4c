"""Restored terms whose coefficients' exponents are far outside those of any
circuit."""
from __future__ import annotations

import numpy as np
import pytest

from stab_decomp_simulator_rust_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def with_exponents(pkg, n, t, seed, change):
    d = pkg.QuantumState.from_gates(n, W.random_clifford_t_circuit(n, 20 * n, t, seed)).export_terms()
    d["coef_r"] = change(d["coef_r"].astype(np.int64)).astype(np.int32)
    return d


@pytest.mark.parametrize("low,high", [(-400, 2 ** 31 - 64), (-400, 2 ** 30), (-40, 2 ** 20 + 1), (0, 2 ** 31 - 64)])
def test_vector_with_exponents_that_overflow_their_difference(gpu_pkg, low, high):
    """Every second term is 2^(-high/2): nothing is left of it."""
    n = 10
    d = with_exponents(gpu_pkg, n, 12, 5500, lambda r: np.where(np.arange(len(r)) % 2, high, r + low))
    keep = {k: v[::2] if isinstance(v, np.ndarray) and k != "global_factor" else v for k, v in d.items()}
    got = gpu_pkg.QuantumState.from_terms(d).to_statevector()
    want = gpu_pkg.QuantumState.from_terms(dict(keep, coef_r=keep["coef_r"] - np.int32(low))).to_statevector()
    want = want * 2.0 ** (-low / 2)
    np.testing.assert_allclose(got, want, rtol=0, atol=1e-13 * np.abs(want).max())
