"""Exported terms on both sides of the size from which output pages are mapped ahead of the copy."""
from __future__ import annotations

import numpy as np
import pytest

from stab_decomp_simulator_rust_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chi", [1, 85, 86, 400, 1100])  # three matrices of 4 KB a term: 1 MB at 86, several parts at 1,100
def test_export_equals_its_parts(gpu_pkg, chi):
    st = gpu_pkg.QuantumState.from_gates(64, W.random_clifford_t_circuit(64, 800, 26, 6100)).select(range(chi))
    d = st.export_terms()
    again = gpu_pkg.QuantumState.from_terms(d).export_terms()
    parts = [st.select(range(a, min(a + 60, chi))).export_terms() for a in range(0, chi, 60)]
    for k in ("G", "F", "M", "gamma", "v", "s", "phase", "coef_phase", "coef_r", "coef_zero"):
        np.testing.assert_array_equal(d[k], np.concatenate([p[k] for p in parts]))
        np.testing.assert_array_equal(d[k], again[k])
