"""State vectors on both sides of the number of terms from which the amplitude
kernels are used: the same as the sum of the vectors of two parts."""
from __future__ import annotations

import numpy as np
import pytest

from stab_decomp_simulator_rust_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def limit(n):
    return int((50 if n <= 12 else 65) / max(0.6 + 0.13 * n, 2.3e-5 * 2 ** n))


@pytest.mark.parametrize("n", [1, 8, 12, 13, 16, 18, 20])
def test_vector_of_parts(gpu_pkg, n):
    d = gpu_pkg.QuantumState.from_gates(n, W.random_clifford_t_circuit(n, 12 * n, 24, 6200 + n)).export_terms()
    d["coef_r"] = d["coef_r"] + np.arange(len(d["coef_r"]), dtype=np.int32) % 3  # odd and even differences
    d["global_factor"] = np.asarray([0.6, -0.8])
    st = gpu_pkg.QuantumState.from_terms(d)
    for chi in (1, limit(n), limit(n) + 1, limit(n) + 2):
        assert chi <= st.stabilizer_rank
        whole = st.select(range(chi)).to_statevector()
        cut = chi // 2
        parts = sum((st.select(r).to_statevector() for r in (range(cut), range(cut, chi)) if len(r)))
        # exact sums, three roundings of values below 100
        np.testing.assert_allclose(whole, parts, rtol=0, atol=1e-13)


@pytest.mark.parametrize("spread", [40, 90, 100, 101, 102, 120])
def test_wide_exponents(gpu_pkg, spread):
    """Integers up to 2^52 in the one launch, FP64 beyond: terms of 1 and of 2^-(spread/2)."""
    n = 6
    h = np.asarray([(W.OP["H"], q, 0, 0) for q in range(n)], np.uint32)
    a, b = (gpu_pkg.QuantumState.from_gates(n, g).export_terms() for g in (h, h[:-1]))
    d = {k: np.concatenate([a[k], b[k]]) for k in
         ("G", "F", "M", "gamma", "v", "s", "phase", "coef_phase", "coef_r", "coef_zero")}
    d["coef_r"] = d["coef_r"] + np.asarray([0, spread], np.int32)
    got = gpu_pkg.QuantumState.from_terms(dict(d, n=n, global_factor=np.asarray([1.0, 0.0]))).to_statevector()
    want = np.full(64, 0.125)
    want[:32] += 2.0 ** (-(spread + 5) / 2)
    np.testing.assert_allclose(got, want, rtol=4e-16, atol=0)
