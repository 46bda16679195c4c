"""Equal terms and dozens of others that each break a stabilizer of their own:
more of them than a search for common stabilizers can be told to sample."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import random_full_circuit
from stab_decomp_simulator_rust_gb300 import workloads as W
from test_gpu_reduction import noalloc

pytestmark = pytest.mark.gpu


def state(pkg, n, chi, outliers, seed):
    one = pkg.QuantumState.from_gates(n, W.random_clifford_t_circuit(n, 15 * n, 0, seed)).export_terms()
    d = {k: (np.repeat(v, chi, axis=0) if isinstance(v, np.ndarray) and k != "global_factor" else v)
         for k, v in one.items()}
    at = np.random.default_rng(seed).permutation(chi)[:outliers]
    for j, i in enumerate(at):  # the j-th generator's sign
        d["s"][i, j] ^= 1
    d["global_factor"] = np.asarray([1.0 / chi, 0.0])
    return pkg.QuantumState.from_terms(d)


# 32 outliers can all be sampled, 33 and more cannot
@pytest.mark.parametrize("n,outliers", [(40, 32), (40, 33), (60, 50)])
def test_more_outliers_than_are_sampled(gpu_pkg, n, outliers):
    st = state(gpu_pkg, n, 2000, outliers, 91)
    ps = [gpu_pkg.PauliString.dense(p) for p in W.random_dense_paulis(n, 5, 92)]
    ps += [gpu_pkg.PauliString.sparse([3], [q]) for q in range(0, n, 9)] + [gpu_pkg.PauliString.identity()]

    def check(s):
        want = [noalloc(s, p) for p in ps]
        for _ in range(2):
            np.testing.assert_allclose(s.exp_values(ps), want, rtol=0, atol=1e-12)

    check(st)
    np.testing.assert_array_equal(gpu_pkg.BatchPlan([st], [ps]).run()[0], st.exp_values(ps))
    other = state(gpu_pkg, n, 2000, outliers, 91)
    check(other)
    copies = [st.clone(), other, state(gpu_pkg, n, 2000, outliers, 91)]
    qargs = [1, 5, 8, 20, 33]
    bits = [list(c.measure(qargs, 17)) for c in copies]
    assert bits[0] == bits[1] == bits[2]
    for c in copies:
        for q, b in zip(qargs, bits[0]):
            assert abs(c.exp_value(gpu_pkg.PauliString.sparse([3], [q])) - (-1) ** int(b)) <= 1e-12
    st.apply_gates(random_full_circuit(n, 40, 0, 93))
    check(st)
