"""What a state's pairs are summed by follows its terms: term tables while they
have few free variables, quadratic forms after gates that free them."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import random_full_circuit
from stab_decomp_simulator_rust_gb300 import workloads as W
from test_gpu_reduction import noalloc

pytestmark = pytest.mark.gpu


def shallow_terms(pkg, n, chi, hs, seed):
    """Unrelated terms of circuits with `hs` H gates each: at most that many free variables."""
    rng = np.random.default_rng(seed)
    circuits = []
    for _ in range(chi):
        g = W.random_clifford_t_circuit(n, 12 * n, 0, int(rng.integers(1 << 30)))
        drop = (g[:, 0] == W.OP["H"]) & (np.cumsum(g[:, 0] == W.OP["H"]) > hs)
        circuits.append((n, g[~drop]))
    parts = [s.export_terms() for s in pkg.QuantumState.from_gates_many(circuits)]
    d = {k: np.concatenate([p[k] for p in parts]) for k in
         ("G", "F", "M", "gamma", "v", "s", "phase", "coef_phase", "coef_r", "coef_zero")}
    return pkg.QuantumState.from_terms(dict(d, n=n, global_factor=np.asarray([1.0 / chi, 0.0])))


# without common stabilizers, and with eight of them
@pytest.mark.parametrize("extra", [0, 8])
def test_choice_after_gates(gpu_pkg, extra):
    n, chi = 44, 260
    st = shallow_terms(gpu_pkg, n, chi, 12, 6000)
    if extra:
        st = st.kron(gpu_pkg.QuantumState.from_gates(extra, np.zeros((0, 4), np.uint32)))
    n += extra
    ps = [gpu_pkg.PauliString.dense(p) for p in W.random_dense_paulis(n, 3, 6001)]
    ps += [gpu_pkg.PauliString.sparse([3], [q]) for q in range(0, n, 6)] + [gpu_pkg.PauliString.identity()]

    def check():
        want = [noalloc(st, p) for p in ps]
        plan = gpu_pkg.BatchPlan([st], [ps])
        for got in (plan.run()[0], st.exp_values(ps), st.exp_values(ps)):
            np.testing.assert_allclose(got, want, rtol=0, atol=1e-12)
        return plan.tiling

    assert check()["chunk_rows64"] > 0  # a launch over tables
    diagonal = random_full_circuit(n, 200, 0, 6002)
    st.apply_gates(diagonal[np.isin(diagonal[:, 0], [W.OP[k] for k in ("S", "Z", "X", "CX", "CZ")])])
    assert check()["chunk_rows64"] > 0  # no gate of these changes how many variables are free
    st.apply_gates(random_full_circuit(n, 30 * n, 0, 6003))
    st.exp_values(ps)
    assert check()["chunk_rows64"] == 0  # forms
