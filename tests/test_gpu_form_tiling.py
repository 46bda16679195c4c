"""nsg_set_pair_tiling on sums over quadratic forms, a pair per lane and a pair
per warp: any chunk and any number of tasks give the same values."""
from __future__ import annotations

import numpy as np
import pytest

from stab_decomp_simulator_rust_gb300 import workloads as W
from stab_decomp_simulator_rust_gb300.state import set_pair_tiling
from test_gpu_reduction import noalloc, stabilizers

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _default_tiling():
    yield
    set_pair_tiling(0, 0)


@pytest.mark.parametrize("n,t,terms", [(44, 20, None), (40, 36, 500)])  # up to 32 qubits left, and more
def test_values_do_not_depend_on_the_tiling(gpu_pkg, n, t, terms):
    gates = W.random_clifford_t_circuit(n, 20 * n, t, 4900 + n)
    st = gpu_pkg.QuantumState.from_gates(n, gates)
    if terms:
        st = st.select(sorted(np.random.default_rng(n).permutation(st.stabilizer_rank)[:terms].tolist()))
    ps = [gpu_pkg.PauliString.dense(p) for p in stabilizers(n, gates, 40, 4901)] + [gpu_pkg.PauliString.identity()]
    want = [noalloc(st, p) for p in ps]
    # exact dyadic terms of at most 10^5 pairs, a few roundings of the sum
    for chunk, tasks in [(0, 0), (1, 1), (1, 1024), (7, 3), (32, 64), (64, 1), (65, 200), (1024, 1024)]:
        set_pair_tiling(chunk, tasks)
        for precision in (0, 1):
            np.testing.assert_allclose(st.exp_values(ps, precision), want, rtol=0, atol=1e-13)
