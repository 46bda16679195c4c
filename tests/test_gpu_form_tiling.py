"""nsg_set_pair_tiling on sums over quadratic forms, a pair per lane and a pair
per warp: any chunk and any number of tasks give the same values."""
from __future__ import annotations

import numpy as np
import pytest

from stab_decomp_simulator_rust_gb300.state import set_pair_tiling
from term_sets import unrelated_terms
from test_gpu_reduction import noalloc

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _default_tiling():
    yield
    set_pair_tiling(0, 0)


@pytest.mark.parametrize("n,extra", [(31, 9), (40, 0)])  # qubits left: 31 of 40, and 40
def test_values_do_not_depend_on_the_tiling(gpu_pkg, n, extra):
    st = gpu_pkg.QuantumState.from_terms(unrelated_terms(gpu_pkg, n, 300, 4902))
    if extra:
        st = st.kron(gpu_pkg.QuantumState.from_gates(extra, np.zeros((0, 4), np.uint32)))
    rng = np.random.default_rng(n)
    ps = [gpu_pkg.PauliString.sparse([3] * 3, rng.permutation(n + extra)[:3]) for _ in range(40)]
    ps += [gpu_pkg.PauliString.identity()]
    want = [noalloc(st, p) for p in ps]
    # exact dyadic terms of at most 10^5 pairs, a few roundings of the sum
    for chunk, tasks in [(0, 0), (1, 1), (1, 1024), (7, 3), (32, 64), (64, 1), (65, 200), (1024, 1024)]:
        set_pair_tiling(chunk, tasks)
        for precision in (0, 1):
            np.testing.assert_allclose(st.exp_values(ps, precision), want, rtol=0, atol=1e-13)
