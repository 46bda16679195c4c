"""A plan whose graph could not be made again: the run that fails says so, and
the next one has the values of the states as they are."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import random_full_circuit
from stab_decomp_simulator_rust_gb300 import workloads as W
from test_gpu_reduction import TOL, noalloc, observables

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gates_after", [False, True])
def test_run_after_a_failed_rebuild(gpu_pkg, gates_after):
    from stab_decomp_simulator_rust_gb300 import NecstarError, _ffi
    L = _ffi.load()
    specs = [(36, 20), (24, 9)]  # reduced; a few terms, summed by tables
    made = [(n, W.random_clifford_t_circuit(n, 20 * n, t, 4700 + n)) for n, t in specs]
    states = gpu_pkg.QuantumState.from_gates_many(made)
    ps = [observables(gpu_pkg, n, g, n) for n, g in made]
    plan = gpu_pkg.BatchPlan(states, ps)
    plan.run()

    def layer(seed):
        for (n, _), s in zip(specs, states):
            s.apply_gates(random_full_circuit(n, 10, 0, seed))

    layer(4710)
    plan.run()  # without the graph
    _ffi.check(L.nsg_debug_set_wait(1 << 10, 16))  # table launches run out of time
    try:
        with pytest.raises(NecstarError) as e:
            plan.run()
        assert e.value.code == _ffi.header_constants()["NSG_ERR_TIMEOUT"]
    finally:
        _ffi.check(L.nsg_debug_set_wait(0, 0))
    if gates_after:
        states[1].apply_gates(random_full_circuit(24, 10, 0, 4711))
    for _ in range(3):
        for got, s, p in zip(plan.run(), states, ps):
            np.testing.assert_allclose(got, [noalloc(s, x) for x in p], rtol=0, atol=TOL)
