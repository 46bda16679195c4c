"""Edges of the pair sums: exponents further apart than a chunk's integers hold,
states that came from more than 64 qubits, and states used by several threads at once."""
from __future__ import annotations

import threading

import numpy as np
import pytest

from conftest import random_full_circuit
from stab_decomp_simulator_rust_gb300 import workloads as W
from term_sets import unrelated_terms
from test_gpu_reduction import noalloc, observables

pytestmark = pytest.mark.gpu


# up to 32 qubits left (a pair per lane), and more (a pair per warp); the integers hold 44 powers of two
@pytest.mark.parametrize("n,extra", [(30, 10), (40, 0)])
@pytest.mark.parametrize("spread", [86, 90, 130, 300])
def test_exponents_beyond_a_chunk(gpu_pkg, n, extra, spread):
    """Every third term 2^-(spread/2), every seventh 2^-spread: in turns, so that most chunks hold all three."""
    d = unrelated_terms(gpu_pkg, n, 300, 6502)
    i = np.arange(len(d["phase"]))
    d["coef_r"] = (d["coef_r"] + spread * (i % 3 == 1) + 2 * spread * (i % 7 == 3)).astype(np.int32)
    st = gpu_pkg.QuantumState.from_terms(d)
    if extra:
        st = st.kron(gpu_pkg.QuantumState.from_gates(extra, np.zeros((0, 4), np.uint32)))
    ps = [gpu_pkg.PauliString.sparse([3], [q]) for q in range(0, n + extra, 3)]
    ps += [gpu_pkg.PauliString.dense(p) for p in W.random_dense_paulis(n + extra, 4, 6501)] + [gpu_pkg.PauliString.identity()]
    want = np.asarray([noalloc(st, p) for p in ps])
    for precision in (0, 1):
        np.testing.assert_allclose(st.exp_values(ps, precision), want, rtol=0, atol=1e-13 * max(1.0, want[-1]))


@pytest.mark.parametrize("n,left", [(70, 64), (70, 40), (66, 20), (80, 12)])
def test_states_from_more_than_64_qubits(gpu_pkg, n, left):
    """Two words a row remain after the discards; reduced, as they are, and from amplitudes."""
    t = 20
    inner = W.random_clifford_t_circuit(left, 15 * left, t, 6600 + left)
    wide = gpu_pkg.QuantumState.from_gates(n, inner)
    assert wide.num_qubits == n
    for q in range(n - 1, left - 1, -1):  # they are in |0>
        wide.project_unnormalized(q, False)
        wide.discard(q)
    st = gpu_pkg.QuantumState.from_gates(left, inner)
    ps = observables(gpu_pkg, left, inner, 4, 5)
    extra = random_full_circuit(left, 40, 0, 6700)
    for _ in range(2):
        want = [noalloc(st, p) for p in ps]
        np.testing.assert_allclose(wide.exp_values(ps), want, rtol=0, atol=1e-12)
        np.testing.assert_allclose(gpu_pkg.BatchPlan([wide], [ps]).run()[0], want, rtol=0, atol=1e-12)
        if left <= 20:
            np.testing.assert_allclose(wide.to_statevector(), st.to_statevector(), rtol=0, atol=1e-12)
            assert wide.sample_raw(range(10), 100, 3) == st.sample_raw(range(10), 100, 3)
        wide.apply_gates(extra)
        st.apply_gates(extra)


def test_states_in_threads(gpu_pkg):
    """Every thread makes, evaluates, changes and frees states of its own, all from one pool."""
    specs = [(16, 8), (36, 20), (22, 21), (48, 18)]
    ps = {n: [gpu_pkg.PauliString.dense(p) for p in W.random_dense_paulis(n, 6, n)] + [gpu_pkg.PauliString.identity()]
          for n, _ in specs}

    def work(n, t, seed):
        out = []
        for k in range(4):
            st = gpu_pkg.QuantumState.from_gates(n, W.random_clifford_t_circuit(n, 12 * n, t, 6800 + 10 * seed + k))
            out.append(st.exp_values(ps[n]))
            st.apply_gates(random_full_circuit(n, 30, 0, k))
            out.append(st.exp_values(ps[n]))
            plan = gpu_pkg.BatchPlan([st], [ps[n]])
            out.append(plan.run()[0])
            out.append(np.asarray(st.measure(range(5), seed)))
            out.append(st.exp_values(ps[n]))
            if n <= 22:
                out.append(st.to_statevector())
        return out

    jobs = [(n, t, s) for s, (n, t) in enumerate(specs * 2)]
    want = [work(*j) for j in jobs]
    got = [None] * len(jobs)

    def run(i):
        got[i] = work(*jobs[i])

    threads = [threading.Thread(target=run, args=(i,)) for i in range(len(jobs))]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    for a, b in zip(got, want):
        assert a is not None and len(a) == len(b)
        for x, y in zip(a, b):
            np.testing.assert_array_equal(x, y)
