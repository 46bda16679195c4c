"""Sampling of more than eight qubits where the outcomes' exact weights pass 64
bits: two terms on all but one and on all qubits, 2^spread apart in weight."""
from __future__ import annotations

import numpy as np
import pytest

from stab_decomp_simulator_rust_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def two_terms(pkg, n, spread):
    """|+⟩^(n-1) ⊗ |0⟩ + 2^(-spread/2)·|+⟩^n."""
    h = np.asarray([(W.OP["H"], q, 0, 0) for q in range(n)], np.uint32)
    a, b = (pkg.QuantumState.from_gates(n, g).export_terms() for g in (h[:-1], h))
    d = {k: np.concatenate([a[k], b[k]]) for k in
         ("G", "F", "M", "gamma", "v", "s", "phase", "coef_phase", "coef_r", "coef_zero")}
    d["coef_r"] = d["coef_r"] + np.asarray([0, spread], np.int32)
    return pkg.QuantumState.from_terms(dict(d, n=n, global_factor=np.asarray([1.0, 0.0])))


# sums of weights of 2^(n + spread) and a little more on both sides of 2^62 and
# 2^63; 44 is the largest spread that the amplitudes' integers hold
@pytest.mark.parametrize("n,spread,k", [(20, 30, 9), (19, 41, 9), (19, 42, 19), (19, 43, 12), (20, 41, 20), (20, 42, 10),
                                        (20, 43, 9), (20, 44, 20), (21, 44, 9), (22, 44, 12), (22, 44, 20), (22, 46, 9)])
def test_weights_beyond_64_bits(gpu_pkg, n, spread, k):
    st = two_terms(gpu_pkg, n, spread)
    qargs = [n - 1] + [int(q) for q in np.random.default_rng(n).permutation(n - 1)[:k - 1]]
    shots = 100000
    vals, counts = st.sample_raw(qargs, shots, 5)
    vals, counts = np.asarray(vals), np.asarray(counts)
    assert counts.sum() == shots and len(set(vals.tolist())) == len(vals)
    p = np.abs(st.to_statevector()) ** 2
    p /= p.sum()
    for i, q in enumerate(qargs):
        want = p.reshape(-1, 2, 1 << q)[:, 1].sum()
        freq = counts[(vals >> i) & 1 == 1].sum() / shots
        assert abs(freq - want) <= 6 * np.sqrt(want * (1 - want) / shots), q
