"""Restored terms whose coefficients' exponents are far outside those of any
circuit."""
from __future__ import annotations

import numpy as np
import pytest

from stab_decomp_simulator_rust_gb300 import workloads as W
from term_sets import unrelated_terms

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


def noalloc(st, p):
    import ctypes as C
    from stab_decomp_simulator_rust_gb300 import _ffi
    out = C.c_double()
    a = p.abi()
    _ffi.check(_ffi.load().nsg_exp_value_noalloc(st._h, C.byref(a), C.byref(out)))
    return out.value


# summed a pair per lane, and (more than 32 qubits left) a pair per warp
@pytest.mark.parametrize("n,t", [(34, 20), (40, 0)])
@pytest.mark.parametrize("shift", [-960, 960, 986])
def test_values_near_the_ends_of_the_exponents(gpu_pkg, n, t, shift):
    """Pair terms down to 2^-1019 and up to 2^960: the values of the state without the shift, scaled."""
    if t:
        d = with_exponents(gpu_pkg, n, t, 5600 + n, lambda r: r + shift)
    else:
        d = unrelated_terms(gpu_pkg, n, 300, 5602)
        d["coef_r"] = d["coef_r"] + np.int32(shift)
    st = gpu_pkg.QuantumState.from_terms(d)
    base = gpu_pkg.QuantumState.from_terms(dict(d, coef_r=d["coef_r"] - np.int32(shift)))
    ps = [gpu_pkg.PauliString.identity()] + [gpu_pkg.PauliString.sparse([3], [q]) for q in range(0, n, 7)]
    want = [noalloc(base, p) for p in ps]
    scale = 2.0 ** -shift
    np.testing.assert_allclose(st.exp_values(ps) / scale, want, rtol=0, atol=1e-12 * want[0])
    np.testing.assert_allclose(st.exp_values(ps, gpu_pkg.PRECISION_MIXED) / scale, want, rtol=0, atol=1e-12 * want[0])
