"""nsg_profile_launch: the kernel and the width of the launch with the most pairs."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from stab_decomp_simulator_rust_gb300 import workloads as W
from term_sets import unrelated_terms

pytestmark = pytest.mark.gpu


def profiled(fn):
    from stab_decomp_simulator_rust_gb300 import _ffi
    L = _ffi.load()
    _ffi.check(L.nsg_profile_enable(1))
    _ffi.check(L.nsg_profile_read(None, None, None))
    fn()
    kernel, width = C.c_int32(), C.c_int32()
    _ffi.check(L.nsg_profile_launch(C.byref(kernel), C.byref(width)))
    _ffi.check(L.nsg_profile_read(None, None, None))
    _ffi.check(L.nsg_profile_enable(0))
    return kernel.value, width.value


def test_kernel_and_width(gpu_pkg):
    ident = gpu_pkg.PauliString.identity()

    few = gpu_pkg.QuantumState.from_gates(30, W.random_clifford_t_circuit(30, 600, 8, 7000))
    zeros = gpu_pkg.QuantumState.from_gates(14, np.zeros((0, 4), np.uint32))  # 14 common stabilizers
    narrow = gpu_pkg.QuantumState.from_terms(unrelated_terms(gpu_pkg, 30, 300, 7002)).kron(zeros)
    wide = gpu_pkg.QuantumState.from_terms(unrelated_terms(gpu_pkg, 40, 300, 7001))
    assert profiled(lambda: few.exp_value(ident)) == (0, 30)
    assert profiled(lambda: wide.exp_value(ident)) == (1, 40)
    assert profiled(lambda: narrow.exp_value(ident)) == (2, 30)
    # tables at the reduced width where exact counts are asked for, and the larger of several launches
    assert profiled(lambda: narrow.exp_value_counts([ident])) == (0, 30)
    assert profiled(lambda: gpu_pkg.exp_values_multi([few, narrow], [[ident], [ident]])) == (2, 30)
    assert profiled(lambda: None) == (-1, 0)
