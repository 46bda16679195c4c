"""The common stabilizers that a state carries through projections and gates."""
from __future__ import annotations

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(not shutil.which("g++"), reason="needs g++")
def test_generators_stay_independent(tmp_path):
    exe = str(tmp_path / "check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "stab_decomp_simulator_rust_gb300", "csrc"),
                    "-I", "/usr/local/cuda/include",
                    os.path.join(ROOT, "tests", "cpp", "common_group_projections_check.cpp"), "-o", exe], check=True)
    run = subprocess.run([exe], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout
