"""The plan's integer evaluation of a near-identity SHIFT's phase (geom.cuh, tiny_phase) decides
nothing that it gets wrong: zeros, the largest and smallest W, infinities and NaN, on the host."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_tiny_phase_limits(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    exe = str(tmp_path / "phase_limits")
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(HERE, "..", "sde_gb300", "csrc"),
                    os.path.join(HERE, "phase_limits.cpp"), "-o", exe, "-lm"], check=True)
    out = subprocess.run([exe], capture_output=True, text=True)
    decided, bad = (int(x) for x in out.stdout.split())
    assert bad == 0, out.stderr
    assert decided >= 10
