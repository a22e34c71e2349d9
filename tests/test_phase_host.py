"""The plan's integer evaluation of the phase that a near-identity SHIFT leaves (geom.cuh,
tiny_phase) against the DOUBLE products it stands in for, bit for bit, on the host."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_tiny_phase_matches_double(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    exe = str(tmp_path / "phase_check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(HERE, "..", "sde_gb300", "csrc"),
                    os.path.join(HERE, "phase_check.cpp"), "-o", exe, "-lm"], check=True)
    out = subprocess.run([exe, "20000000"], capture_output=True, text=True)
    cases, decided, bad = (int(x) for x in out.stdout.split())
    assert bad == 0, out.stderr
    assert decided > 0.5 * cases
