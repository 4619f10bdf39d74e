"""Turns of kernels whose blocks wait for one another (host logic, no GPU)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_kernels_at_work_fit_the_device(tmp_path):
    exe = str(tmp_path / "sm_turns")
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", os.path.join(ROOT, "yafel_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cxx", "sm_turns.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
