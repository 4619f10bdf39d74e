"""Queues of a batch's resident systems (host logic, no GPU)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_waits_for_a_group_are_bounded(tmp_path):
    exe = str(tmp_path / "resident_queues")
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", os.path.join(ROOT, "yafel_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cxx", "resident_queues.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
