"""build_closure at its limits (tests/closure_limits_check.cpp): refused graphs
cost no more memory than accepted ones, and running out of memory on any thread
is an error of the call, not of the process."""
import os
import subprocess

from conftest import ROOT

HERE = os.path.dirname(os.path.abspath(__file__))


def test_closure_limits(tmp_path):
    exe = str(tmp_path / "closure_limits_check")
    csrc = os.path.join(ROOT, "chsga_b200", "csrc")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fopenmp", "-I", csrc, "-I", os.path.join(ROOT, "include"),
                    "-o", exe, os.path.join(HERE, "closure_limits_check.cpp"), os.path.join(csrc, "closure.cpp")],
                   check=True, timeout=300)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "OK" in r.stdout, (r.returncode, r.stdout + r.stderr)
