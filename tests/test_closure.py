"""Closure lists and bit-row words checked on the host
(tests/closure_check.cpp): the lists give the level-by-level sweep result on
random raw scores, the word operations the scalar recurrences."""
import os
import subprocess

from conftest import ROOT

HERE = os.path.dirname(os.path.abspath(__file__))


def test_closure_lists_and_bit_words(tmp_path):
    exe = str(tmp_path / "closure_check")
    lib = os.path.join(ROOT, "chsga_b200", "lib")
    csrc = os.path.join(ROOT, "chsga_b200", "csrc")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fopenmp", "-I", csrc, "-I", os.path.join(ROOT, "include"),
                    "-o", exe, os.path.join(HERE, "closure_check.cpp"), os.path.join(csrc, "closure.cpp"),
                    os.path.join(csrc, "device_graph.cpp"), "-L", lib, "-lchsga", "-Wl,-rpath," + lib],
                   check=True, timeout=300)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.startswith("OK")
