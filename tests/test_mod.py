"""The remainders and the fraction that the step kernels take positions from are
exact for every divisor, and a run's buckets hold every draw that falls in it."""
import os
import subprocess

from conftest import ROOT


def test_mod_by_and_fraction_are_exact(tmp_path):
    exe = tmp_path / "mod"
    subprocess.run(["/usr/bin/g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "gowalker_b200", "csrc"),
                    "-o", str(exe), os.path.join(ROOT, "tests", "cuda", "mod_check.cpp")], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=240)
    assert out.returncode == 0 and out.stdout.startswith("ok"), out.stdout
