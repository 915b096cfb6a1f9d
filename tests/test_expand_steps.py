"""The split of an Expand into band passes (vlsg_expand.h), compiled for the
host and checked on lines of cells."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_passes_equal_cycles(tmp_path):
    exe = str(tmp_path / "expand_steps")
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-ffp-contract=off",
                           "-I", os.path.join(ROOT, "viennals_b200", "csrc"),
                           os.path.join(ROOT, "tests", "cpp", "expand_steps.cpp"), "-o", exe])
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
