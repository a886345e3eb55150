"""The F_p2 forms of fp2.cuh at the ends of their ranges, on the CPU."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_forms_at_their_bounds(tmp_path):
    exe = str(tmp_path / "field_bounds_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I" + os.path.join(ROOT, "virgo_b200", "csrc"),
                    os.path.join(ROOT, "tests", "field_bounds_check.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    assert "cases agree" in out
