"""The launch shapes of the leaf-hash chains, on the CPU."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_chain_shapes(tmp_path):
    exe = str(tmp_path / "leaf_shape_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I" + os.path.join(ROOT, "virgo_b200", "csrc"),
                    os.path.join(ROOT, "tests", "leaf_shape_check.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    assert "shapes agree" in out
