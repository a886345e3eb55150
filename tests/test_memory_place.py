"""Which leaves a Merkle tree's kernel reads where they are: the decision on the
CPU, and on the GPU leaves that have to be copied first (off 16-byte
boundaries)."""
import ctypes
import hashlib
import os
import subprocess

import numpy as np
import pytest

import virgo_b200 as vb

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_places(tmp_path):
    exe = str(tmp_path / "memory_place_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I" + os.path.join(ROOT, "virgo_b200", "csrc"),
                    os.path.join(ROOT, "tests", "memory_place_check.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    assert "places agree" in out


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 3, 64, 1000, 20000])
def test_tree_of_copied_leaves(n):
    leaves = np.random.default_rng(n).integers(0, 256, (n, 32), dtype=np.uint8)
    size = 1 << (n - 1).bit_length()
    level = [r.tobytes() for r in leaves] + [hashlib.sha3_256(bytes(64)).digest()] * (size - n)
    while len(level) > 1:
        level = [hashlib.sha3_256(level[i] + level[i + 1]).digest() for i in range(0, len(level), 2)]
    ctx = vb.Context(0)
    try:
        for off in (0, 8):
            src, dst = ctx.buffer(np.concatenate([np.zeros(off, np.uint8), leaves.reshape(-1)])), ctx.buffer(2 * size * 32)
            vb.check(vb.lib().vg_merkle_tree(ctx.h, ctypes.c_void_p(src.p.value + off), n, dst.p), "vg_merkle_tree")
            got = dst.download(np.zeros((2 * size, 32), np.uint8))
            assert got[1].tobytes() == level[0] and (got[size:size + n] == leaves).all(), off
    finally:
        ctx.close()
