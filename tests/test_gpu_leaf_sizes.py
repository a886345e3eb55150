"""Leaf chains in every CTA size, up to sets of more than 24 warps per
scheduler (454656 chains), where 256 threads run too: against hashlib at sampled
leaves and against the 64-thread form everywhere."""
import hashlib

import numpy as np
import pytest

import _oracle as O
import virgo_b200 as vb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("log_n,slices", [(3, 65), (13, 3), (16, 3), (17, 2), (18, 2), (20, 2), (21, 1)])
def test_leaf_chain_cta_sizes(kind, log_n, slices):
    n, half = 1 << log_n, 1 << (log_n - 1)
    h = hashlib.sha256 if kind else hashlib.sha3_256
    ctx = vb.Context(0, kind)
    try:
        c = O.fe_random(log_n, slices * n)
        cw = ctx.buffer(c)
        got = {}
        for threads in (64, 128, 256):
            vb.tune_set(0, leaf_threads=threads)
            leaves = ctx.buffer(half * 32)
            vb.check(vb.lib().vg_leaf_chain(ctx.h, cw.p, slices, n, leaves.p), "vg_leaf_chain")
            got[threads] = leaves.download(np.zeros((half, 32), np.uint8))
            assert (got[threads] == got[64]).all(), threads
        v = c.reshape(slices, n, 2)
        for k in sorted({0, 1, half // 2, half // 2 - 1, half - 1}):
            d = bytes(32)
            for s in range(slices):
                d = h(v[s, k].tobytes() + v[s, k + half].tobytes() + d).digest()
            assert got[64][k].tobytes() == d, k
    finally:
        vb.tune_reset(0)
        ctx.close()
