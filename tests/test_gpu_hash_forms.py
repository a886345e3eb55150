"""Leaf chains on threads, on pairs of lanes and on a mixture of both, and the
subtree form of Merkle trees, against hashlib and against the fully unrolled
one-thread permutation."""
import ctypes
import hashlib

import numpy as np
import pytest

import _oracle as O
import virgo_b200 as vb
from virgo_b200 import transcript

pytestmark = pytest.mark.gpu


def chains(ctx, cw, n, slices):
    leaves = ctx.buffer(max(1, n // 2) * 32)
    vb.check(vb.lib().vg_leaf_chain(ctx.h, cw.p, slices, n, leaves.p), "vg_leaf_chain")
    return leaves.download(np.zeros((n // 2, 32), np.uint8))


@pytest.mark.parametrize("log_n,slices", [(1, 1), (2, 3), (5, 65), (6, 65), (9, 65), (14, 65), (15, 2), (16, 5), (17, 4),
                                          (18, 3)])
def test_leaf_chain_forms(log_n, slices):
    # 2^14: pairs only; 2^15, 2^16: threads; 2^17: three warps per scheduler on
    # threads and the rest on pairs
    n, half = 1 << log_n, 1 << (log_n - 1)
    ctx = vb.Context(0)
    try:
        c = O.fe_random(log_n, slices * n)
        cw = ctx.buffer(c)
        got = chains(ctx, cw, n, slices)
        vb.tune_set(0, leaf_rot=0)
        plain = chains(ctx, cw, n, slices)
        assert (got == plain).all()
        v = c.reshape(slices, n, 2)
        for k in sorted({0, min(1, half - 1), half // 2, half - 1}):
            h = bytes(32)
            for s in range(slices):
                h = hashlib.sha3_256(v[s, k].tobytes() + v[s, k + half].tobytes() + h).digest()
            assert got[k].tobytes() == h, k
    finally:
        vb.tune_reset(0)
        ctx.close()


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("n", [1, 2, 3, 16, 63, 64, 65, 128, 129, 255, 1024, 8192, 16384, 16385, 40000])
def test_merkle_subtrees(kind, n):
    h = hashlib.sha3_256 if kind == 0 else hashlib.sha256
    leaves = np.random.default_rng(n).integers(0, 256, (n, 32), dtype=np.uint8)
    size = 1 << (n - 1).bit_length()
    tree = [bytes(32)] * size + [r.tobytes() for r in leaves] + [h(bytes(64)).digest()] * (size - n)
    for i in range(size - 1, 0, -1):
        tree[i] = h(tree[2 * i] + tree[2 * i + 1]).digest()
    ctx = vb.Context(0, kind)
    try:
        src, dst = ctx.buffer(leaves), ctx.buffer(2 * size * 32)
        vb.check(vb.lib().vg_merkle_tree(ctx.h, src.p, n, dst.p), "vg_merkle_tree")
        got = dst.download(np.zeros((2 * size, 32), np.uint8))
        assert got.tobytes() == b"".join(tree)
    finally:
        ctx.close()


@pytest.mark.parametrize("log_in", [10, 16, 17, 18])
@pytest.mark.parametrize("gates", [2, 1 << 20])
def test_proof_leaves_are_chains_of_all_slices(log_in, gates):
    """A proof's committed leaves, whether their chains ran in one launch (the
    circuits with 2^20 gates, up to 2^17 values) or went on after the mask
    slice came (the others): on pairs, on threads and, for 2^18 values, on both."""
    rng = np.random.default_rng(log_in)
    n = 1 << log_in
    layers = [(np.full(n, 3, np.uint8), rng.integers(0, 1 << 20, n), np.zeros(n, np.int64)),
              (rng.integers(0, 2, gates).astype(np.uint8), rng.integers(0, n, gates), rng.integers(0, n, gates))]
    s = vb.Session(layers)
    try:
        for seed in (3, 4):
            recs = transcript.parse(s.prove(seed)[1])
            roots = [d for t, d in recs if t == "C"][:2]
            first = [d for t, d in recs if t == "I"]
            assert len(first) >= 10 and len(first) % 2 == 0
            for i, d in enumerate(first):   # l and h in turn
                counts = int.from_bytes(d[8:16], "little")
                nv, nd = counts >> 16, counts & 0xffff
                assert nv == 65 and len(d) == 16 + 32 * (nv + nd)
                values, nodes = d[16:16 + 32 * nv], d[16 + 32 * nv:]
                h = bytes(32)
                for k in range(nv):
                    h = hashlib.sha3_256(values[32 * k:32 * k + 32] + h).digest()
                assert h == nodes[-32:]
                if i < 2:
                    assert roots[i] in _folds(h, [nodes[32 * k:32 * k + 32] for k in range(nd - 1)])
    finally:
        s.close()


def _folds(h, siblings):
    """The roots that a leaf digest and its siblings can have, left and right
    siblings together (the position is not in the record)."""
    level = {h}
    for x in siblings:
        level = {hashlib.sha3_256(p).digest() for a in level for p in (a + x, x + a)}
    return level
