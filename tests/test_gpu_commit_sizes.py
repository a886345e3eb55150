"""Whole commitments at the sizes on both sides of the second stream's limit
(2^20 values) and below it, from host and from device arrays, both hashes:
every root, sum and answer equals the step API's, whose kernels run one after
another on one stream."""
import ctypes

import numpy as np
import pytest

import _oracle as O
import virgo_b200 as vb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("log_len", [12, 14, 16, 17, 18, 19, 20])
def test_commit_all_equals_steps(log_len, kind):
    L = vb.lib()
    n, S, levels, n_mask = 1 << log_len, 1 << (log_len - 1), log_len - 6, 50
    gap = 1
    while gap * 2 <= S // n_mask:
        gap *= 2
    M = S // gap
    priv, mask, pub, pub_mask, fri_r = (O.fe_random(log_len + k, m) for k, m in enumerate((n, n_mask, n, M, levels)))
    which = np.array([0, 1] + [2 + t for t in range(levels)], np.int32)
    pos = (np.random.default_rng(log_len).integers(0, 1 << 40, len(which)) % (S // 2)).astype(np.int64)
    nq = len(which)

    ctx = vb.Context(0, kind)
    pc = ctypes.c_void_p()
    try:
        vb.check(L.vg_pc_create(ctx.h, ctypes.byref(pc)))
        # the steps
        roots = np.zeros((2 + levels, 32), np.uint8)
        sums, inner = np.zeros((65, 2), np.uint64), np.zeros(2, np.uint64)
        vb.check(L.vg_pc_encode_private(pc, vb.ptr(priv), log_len, vb.ptr(mask), n_mask, None))
        vb.check(L.vg_pc_init_commit(pc, 0, vb.ptr(roots[0:])))
        vb.check(L.vg_pc_encode_public(pc, vb.ptr(pub), vb.ptr(pub_mask), M, vb.ptr(sums), vb.ptr(inner)))
        vb.check(L.vg_pc_init_commit(pc, 1, vb.ptr(roots[1:])))
        for t in range(levels):
            vb.check(L.vg_pc_fri_step(pc, vb.to_fe(fri_r[t]), vb.ptr(roots[2 + t:])))
        vals, paths = np.zeros((nq * 130, 2), np.uint64), np.zeros((nq * 32, 32), np.uint8)
        vb.check(L.vg_pc_query_batch(pc, nq, vb.ptr(which), vb.ptr(pos), vb.ptr(vals), vb.ptr(paths), None))

        dev = [ctx.buffer(priv), ctx.buffer(pub)]
        for a, b in ((vb.ptr(priv), vb.ptr(pub)), (dev[0].p, dev[1].p)):
            r2, s2, i2 = np.zeros_like(roots), np.zeros_like(sums), np.zeros_like(inner)
            fin, v2, p2 = np.zeros((65 * 32, 2), np.uint64), np.zeros_like(vals), np.zeros_like(paths)
            vb.check(L.vg_pc_commit_all(pc, a, log_len, vb.ptr(mask), n_mask, b, vb.ptr(pub_mask), M, vb.ptr(fri_r), levels, nq,
                                        vb.ptr(which), vb.ptr(pos), vb.ptr(r2), vb.ptr(s2), vb.ptr(i2), vb.ptr(fin), vb.ptr(v2),
                                        vb.ptr(p2)), "vg_pc_commit_all")
            for x, y in ((roots, r2), (sums, s2), (inner, i2), (vals, v2), (paths, p2)):
                assert (x == y).all()
        for d in dev:
            d.free()
    finally:
        if pc:
            L.vg_pc_destroy(pc)
        ctx.close()
