"""The rows of an answer's path beyond its depth are zero, whatever the buffers
held before."""
import ctypes

import numpy as np
import pytest

import _oracle as O
import virgo_b200 as vb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log_len,levels", [(11, 5), (14, 8)])
def test_unused_path_rows_are_zero(log_len, levels):
    S = 1 << (log_len - 1)
    gap = 1
    while gap * 2 <= S // 40:
        gap *= 2
    M, which = S // gap, np.array([0, 1] + [2 + t for t in range(levels)], np.int32)
    nq, pos = len(which), np.arange(len(which), dtype=np.int64)
    roots, sums, inner = np.zeros((2 + levels, 32), np.uint8), np.zeros((65, 2), np.uint64), np.zeros(2, np.uint64)
    fin, vals = np.zeros((65 * (S >> levels), 2), np.uint64), np.zeros((nq * 130, 2), np.uint64)
    ctx = vb.Context(0)
    pc = ctypes.c_void_p()
    L = vb.lib()
    try:
        junk = ctx.buffer(np.full(1 << 20, 255, np.uint8))   # freed memory the answers' buffer may be made of
        junk.free()
        vb.check(L.vg_pc_create(ctx.h, ctypes.byref(pc)))
        a = [O.fe_random(k, n) for k, n in ((1, 2 * S), (2, 40), (3, 2 * S), (4, M), (5, levels))]
        paths = np.full((nq, 32, 32), 255, np.uint8)
        vb.check(L.vg_pc_commit_all(pc, vb.ptr(a[0]), log_len, vb.ptr(a[1]), 40, vb.ptr(a[2]), vb.ptr(a[3]), M, vb.ptr(a[4]),
                                    levels, nq, vb.ptr(which), vb.ptr(pos), vb.ptr(roots), vb.ptr(sums), vb.ptr(inner),
                                    vb.ptr(fin), vb.ptr(vals), vb.ptr(paths)), "vg_pc_commit_all")
        again, lens = np.full((nq, 32, 32), 255, np.uint8), np.zeros(nq, np.int32)
        vb.check(L.vg_pc_query_batch(pc, nq, vb.ptr(which), vb.ptr(pos), vb.ptr(vals), vb.ptr(again), vb.ptr(lens)))
        assert (paths == again).all()
        for q, w in enumerate(which):
            used = (log_len - 2 if w < 2 else log_len - (w - 2) - 3) + 1
            assert lens[q] == used and paths[q, :used].any(1).all() and not paths[q, used:].any(), q
    finally:
        if pc:
            L.vg_pc_destroy(pc)
        ctx.close()
