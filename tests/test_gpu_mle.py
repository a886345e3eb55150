"""vg_mle_eval at the edges of its table splits (fewer than 2^8 entries, one
CTA, one chunk per CTA, chunks of several rows, looping CTAs), device and host
inputs, against Python integers and the allocation-free entry point."""
import ctypes
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

import virgo_b200 as vb

P = vb.P


def mle(vals, r):
    t = [(int(re), int(im)) for im, re in vals]
    for im, re in r:
        c, d = int(re), int(im)
        t = [((x[0] + (y[0] - x[0]) * c - (y[1] - x[1]) * d) % P, (x[1] + (y[0] - x[0]) * d + (y[1] - x[1]) * c) % P)
             for x, y in zip(t[::2], t[1::2])]
    return t[0]


@pytest.mark.gpu
@pytest.mark.parametrize("log_n", [0, 1, 3, 4, 5, 7, 8, 9, 11, 12, 13, 16, 17, 19, 21, 22])
def test_mle_eval_sizes(log_n):
    L = vb.lib()
    rng = np.random.default_rng(log_n)
    vals = rng.integers(0, P, (1 << log_n, 2), dtype=np.uint64)
    vals[0] = P - 1   # largest canonical entry
    r = rng.integers(0, P, (max(1, log_n), 2), dtype=np.uint64)
    ctx = vb.Context(0)
    try:
        dev = ctx.buffer(vals)
        out = np.zeros((4, 2), np.uint64)
        for k in range(2):   # the second call finds the context's sums as the first left them
            vb.check(L.vg_mle_eval(ctx.h, dev.p, 1 << log_n, vb.ptr(r), log_n, vb.ptr(out[k:])), "device")
        vb.check(L.vg_mle_eval(ctx.h, vb.ptr(vals), 1 << log_n, vb.ptr(r), log_n, vb.ptr(out[2:])), "host")
        L.vg_mle_eval_noalloc.argtypes = [ctypes.c_void_p, ctypes.c_long, ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p]
        vb.check(L.vg_mle_eval_noalloc(dev.p, 1 << log_n, vb.ptr(r), log_n, vb.ptr(out[3:])), "no alloc")
        assert (out == out[0]).all()
        if log_n <= 13:
            assert (int(out[0][1]), int(out[0][0])) == mle(vals, r[:log_n])
    finally:
        ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("log_n", [3, 16, 18, 20])
def test_contexts_that_follow_one_another_in_threads(log_n):
    """Pinned blocks change hands between contexts of several threads: every
    evaluation of a host table is its own table's."""
    rng = np.random.default_rng(log_n)
    r = rng.integers(0, P, (log_n, 2), dtype=np.int64)
    tables = [rng.integers(0, P, (1 << log_n, 2), dtype=np.int64) for _ in range(4)]

    def evaluate(ctx, vals):
        out = np.zeros((1, 2), np.int64)
        vb.check(vb.lib().vg_mle_eval(ctx.h, vals, 1 << log_n, r.ctypes.data_as(ctypes.c_void_p), log_n,
                                      out.ctypes.data_as(ctypes.c_void_p)), "vg_mle_eval")
        return out.tobytes()

    def value(t):
        ctx = vb.Context(0)
        try:
            return evaluate(ctx, t.ctypes.data_as(ctypes.c_void_p))
        finally:
            ctx.close()

    ctx = vb.Context(0)
    on_device = [ctx.buffer(t) for t in tables]
    want = [evaluate(ctx, b.p) for b in on_device]
    for b in on_device:
        b.free()
    ctx.close()
    with ThreadPoolExecutor(4) as pool:
        for _ in range(4):
            assert list(pool.map(value, tables)) == want
