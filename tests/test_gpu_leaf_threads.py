"""Leaf chains launched from several host threads at once, each on a context of
its own, at sizes whose launches are the same kernel with different shared
memory (room for two, four or any number of CTAs on an SM: 115712, 57344 and 0
bytes): every launch is accepted and every digest is the one computed alone."""
import threading

import numpy as np
import pytest

import _oracle as O
import virgo_b200 as vb

pytestmark = pytest.mark.gpu

SLICES = 2


def _chain(ctx, cw, log_n, leaves):
    return vb.lib().vg_leaf_chain(ctx.h, cw.p, SLICES, 1 << log_n, leaves.p)


@pytest.mark.parametrize("sizes", [(15, 16), (15, 18), (15, 16, 18), (15, 15, 16, 17, 18)])
def test_leaf_chains_of_different_sizes_from_threads(sizes):
    work, errors = [], []
    start = threading.Barrier(len(sizes))
    try:
        for i, log_n in enumerate(sizes):
            ctx = vb.Context(0)
            cw = ctx.buffer(O.fe_random(100 * i + log_n, SLICES << log_n))
            leaves = ctx.buffer(32 << (log_n - 1))
            vb.check(_chain(ctx, cw, log_n, leaves), "vg_leaf_chain")
            want = leaves.download(np.zeros((1 << (log_n - 1), 32), np.uint8))
            work.append((ctx, cw, log_n, leaves, want))

        def run(ctx, cw, log_n, leaves, want):
            start.wait()
            for _ in range(10):
                for _ in range(40):
                    if _chain(ctx, cw, log_n, leaves) != 0:
                        errors.append((log_n, vb.lib().vg_last_error()))
                        return
                got = leaves.download(np.zeros_like(want))
                if not (got == want).all():
                    errors.append((log_n, "digests"))
                    return

        threads = [threading.Thread(target=run, args=w) for w in work]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not errors, errors
    finally:
        for w in work:
            w[0].close()
