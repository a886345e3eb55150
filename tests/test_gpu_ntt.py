"""The transform's step sizes, skipped stages and root permutations against the
oracle: every size up to 2^11 (each mix of 8-, 4- and 2-point steps), input
lengths on both sides of the power of two where a stage begins to have work,
and roots w, w^3, w^5, w^7 (the four primitive 8th roots)."""
import numpy as np
import pytest

import _oracle as O
import virgo_b200 as vb

pytestmark = pytest.mark.gpu
P = vb.P


def power(w, e):
    a, b, r = int(w[1]), int(w[0]), (1, 0)
    for _ in range(e):
        r = ((r[0] * a - r[1] * b) % P, (r[0] * b + r[1] * a) % P)
    return np.array([r[1], r[0]], np.uint64)


def check(ctx, log_n, in_len, batch, root):
    n = 1 << log_n
    co = O.fe_random(log_n * 131 + in_len, batch * max(1, in_len))
    co[0] = P - 1
    src, dst = ctx.buffer(co), ctx.buffer(batch * n * 16)
    vb.check(vb.lib().vg_ntt(ctx.h, src.p, in_len, in_len, dst.p, log_n, n, batch, vb.to_fe(root), 0), "vg_ntt")
    got = dst.download(np.zeros((batch * n, 2), np.uint64))
    for b in (0, batch - 1):
        exp = O.fft(co[b * in_len:(b + 1) * in_len], n, root)
        assert (got[b * n:(b + 1) * n] == exp).all(), (log_n, in_len, batch, b)


@pytest.mark.parametrize("log_n", list(range(1, 15)) + [16])
def test_ntt_steps_and_padding(log_n):
    ctx = vb.Context(0)
    try:
        n, w = 1 << log_n, O.root_of_unity(log_n)
        lens = sorted({1, 2, 3, n >> 5, (n >> 5) + 1, n >> 3, (n >> 3) + 1, (n >> 1) - 1, n} & set(range(1, n + 1)))
        for i, in_len in enumerate(lens):
            check(ctx, log_n, in_len, 1 + (i % 3) * 4, w)
        for k in (3, 5, 7):
            check(ctx, log_n, n, 2, power(w, k))
    finally:
        ctx.close()


@pytest.mark.parametrize("shape", [{"ntt_max_log": 6, "ntt_tile_log": 10}, {"ntt_max_log": 8, "ntt_tile_log": 13}])
def test_ntt_shapes(shape):
    """Other factorisations (three and more passes, small last factors)."""
    ctx = vb.Context(0)
    try:
        vb.tune_set(0, **shape)
        for log_n, in_len, batch in [(7, 128, 3), (13, 8192, 2), (14, 100, 5), (17, 1 << 12, 1)]:
            check(ctx, log_n, in_len, batch, O.root_of_unity(log_n))
    finally:
        vb.tune_reset(0)
        ctx.close()
