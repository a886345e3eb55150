"""The edge sets behind the phase gathers at the sizes where their build can go
wrong: keys with as many edges as one thread, one warp or one launch's split
takes, more split keys than travel with the counts, sets that outgrow one edge
per gate, layers of two gates and key ranges beyond one tile per CTA.  The
scatter path, which uses no edge sets, has to give the same transcript."""
import numpy as np
import pytest
import virgo_b200 as vb

pytestmark = pytest.mark.gpu


def _inputs(rng, n):
    return np.full(n, 3, np.uint8), rng.integers(0, 1 << 20, n), np.zeros(n, np.int64)


def _gates(rng, n, prev, u=None):
    t = rng.choice([0, 1, 7, 8, 9], n).astype(np.uint8)
    return t, rng.integers(0, prev, n) if u is None else u, rng.integers(0, prev, n)


def _repeat(counts, n):
    """n wires: key k counts[k] times, the rest spread over the keys after them"""
    u = np.repeat(np.arange(len(counts)), counts)
    return np.concatenate([u, len(counts) + np.arange(n - len(u)) % 64])


def _sums(rng, n, prev, width):
    t, u, v = _gates(rng, n, prev)
    a = rng.integers(0, prev - width + 1, n)
    t[::2], u[::2], v[::2] = 5, a[::2], a[::2] + width          # u .. v - 1
    t[::8], v[::8] = 12, a[::8] + min(width, 60) - 1             # u .. v, weighted
    return t, u, v


def _layers(case):
    rng = np.random.default_rng(11)
    x = _inputs(rng, 1 << 10)
    if case == "two gates":
        return [x, _gates(rng, 2, 1 << 10), _gates(rng, 2, 2), _gates(rng, 2, 2)]
    if case == "list limits":   # 63, 64, 65 edges; 32768 and 32769
        return [x, _gates(rng, 1 << 17, 1 << 10, _repeat([63, 64, 65, 0, 32768, 32769], 1 << 17)), _gates(rng, 4, 1 << 17)]
    if case == "many split keys":
        return [x, _gates(rng, 1 << 19, 1 << 10, _repeat([40000] * 12, 1 << 19)), _gates(rng, 4, 1 << 19)]
    if case == "sums outgrow the layer":
        return [x, _sums(rng, 1 << 11, 1 << 10, 700), _sums(rng, 1 << 9, 1 << 11, 2), _gates(rng, 2, 1 << 9)]
    return [x, _gates(rng, 1 << 22, 1 << 10), _gates(rng, 1 << 10, 1 << 22), _gates(rng, 2, 1 << 10)]


@pytest.mark.parametrize("case", ["two gates", "list limits", "many split keys", "sums outgrow the layer", "wide keys"])
def test_gathers_equal_scatters(case, monkeypatch):
    layers = _layers(case)
    s = vb.Session(layers)
    try:
        monkeypatch.setenv("VIRGO_PHASE_TABLES", "atomic")
        s.load(layers)
        want = s.prove(5)[1]
        monkeypatch.delenv("VIRGO_PHASE_TABLES")
        for _ in range(2):   # after the scatters, then into the same buffers
            s.load(layers)
            assert s.prove(5)[1] == want
    finally:
        s.close()
