"""A proof file holds the proof and nothing else of the process: the same bytes
whatever the sessions before it left in the buffers, zeros in the places that a
record or a path does not use."""
import numpy as np
import pytest

import virgo_b200 as vb
from virgo_b200 import circuits

pytestmark = pytest.mark.gpu


def _file(s, seed, path):
    s.prove(seed)
    s.write_proof(str(path))
    return path.read_bytes()


def test_proof_files_are_the_proof_alone(tmp_path):
    small, large = circuits.random_layered([9, 11, 8], seed=2), circuits.random_layered([16, 12, 17, 9], seed=4)
    s = vb.Session(small)
    try:
        first = _file(s, 7, tmp_path / "a")
        s.load(large)   # other records, deeper paths, into the same buffers
        _file(s, 8, tmp_path / "b")
        s.load(small)
        assert _file(s, 7, tmp_path / "c") == first
    finally:
        s.close()
    i32 = lambda o: int.from_bytes(first[o:o + 4], "little")  # noqa: E731
    depth = i32(12)
    bl = [i32(16 + 4 * i) for i in range(depth)]
    o = 16 + 4 * depth
    nrec, levels, nq, n_final = i32(o), i32(o + 4), i32(o + 8), int.from_bytes(first[o + 12:o + 20], "little")
    rec = np.frombuffer(first, np.uint64, 18 * nrec, o + 24).reshape(nrec, 18)
    last = np.cumsum([0] + [bl[i - 1] for i in range(depth - 1, 0, -1) for _ in range(2)])[1:]
    assert last[-1] == nrec - 1
    inner = np.setdiff1d(np.arange(1, nrec), last)
    assert not rec[0, 2:].any() and not rec[inner, 6:].any()
    # set everywhere but in the relay layer's second phase, whose tables are zero
    assert rec[inner[inner < nrec - bl[0]], :6].any(1).all() and rec[last[:-1], 6:].any(1).all()
    which = np.frombuffer(first, np.int32, nq, o + 24 + 144 * nrec + 32 * (2 + levels) + 66 * 16 + 16 * levels + 65 * 16 * n_final)
    paths = np.frombuffer(first, np.uint8, nq * 1024, len(first) - nq * 1024).reshape(nq, 32, 32)
    for q, w in enumerate(which):
        used = (bl[0] - 2 if w < 2 else bl[0] - (w - 2) - 3) + 1
        assert paths[q, :used].any(1).all() and not paths[q, used:].any(), q
