"""Proofs whose launch sequences are being captured while another thread makes
and closes sessions, each the last one of its circuit: every proof is made and
is the one made alone."""
import threading

import pytest

import virgo_b200 as vb
from virgo_b200 import circuits

pytestmark = pytest.mark.gpu


def _disturbed(disturb, rounds):
    """`rounds` new sessions in each of three threads, three proofs each (the
    second captures), while a fourth thread calls disturb() over and over."""
    layers = [circuits.random_layered([12, 13, 11], seed=k) for k in range(3)]
    want = []
    for l in layers:
        s = vb.Session(l)
        want.append([s.prove(k)[1] for k in range(3)])
        s.close()
    errors, captures, stop = [], [], threading.Event()

    def prove(i):
        try:
            for _ in range(rounds):
                s = vb.Session(layers[i])
                try:
                    for k in range(3):
                        st, blob = s.prove(k)
                        captures.append(st.graph_captures)
                        if blob != want[i][k]:
                            errors.append("another proof")
                finally:
                    s.close()
        except Exception as e:  # noqa: BLE001
            errors.append(repr(e))

    def other():
        while not stop.is_set():
            disturb()

    threads = [threading.Thread(target=prove, args=(i,)) for i in range(3)]
    back = threading.Thread(target=other)
    back.start()
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    stop.set()
    back.join()
    assert not errors, errors[:3]
    return captures


def test_proofs_beside_sessions_that_close():
    small = circuits.random_layered([6, 5], seed=9)

    def come_and_go():
        s = vb.Session(small)
        s.close()

    captures = _disturbed(come_and_go, 12)
    assert sum(captures) > 0
