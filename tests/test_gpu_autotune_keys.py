"""The autotuner proves nothing for the keys that are accepted without effect:
their values have one time, the settings in force stay."""
import pytest

import virgo_b200 as vb
from virgo_b200 import circuits

pytestmark = pytest.mark.gpu


def test_keys_without_effect_are_not_timed():
    s = vb.Session(circuits.random_layered([8, 7], seed=3))
    try:
        vb.tune_reset(0)
        vb.tune_set(0, group_split=1)
        chosen, trials = vb.autotune([s], seed=2, reps=1)
        for key, kept in (("group_split", 1), ("lazy_fold", 0)):
            mine = [t for t in trials if t[0] == key]
            assert sorted(t[1] for t in mine) == [0, 1]
            assert mine[0][2] == mine[1][2] > 0
            assert [t[1] for t in mine if t[3]] == [kept] and chosen[key] == kept
    finally:
        vb.tune_reset(0)
        s.close()
