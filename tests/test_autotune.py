"""The plans that the autotuner compares with the engine's own choice."""
import pytest


@pytest.mark.parametrize("b", [1, 4, 5, 32, 33, 64, 65, 100, 128, 1024])
def test_candidates_cover_what_the_engine_chooses_from(b):
    from altopir_b200 import autotune
    plans = autotune.candidates(b)
    limb_cols = 4 * ((b + 3) // 4 * 4)
    assert len(set(plans)) == len(plans) and (0, -1, 0, 0) in plans
    pair = [p for p in plans if p[0] == 1]
    assert bool(pair) == (limb_cols > 16)
    # wide units, and the split by rounds for both kinds of units, from the first batch that can take them
    above = limb_cols > 256
    assert ((1, 1, 256, 0) in plans) == above and ((1, 0, 256, 0) in plans) == above
    assert any(p[1] == 1 for p in plans) == above and any(p[3] == 0 for p in pair) == above
