"""Candidates of the launch-shape tuner (CPU: nothing is timed)."""
import pytest

from heterogeneous_mhd_gb300 import autotune


@pytest.mark.parametrize("n", [32, 48, 64, 96, 128, 192, 256, 512])
def test_the_planners_own_choice_is_a_candidate(n):
    """What tune() keeps is never slower than no tuning: the planner may run a kernel that the
    knobs' candidates leave out (the warp-per-pencil one for 32, 96 and 192 cells)."""
    fx, adv = autotune.candidates(n)
    assert {} in adv and len(fx) >= 3
    assert autotune.batch_candidates(n)[0] == {}
