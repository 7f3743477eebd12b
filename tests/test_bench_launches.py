"""The bench's kernel count per step attempt on the mixed path against the integrator's stage
schedule (record_step in ceda_demonstrations_gb300/csrc/lsrk.cu): stage 1, then stages 2..s
in groups of ks (a shorter last group; a last group of one stage is a single-stage launch),
then the step end."""
import os
import sys

import pytest

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import bench  # noqa: E402


def schedule(s, ks):
    launches, j = 2, 2  # stage 1 and the step end
    while j <= s:
        g = min(ks, s - j + 1)
        launches += 1
        j += g if g >= 2 else 1
    return launches


@pytest.mark.parametrize("ks", [1, 2, 3, 4])
def test_step_launches_follow_the_stage_schedule(ks):
    for s in range(2, 201):
        want = s + 1 if ks == 1 else schedule(s, ks)
        assert bench.step_launches(s, ks) == want, (s, ks)
    assert bench.step_launches(196, 4) == 51  # the 8192^2 workload's steps


def test_step_launches_with_groups_of_eight():
    """Groups of eight while eight stages remain, then groups of four, a last single stage alone."""
    for s in range(2, 201):
        launches, j = 2, 2
        while j <= s:
            left = s - j + 1
            j += 8 if left >= 8 else min(4, left)
            launches += 1
        assert bench.step_launches(s, 8) == launches, s
