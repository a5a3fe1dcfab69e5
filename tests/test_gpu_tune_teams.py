"""Tuning a plan of a few FP64 trains can keep the team per train that it
starts with (two to three times as fast as one CTA per train)."""
import pytest

from oracle import pyoracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [2, 3])
def test_tuning_can_keep_the_teams(ttg, count):
    xs = [O.random([4] * 8, 60, 90 + i, fan_in_scale=True) for i in range(count)]
    plan = ttg.Plan("round", xs, opts=ttg.RoundOptions(eps=1e-8))
    plan.upload()
    assert plan.schedule() == "teams"
    assert plan.autotune() == "teams x%d" % count
    assert plan.schedule() == "teams"
