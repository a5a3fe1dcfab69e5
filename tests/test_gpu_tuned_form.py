"""A tuned mixed plan rounds as the untuned one: which form a df64
factorisation takes does not depend on the CTAs per SM."""
import numpy as np
import pytest

from oracle import pyoracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count,modes,r", [(460, [8] * 6, 96), (310, [16] * 4, 80)])
def test_tuned_mixed_plan_is_bit_equal(ttg, count, modes, r):
    # tallest panels: 768 rows (beyond 38 KB of staging), 1280 (beyond 56 KB)
    base = [O.random(modes, r, 80 + i, fan_in_scale=True) for i in range(8)]
    xs = [[c * (1.0 + 1e-3 * i) for c in base[i % 8]] for i in range(count)]
    plan = ttg.Plan("round", xs, opts=ttg.RoundOptions(eps=1e-3, max_rank=r // 2,
                                                       precision=ttg.precision.mixed))
    plan.upload()
    plan.run()
    want = plan.download()
    plan.autotune()
    plan.run()
    for a, b in zip(want, plan.download()):
        assert all(np.array_equal(p, q) for p, q in zip(a, b))
