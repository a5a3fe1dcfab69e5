"""Where the default schedule of a lone train changes: long trains of small
cores with a few large ones stay on one CTA, whose steps cost no grid barriers."""
import numpy as np
import pytest

from oracle import pyoracle as O

pytestmark = pytest.mark.gpu

FP64_TOL, MIXED_TOL = 1e-11, 1e-10  # as in the parity tests


def _bump(d, n, base, top):
    """Ranks `base`, rising by factors of n to `top` and back in the middle."""
    up = [base]
    while up[-1] < top:
        up.append(min(up[-1] * n, top))
    mid = up[1:] + [top] + up[1:][::-1]
    left = (d - 1 - len(mid)) // 2
    r = [1] + [base] * left + mid + [base] * (d - 1 - left - len(mid)) + [1]
    for k in range(d):
        r[k + 1] = min(r[k + 1], r[k] * n)
    for k in reversed(range(d)):
        r[k] = min(r[k], r[k + 1] * n)
    g = np.random.default_rng(9)
    return [g.standard_normal((r[k], n, r[k + 1])) / (r[k] * n) ** 0.5 for k in range(d)]


@pytest.mark.parametrize("d,n,base,top,fp64,mixed", [
    (60, 8, 2, 18, "per_tt", "per_tt"), (300, 2, 2, 32, "per_tt", "per_tt"),
    (60, 8, 10, 18, "per_tt", "whole_gpu"), (60, 8, 14, 18, "whole_gpu", "whole_gpu"),
    (12, 2, 10, 33, "per_tt", "per_tt")])
def test_schedule_of_a_lone_train(ttg, d, n, base, top, fp64, mixed):
    x = _bump(d, n, base, top)
    for prec, want, tol in (("fp64", fp64, FP64_TOL), ("mixed", mixed, MIXED_TOL)):
        o = ttg.RoundOptions(eps=1e-8, precision=ttg.precision[prec])
        plan = ttg.Plan("round", [x], opts=o)
        assert plan.schedule() == want
        plan.close()
        y, ref = ttg.round(x, o), O.round(x, 1e-8)
        assert O.ranks(y) == O.ranks(ref) and O.rel_err(y, ref) <= tol
