"""FP64 per-TT sweeps of narrow unfoldings on both sides of the lines where the
blocked Householder routines give way to the unblocked ones (3, 12 and 16
columns; 40 and 80 rows a column), single columns and copies of few columns."""
import numpy as np
import pytest

from oracle import pyoracle as O

pytestmark = pytest.mark.gpu

FP64_TOL, MIXED_TOL = 1e-11, 1e-10  # as in the parity tests


@pytest.mark.parametrize("n,r", [(2, 1), (5000, 1), (3, 2), (600, 2), (40, 3), (41, 3), (40, 8),
                                 (41, 8), (40, 11), (41, 11), (80, 12), (81, 12), (80, 15), (81, 15),
                                 (81, 16)])
@pytest.mark.parametrize("gauge", ["none", "right_canonical"])
def test_narrow_unfoldings(ttg, n, r, gauge):
    a = O.random([n] * 4, r, 71, fan_in_scale=True)
    u = [np.array(c) for c in a]
    u[0] = 1e-2 * O.random([n] * 4, r, 72, fan_in_scale=True)[0]
    # Bonds of rank r as they are, and of rank 2 r cut back to r.
    for x in (a, O.add(a, u)):
        ref = O.round(x, 1e-8, gauge=gauge)
        for prec, tol in (("fp64", FP64_TOL), ("mixed", MIXED_TOL)):
            y = ttg.round(x, ttg.RoundOptions(eps=1e-8, gauge=ttg.round_gauge[gauge],
                                              precision=ttg.precision[prec],
                                              schedule=ttg.schedule.per_tt))
            assert O.ranks(y) == O.ranks(ref)
            assert O.rel_err(y, ref) <= tol
