"""The per-TT sweep's blocked FP64 Householder routines at their edges: ranks
around the 16-reflector blocks, matrices in shared memory, staged by panels
and too tall for either, more columns than rows, truncated bonds (Q applied
instead of formed); and the df64 Jacobi sweeps of truncated bonds."""
import numpy as np
import pytest

from oracle import pyoracle as O

pytestmark = pytest.mark.gpu

# As in the parity tests.
FP64_TOL, MIXED_TOL = 1e-11, 1e-10


@pytest.mark.parametrize("modes,r,s", [
    ([2], 1, 0), ([3, 2], 2, 1), ([4] * 5, 1, 0), ([4] * 5, 15, 0), ([4] * 6, 16, 0),
    ([4] * 6, 17, 0), ([4] * 6, 31, 2), ([9] * 4, 48, 33), ([2] * 14, 40, 24), ([8] * 5, 60, 40),
    ([7, 130, 5], 33, 0), ([3, 1900, 4, 3], 9, 3)])
@pytest.mark.parametrize("gauge", ["none", "right_canonical"])
def test_cta_qr_edges(ttg, modes, r, s, gauge):
    x = O.random(modes, r, 31, fan_in_scale=True)
    if s:
        x = O.add(x, O.random(modes, s, 32, fan_in_scale=True))
    o = dict(eps=1e-8, gauge=ttg.round_gauge[gauge], schedule=ttg.schedule.per_tt)
    y = ttg.round(x, ttg.RoundOptions(**o))
    ref = O.round(x, 1e-8, gauge=gauge)
    assert O.ranks(y) == O.ranks(ref)
    assert O.rel_err(y, ref) <= FP64_TOL
    if gauge == "right_canonical":
        for c in y[1:]:
            m = c.reshape(c.shape[0], -1)
            assert np.max(np.abs(m @ m.T - np.eye(m.shape[0]))) <= FP64_TOL


@pytest.mark.parametrize("r,n,d,cap", [(5, 3, 6, 0), (16, 4, 6, 0), (33, 4, 6, 0), (48, 4, 6, 40),
                                       (70, 5, 5, 0)])
def test_truncated_bonds_in_both_precisions(ttg, r, n, d, cap):
    # x + update in x's own bond spaces: every bond is cut to half (or to cap),
    # so the SVD, its polish sweeps and the application of Q decide the result.
    x = O.random([n] * d, r, 41, fan_in_scale=True)
    u = [np.array(c) for c in x]
    u[0] = 1e-2 * O.random([n] * d, r, 42, fan_in_scale=True)[0]
    t = O.add(x, u)
    ref = O.round(t, 1e-9, cap)
    for prec, tol in (("fp64", FP64_TOL), ("mixed", MIXED_TOL)):
        y = ttg.round(t, ttg.RoundOptions(eps=1e-9, max_rank=cap, precision=ttg.precision[prec],
                                          schedule=ttg.schedule.per_tt))
        assert O.ranks(y) == O.ranks(ref)
        assert O.rel_err(y, ref) <= tol
