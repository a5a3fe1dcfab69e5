"""The whole-GPU sweeps' Q that is formed during the next QR: long trains,
steps after it that have no QR (fewer rows than columns, max_rank), bonds that
are cut between kept ones, a next QR too large to share the shared memory, and
the streaming product."""
import numpy as np
import pytest

from oracle import pyoracle as O

pytestmark = pytest.mark.gpu

# Both schedules round to within eps of x, so to within 2 eps of each other, and
# their arithmetic's error is that of the whole-GPU parity tests.
FP64_TOL, MIXED_TOL = 1e-11, 1e-10


@pytest.mark.parametrize("modes,r,s,max_rank", [
    ([4] * 9, 70, 0, 0), ([6] * 8, 17, 0, 0), ([4] * 8, 40, 30, 0), ([3] * 9, 66, 0, 50),
    ([16] * 5, 250, 0, 0), ([2, 40, 2, 2, 40, 2, 40, 2], 90, 0, 0), ([70, 2, 70], 64, 0, 0)])
@pytest.mark.parametrize("gauge", ["none", "right_canonical"])
@pytest.mark.parametrize("prec,tol", [("fp64", FP64_TOL), ("mixed", MIXED_TOL)])
def test_q_formed_during_the_next_qr(ttg, modes, r, s, max_rank, gauge, prec, tol):
    x = O.random(modes, r, 31, fan_in_scale=True)
    if s:  # a middle bond that is cut: a term at 1e-3 eps
        y = O.random(modes, s, 32, fan_in_scale=True)
        y[0] = y[0] * 1e-9
        x = O.add(x, y)
    o = dict(eps=1e-6 if s else 1e-10, max_rank=max_rank, gauge=ttg.round_gauge[gauge],
             precision=ttg.precision[prec])
    y = ttg.round(x, ttg.RoundOptions(schedule=ttg.schedule.whole_gpu, **o))
    z = ttg.round(x, ttg.RoundOptions(schedule=ttg.schedule.per_tt, **o))
    assert O.ranks(y) == O.ranks(z)
    assert O.rel_err(y, z) <= 2 * o["eps"] + tol
    for c in (y[1:] if gauge == "right_canonical" else []):
        m = c.reshape(c.shape[0], -1)
        assert np.max(np.abs(m @ m.T - np.eye(m.shape[0]))) <= tol


@pytest.mark.parametrize("prec,tol", [("fp64", FP64_TOL), ("mixed", MIXED_TOL)])
def test_streaming_product(ttg, prec, tol):
    rng = np.random.default_rng(33)
    d, n, ra, rx = 9, 3, 6, 14
    a = [rng.standard_normal((1 if k == 0 else ra, n, n, 1 if k == d - 1 else ra)) / ra
         for k in range(d)]
    x = O.random([n] * d, rx, 34, fan_in_scale=True)
    o = dict(eps=1e-10, method=ttg.round_method.svd_streaming, precision=ttg.precision[prec])
    y = ttg.matvec_round(a, x, ttg.RoundOptions(schedule=ttg.schedule.whole_gpu, **o))
    z = ttg.matvec_round(a, x, ttg.RoundOptions(schedule=ttg.schedule.per_tt, **o))
    assert O.ranks(y) == O.ranks(z) and O.rel_err(y, z) <= 2 * o["eps"] + tol
