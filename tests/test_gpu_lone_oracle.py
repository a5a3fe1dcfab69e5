"""The default schedule of a lone medium train and of a few FP64 ones against
the oracle, where nothing is cut off and only rounding separates the two."""
import numpy as np
import pytest

from oracle import pyoracle as O

pytestmark = pytest.mark.gpu

# As in the whole-GPU parity tests.
FP64_TOL, MIXED_TOL = 1e-11, 1e-10


@pytest.mark.parametrize("modes,r,gauge", [
    ([4] * 7, 22, "none"), ([4] * 7, 23, "none"), ([4] * 7, 23, "right_canonical"),
    ([2] * 12, 33, "none"), ([20, 3, 20, 2], 40, "none"), ([5, 3, 7, 4, 6], 63, "right_canonical")])
@pytest.mark.parametrize("prec,tol", [("fp64", FP64_TOL), ("mixed", MIXED_TOL)])
def test_lone_train(ttg, modes, r, gauge, prec, tol):
    x = O.random(modes, r, 41, fan_in_scale=True)
    y = ttg.round(x, ttg.RoundOptions(eps=1e-8, gauge=ttg.round_gauge[gauge],
                                      precision=ttg.precision[prec]))
    ref = O.round(x, 1e-8, gauge=gauge)
    assert O.ranks(y) == O.ranks(ref) and O.rel_err(y, ref) <= tol


@pytest.mark.parametrize("count,rmin,rmax", [(2, 40, 60), (3, 20, 112), (30, 23, 50), (31, 30, 40)])
def test_few_trains(ttg, count, rmin, rmax):
    rng = np.random.default_rng(44)
    xs = [O.random([int(v) for v in rng.integers(3, 9, int(rng.integers(4, 8)))],
                   rmin + i % (rmax - rmin + 1) if i else rmax, 60 + i, fan_in_scale=True)
          for i in range(count)]
    for x, y in zip(xs, ttg.round_batch(xs, ttg.RoundOptions(eps=1e-8))):
        ref = O.round(x, 1e-8)
        assert O.ranks(y) == O.ranks(ref) and O.rel_err(y, ref) <= FP64_TOL
