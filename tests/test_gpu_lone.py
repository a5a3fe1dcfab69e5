"""A lone medium train (spread over part of the GPU from 2048 doubles per core
on) and a few FP64 ones (a team of CTAs each) in the default schedule, against
one CTA per train."""
import threading

import numpy as np
import pytest

from oracle import pyoracle as O

pytestmark = pytest.mark.gpu

# As in the whole-GPU parity tests, on top of the two roundings' own eps.
FP64_TOL, MIXED_TOL = 1e-11, 1e-10


@pytest.mark.parametrize("modes,r,gauge", [
    ([4] * 7, 22, "none"), ([4] * 7, 23, "none"), ([4] * 7, 23, "right_canonical"),
    ([2] * 12, 33, "none"), ([20, 3, 20, 2], 40, "none"), ([5, 3, 7, 4, 6], 63, "right_canonical")])
@pytest.mark.parametrize("prec,tol", [("fp64", FP64_TOL), ("mixed", MIXED_TOL)])
@pytest.mark.parametrize("cut", [False, True])
def test_lone_train(ttg, modes, r, gauge, prec, tol, cut):
    x = O.random(modes, r, 41, fan_in_scale=True)
    o = dict(eps=1e-8, max_rank=r // 2 if cut else 0, gauge=ttg.round_gauge[gauge],
             precision=ttg.precision[prec])
    y = ttg.round(x, ttg.RoundOptions(**o))
    z = ttg.round(x, ttg.RoundOptions(schedule=ttg.schedule.per_tt, **o))
    assert O.ranks(y) == O.ranks(z)
    assert O.rel_err(y, z) <= 2 * o["eps"] + tol


@pytest.mark.parametrize("count,rmin,rmax,cut", [
    (2, 40, 60, 0), (3, 20, 112, 0), (7, 30, 112, 25), (30, 23, 50, 20), (31, 30, 40, 0)])
def test_few_trains(ttg, count, rmin, rmax, cut):
    rng = np.random.default_rng(44)
    xs = [O.random([int(v) for v in rng.integers(3, 9, int(rng.integers(4, 8)))],
                   rmin + i % (rmax - rmin + 1) if i else rmax, 60 + i, fan_in_scale=True)
          for i in range(count)]
    o = dict(eps=1e-8, max_rank=cut)
    ys = ttg.round_batch(xs, ttg.RoundOptions(**o))
    zs = ttg.round_batch(xs, ttg.RoundOptions(schedule=ttg.schedule.per_tt, **o))
    for y, z in zip(ys, zs):
        assert O.ranks(y) == O.ranks(z)
        assert O.rel_err(y, z) <= 2 * o["eps"] + FP64_TOL


def test_lone_trains_in_threads(ttg):
    xs = [O.random([4] * 6, 30 + i, 50 + i, fan_in_scale=True) for i in range(6)]
    want = [ttg.round(x, ttg.RoundOptions(eps=1e-8)) for x in xs]
    got = [None] * len(xs)

    def call(i):
        got[i] = ttg.round(xs[i], ttg.RoundOptions(eps=1e-8))
    ts = [threading.Thread(target=call, args=(i,)) for i in range(len(xs))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for a, b in zip(want, got):
        assert all(np.array_equal(p, q) for p, q in zip(a, b))
