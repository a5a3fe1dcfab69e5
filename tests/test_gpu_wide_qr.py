"""The blocked QR of the whole-GPU schedule at its edges: ranks around its
16-reflector blocks, panels of one slab and of 32, more columns than rows,
square and very tall unfoldings, both gauges and precisions, and teams."""
import numpy as np
import pytest

from oracle import pyoracle as O

pytestmark = pytest.mark.gpu

# As in the whole-GPU parity tests.
FP64_TOL, MIXED_TOL = 1e-11, 1e-10


def _sum_of(modes, r, s):
    a = O.random(modes, r, 21, fan_in_scale=True)
    return O.add(a, O.random(modes, s, 22, fan_in_scale=True)) if s else a


@pytest.mark.parametrize("modes,r,s", [
    ([4] * 5, 1, 0), ([4] * 5, 15, 0), ([4] * 5, 16, 0), ([4] * 5, 9, 8), ([5] * 5, 33, 0),
    ([9] * 4, 81, 0), ([2] * 12, 40, 24), ([64, 3, 65], 40, 0), ([3, 4100, 2, 3], 6, 3),
    ([7, 6, 5, 6, 7], 42, 30)])
@pytest.mark.parametrize("gauge", ["none", "right_canonical"])
def test_blocked_qr_edges(ttg, modes, r, s, gauge):
    x = _sum_of(modes, r, s)
    for prec, tol in (("fp64", FP64_TOL), ("mixed", MIXED_TOL)):
        y = ttg.round(x, ttg.RoundOptions(eps=1e-8, gauge=ttg.round_gauge[gauge],
                                          precision=ttg.precision[prec],
                                          schedule=ttg.schedule.whole_gpu))
        ref = O.round(x, 1e-8) if gauge == "none" else O.round(x, 1e-8, gauge="right_canonical")
        assert O.ranks(y) == O.ranks(ref)
        assert O.rel_err(y, ref) <= tol
        for c in (y[1:] if gauge == "right_canonical" else []):
            m = c.reshape(c.shape[0], -1)
            assert np.max(np.abs(m @ m.T - np.eye(m.shape[0]))) <= tol


def test_blocked_qr_in_teams(ttg):
    tts = [O.random([4, 6, 5, 6, 4], 24 + 5 * i, 60 + i, fan_in_scale=True) for i in range(9)]
    ys = ttg.round_batch(tts, ttg.RoundOptions(eps=1e-8, schedule=ttg.schedule.teams))
    for x, y in zip(tts, ys):
        ref = O.round(x, 1e-8)
        assert O.ranks(y) == O.ranks(ref) and O.rel_err(y, ref) <= FP64_TOL


def test_near_threshold_bonds_keep_the_elimination(ttg):
    # A smallest singular value between eps and the inverse test's reach: the
    # bond must come out as before, whatever test decides it.
    x = O.random([8] * 5, 40, 77, fan_in_scale=True)
    scale = np.ones(40)
    scale[-1] = 1e-7
    x[2] = x[2] * scale[None, None, :]
    for prec in ("fp64", "mixed"):
        o = dict(eps=1e-12, precision=ttg.precision[prec])
        y = ttg.round(x, ttg.RoundOptions(schedule=ttg.schedule.whole_gpu, **o))
        z = ttg.round(x, ttg.RoundOptions(schedule=ttg.schedule.per_tt, **o))
        assert O.ranks(y) == O.ranks(z) == O.ranks(O.round(x, 1e-12))
        assert O.rel_err(y, z) <= MIXED_TOL
