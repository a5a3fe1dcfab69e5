"""A NaN of either sign anywhere in a train is reported, also where it is all
that stands below the diagonal of a bond's only column."""
import numpy as np
import pytest

from oracle import pyoracle as O

pytestmark = pytest.mark.gpu

NANS = {"+nan": np.array([0x7ff8000000000000], np.uint64).view(np.float64)[0],
        "-nan": np.array([0xfff8000000000000], np.uint64).view(np.float64)[0]}


@pytest.mark.parametrize("nan", sorted(NANS))
@pytest.mark.parametrize("sched", ["auto", "per_tt", "whole_gpu"])
@pytest.mark.parametrize("gauge", ["none", "right_canonical"])
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("modes,r", [([4, 5, 3, 4], 1), ([4] * 6, 9), ([4] * 5, 70)])
def test_nan_of_either_sign(ttg, modes, r, prec, gauge, sched, nan):
    for k in range(len(modes)):
        for at in (0, -1):
            x = [c.copy() for c in O.random(modes, r, 7, fan_in_scale=True)]
            x[k][-1, at, -1] = NANS[nan]
            with pytest.raises(ttg.TTGError) as e:
                ttg.round(x, ttg.RoundOptions(eps=1e-8, gauge=ttg.round_gauge[gauge],
                                              precision=ttg.precision[prec],
                                              schedule=ttg.schedule[sched]))
            assert e.value.status == 5, (k, at)
