"""A call that is refused for want of memory leaves nothing for the next one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_next_call_after_out_of_memory(ttg):
    # One core of 8 x 120 000 x 8: its work matrices of (8 n)^2 entries would take
    # 15 TB, which the allocation refuses at once.
    g = np.random.default_rng(1)
    x = [g.standard_normal(s) for s in ((1, 8, 8), (8, 120000, 8), (8, 8, 1))]
    with pytest.raises(ttg.TTGError) as e:
        ttg.round(x, ttg.RoundOptions(eps=1e-8, schedule=ttg.schedule.per_tt))
    assert e.value.status == 8  # TTG_ERR_OOM
    y = [c[:, :3, :] for c in x]
    assert len(ttg.soft_threshold(y, 1e-3)) == 3
    from tensor_train_gb300.mlp import RankModel
    assert RankModel(4, 16).forward(np.zeros((2, 4), np.float32)).shape == (2,)
