"""What large calls leave allocated: an evaluation's buffers and the work buffers
of sweeps over several CTAs are kept to 1 GiB on the device."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KEPT = 1 << 30
SLACK = 64 << 20  # contexts, modules, allocation granularity


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _train(modes, ranks):
    r = [1] + ranks + [1]
    g = np.random.default_rng(3)
    return [g.standard_normal((r[k], n, r[k + 1])) for k, n in enumerate(modes)]


def test_evaluation_gives_its_buffers_back(ttg):
    x = _train([3, 4], [2])
    ttg.eval_batch(x, np.zeros((4, 2), np.int32))
    before = _free()
    idx = np.zeros((1 << 27, 2), np.int32)  # 1 GiB up, 1 GiB down
    idx[-1] = (2, 3)
    v = ttg.eval_batch(x, idx)
    assert abs(v[-1] - float(x[0][0, 2] @ x[1][:, 3, 0])) <= 1e-15 * np.abs(x[0]).max() * 8
    assert before - _free() <= KEPT + SLACK


def test_team_sweeps_give_their_work_buffers_back(ttg):
    xs = [_train([128, 64, 128], [128, 128])] * 32  # 1 M doubles in each middle core
    before = _free()
    plan = ttg.Plan("round", xs, opts=ttg.RoundOptions(eps=1e-8, schedule=ttg.schedule.per_tt))
    rest = before - _free()  # all that a call takes beside the work buffers
    plan.close()
    assert before - _free() <= SLACK
    ttg.round_batch(xs, ttg.RoundOptions(eps=1e-8, schedule=ttg.schedule.teams))
    assert before - _free() <= rest + KEPT + SLACK
