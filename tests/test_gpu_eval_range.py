"""eval_batch of trains whose left-to-right products stay in FP64's range
while products of their last sites alone leave it: the values are those of
the left-to-right order, with few indices and with many."""
import numpy as np
import pytest

from oracle import pyoracle as O

pytestmark = pytest.mark.gpu

U = 1.2e-16  # as in test_gpu_eval_tables


def _indices(modes, m):
    rng = np.random.default_rng(m)
    return np.stack([rng.integers(0, n, m) for n in modes], axis=1).astype(np.int32)


def _check(ttg, x, idx):
    v = ttg.eval_batch(x, idx)
    ref = O.eval_batch(x, idx)
    size = O.eval_batch([np.abs(c) for c in x], idx)
    terms = sum(c.shape[0] for c in x) + len(x)
    assert np.all(np.isfinite(ref)) and np.any(ref != 0)
    assert np.all(np.abs(v - ref) <= terms * U * size)


# Powers of ten that the sites carry; every running product from the left
# stays in 1e+-300.
LATE = [
    ([4] * 8, [250, 0, 0, 0, -100, -100, -100, -100]),
    ([4] * 8, [-250, 0, 0, 0, 100, 100, 100, 100]),
    ([4] * 10, [0, 0, 0, 150, 150, 0, 0, 0, -170, -170]),
    ([4] * 10, [0, 0, 0, -150, -150, 0, 0, 0, 170, 170]),
    ([3, 5, 2, 7, 4, 3, 6, 2, 5, 3, 4, 2], [0, 120, 120, 0, 0, 0, -90, -90, -90, -90, 0, 90]),
    ([2] * 40, [-280] + [0] * 19 + [30] * 18 + [0] * 2),
    ([4] * 12, [0, 0, -150, 150, 150, 150, 0, -250, 0, 0, 0, 0]),
]


@pytest.mark.parametrize("modes,scales", LATE)
@pytest.mark.parametrize("r", [1, 7, 40])
@pytest.mark.parametrize("m", [1, 33, 30000, 70000])
def test_sites_out_of_range_among_themselves(ttg, modes, scales, r, m):
    x = [c * 10.0 ** s for c, s in zip(O.random(modes, r, 3, fan_in_scale=True), scales)]
    _check(ttg, x, _indices(modes, m))


@pytest.mark.parametrize("m", [1, 33, 30000, 70000])
def test_one_term_of_a_sum_out_of_range(ttg, m):
    # Block-diagonal cores: the largest entries of the last sites belong to
    # the other term, so their products stay near one.
    modes = [4] * 8
    a = O.random(modes, 5, 3, fan_in_scale=True)
    b = [c * 10.0 ** s for c, s in zip(O.random(modes, 6, 4, fan_in_scale=True),
                                       [200, 0, 0, 0, -170, 0, -170, 130])]
    a[0] = a[0] * 0.0
    _check(ttg, O.add(a, b), _indices(modes, m))


@pytest.mark.parametrize("m", [33, 70000])
def test_exact_zeros_and_infinities(ttg, m):
    modes = [4] * 10
    idx = _indices(modes, m)
    x = O.random(modes, 6, 3, fan_in_scale=True)
    for c in x[1:-1]:
        c[:, 1, :] = 0.0
    _check(ttg, x, idx)
    x[7][2, 3, 1] = np.inf
    v, ref = ttg.eval_batch(x, idx), O.eval_batch(x, idx)
    assert np.array_equal(np.isnan(v), np.isnan(ref))
    assert np.array_equal(np.where(np.isinf(ref), ref, 0), np.where(np.isinf(v), v, 0))


def test_a_value_alone_and_among_others(ttg):
    modes, scales = LATE[0]
    x = [c * 10.0 ** s for c, s in zip(O.random(modes, 7, 3, fan_in_scale=True), scales)]
    idx = _indices(modes, 3000)
    v = ttg.eval_batch(x, idx)
    for i in (0, 17, 2999):
        assert ttg.eval_batch(x, idx[i:i + 1])[0] == v[i]
