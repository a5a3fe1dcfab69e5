"""eval_batch with and without product tables: sample counts around the sizes
at which tables appear, uneven modes and ranks, a single core, out-of-range
indices, and trains whose products would leave FP64's range."""
import numpy as np
import pytest

from oracle import pyoracle as O

pytestmark = pytest.mark.gpu

# A value is a sum of products formed in another order: its error is below
# (sum of ranks) u times the same value of the train of absolute entries.
U = 1.2e-16


def _check(ttg, x, idx):
    v = ttg.eval_batch(x, idx)
    ref = O.eval_batch(x, idx)
    size = O.eval_batch([np.abs(c) for c in x], idx)
    terms = sum(c.shape[0] for c in x) + len(x)
    assert np.all(np.abs(v - ref) <= terms * U * size)


@pytest.mark.parametrize("modes,r,m", [
    ([7], 1, 5), ([3, 4], 2, 9), ([4] * 10, 16, 33), ([4] * 10, 16, 3000), ([2] * 24, 33, 20000),
    ([4] * 12, 64, 70000), ([3, 2, 5, 4, 7, 2, 6, 3, 8, 5, 2], 31, 40000), ([8] * 7, 5, 1),
    ([5] * 6, 97, 5000), ([2] * 300, 2, 64)])
def test_eval_against_the_oracle(ttg, modes, r, m):
    x = O.random(modes, r, 3, fan_in_scale=True)
    rng = np.random.default_rng(len(modes) * m)
    idx = np.stack([rng.integers(0, n, m) for n in modes], axis=1).astype(np.int32)
    _check(ttg, x, idx)


def test_eval_tables_keep_range_and_errors(ttg):
    modes = [4] * 12
    rng = np.random.default_rng(5)
    idx = rng.integers(0, 4, (30000, 12)).astype(np.int32)
    x = O.random(modes, 24, 9, fan_in_scale=True)
    # 1e200, 1e200, 1e-200, 1e-200, ...: neighbouring cores' products overflow
    # although every running vector product is finite.
    wild = [c * s for c, s in zip(x, ([1.0, 1e-200, 1e200, 1e200, 1e-200, 1e-200, 1e200] + [1.0] * 5))]
    v, ref = ttg.eval_batch(wild, idx), O.eval_batch(wild, idx)
    assert np.all(np.isfinite(v)) and np.allclose(v, ref, rtol=1e-9, atol=1e-12 * np.abs(ref).max())
    # an infinity in an entry no index asks for stays out of every value
    x[5][:, 3, :] = np.inf
    some = idx[idx[:, 5] != 3]
    assert np.all(np.isfinite(ttg.eval_batch(x, some)))
    bad = idx.copy()
    bad[777, 6] = 4
    with pytest.raises(ttg.TTGError):
        ttg.eval_batch(O.random(modes, 24, 9, fan_in_scale=True), bad)
