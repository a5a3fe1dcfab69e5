"""inner and norm over the grid: ranks at the edges of the 16 x 16 tiles,
sliced and unsliced inner dimensions, more tiles than CTAs, a single core."""
import numpy as np
import pytest

from oracle import pyoracle as O

pytestmark = pytest.mark.gpu

# FP64 chains: every entry of an environment is a sum of at most n r terms,
# so a chain's error is below d (n r) u times the norms' product.
U = 1.2e-16


@pytest.mark.parametrize("modes,ra,rb", [
    ([5], 1, 1), ([3, 4], 1, 2), ([4] * 5, 15, 16), ([4] * 5, 17, 33), ([2, 7, 3, 5, 2, 6], 31, 9),
    ([3] * 9, 96, 64), ([8, 8, 8, 8], 64, 200), ([6] * 6, 130, 131)])
def test_inner_edges(ttg, modes, ra, rb):
    a, b = O.random(modes, ra, 7, fan_in_scale=True), O.random(modes, rb, 8, fan_in_scale=True)
    na, nb = O.norm(a), O.norm(b)
    terms = max(modes) * max(max(O.ranks(a)), max(O.ranks(b)))
    tol = len(modes) * terms * U
    assert abs(ttg.inner(a, b) - O.inner(a, b)) <= tol * na * nb
    assert abs(ttg.norm(a) - na) <= tol * na
    assert ttg.inner(a, b) == ttg.inner(a, b)
