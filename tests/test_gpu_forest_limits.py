"""kd-tree builds of uneven splits (nearly every one cuts a few records off)
at the sizes where the build changes hands, wherever the node limit has room
for any tree: a binary tree over n records has at most 2 n - 1 nodes.  No
error is accepted there; the order is the oracle's, element for element."""
import numpy as np
import pytest

from test_gpu_forest import points

pytestmark = pytest.mark.gpu


def fits(n, leaf):
    return min(1 + 4 * (n // leaf) + 4096, 2 * n + 17) >= 2 * n - 1


CASES = [(dim, leaf, n) for dim, leaf in [(3, 10), (3, 20), (6, 40), (6, 2)]
         for n in [1, 11, 41, 255, 256, 257, 2039, 2047, 2048, 2049, 4097, 20011] if fits(n, leaf)]


@pytest.mark.parametrize("dim,leaf,n", CASES)
def test_uneven_splits(rk, oracle, dim, leaf, n):
    p = points(rk, n, "cusp")
    assert np.array_equal(rk.tree_order(p, dim, leaf)["id"],
                          oracle.tree_order(p, dim, leaf)["id"])

