"""kd-tree builds at the sizes where the build changes hands: trees of one
leaf, the two classes of block-built subtrees (256 and 2,048 records) and
their neighbours, and a small leaf size, whose tables bound the subtree
instead.  The permutation must be the oracle's element for element (the
boxes, node links and limits decide it, so they are checked with it)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def points(rk, n, kind):
    rng = np.random.default_rng(1000 + n)
    p = np.zeros(n, rk.PARTICLE)
    p["id"] = np.arange(n)
    if kind == "uniform":
        p["pos"] = rng.random((n, 6))
    elif kind == "cusp":  # nearly every split cuts a few records off
        p["pos"] = rng.choice([-1.0, 1.0], (n, 6)) * rng.random((n, 6)) ** 8
    else:  # repeated values, a run of coincident records
        p["pos"] = rng.integers(0, 3, (n, 6))
        p["pos"][n // 3: n // 2] = -0.0
    return p


@pytest.mark.parametrize("kind", ["uniform", "cusp", "ties"])
@pytest.mark.parametrize("dim,leaf", [(3, 10), (3, 20), (6, 40), (6, 2)])
@pytest.mark.parametrize("n", [1, 11, 41, 255, 256, 257, 2047, 2048, 2049, 4097, 20011])
def test_tree_order_at_class_edges(rk, oracle, kind, dim, leaf, n):
    p = points(rk, n, kind)
    try:
        got = rk.tree_order(p, dim, leaf)
    except rk.RockstarError as e:
        # many records cut off one at a time: the build's stated node limit
        assert e.code == -4 and "node capacity" in str(e) and kind == "cusp"
        return
    assert np.array_equal(got["id"], oracle.tree_order(p, dim, leaf)["id"])
