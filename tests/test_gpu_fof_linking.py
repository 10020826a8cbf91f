"""3D FOF with linking lengths that no run is configured with but the call
takes: negative (the reference's searches then find the same leaf points and
never take a node whole) and not a number (they take the whole tree).  The
output is the oracle's, byte for byte, and the call comes back: a run of
dense particles always holds its first one, whatever the reach compares to."""
import numpy as np
import pytest

from test_gpu_fof_ties import R, same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [17, 33, 500, 4097])
def test_negative(rk, oracle, n):
    rng = np.random.default_rng(n)
    same(rk, oracle, 32 + rng.normal(size=(n, 3)) * 0.3, -R)


@pytest.mark.parametrize("seed", range(3))
def test_negative_on_a_lattice(rk, oracle, seed):
    rng = np.random.default_rng(seed)
    same(rk, oracle, 32 + R * rng.integers(0, 4, (700, 3)), -R)


@pytest.mark.parametrize("n", [17, 33, 500])
def test_not_a_number(rk, oracle, n):
    rng = np.random.default_rng(n)
    same(rk, oracle, 32 + rng.normal(size=(n, 3)) * 3, float("nan"))


@pytest.mark.parametrize("link", [float("inf"), 1e30])
def test_unbounded(rk, oracle, link):
    rng = np.random.default_rng(3)
    same(rk, oracle, 32 + rng.normal(size=(500, 3)) * 3, link)
