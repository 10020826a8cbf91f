"""3D FOF with whole tree nodes at exactly the linking length of the dense
particles: the reference takes a node whole when its far corner is at r, so
the points of a child that starts there belong to the sphere too.  Coincident
positions on lattices whose step divides r exactly; rockstar()'s output
against the oracle, byte for byte."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

R = 0.25  # the linking length: a quarter of the mean spacing of 1, exact in float


def same(rk, oracle, x, link=R):
    rng = np.random.default_rng(len(x))
    c = rk.Config(box_size=64.0, particle_mass=0.0, total_particles=64 ** 3)
    c.particle_mass = float(rk.setup_config(c).particle_mass)
    c.fof_linking_length = link
    p = np.zeros(len(x), rk.PARTICLE)
    p["id"] = np.arange(len(x))
    p["pos"][:, :3] = x
    p["pos"][:, 3:] = rng.normal(size=(len(x), 3)) * 100
    oracle.setup(c)
    ro, roff, rsz = oracle.fof(p)
    g, off, sz = rk.rockstar_fof(p, c)
    assert g.tobytes() == ro.tobytes()
    assert np.array_equal(off, roff) and np.array_equal(sz, rsz)
    return roff, rsz


def test_two_sites_at_the_linking_length(rk, oracle):
    """40 particles at one site, 40 at r from it, 12 at 1.9 r from the second
    site only: two groups, for the second site's particles are skipped by
    the first's and do not link the 12."""
    x = np.full((92, 3), 32.0)
    x[40:, 0] += R
    x[80:, 1] -= 1.9 * R
    _, sz = same(rk, oracle, x)
    assert sorted(sz) == [12, 80]


@pytest.mark.parametrize("seed", range(12))
def test_lattice_of_step_r(rk, oracle, seed):
    rng = np.random.default_rng(seed)
    n, k = int(rng.integers(300, 2000)), int(rng.integers(3, 6))
    same(rk, oracle, 32 + R * rng.integers(0, k, (n, 3)))


@pytest.mark.parametrize("seed", range(12))
@pytest.mark.parametrize("step", [0.125, 0.0625])
def test_clump_on_a_lattice(rk, oracle, seed, step):
    rng = np.random.default_rng(100 + seed)
    n = int(rng.integers(2700, 3200))
    same(rk, oracle, np.round((rng.normal(size=(n, 3)) * 0.3 + 32) / step) * step)


@pytest.mark.parametrize("n,sites", [(17, 1), (40, 1), (300, 5), (3000, 40)])
def test_linking_length_of_zero(rk, oracle, n, sites):
    """Only coincident positions link, through the node shortcut alone."""
    rng = np.random.default_rng(n)
    same(rk, oracle, rng.integers(0, 8, (sites, 3))[rng.integers(0, sites, n)] + 20.0, 0.0)
