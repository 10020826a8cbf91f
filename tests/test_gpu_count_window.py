"""The neighbour counts that make a particle dense (more than 16 in its sphere):
17 are looked for first among the 32 particles on either side in tree order.
Clumps of 15 to 20 particles, closer than the linking length or spread over
it, put counts on both sides of the limit, within a window and across several;
the particle counts put the window at the ends of the array and of a block.
rockstar()'s output is compared with the oracle byte for byte."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spread", [0.2, 0.55])
@pytest.mark.parametrize("n", [1, 16, 17, 18, 33, 127, 128, 129, 161, 1000, 20011])
def test_dense_limit(rk, oracle, n, spread):
    rng = np.random.default_rng(n)
    box = 10.0 * n ** (1 / 3)
    c = rk.Config(box_size=box, particle_mass=0.0, total_particles=n)
    st = rk.setup_config(c)
    link = st.avg_particle_spacing * st.fof_linking_length
    clump = np.repeat(np.arange(n), rng.integers(15, 21, n))[:n]
    p = np.zeros(n, rk.PARTICLE)
    p["id"] = np.arange(n)
    p["pos"][:, :3] = rng.random((n, 3))[clump] * box + \
        (rng.random((n, 3)) - 0.5) * 2 * spread * link
    p["pos"][:, 3:] = rng.normal(size=(n, 3)) * 100
    rng.shuffle(p["pos"])
    c.particle_mass = float(st.particle_mass)
    oracle.setup(c)
    ro, roff, rsz = oracle.fof(p)
    g, off, sz = rk.rockstar_fof(p, c)
    assert g.tobytes() == ro.tobytes()
    assert np.array_equal(off, roff) and np.array_equal(sz, rsz)
