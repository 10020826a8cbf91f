"""The partition sort by union-find label at the sizes where it changes hands
(one block up to 256 and up to 2,048 elements, rounds over all elements
above): clumps and loose particles in a count at each edge.  rockstar()'s
output is the sorted particles, compared with the oracle byte for byte."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3, 64, 255, 256, 257, 1000, 2047, 2048, 2049, 4500, 30011])
@pytest.mark.parametrize("mean", [3, 60])
def test_sorted_by_label_at_class_edges(rk, oracle, n, mean):
    rng = np.random.default_rng(n * 7 + mean)
    box = 10.0 * n ** (1 / 3)
    c = rk.Config(box_size=box, particle_mass=0.0, total_particles=n)
    st = rk.setup_config(c)
    link = st.avg_particle_spacing * st.fof_linking_length
    p = np.zeros(n, rk.PARTICLE)
    p["id"] = np.arange(n)
    clump = np.sort(rng.integers(0, max(1, n // mean), n))
    p["pos"][:, :3] = rng.random((n, 3))[clump] * box + rng.normal(size=(n, 3)) * 0.3 * link
    p["pos"][:, 3:] = rng.normal(size=(n, 3)) * 100
    rng.shuffle(p["pos"])
    c.particle_mass = float(st.particle_mass)
    oracle.setup(c)
    ro, roff, rsz = oracle.fof(p)
    g, off, sz = rk.rockstar_fof(p, c)
    assert g.tobytes() == ro.tobytes()
    assert np.array_equal(off, roff) and np.array_equal(sz, rsz)
