"""The next-closest searches, 16 lanes a query, at the sizes where they change
shape: groups of one leaf (up to 40 particles), of two, and of several levels,
and samples at random positions (above 10,000).  On a coarse lattice many
particles coincide or are equally far, so a zero distance in the own leaf is
left out, one in another leaf counts, and whole nodes are a point.  The linking
lengths of the 6D hierarchy are compared with the oracle bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lattice", [0, 3, 12])
@pytest.mark.parametrize("n", [20, 40, 41, 81, 330, 2500, 10050])
def test_linking_lengths(rk, oracle, n, lattice):
    rng = np.random.default_rng(n + lattice)
    box = 20.0 * n ** (1 / 3)
    c = rk.Config(box_size=box, particle_mass=0.0, total_particles=n)
    st = rk.setup_config(c)
    link = st.avg_particle_spacing * st.fof_linking_length
    u = rng.random((n, 6))
    if lattice:
        u = np.floor(u * lattice) / lattice
    p = np.zeros(n, rk.PARTICLE)
    p["id"] = np.arange(n)
    # within a third of the linking length on each axis: one group
    p["pos"][:, :3] = box / 2 + u[:, :3] * link / 3
    p["pos"][:, 3:] = u[:, 3:] * 300
    c.particle_mass = float(st.particle_mass)
    oracle.setup(c)
    fp, off, sz = oracle.fof(p)
    assert len(sz) == 1
    oracle.find_subs(fp, off, sz)
    ol, on, otr = oracle.hierarchy()
    want = sorted(zip(ol.tolist(), on.tolist(), otr.tolist()))
    for batched in (False, True):
        rk.find_subs(fp, off, sz, c, batched=batched)
        gl, gn, gtr = rk.debug_hierarchy()
        assert sorted(zip(gl.tolist(), gn.tolist(), gtr.tolist())) == want
