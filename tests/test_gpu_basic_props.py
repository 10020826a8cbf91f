"""Basic halo properties by size class in the batched form: a warp up to 1,024
particles, a block per coordinate up to bp_big (16,384), chunks above.  One clump
of a size at each edge; the halos of the plain form, whose sums are in the
reference's order, must come out with the same members, links and integers, and
every float within 1e-4 (FP64 sums in another order differ by 1e-13; a halo
whose near-tie goes the other way is allowed, as in the other batched tests)."""
import numpy as np
import pytest

import halo_compare as HC

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [33, 1023, 1024, 1025, 1290, 16384, 16385])
def test_size_classes(rk, n):
    rng = np.random.default_rng(n)
    box = 20.0 * n ** (1 / 3)
    c = rk.Config(box_size=box, particle_mass=0.0, total_particles=n)
    st = rk.setup_config(c)
    link = st.avg_particle_spacing * st.fof_linking_length
    p = np.zeros(n, rk.PARTICLE)
    p["id"] = np.arange(n)
    p["pos"][:, :3] = box / 2 + rng.random((n, 3)) * link / 3
    p["pos"][:, 3:] = rng.normal(size=(n, 3)) * 100
    c.particle_mass = float(st.particle_mass)
    fp, off, sz = rk.rockstar_fof(p, c)
    assert list(sz) == [n]
    ref = rk.find_subs(fp, off, sz, c)
    got = rk.find_subs(fp, off, sz, c, batched=True)
    ua, ub, worst, bad = HC.compare(HC.halo_sets(ref[0], ref[1]), ref[1],
                                    HC.halo_sets(got[0], got[1]), got[1], 1e-4, ref_E=ref[2],
                                    got_E=got[2])
    assert ua == 0 and ub == 0
    assert len({h for _, h, _ in bad}) <= 0.05 * len(ref[1]) + 1, bad[:10]
