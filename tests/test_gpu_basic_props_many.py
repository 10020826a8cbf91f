"""Basic halo properties by size class in the batched form (a warp up to 1,024
particles, a block per coordinate up to bp_big, chunks above), many clumps of
a size at a time, bp_big set on both sides of some of them: the plain form's sums are in the reference's order, so each
clump's halo must have the same members, links, integers and floats within
1e-4 (FP64 sums in another order differ by 1e-13).  A near-tie may go the other
way in one clump in twenty, the share the other batched tests allow: a class
that is summed wrongly fails in all of them."""
import numpy as np
import pytest

import halo_compare as HC

pytestmark = pytest.mark.gpu


@pytest.fixture
def class_edge(rk):
    old = rk.get_tuning()
    yield lambda big: (rk.set_tuning("bp_big", big), rk.set_tuning("bp_chunk", 256))
    for k in ("bp_big", "bp_chunk"):
        rk.set_tuning(k, old[k])


@pytest.mark.parametrize("n,clumps,big", [(33, 64, 0), (1023, 40, 0), (1024, 40, 0), (1025, 40, 0),
                                          (1290, 40, 0), (1290, 40, 1289), (1290, 40, 1290),
                                          (16385, 20, 0)])
def test_every_clump(rk, class_edge, n, clumps, big):
    if big:
        class_edge(big)
    rng = np.random.default_rng(n)
    total = n * clumps
    box = 20.0 * total ** (1 / 3)
    c = rk.Config(box_size=box, particle_mass=0.0, total_particles=total)
    st = rk.setup_config(c)
    link = st.avg_particle_spacing * st.fof_linking_length
    p = np.zeros(total, rk.PARTICLE)
    p["id"] = np.arange(total)
    k = np.repeat(np.arange(clumps), n)
    site = np.stack([k % 4, k // 4 % 4, k // 16], 1) + 0.5
    p["pos"][:, :3] = site * box / 5 + rng.random((total, 3)) * link / 3
    p["pos"][:, 3:] = rng.normal(size=(total, 3)) * 100
    c.particle_mass = float(st.particle_mass)
    fp, off, sz = rk.rockstar_fof(p, c)
    assert list(sz) == [n] * clumps
    ref = rk.find_subs(fp, off, sz, c)
    got = rk.find_subs(fp, off, sz, c, batched=True)
    sets = HC.halo_sets(ref[0], ref[1])
    ua, ub, worst, bad = HC.compare(sets, ref[1], HC.halo_sets(got[0], got[1]), got[1], 1e-4,
                                    ref_E=ref[2], got_E=got[2])
    assert ua == 0 and ub == 0
    clump = {i: int(np.frombuffer(ids, np.int64)[0]) // n for ids, i in sets.items()}
    assert set(clump.values()) == set(range(clumps))
    if n < 2000:  # most of the small clumps are one halo of just this size
        assert sum(ref[1][i]["num_p"] == n for i in clump) >= clumps / 4
    assert len({clump[h] for _, h, _ in bad}) <= 0.05 * clumps, bad[:10]
