"""The scans over a node's halos for each halo's best parent (a warp per halo) and
each particle's nearest halo: Morton buckets of 32 and 1,024 against the plain
scan of the list, which is taken by nodes of at most asc_bucket_min halos.  Both
must leave the same bytes, in both forms of find_subs."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cfg,scale", [(5, 0.01), (5, 0.06), (2, 1 / 8), (3, 0.003)])
@pytest.mark.parametrize("batched", [False, True])
def test_buckets_against_list(rk, cfg, scale, batched):
    p, box, mp, _ = rk.synth(cfg, scale)
    c = rk.Config(particle_mass=mp, box_size=box, total_particles=len(p))
    fp, off, sz = rk.rockstar_fof(p, c)
    old = rk.get_tuning()["asc_bucket_min"]
    out = []
    try:
        for bmin in (1 << 20, 32, old):
            rk.set_tuning("asc_bucket_min", bmin)
            out.append(rk.find_subs(fp, off, sz, c, batched=batched))
    finally:
        rk.set_tuning("asc_bucket_min", old)
    for got in out[1:]:
        for a, b in zip(out[0], got):
            assert a.tobytes() == b.tobytes()
