"""The grouped later-dense lists of the 3D FOF: counts of dense particles
around a group of 32, grid positions whose pair distances equal the linking
length (where the reference takes or leaves a pair by its node shortcut), and
lists walked several chunks of groups at a time.  rockstar()'s whole output
against the oracle, byte for byte."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def same(rk, oracle, p, c):
    oracle.setup(c)
    ro, roff, rsz = oracle.fof(p)
    g, off, sz = rk.rockstar_fof(p, c)
    assert g.tobytes() == ro.tobytes()
    assert np.array_equal(off, roff) and np.array_equal(sz, rsz)


def clump(rk, n, grid, seed=0):
    """n particles in a ball of three linking lengths; on a grid of an eighth
    of the linking length, many pairs are exactly that length apart."""
    rng = np.random.default_rng(seed + n)
    c = rk.Config(box_size=64.0, particle_mass=0.0, total_particles=64 ** 3)
    st = rk.setup_config(c)
    c.particle_mass = float(st.particle_mass)
    c.fof_linking_length = 0.25  # a quarter of the mean spacing of 1: exact in float
    p = np.zeros(n, rk.PARTICLE)
    p["id"] = np.arange(n)
    x = rng.normal(size=(n, 3)) * 0.3 + 32.0
    if grid:
        x = np.round(x * 32) / 32
    p["pos"][:, :3] = x
    p["pos"][:, 3:] = rng.normal(size=(n, 3)) * 100
    return p, c


@pytest.mark.parametrize("grid", [False, True])
@pytest.mark.parametrize("n", [18, 33, 64, 65, 500, 4097, 20000])
def test_group_edges(rk, oracle, n, grid):
    p, c = clump(rk, n, grid)
    same(rk, oracle, p, c)


@pytest.mark.parametrize("cfg_id,scale", [(2, 1 / 16), (3, 0.005)])
def test_lists_in_several_chunks(rk, cfg_id, scale, monkeypatch):
    """Every group takes a list chunk of 128 entries, so a third as many
    chunks as groups is too few for the whole list."""
    p, box, mp, _ = rk.synth(cfg_id, scale)
    cfg = rk.Config(particle_mass=mp, box_size=box, total_particles=len(p))
    whole = rk.rockstar_fof(p, cfg)
    st = rk.last_stats()
    groups = st["dense"] // 32
    monkeypatch.setenv("RSG_FOF_LIST_ENTRIES", str(groups // 3 * 128))
    parts = rk.rockstar_fof(p, cfg)
    assert rk.last_stats()["dense_pairs"] == st["dense_pairs"]
    for a, b in zip(whole, parts):
        assert a.tobytes() == b.tobytes()
