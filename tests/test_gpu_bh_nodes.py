"""Node pass of the Barnes-Hut tree (mass centres by climbing from the
leaves, opening radii of every node in one launch) at the sizes where its
kernels change hands: one leaf, one split, a warp's remainder, the block
form above 4,096 records with a partial buffer, the chunked form above
65,536.  Form 0 is compared with the oracle bit for bit; form 1 with form 0
within 1e-5 relative, the bound stated for the FP32 terms (a few FP32
roundings of a Kahan-compensated sum: 2.4e-7 measured)."""
import numpy as np
import pytest

from test_gpu_potential import nfw_like

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,dup", [(1, 0), (10, 0), (11, 0), (43, 0), (4095, 0), (4097, 0),
                                   (9001, 25)])
def test_form0_bit_for_bit(rk, oracle, n, dup):
    po = nfw_like(n, 100 + n, dup=dup).view(rk.POTENTIAL)
    cfg = rk.Config(particle_mass=1e9, force_res=0.003)
    oracle.setup(cfg)
    ref = oracle.compute_potential(po)
    got = rk.compute_potential(po, cfg, form=0)
    assert np.array_equal(got["pos"], ref["pos"])
    assert got["pe"].tobytes() == ref["pe"].tobytes()


@pytest.mark.parametrize("n", [11, 4097, 65535, 70001])
def test_form1_against_form0(rk, n):
    po = nfw_like(n, 7 + n).view(rk.POTENTIAL)
    cfg = rk.Config(particle_mass=1e9, force_res=0.003)
    a = rk.compute_potential(po, cfg, form=0)
    b = rk.compute_potential(po, cfg, form=1)
    assert np.array_equal(a["pos"], b["pos"])
    assert (np.abs(b["pe"] - a["pe"]) / np.abs(a["pe"])).max() <= 1e-5
