"""The id sort where its route changes: ids whose range shares a word with the
record index or does not, one id, records aligned to 16 bytes or only to 8,
and counts around a block of the gather.  The order is numpy's stable sort
(equal ids keep their input order), byte for byte."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [0, 8])
@pytest.mark.parametrize("lo,hi", [(0, 7), (-5, 1 << 40), (0, 1 << 57),
                                   (-(1 << 63), (1 << 63) - 1), (12, 13)])
@pytest.mark.parametrize("n", [2, 255, 1023, 1025, 70001])
def test_sorted_stably(rk, n, lo, hi, shift):
    import torch
    rng = np.random.default_rng(n)
    p = np.zeros(n, rk.PARTICLE)
    p["id"] = rng.integers(lo, hi, n)
    p["pos"] = rng.random((n, 6))
    want = p[np.argsort(p["id"], kind="stable")]
    buf = torch.zeros(n * 32 + 16, dtype=torch.uint8, device="cuda")
    d = buf[shift:shift + n * 32]
    d.copy_(torch.from_numpy(p.view(np.uint8)))
    rk.sort_by_id_device(d)
    assert d.cpu().numpy().tobytes() == want.tobytes()
