"""The id sort on both sides of its key widths: 4-byte keys for an id range
below 2^32, 8-byte keys from there on, both ends of the range among the ids
(negative ones too).  The order is numpy's stable sort, byte for byte."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [0, 8])
@pytest.mark.parametrize("lo", [0, -(1 << 31), (1 << 62), -(1 << 63)])
@pytest.mark.parametrize("span", [(1 << 32) - 2, (1 << 32) - 1, 1 << 32, (1 << 32) + 1])
@pytest.mark.parametrize("n", [2, 1025, 70001])
def test_both_ends_present(rk, n, span, lo, shift):
    import torch
    rng = np.random.default_rng(n)
    p = np.zeros(n, rk.PARTICLE)
    p["id"] = lo + rng.integers(0, span, n, endpoint=True)
    p["id"][rng.permutation(n)[:2]] = [lo + span, lo]
    p["pos"] = rng.random((n, 6))
    assert int(p["id"].max()) - int(p["id"].min()) == span
    want = p[np.argsort(p["id"], kind="stable")]
    buf = torch.zeros(n * 32 + 16, dtype=torch.uint8, device="cuda")
    d = buf[shift:shift + n * 32]
    d.copy_(torch.from_numpy(p.view(np.uint8)))
    rk.sort_by_id_device(d)
    assert d.cpu().numpy().tobytes() == want.tobytes()
