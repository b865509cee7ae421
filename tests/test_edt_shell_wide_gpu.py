"""The general-width shell search on planes of more than 50 K voxels, with items that it finishes
and items that it leaves (inside objects, and where single voxels stay open), bit for bit
against the oracle."""

import numpy as np
import pytest
import torch

import oracle
import torchmorph_gb300 as tm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(2, 1, 9, 180, 256), (1, 1, 5, 254, 252), (1, 2, 12, 210, 240)])
@pytest.mark.parametrize("kind", ["noise50", "noise97", "ball", "mixed"])
def test_wide_planes(cuda, shape, kind):
    r = np.random.default_rng(sum(shape))
    x = r.random(shape) < (0.97 if kind == "noise97" else 0.5)
    if kind in ("ball", "mixed"):  # one item (ball: every item) with a large object
        z, y, w = np.ogrid[:shape[2], :shape[3], :shape[4]]
        ball = (z - 4) ** 2 + (y - 90) ** 2 + (w - 100) ** 2 < 70 ** 2
        for b in range(shape[0] if kind == "ball" else 1):
            x[b, 0] |= ball
    t = torch.from_numpy(x).cuda()
    d, idx = tm.euclidean_distance_transform(t, return_indices=True)
    _, od, oi = oracle.edt(x, None)
    np.testing.assert_array_equal(d.cpu().numpy(), od.astype(np.float32))
    np.testing.assert_array_equal(idx.cpu().numpy(), oi)
