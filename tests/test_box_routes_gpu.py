"""Binary and grey boxes on either side of the lines between walkers, bit tiles and byte tiles, and
windows of one column, which have no row pass: against the oracle."""

import numpy as np
import pytest
import torch

import oracle
import torchmorph_gb300 as tm
from torchmorph_gb300 import ragged

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(3, 3), (5, 5), (13, 5), (33, 1), (1, 65), (1, 66), (35, 1), (6, 11), (9, 45),
                                  (45, 45), (2, 40)])
@pytest.mark.parametrize("shape", [(2, 1, 70, 144), (1, 1, 33, 301)])
def test_binary_boxes(cuda, shape, size):
    x = np.random.default_rng(sum(size)).random(shape) < 0.7
    box = np.ones(size, bool)
    t = torch.from_numpy(x).cuda()
    for dilation, op in ((False, tm.binary_erosion), (True, tm.binary_dilation)):
        got = op(t, structure=torch.from_numpy(box)).cpu().numpy()
        np.testing.assert_array_equal(got, oracle.binary(x, box, dilation=dilation).astype(bool))


@pytest.mark.parametrize("size", [(3, 3), (5, 5)])
def test_binary_boxes_above_the_walkers_line(cuda, size):
    """One batch of 1.2 M words and one below, the same rows in both."""
    x = np.random.default_rng(3).random((10, 1, 2048, 2048)) < 0.6
    box = torch.ones(size, dtype=torch.bool)
    t = torch.from_numpy(x).cuda()
    all_of_them, some = tm.binary_erosion(t, structure=box), tm.binary_erosion(t[:4], structure=box)
    assert torch.equal(all_of_them[:4], some)
    assert torch.equal(tm.binary_opening(t, structure=box)[:4], tm.binary_opening(t[:4], structure=box))
    exp = oracle.binary(x[:1], box.numpy(), dilation=False).astype(bool)
    np.testing.assert_array_equal(some[:1].cpu().numpy(), exp)


@pytest.mark.parametrize("size", [(2, 1), (3, 1), (7, 1), (8, 1), (65, 1), (201, 1), (1, 2), (2, 2), (3, 2), (2, 33), (4, 60)])
@pytest.mark.parametrize("mode", ["reflect", "constant", "wrap"])
def test_grey_windows(cuda, size, mode):
    x = np.random.default_rng(sum(size)).random((2, 1, 41, 137)).astype(np.float32)
    st = np.zeros(size, np.float32)
    t = torch.from_numpy(x).cuda()
    batch = ragged.RaggedBatch.from_images([t[0, 0], t[1, 0, :19, :70]])
    for dilation, op, rop in ((False, tm.grey_erosion, ragged.grey_erosion), (True, tm.grey_dilation, ragged.grey_dilation)):
        exp = oracle.grey(x, st, dilation=dilation, mode=mode, cval=0.25)
        np.testing.assert_array_equal(op(t, size=size, mode=mode, cval=0.25).cpu().numpy(), exp)
        if size[0] <= 100:
            out = rop(batch, size=size, mode=mode, cval=0.25)
            np.testing.assert_array_equal(out[0].cpu().numpy(), exp[0, 0])
            part = oracle.grey(np.ascontiguousarray(x[1:, :, :19, :70]), st, dilation=dilation, mode=mode, cval=0.25)
            np.testing.assert_array_equal(out[1].cpu().numpy(), part[0, 0])
